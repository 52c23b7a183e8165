"""GPU: the norm backwards of row lengths that are not whole packets and need just under 48 KB of dynamic shared memory.  Each
runs in a process of its own: the limit that a launch asks for stays with the kernel, so any longer row of that kind run
before would hide a call that forgot to ask."""
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

CHILD = """
import sys, torch
sys.path.insert(0, sys.argv[1])
from conftest import load_package
t = load_package()
op, M, N = sys.argv[2], int(sys.argv[3]), 5
g = torch.Generator("cuda").manual_seed(M)
X, dY = (torch.randn(N, M, generator=g, device="cuda", dtype=torch.float32) for _ in range(2))
W, B = torch.randn(M, generator=g, device="cuda") * 0.1 + 1, torch.zeros(M, device="cuda")
x = X.double().requires_grad_(); w = W.double().requires_grad_(); b = B.double().requires_grad_()
if op == "rms":
    cp = t.allocate_checkpoints_rms_norm(X, W)
    t.rms_norm(X, W, eps=1e-5, checkpoints=cp)
    got = t.grad_rms_norm(dY, X, W, checkpoints=cp)
    y = x * torch.rsqrt((x * x).mean(-1, keepdim=True) + 1e-5) * w
else:
    cp = t.allocate_checkpoints_layer_norm(X, W, B)
    t.layer_norm(X, W, B, eps=1e-5, checkpoints=cp)
    got = t.grad_layer_norm(dY, X, W, B, checkpoints=cp)
    y = torch.nn.functional.layer_norm(x, (M,), w, b, 1e-5)
y.backward(dY.double())
for a, r in zip(got, (x.grad, w.grad, b.grad)):
    assert float((a.double() - r).abs().max()) <= 1e-5 * float(r.abs().max()) + 1e-6
"""


# 12 bytes per element (RMSNorm) or 16 (LayerNorm): lengths whose request fits 48 KB, but not together with the kernel's static part
@pytest.mark.parametrize("op,M", [("rms", 4081), ("rms", 4095), ("layer", 3057), ("layer", 3071)])
def test_first_call_of_a_process(op, M):
    r = subprocess.run([sys.executable, "-c", CHILD, str(Path(__file__).resolve().parent), op, str(M)], capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
