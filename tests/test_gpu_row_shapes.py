"""GPU parity: the row kernels at the edges of their launch shapes — rows that start inside a 16-byte packet, rows too long
for one CTA's registers, norm backward with several rows per CTA, with more than one packet per thread, and with fewer
partial rows or tokens than CTAs."""
import numpy as np
import pytest
import torch

from gpu_util import back, check, draw

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", ["f32", "bf16", "f16"])
@pytest.mark.parametrize("M,N", [(1, 5), (7, 9), (9, 3), (63, 4), (513, 3), (2049, 3), (4095, 3), (8193, 2), (65533, 2), (65544, 2),
                                 (70001, 2), (131072, 1), (12292, 18), (33001, 30), (40000, 74), (33000, 150)])
def test_softmax_rows(tylo, oracle, M, N, dt):
    rng = np.random.default_rng(M + N)
    buf = torch.full((N * M + 32,), 7.0, device="cuda", dtype={"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}[dt])
    X, X64 = draw(rng, (N, M), dt, scale=2.0)
    Y = buf[:N * M].view(N, M)
    tylo.softmax_(Y, X)
    assert bool((buf[N * M:] == 7.0).all())          # nothing beyond the last row is written
    check(Y, oracle.softmax_ref(X64), dt, "softmax")
    dY, dY64 = draw(rng, (N, M), dt)
    check(tylo.grad_softmax(dY, Y), oracle.softmax_bwd_ref(dY64, back(Y)), dt, "softmax bwd")


@pytest.mark.parametrize("M", [9, 4097, 70001, 131072])
def test_softmax_minus_infinity(tylo, oracle, M):
    X = torch.randn(3, M, device="cuda")
    X[0, 1:] = float("-inf")                          # one entry left
    X[1, ::2] = float("-inf")
    X[2, :-1] = float("-inf")
    check(tylo.softmax(X), oracle.softmax_ref(back(X)), "f32", "softmax")


# one length per kernel and per way a row is moved: a warp, several warps, the long two-pass rows, each in whole packets and not
@pytest.mark.parametrize("dt", ["f32", "bf16", "f16"])
@pytest.mark.parametrize("M", [40, 61, 1000, 1001, 8192, 8195, 16392, 16401, 32768, 32771, 65600, 70001])
def test_softmax_not_finite(tylo, M, dt):
    X = torch.randn(9, M, device="cuda").to({"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}[dt])
    X[0, M // 3] = float("nan")
    X[1, M - 1] = float("inf")
    X[2, :] = float("-inf")
    X[2, M // 2] = float("nan")
    X[3, :] = float("nan")
    X[4, :] = float("-inf")
    X[4, 0] = float("inf")
    X[5, :] = float("-inf")                           # the one row that is defined to be zeros
    X[6, ::2] = torch.finfo(X.dtype).min              # masked by the lowest value, in part
    if dt != "bf16" or M > 32768:                     # (bf16 rows in registers: the lowest value times log2(e) is -Inf)
        X[7, :] = torch.finfo(X.dtype).min            # and throughout
    Y = tylo.softmax(X)
    assert bool(Y[:5].isnan().all())
    assert bool((Y[5] == 0).all())
    ref = torch.softmax(X[6:].double(), -1)
    tol = {"f32": 1e-5, "bf16": 2.0 ** -8, "f16": 2.0 ** -10}[dt] * float(ref.max())       # an ulp of the largest result
    assert float((Y[6:].double() - ref).abs().max()) <= tol


def test_softmax_row_beyond_int_packets(tylo):
    """One row of 2^31 packets: forward at a length that is no whole number of them, backward at one that is."""
    torch.cuda.empty_cache()
    if torch.cuda.mem_get_info()[0] < 115e9:
        pytest.skip("needs 105 GB")
    M = 2 ** 33
    buf = torch.empty(3, M + 4, device="cuda")
    at = torch.tensor([5, 2 ** 32 + 1, M - 1, M + 2], device="cuda")
    x = torch.tensor([0.0, 1.0, 2.0, 0.5], device="cuda")
    X, Y = buf[0, :M + 3].view(1, -1), buf[1, :M + 3].view(1, -1)
    X.fill_(float("-inf"))
    X[0, at] = x
    Y.fill_(7.0)
    tylo.softmax_(Y, X)
    assert torch.allclose(Y[0, at], x.softmax(0), rtol=1e-6, atol=0)
    Y[0, at] = 0.0
    assert not Y.any()
    Y, dY, dX = buf[0, :M].view(1, -1), buf[1, :M].view(1, -1), buf[2, :M].view(1, -1)
    at, y, g = at[:3], torch.tensor([0.25, 0.5, 0.25], device="cuda"), torch.tensor([1.0, 2.0, -3.0], device="cuda")
    Y.zero_(); dY.fill_(1.0); dX.fill_(7.0)
    Y[0, at], dY[0, at] = y, g
    tylo.grad_softmax_(tylo.Duplicated(Y, dY), tylo.Duplicated(dX, dX))
    assert torch.allclose(dX[0, at], y * (g - (y * g).sum()), rtol=1e-6, atol=0)
    dX[0, at] = 0.0
    assert not dX.any()
    del buf, X, Y, dY, dX
    torch.cuda.empty_cache()


# packets per row (f32: 4 elements, 16-bit: 8): one warp, a warp and one, eight rows per CTA, ragged thread counts, 1,024 and
# beyond (two and four packets per thread), and lengths that are not a multiple of the packet
@pytest.mark.parametrize("dt", ["f32", "bf16"])
@pytest.mark.parametrize("M,N,groups", [(8, 40, 296), (256, 700, 296), (264, 31, 3), (520, 5000, 296), (4104, 301, 296), (8192, 3, 1),
                                        (8200, 17, 5), (12288, 200, 296), (16384, 9, 296), (16392, 3, 296), (1, 7, 296), (1001, 333, 296),
                                        (33001, 2, 296), (2056, 310, 296), (3080, 30, 296), (5128, 160, 296), (6152, 9, 7),
                                        (7176, 5, 296), (6251, 3, 296), (7043, 300, 296), (9401, 5, 3)])
def test_norm_rows(tylo, oracle, M, N, groups, dt):
    rng = np.random.default_rng(M + N)
    eps = 1e-5
    X, X64 = draw(rng, (N, M), dt, shift=0.3)
    W, W64 = draw(rng, (M,), dt, scale=0.1, shift=1.0)
    B, B64 = draw(rng, (M,), dt, scale=0.1)
    dY, dY64 = draw(rng, (N, M), dt)
    cp = tylo.allocate_checkpoints_rms_norm(X, W)
    check(tylo.rms_norm(X, W, eps=eps, offset=0.25, checkpoints=cp), oracle.rms_norm_ref(X64, W64, eps=eps, offset=0.25), dt, "rms")
    sc = tylo.allocate_scratchspace_grad_rms_norm(X, W, N_GROUPS=groups)
    dX, dW = tylo.grad_rms_norm(dY, X, W, checkpoints=cp, offset=0.25, scratch=sc)
    dXr, dWr, _ = oracle.rms_norm_bwd_ref(dY64, X64, W64, eps=eps, offset=0.25)
    check(dX, dXr, dt, "rms dX"); check(dW, dWr, dt, "rms dW", scale_hint=4 * float(np.abs(dWr).max()))
    if M == 1:
        return                                        # LayerNorm of one element: 0 / sqrt(eps) against rounding noise
    cpl = tylo.allocate_checkpoints_layer_norm(X, W, B)
    check(tylo.layer_norm(X, W, B, eps=eps, checkpoints=cpl), oracle.layer_norm_ref(X64, W64, B64, eps=eps), dt, "ln")
    sc = tylo.allocate_scratchspace_grad_layer_norm(X, W, B, N_GROUPS=groups)
    dX, dW, dB = tylo.grad_layer_norm(dY, X, W, B, checkpoints=cpl, scratch=sc)
    dXr, dWr, dBr, _, _ = oracle.layer_norm_bwd_ref(dY64, X64, W64, eps=eps)
    check(dX, dXr, dt, "ln dX")
    check(dW, dWr, dt, "ln dW", scale_hint=4 * float(np.abs(dWr).max()))
    check(dB, dBr, dt, "ln dB", scale_hint=4 * float(np.abs(dBr).max()))


def test_norm_backward_of_the_most_rows(tylo):
    """2^31 - 1 rows, the most that are accepted: the rows asked for ahead of the last ones lie beyond what an int holds."""
    M, N, tail = 8, 2 ** 31 - 1, 20000
    torch.cuda.empty_cache()
    if torch.cuda.mem_get_info()[0] < 125e9:
        pytest.skip("needs 115 GB")
    X, dY, dX = (torch.ones(N, M, device="cuda", dtype=torch.bfloat16) for _ in range(3))
    g = torch.Generator("cuda").manual_seed(1)
    for t in (X, dY):
        t[-tail:] = torch.randn(tail, M, generator=g, device="cuda").bfloat16()
    W, dW = torch.ones(M, device="cuda", dtype=torch.bfloat16), torch.empty(M, device="cuda", dtype=torch.bfloat16)
    cp = tylo.allocate_checkpoints_rms_norm(X, W)
    tylo.rms_norm_(dX, X, W, eps=1e-6, checkpoints=cp)
    d = tylo.Duplicated
    tylo.grad_rms_norm_(d(dX, dY), d(X, dX), d(W, dW), checkpoints=cp, scratch=tylo.allocate_scratchspace_grad_rms_norm(X, W))
    x = X[-tail:].double().requires_grad_()
    y = x * torch.rsqrt((x * x).mean(-1, keepdim=True) + 1e-6)
    y.backward(dY[-tail:].double())
    err = (dX[-tail:].double() - x.grad).abs()
    assert bool((err <= 2.0 ** -8 * x.grad.abs() + 1e-4).all())        # an ulp of bf16
    assert bool((dX[:tail].float().abs() < 1e-5).all())               # rows of ones: dY is parallel to X
    del X, dY, dX, cp
    torch.cuda.empty_cache()
