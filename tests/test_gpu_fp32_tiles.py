"""GPU parity: the register-tiled fp32 attention kernels at the edges of their 64-row tiles, their two groups of streamed
tiles (an odd number of them, fewer than two), padded head dims (32 / 64 / 128)."""
import numpy as np
import pytest

from gpu_util import check, draw

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("D", [4, 32, 36, 64, 100, 128])
@pytest.mark.parametrize("B,H,Hkv,Sq,Sk,pos", [(1, 1, 1, 1, 1, 0), (2, 4, 2, 63, 65, 2), (1, 2, 2, 64, 64, 0),
                                               (1, 3, 1, 129, 200, 71), (2, 2, 2, 200, 129, 0)])
def test_tiles(tylo, oracle, B, H, Hkv, Sq, Sk, pos, D, causal):
    rng = np.random.default_rng(Sq + Sk + D)
    Q, Q64 = draw(rng, (B, H, Sq, D), "f32"); K, K64 = draw(rng, (B, Hkv, Sk, D), "f32"); V, V64 = draw(rng, (B, Hkv, Sk, D), "f32")
    dO, dO64 = draw(rng, (B, H, Sq, D), "f32")
    mask = tylo.CausalMask() if causal else None
    okw = dict(mask=oracle.MaskSpec(causal=True) if causal else None, input_pos=pos)
    cp = tylo.allocate_checkpoints_flex_attention(Q, K, V)
    O = tylo.flex_attention(Q, K, V, mask_mod=mask, input_pos=pos, checkpoints=cp)
    check(O, oracle.flex_ref(Q64, K64, V64, **okw), "f32", "O")
    got = tylo.grad_flex_attention(dO, Q, K, V, O, checkpoints=cp, mask_mod=mask, input_pos=pos)
    for g, ref, name in zip(got, oracle.flex_bwd_ref(dO64, Q64, K64, V64, **okw), ("dQ", "dK", "dV")):
        check(g, ref, "f32", name)
