"""GPU parity: the register-tiled fp32 attention kernels at the edges of their 64-row tiles, of their groups of streamed
tiles (four at head dims up to 64, two above: a number of tiles that is no multiple of them, fewer than them), of padded head
dims (32 / 64 / 128), and on both sides of the lines to the general kernels (32 and 64 keys)."""
import numpy as np
import pytest
import torch

from gpu_util import back, check, draw

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


def _mask(name, t, o, n):
    ids = (np.arange(n) * 5 // n).astype(np.int32)
    docs = t.DocumentMask(torch.from_numpy(ids).cuda())
    if name == "causal & window & document":
        return t.CausalMask() & t.SlidingWindowMask(20) & docs, o.MaskSpec(causal=True, window=20, doc_q=ids)
    if name == "prefix & document":
        return t.PrefixMask(37) & docs, o.MaskSpec(prefix=37, doc_q=ids)
    if name == "prefix_lm":
        return t.prefix_lm(19), o.MaskSpec(prefix_or_causal=19)
    if name == "window | document":
        return t.SlidingWindowMask(9) | docs, o.MaskAny(o.MaskSpec(window=9), o.MaskSpec(doc_q=ids))
    return None, None


# every mask term as the bits of a column of pairs, from the queries' side and from the keys', with each order of the score mods
@pytest.mark.parametrize("mask", ["none", "causal & window & document", "prefix & document", "prefix_lm", "window | document"])
@pytest.mark.parametrize("score", ["none", "alibi, then soft cap", "soft cap, then alibi", "bias, then soft cap"])
@pytest.mark.parametrize("B,H,Hkv,Sq,Sk,D", [(1, 2, 1, 32, 32, 64), (1, 2, 2, 33, 33, 32), (2, 4, 2, 64, 64, 64), (40, 8, 8, 20, 30, 32),
                                             (1, 2, 1, 65, 130, 128), (2, 3, 1, 150, 100, 36)])
def test_masks_and_mods(tylo, oracle, B, H, Hkv, Sq, Sk, D, score, mask):
    t, o = tylo, oracle
    rng = np.random.default_rng(Sq + Sk + D)
    Q, Q64 = draw(rng, (B, H, Sq, D), "f32"); K, K64 = draw(rng, (B, Hkv, Sk, D), "f32"); V, V64 = draw(rng, (B, Hkv, Sk, D), "f32")
    dO, dO64 = draw(rng, (B, H, Sq, D), "f32")
    m, om = _mask(mask, t, o, max(Sq, Sk))
    slopes = torch.tensor([0.25 * 2.0 ** -h for h in range(H)], device="cuda")
    table, table64 = draw(rng, (1, H, Sq, Sk), "f32")
    alibi = (t.AliBiScore(slopes), ("alibi", back(slopes)))
    cap = (t.SoftCapScore(3.0), ("softcap", 3.0))
    chain = {"none": [], "alibi, then soft cap": [alibi, cap], "soft cap, then alibi": [cap, alibi],
             "bias, then soft cap": [(t.BiasScore(table), ("bias", table64)), cap]}[score]
    sm = chain[1][0] @ chain[0][0] if chain else None
    kw = dict(mask_mod=m, score_mod=sm)
    okw = dict(mask=om, score=o.ScoreSpec([c[1] for c in chain]) if chain else None)
    cp = t.allocate_checkpoints_flex_attention(Q, K, V)
    O = t.flex_attention(Q, K, V, checkpoints=cp, **kw)
    check(O, o.flex_ref(Q64, K64, V64, **okw), "f32", "O")
    got = t.grad_flex_attention(dO, Q, K, V, O, checkpoints=cp, **kw)
    for g, ref, name in zip(got, o.flex_bwd_ref(dO64, Q64, K64, V64, **okw), ("dQ", "dK", "dV")):
        check(g, ref, "f32", name)


def test_error_against_64_bits(tylo):
    """Rounding over long sums.  The bounds are 1.2 times what sums of at most 32 terms give (attn_generic.cu on the same inputs:
    O 2.97e-7, dQ 4.28e-7, dK 4.40e-7, dV 4.20e-7, relative 2-norm); accumulators that run through all rows of a head, or through
    half of the head dim per packed lane, gave 5.1e-7, 6.1e-7, 5.9e-7 and 5.7e-7."""
    g = torch.Generator("cuda").manual_seed(5)
    Q, K, V, dO = (torch.randn(2, h, 1200, 128, generator=g, device="cuda") for h in (8, 4, 4, 8))
    cp = tylo.allocate_checkpoints_flex_attention(Q, K, V)
    O = tylo.flex_attention(Q, K, V, checkpoints=cp)
    got = (O, *tylo.grad_flex_attention(dO, Q, K, V, O, checkpoints=cp))
    q, k, v = (x.double().requires_grad_() for x in (Q, K, V))
    ref = (q @ k.repeat_interleave(2, 1).transpose(-1, -2) / 128 ** 0.5).softmax(-1) @ v.repeat_interleave(2, 1)
    ref.backward(dO.double())
    for a, b, bound, name in zip(got, (ref.detach(), q.grad, k.grad, v.grad), (3.6e-7, 5.1e-7, 5.3e-7, 5.0e-7), ("O", "dQ", "dK", "dV")):
        err = float((a.double() - b).norm() / b.norm())
        assert err <= bound, f"{name}: {err:.2e} > {bound:.1e}"


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("D", [32, 64, 128])
def test_ragged_backward(tylo, oracle, D, causal):
    """Lengths of none, one, a tile less one, a tile and one, and all rows: each batch entry against the oracle on its own keys and
    query blocks; keys beyond a length and query blocks beyond one get gradients of exactly zero."""
    lens = [0, 1, 63, 65, 200]
    B, H, Hkv, S = len(lens), 4, 2, 200
    rng = np.random.default_rng(D)
    Q, Q64 = draw(rng, (B, H, S, D), "f32"); K, K64 = draw(rng, (B, Hkv, S, D), "f32"); V, V64 = draw(rng, (B, Hkv, S, D), "f32")
    dO, dO64 = draw(rng, (B, H, S, D), "f32")
    n = torch.tensor(lens, dtype=torch.int32, device="cuda")
    kw = dict(causal=causal, k_lengths=n, q_lengths=n)
    cp = tylo.allocate_checkpoints_attention(Q, K, V)
    O = torch.zeros_like(Q)
    tylo.attention_(O, Q, K, V, checkpoints=cp, **kw)
    dQ, dK, dV = tylo.grad_attention(dO, Q, K, V, O, checkpoints=cp, **kw)
    for b, k in enumerate(lens):
        q = min(S, -(-k // 64) * 64)                  # query blocks of 64 rows that start below the length
        assert not dQ[b, :, q:].any() and not dK[b, :, k:].any() and not dV[b, :, k:].any() and not O[b, :, q:].any()
        if k == 0:
            continue
        okw = dict(mask=oracle.MaskSpec(causal=True) if causal else None)
        args = (Q64[b:b + 1, :, :q], K64[b:b + 1, :, :k], V64[b:b + 1, :, :k])
        check(O[b:b + 1, :, :q], oracle.flex_ref(*args, **okw), "f32", f"O of length {k}")
        ref = oracle.flex_bwd_ref(dO64[b:b + 1, :, :q], *args, **okw)
        check(dV[b:b + 1, :, :k], ref[2], "f32", f"dV of length {k}")
        if k == 1:
            # one key: dS = P (dP - Delta) is a difference of two equal sums of D products, dQ and dK are zero but for its rounding,
            # at most D 2^-24 of the largest product in either sum
            e = 2 * D * 2.0 ** -24 * np.abs(dO64[b]).max() * np.abs(V64[b]).max() * D ** -0.5
            assert float(dQ[b].abs().max()) <= e * np.abs(K64[b]).max()
            assert float(dK[b].abs().max()) <= e * np.abs(Q64[b]).max() * q * H / Hkv
            continue
        for g, r, name in ((dQ[b:b + 1, :, :q], ref[0], "dQ"), (dK[b:b + 1, :, :k], ref[1], "dK")):
            check(g, r, "f32", f"{name} of length {k}")
