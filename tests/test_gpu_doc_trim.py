"""GPU: key and query tiles dropped because their span of document ids does not meet the owned rows' span.  Dropping is exact,
so a call that may skip tiles equals one that may not (block_sparse=False), bit for bit, for packed documents, for ids in
no order, for ids that meet nowhere and with a shifted query position."""
import pytest
import torch

pytestmark = pytest.mark.gpu

S = 2100


def _ids(kind, n):
    g = torch.Generator().manual_seed(n)
    pos = torch.arange(n)
    if kind == "packed":
        return (pos // 170).to(torch.int32)
    if kind == "one long":
        return (pos >= 60).to(torch.int32) + (pos >= 2050).to(torch.int32)
    if kind == "descending":
        return (-(pos // 300)).to(torch.int32)
    if kind == "shuffled blocks":
        return torch.randperm(n // 64 + 1, generator=g)[pos // 64].to(torch.int32) // 3
    return torch.randint(-5, 5, (n,), generator=g).to(torch.int32)          # no order at all


@pytest.mark.parametrize("window", [0, 500])
@pytest.mark.parametrize("pos", [0, 129])
@pytest.mark.parametrize("kind", ["packed", "one long", "descending", "shuffled blocks", "random"])
@pytest.mark.parametrize("Hkv", [1, 2])            # two heads of a group per work item, or two row blocks of one head
def test_trim_is_exact(tylo, Hkv, kind, pos, window):
    g = torch.Generator("cuda").manual_seed(3)
    B, H, D = 2, 2, 64
    Q, K, V, dO = (torch.randn(B, h, S, D, generator=g, device="cuda").bfloat16() for h in (H, Hkv, Hkv, H))
    table = torch.stack([_ids(kind, S + pos), _ids(kind, S + pos) + (1000 if kind == "random" else 0)]).cuda()
    doc_kv = table.clone()
    if kind == "random":
        doc_kv[1] -= 1000                          # batch entry 1: no pair shares a document
    mask = tylo.CausalMask() & tylo.DocumentMask(table, doc_kv)
    if window:
        mask = tylo.SlidingWindowMask(window) & mask
    res = []
    for sparse in (True, False):
        kw = dict(mask_mod=mask, block_sparse=sparse, input_pos=pos)
        cp = tylo.allocate_checkpoints_flex_attention(Q, K, V)
        O = tylo.flex_attention(Q, K, V, checkpoints=cp, **kw)
        res.append((O, cp.M, cp.L) + tuple(tylo.grad_flex_attention(dO, Q, K, V, O, checkpoints=cp, **kw)))
    assert tylo.device_status() == 0
    for a, b in zip(*res):
        assert torch.equal(a, b)
