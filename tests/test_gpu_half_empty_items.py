"""GPU parity: work items whose second Q tile has no rows, several of them per CTA.  With one query head per KV head
an item is 256 rows of one head, so Sq mod 256 in 1..128 leaves the last item of every head half empty; with more items
than SMs a CTA walks several such items in a row."""
import numpy as np
import pytest

from gpu_util import check, draw

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("Sq", [40, 128, 300])      # one half-empty item per head; a full tile and an empty one; full + half
def test_half_empty_items(tylo, oracle, Sq, causal):
    B, H, D = 8, 64, 64                              # 512 heads: at least three items per SM
    rng = np.random.default_rng(Sq)
    Q, Q64 = draw(rng, (B, H, Sq, D), "bf16"); K, K64 = draw(rng, (B, H, Sq, D), "bf16"); V, V64 = draw(rng, (B, H, Sq, D), "bf16")
    O = tylo.attention(Q, K, V, causal=causal)
    assert tylo.device_status() == 0
    for b in (0, B // 2, B - 1):
        check(O[b:b + 1], oracle.attn_ref(Q64[b:b + 1], K64[b:b + 1], V64[b:b + 1], causal=causal), "bf16", f"batch entry {b}")
