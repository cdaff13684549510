"""The training-free block score where a KV head's query heads and its key-block tiles are shared between CTAs:
groups of heads (whole, with a remainder), shares of the tiles (more than there are visible ones), ragged chunks."""
import pytest
import torch

from oracle import compact_oracle as co

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Q,K,Hq,Hkv,bs", [
    (300, 20012, 28, 4, 128),   # seven heads do not fit beside the key tiles: 4 + 3
    (128, 32768, 16, 1, 128),   # two heads a group, the key tiles shared as well
    (64, 40000, 4, 1, 64),      # one q-block: every key tile a CTA of its own
    (200, 1000, 10, 2, 64),     # five heads in passes of 4 + 1, one key tile
    (2560, 5120, 28, 4, 128),   # enough q-blocks: groups only
])
def test_shared_heads_and_tiles(Q, K, Hq, Hkv, bs):
    from compactattention_b200 import ops
    g = torch.Generator().manual_seed(Q + K)
    q = torch.randn((1, Q, Hq, 128), generator=g).to(torch.bfloat16)
    mean_k = torch.randn((1, -(-K // bs), Hkv, 128), generator=g).to(torch.bfloat16)
    raw, mx, _ = ops.flashprefill_score(q.cuda(), mean_k.cuda(), K, bs, normalize=False)
    want_raw, want_mx = co.flashprefill_block_score_raw(q, mean_k, K, bs)
    fin = torch.isfinite(want_mx)
    assert torch.equal(torch.isfinite(mx.cpu()), fin)
    # fp32 sums of 128 products of 16-bit values, and of up to 128 exponentials
    assert torch.allclose(mx.cpu()[fin], want_mx[fin], rtol=1e-4, atol=1e-4)
    assert torch.allclose(raw.cpu()[fin], want_raw[fin], rtol=1e-3, atol=1e-5)
