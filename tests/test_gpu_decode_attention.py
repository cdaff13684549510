"""Attention of few query rows (Q * G <= 16 rows per KV head) against the CPU oracle: edges of the 64-token
sub-blocks, every cut of a row (one CTA, a cluster, several clusters), tables with empty rows, page tables."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from compactattention_b200 import ops as _ops
    return _ops


def _check(out, lse, want, want_lse):
    # one 16-bit rounding of each probability and of the output: 2^-9 (bf16) of a mean of ~N(0, 1) values, taken
    # four times over for the largest of up to 1e5 entries; log-sum-exp stays in fp32
    err = (out.float().cpu() - want).abs()
    assert err.max().item() < 2e-2 and err.mean().item() < 2e-3, (err.max().item(), err.mean().item())
    assert (lse.cpu() - want_lse).abs().max().item() < 1e-3


@pytest.mark.parametrize("B,Q,K,Hq,Hkv,dtype", [
    (1, 1, 1, 4, 1, torch.bfloat16),       # a first token: one key
    (1, 1, 64, 8, 2, torch.bfloat16),      # exactly one sub-block
    (2, 1, 65, 8, 8, torch.float16),       # G = 1, one token into the second sub-block
    (1, 1, 255, 28, 4, torch.bfloat16),    # G = 7
    (1, 16, 1040, 2, 2, torch.float16),    # 16 tokens of one head
    (1, 3, 700, 10, 2, torch.bfloat16),    # 15 of the 16 rows, causal inside the call
    (3, 2, 4001, 16, 2, torch.float16),    # a cluster per row
    (40, 1, 300, 32, 8, torch.bfloat16),   # more rows than the GPU holds CTAs
    (1, 1, 20000, 4, 1, torch.bfloat16),   # one row: several clusters and the merge launch
    (33, 1, 1100, 2, 1, torch.bfloat16),   # too many rows for clusters of 8 at once: of 4
    (74, 1, 600, 2, 1, torch.float16),     # ... and for clusters of 4: of 2
    (38, 1, 1500, 16, 8, torch.bfloat16),  # more rows than CTAs: clusters in several waves
])
@pytest.mark.parametrize("workspace", [True, False])
def test_dense_decode_matches_oracle(ops, B, Q, K, Hq, Hkv, dtype, workspace):
    from oracle import compact_oracle as co
    g = torch.Generator().manual_seed(K + Q)
    q, k, v = (torch.randn((B, n, h, 128), generator=g).to(dtype) for n, h in ((Q, Hq), (K, Hkv), (K, Hkv)))
    want, want_lse = co.compact_attention(q, k, v, None, None, 64, return_lse=True)
    # a cache of permuted 64-token pages and (where the length allows the view) the contiguous tensors
    pages = -(-K // 64)
    perm = torch.randperm(B * pages, generator=g).to(torch.int32).view(B, pages)
    paged = []
    for t in (k, v):
        full = torch.zeros((B, pages * 64, Hkv, 128), dtype=dtype)
        full[:, :K] = t
        dst = torch.zeros((B * pages, 64, Hkv, 128), dtype=dtype)
        dst[perm.long()] = full.view(B, pages, 64, Hkv, 128)
        paged.append(dst.cuda())
    views = [ops.KvCacheView.from_paged(paged[0], paged[1], perm.cuda())]
    if K >= 64:
        views.append(ops.KvCacheView.from_seq_first(k.cuda(), v.cuda()))
    for kv in views:
        lse = torch.empty((B, Hq, Q), dtype=torch.float32, device="cuda")
        status = torch.zeros(1, dtype=torch.int32, device="cuda")
        out = ops.attn_compact(q.cuda(), kv, K, Hkv, None, None, lse=lse, status=status, use_workspace=workspace)
        assert int(status.item()) == 0
        _check(out, lse, want, want_lse)


@pytest.mark.parametrize("bs,Q,Hq,Hkv", [(64, 1, 8, 2), (128, 4, 4, 1), (64, 2, 28, 4)])
def test_table_decode_matches_oracle(ops, bs, Q, Hq, Hkv):
    from oracle import compact_oracle as co
    B, Pb = 2, 50
    K = Pb * bs + Q
    g = torch.Generator().manual_seed(bs + Q)
    q, k, v = (torch.randn((B, n, h, 128), generator=g).to(torch.bfloat16) for n, h in ((Q, Hq), (K, Hkv), (K, Hkv)))
    counts = torch.randint(0, Pb + 1, (B, Hkv), generator=g).to(torch.int32)
    counts[0, 0] = 0  # a row that reads nothing but the chunk
    counts[1, 0] = Pb // 2  # and one with entries, for the check of clamped ones
    idx = torch.full((B, Hkv, Pb), -1, dtype=torch.int32)
    for b in range(B):
        for h in range(Hkv):
            n = int(counts[b, h])
            idx[b, h, :n] = torch.randperm(Pb, generator=g)[:n].sort().values.to(torch.int32)
    want, want_lse = co.compact_attention(q, k, v, idx, counts, bs, return_lse=True)
    kv = ops.KvCacheView.from_seq_first(k.cuda(), v.cuda())
    lse = torch.empty((B, Hq, Q), dtype=torch.float32, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    wide = torch.zeros((B, Q, Hq, 160), dtype=torch.bfloat16, device="cuda")  # a strided destination
    ops.attn_compact(q.cuda(), kv, K, Hkv, idx.cuda(), counts.cuda(), block_size=bs, out=wide[..., :128], lse=lse, status=status)
    assert int(status.item()) == 0
    _check(wide[..., :128], lse, want, want_lse)
    assert not wide[..., 128:].any()
    # an entry out of range is clamped and reported, as by the kernel for longer chunks
    bad = idx.clone()
    bad[1, 0, 0] = Pb + 3
    ops.attn_compact(q.cuda(), kv, K, Hkv, bad.cuda(), counts.cuda(), block_size=bs, status=status)
    assert int(status.item()) == 2
