"""How the attention kernel deals its work out: causal chunks whose units differ in length, units cut and whole, a
row per CTA and many, more segments per CTA than one planning batch holds.  Against fp32 attention in plain torch."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from compactattention_b200 import ops as _ops
    return _ops


def _reference(q, k, v, past):
    """fp32 causal attention of one sequence, ``q [Q, Hq, D]``, ``k/v [K, Hkv, D]``."""
    group = q.shape[1] // k.shape[1]
    qf, kf, vf = q.float().transpose(0, 1), k.float().repeat_interleave(group, 1).transpose(0, 1), v.float().repeat_interleave(group, 1).transpose(0, 1)
    hidden = torch.arange(k.shape[0], device=q.device).view(1, -1) > past + torch.arange(q.shape[0], device=q.device).view(-1, 1)
    s = (qf @ kf.transpose(1, 2) * q.shape[-1] ** -0.5).masked_fill(hidden, float("-inf"))
    return (s.softmax(-1) @ vf).transpose(0, 1), s.logsumexp(-1)


@pytest.mark.parametrize("B,Q,past,Hq,Hkv,workspace", [
    (1, 4096, 0, 8, 2, True),      # first chunk: units of 1 to 32 steps, cut
    (1, 4096, 0, 8, 2, False),     # the same without a workspace: whole units by their share of the work
    (2, 3000, 0, 28, 4, True),     # 18 tokens to a tile, a ragged end
    (1, 700, 5000, 8, 1, True),    # few long units: cut over many CTAs
    (1, 700, 5000, 8, 1, False),
    (3, 130, 64, 4, 4, True),      # G = 1, a second pair of tiles of one token or none
    (1, 200, 77, 12, 4, True),     # short units, one per CTA
    (128, 320, 0, 64, 8, True),    # 69 units to a CTA: more than one planning batch
])
def test_dense_chunks(ops, B, Q, past, Hq, Hkv, workspace):
    K = past + Q
    g = torch.Generator(device="cuda").manual_seed(Q + past)
    q = torch.randn((B, Q, Hq, 128), generator=g, device="cuda", dtype=torch.bfloat16)
    pages = -(-K // 64)
    k, v = (torch.zeros((B, pages * 64, Hkv, 128), device="cuda", dtype=torch.bfloat16) for _ in range(2))
    for t in (k, v):
        t[:, :K] = torch.randn((B, K, Hkv, 128), generator=g, device="cuda", dtype=torch.bfloat16)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    lse = torch.empty((B, Hq, Q), dtype=torch.float32, device="cuda")
    out = ops.attn_compact(q, ops.KvCacheView.from_seq_first(k, v), K, Hkv, None, None, lse=lse, status=status, use_workspace=workspace)
    assert int(status.item()) == 0
    for b in range(0, B, max(1, B // 8)):
        want, want_lse = _reference(q[b], k[b, :K], v[b, :K], past)
        err = (out[b].float() - want).abs()
        # rows that see few keys have outputs of order 1: a bf16 rounding of P and of the output, 2^-8 of up to ~4
        assert err.max().item() < 3.2e-2 and err.mean().item() < 2e-3, (b, err.max().item(), err.mean().item())
        assert (lse[b] - want_lse).abs().max().item() < 1e-3


def test_rows_of_unequal_length(ops):
    """A block table whose rows keep from none to all of the past blocks: the spans follow the rows' work."""
    B, Q, past, Hq, Hkv, bs = 1, 512, 64 * 200, 16, 4, 64
    K, blocks = past + Q, past // bs
    g = torch.Generator(device="cuda").manual_seed(5)
    q, k, v = (torch.randn((B, n, h, 128), generator=g, device="cuda", dtype=torch.float16) for n, h in ((Q, Hq), (K, Hkv), (K, Hkv)))
    counts = torch.tensor([[0, 3, 77, blocks]], dtype=torch.int32)
    idx = torch.full((B, Hkv, blocks), -1, dtype=torch.int32)
    for h in range(Hkv):
        n = int(counts[0, h])
        idx[0, h, :n] = torch.randperm(blocks, generator=torch.Generator().manual_seed(h))[:n].sort().values.to(torch.int32)
    for workspace in (True, False):
        status = torch.zeros(1, dtype=torch.int32, device="cuda")
        out = ops.attn_compact(q, ops.KvCacheView.from_seq_first(k, v), K, Hkv, idx.cuda(), counts.cuda(), block_size=bs, status=status,
                               use_workspace=workspace)
        assert int(status.item()) == 0
        for h in range(Hkv):
            n = int(counts[0, h])
            tok = torch.cat([(idx[0, h, :n].long().view(-1, 1) * bs + torch.arange(bs)).reshape(-1), torch.arange(past, K)]).cuda()
            want, _ = _reference(q[0, :, h * 4 : h * 4 + 4], k[0, tok, h : h + 1], v[0, tok, h : h + 1], n * bs)
            err = (out[0, :, h * 4 : h * 4 + 4].float() - want).abs()
            assert err.max().item() < 1e-2 and err.mean().item() < 5e-4, (h, workspace, err.max().item())


@pytest.mark.parametrize("B,Q,past,Hq,Hkv,cut", [
    (9, 128, 1152, 32, 8, False),   # a unit to nearly every SM, all of a length
    (1, 1152, 0, 32, 8, False),
    (1, 128, 8192, 32, 8, True),    # few units of 65 steps
])
def test_the_merge_is_launched_where_units_are_cut(ops, B, Q, past, Hq, Hkv, cut):
    from compactattention_b200 import _lib
    K = past + Q
    g = torch.Generator(device="cuda").manual_seed(Q)
    q, k, v = (torch.randn((B, n, h, 128), generator=g, device="cuda", dtype=torch.bfloat16) for n, h in ((Q, Hq), (K, Hkv), (K, Hkv)))
    kv = ops.KvCacheView.from_seq_first(k, v)
    before = _lib.launch_count()
    out = ops.attn_compact(q, kv, K, Hkv, None, None)
    assert _lib.launch_count() - before == (2 if cut else 1)
    whole = ops.attn_compact(q, kv, K, Hkv, None, None, use_workspace=False)
    assert torch.equal(out, whole) != cut  # whole units sum their steps in one order, cut ones in another
