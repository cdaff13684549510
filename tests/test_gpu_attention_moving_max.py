"""Scores whose row maximum moves from KV step to KV step, so that the attention kernel rescales its accumulator between P.V
products and forms P again: units of one step, of one 64-token sub-block, of several, cut and whole.  Against fp32 in plain torch."""
import pytest
import torch

from test_gpu_attention_schedule import _reference

pytestmark = pytest.mark.gpu

# log2 units by which a 128-token step's scores lie above the one before (the kernel rescales from 8 on)
MOVES = {"up": lambda j: 9.0 * j, "down": lambda j: -9.0 * j, "zigzag": lambda j: 14.0 * (j % 2) + 2.0 * j, "below the line": lambda j: 3.0 * j}


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("Q,past,workspace", [(64, 0, True), (100, 28, True), (64, 64, True), (129, 63, False), (256, 1000, False), (256, 3008, True)])
@pytest.mark.parametrize("move", sorted(MOVES))
def test_moving_maximum(move, Q, past, workspace, dtype):
    from compactattention_b200 import ops
    Hq, Hkv, D, K = 8, 2, 128, past + Q
    g = torch.Generator(device="cuda").manual_seed(Q + past)
    level = torch.tensor([MOVES[move](j) for j in range(-(-K // 128))], device="cuda").repeat_interleave(128)[:K]
    q = torch.randn((1, Q, Hq, D), generator=g, device="cuda")
    q[..., 0] = 16.0
    k = torch.randn((1, K, Hkv, D), generator=g, device="cuda")
    k[..., 0] = (level / (16.0 * D ** -0.5 * 1.4427)).view(1, K, 1)
    v = torch.randn((1, K, Hkv, D), generator=g, device="cuda")
    pad = -K % 64
    q, k, v = q.to(dtype), *(torch.nn.functional.pad(t, (0, 0, 0, 0, 0, pad)).to(dtype) for t in (k, v))
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    lse = torch.empty((1, Hq, Q), dtype=torch.float32, device="cuda")
    out = ops.attn_compact(q, ops.KvCacheView.from_seq_first(k, v), K, Hkv, None, None, lse=lse, status=status, use_workspace=workspace)
    assert int(status.item()) == 0
    want, want_lse = _reference(q[0], k[0, :K], v[0, :K], past)
    err = (out[0].float() - want).abs()
    # a row may see one key only, so P's and the output's rounding are of values up to ~4: 2^-8 (bf16) or 2^-11 (f16) of them, twice
    unit = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    assert err.max().item() < 8 * unit and err.mean().item() < 0.5 * unit
    assert (lse[0] - want_lse).abs().max().item() < 1e-5 * want_lse.abs().max().item() + 1e-3
