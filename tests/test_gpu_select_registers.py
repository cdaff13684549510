"""Rows that the rule kernel handles in registers (contiguous f32, at most 2048 key blocks) against the same scores in every other
place of a buffer, which take the general form: the keep bits have to be the same, whatever the scores."""
import pytest
import torch

pytestmark = pytest.mark.gpu

INF = float("inf")


def _scores(kind, shape, g):
    x = torch.randn(shape, generator=g, device="cuda")
    if kind == "outliers":       # the range of a few stretches the bins over the others: one bin holds most
        x[..., ::97] *= 1e4
    elif kind == "ties":
        x = (x * 3).round() / 3
    elif kind == "equal":
        x = torch.full_like(x, -0.75)
    elif kind == "zeros":        # of both signs
        x = torch.where(x > 0.5, x, torch.where(x > 0, 0.0, -0.0))
    elif kind == "not finite":
        x[..., ::50], x[..., 1::61], x[..., 2::71] = INF, -INF, float("nan")
    elif kind == "huge":         # the range itself overflows
        x = x * 3e38
    elif kind == "tiny":         # below the normal numbers
        x = x * 1e-40
    elif kind == "probabilities":
        x = (x * 4).softmax(-1)
    return x.nan_to_num(posinf=3.4e38, neginf=-3.4e38, nan=0.0) if kind == "huge" else x


@pytest.mark.parametrize("Kb", [1, 7, 31, 64, 250, 1016, 2047, 2048])
@pytest.mark.parametrize("kind", ["normal", "outliers", "ties", "equal", "zeros", "not finite", "huge", "tiny", "probabilities"])
def test_registers_and_general_form_agree(kind, Kb):
    from compactattention_b200 import ops
    B, H, Qb = 2, 3, min(5, Kb)
    g = torch.Generator(device="cuda").manual_seed(Kb)
    x = _scores(kind, (B, H, Qb, Kb), g)
    apart = torch.zeros((B, H, Qb, Kb, 2), device="cuda")
    apart[..., 0] = x
    apart = apart[..., 0]
    mask = torch.rand((B, 1, Qb, Kb), generator=g, device="cuda") < 0.7
    rules = [("topk", dict(topk_ratio=(200, 1000), sink=1, local=2)), ("topk", dict(topk_ratio=(1, 100))), ("topk", dict(topk_k=max(1, Kb // 2))),
             ("topk", dict(topk_k=Kb)), ("threshold", dict(threshold=0.3)), ("threshold", dict(threshold=-INF, local=1)),
             ("topk", dict(topk_ratio=(1, 2), rows_voting=1))]
    for rule, kw in rules:
        for valid in (None, mask, torch.zeros_like(mask)):
            got, want = (ops.select_rows(t, Kb - Qb, rule, valid=valid, **kw) for t in (x, apart))
            assert torch.equal(got, want), (rule, kw, valid is not None)
