"""The keep mask's 16-byte loads in the table builder: any nonzero byte keeps a block; lengths, offsets and strides
that the wide loads do not fit take the byte loads."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Kb", [32, 64, 70, 2048])
@pytest.mark.parametrize("offset,step", [(0, 1), (16, 1), (3, 1), (0, 2)])
def test_mask_forms(Kb, offset, step):
    from compactattention_b200 import ops
    B, Hkv, G, Pb = 2, 3, 2, Kb - 2
    g = torch.Generator().manual_seed(Kb + offset)
    room = torch.randint(0, 256, (B, Hkv * G, 1, offset + Kb * step + 16), generator=g).to(torch.uint8)
    room = room * (torch.rand(room.shape, generator=g) < 0.3)
    mask = room.cuda()[..., offset : offset + Kb * step : step]
    table = ops.union_table(mask=mask, num_kv_heads=Hkv, kv_blocks=Kb, past_blocks=Pb)
    keep = (mask.cpu() != 0).any(2).view(B, Hkv, G, Kb).any(2)[..., :Pb]
    for b in range(B):
        for h in range(Hkv):
            want = keep[b, h].nonzero().flatten().to(torch.int32)
            n = int(table.counts[b, h])
            assert n == want.numel() and torch.equal(table.block_idx[b, h, :n].cpu(), want)
