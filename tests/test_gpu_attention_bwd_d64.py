"""The fused backward at head_dim 64 (three Q stages, two dS^T tiles, dQ in TMEM columns of its own), where its rings start,
wrap and end: one item, a few, many; lengths cut inside a tile; query heads divided over CTAs."""
import pytest
import torch

from helpers import compare
from oracle import attention_oracle as ao

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("batch,q_len,hq,hkv,doc", [
    (1, 64, 1, 1, 64),              # one item, half a tile
    (1, 128, 2, 1, 128),            # one tile, the heads of the group divided over two CTAs
    (2, 448, 3, 1, 448),            # up to four query tiles per kv tile and head, three heads in one CTA: rings wrap
    (1, 1600, 2, 2, 700),           # thirteen tiles, the last one half full, several documents
    (3, 192, 8, 8, 50),             # partial tiles only
])
def test_fused_backward_d64(batch, q_len, hq, hkv, doc, dtype):
    from kvax_b200.ops.flash_attention import attention_backward, attention_forward, check_status
    from kvax_b200.ops.mask_creator import build_masks

    d, blocks = 64, (64, 64)
    i = torch.arange(q_len, dtype=torch.int32, device="cuda").repeat(batch, 1)
    seg, pos = i // doc, i % doc
    seg[-1, q_len - q_len // 8:] = -1               # padding at the end of the last row
    g = torch.Generator(device="cuda").manual_seed(11)

    def randn(h):
        return torch.randn(batch, q_len, h, d, generator=g, device="cuda").to(dtype)

    q, k, v, do = randn(hq), randn(hkv), randn(hkv), randn(hq) * (seg != -1)[:, :, None, None]
    masks = build_masks(pos, seg, pos, seg, [(64, 64, False), (64, 64, False), (64, 64, True)], True)
    out, lse, _ = attention_forward(q, k, v, pos, seg, pos, seg, masks[0], blocks, d ** -0.5)
    dq, dk, dv, status = attention_backward(q, k, v, out, do, lse, pos, seg, pos, seg, masks[1], masks[2], blocks, d ** -0.5, mode="fused")
    torch.cuda.synchronize()
    check_status(status, "attention")
    ref = ao.attention_dense_torch(q.float(), k.float(), v.float(), pos, seg, pos, seg, d ** -0.5, dout=do.float())
    rows = (seg != -1)[:, :, None, None].cpu().numpy()
    compare("dq", dq.float().cpu().numpy(), ref["dq"].cpu().numpy(), rows, bf16_output=True)
    compare("dk", dk.cpu().numpy(), ref["dk"].cpu().numpy(), rows)
    compare("dv", dv.cpu().numpy(), ref["dv"].cpu().numpy(), rows)
