"""The tile-list builder at its edges, seen through the attention kernels that walk the lists (dense reference on the GPU):
tiles cut into few and into many runs, more partial tiles than the pool of element masks holds, tiles at the end of
either side, indices instead of positions."""
import numpy as np
import pytest
import torch

from helpers import compare
from oracle import attention_oracle as ao

pytestmark = pytest.mark.gpu


def _tokens(layout, batch, n, rng):
    pos = np.broadcast_to(np.arange(n, dtype=np.int32), (batch, n)).copy()
    if layout == "one_document":                    # diagonal tiles only are partial; the last tiles are cut
        return pos, np.zeros((batch, n), np.int32)
    if layout == "runs_of_9":                       # 14 to 16 runs per tile: the interval path at its limit
        return pos, ((pos // 9) % 3).astype(np.int32)
    if layout == "scattered":                       # a run per token, positions not ascending: token by token, and more
        return rng.permuted(pos, axis=1), rng.integers(0, 3, (batch, n)).astype(np.int32)   # partial tiles than the pool has masks
    seg = np.full((batch, n), -1, np.int32)         # "documents": positions restart, padding at the end
    for b in range(batch):
        at, d = 0, 0
        while at < n - 90:
            m = min(int(rng.integers(20, 700)), n - 90 - at)
            seg[b, at:at + m], pos[b, at:at + m] = d, np.arange(m)
            at, d = at + m, d + 1
        pos[b, at:] = np.arange(n - at)
    return pos, seg


@pytest.mark.parametrize("blocks", [(128, 128), (64, 64)])
@pytest.mark.parametrize("layout,sequential", [("one_document", False), ("runs_of_9", False), ("runs_of_9", True), ("scattered", False),
                                               ("documents", False)])
@pytest.mark.parametrize("q_len,kv_len", [(2240, 2240), (200, 1090)])
def test_lists(layout, sequential, q_len, kv_len, blocks):
    from kvax_b200.ops.flash_attention import attention_backward, attention_forward, check_status
    from kvax_b200.ops.mask_creator import build_masks

    if sequential and q_len != kv_len:
        pytest.skip("indices are positions: queries and keys start at the same token")
    rng = np.random.default_rng(q_len + len(layout))
    batch, hq, hkv, d = 2, 4, 2, 128
    pos, seg = _tokens(layout, batch, kv_len, rng)
    pos, seg = torch.from_numpy(pos).cuda(), torch.from_numpy(seg).cuda()
    qp, qs = pos[:, kv_len - q_len:].contiguous(), seg[:, kv_len - q_len:].contiguous()
    g = torch.Generator(device="cuda").manual_seed(7)

    def randn(n, h):
        return torch.randn(batch, n, h, d, generator=g, device="cuda").to(torch.bfloat16)

    q, k, v = randn(q_len, hq), randn(kv_len, hkv), randn(kv_len, hkv)
    do = randn(q_len, hq) * (qs != -1)[:, :, None, None]
    bq, bk = blocks
    masks = build_masks(qp, qs, pos, seg, [(bq, bk, False), (bk, bq, False), (bq, bk, True)], True)
    scale = d ** -0.5
    out, lse, _ = attention_forward(q, k, v, qp, qs, pos, seg, masks[0], blocks, scale, sequential)
    grads = {m: attention_backward(q, k, v, out, do, lse, qp, qs, pos, seg, masks[1], masks[2], blocks, scale, sequential, mode=m)
             for m in ("fused", "two_kernel")}
    torch.cuda.synchronize()
    check_status(grads["fused"][3], "attention")
    ref = ao.attention_dense_torch(q.float(), k.float(), v.float(), qp, qs, pos, seg, scale, dout=do.float())
    rows, kv_rows = (qs != -1)[:, :, None, None].cpu().numpy(), (seg != -1)[:, :, None, None].cpu().numpy()
    compare("out", out.float().cpu().numpy(), ref["out"].cpu().numpy(), rows, bf16_output=True)
    for mode, (dq, dk, dv, _) in grads.items():
        compare(f"{mode} dq", dq.float().cpu().numpy(), ref["dq"].cpu().numpy(), rows, bf16_output=True)
        compare(f"{mode} dk", dk.cpu().numpy(), ref["dk"].cpu().numpy(), kv_rows)
        compare(f"{mode} dv", dv.cpu().numpy(), ref["dv"].cpu().numpy(), kv_rows)
