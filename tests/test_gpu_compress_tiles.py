"""The tensor-core write kernel for 16-bit vectors at the edges of its tiles, every head_dim it takes."""

import pytest
import torch

from oracle import tq4_oracle as O
from tests.helpers import Prims, index_mismatch, ulp_diff

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [64, 96, 128, 256])
@pytest.mark.parametrize("n_tok,h,dtype,strided", [
    (1201, 3, torch.bfloat16, False),   # just past the line to this kernel; heads that do not divide a tile
    (512, 4, torch.float16, True),     # whole tiles; K and V halves of one tensor
    (1057, 8, torch.bfloat16, True),   # a remainder of one token
])
def test_paged_write_tiles(cuda_lib, d, n_tok, h, dtype, strided):
    from turboquant_vllm.kernels import ops

    pr = Prims(d)
    p = pr.cuda()
    k, v = O.synthetic_kv(n_tok, h, d, seed=n_tok + d, dtype=dtype)
    bs = 16
    nblk = n_tok // bs + 2
    width = h * O.padded_slot_bytes(d)
    slots = torch.randperm(nblk * bs, generator=torch.Generator().manual_seed(d))[:n_tok]
    slots[3] = slots[-1] = -1
    keep = slots >= 0
    ref = torch.zeros(nblk, bs, width, dtype=torch.uint8)
    O.write_paged(k[keep], v[keep], ref, slots[keep], pr.rot, pr.kb, pr.vb)
    kc, vc = k.cuda(), v.cuda()
    if strided:
        kc, vc = torch.cat([kc, vc], dim=1).split(h, dim=1)
    cache = torch.zeros(nblk, bs, width, dtype=torch.uint8, device="cuda")
    ops.tq4_write_paged(kc, vc, cache, slots.cuda(), p["even"], p["odd"], p["kb"], p["vb"])
    got, want = cache.cpu().view(-1, width), ref.view(-1, width)
    kn, vi, vn, end = O.row_layout(h, d)
    for a, b in ((0, kn), (vi, vn)):
        assert index_mismatch(got[:, a:b].contiguous(), want[:, a:b].contiguous()) <= 1e-4
    for a in (kn, vn):
        x, y = (t[:, a:a + 4 * h].contiguous().view(torch.float32) + 1e-30 for t in (got, want))
        assert ulp_diff(x, y).max() <= 4
    assert torch.equal(got[:, end:], want[:, end:])
    if d != 128 or 2 * n_tok * h <= 8192:  # coordinates on a boundary are summed again: the bytes are those of the kernels for few vectors
        parts = torch.zeros_like(cache)
        for i in range(0, n_tok, 32):
            ops.tq4_write_paged(kc[i:i + 32], vc[i:i + 32], parts, slots[i:i + 32].cuda(), p["even"], p["odd"], p["kb"], p["vb"])
        assert torch.equal(cache, parts)
    assert ops.read_and_clear_errors(torch.device("cuda")) == 0


@pytest.mark.parametrize("d,dtype", [(64, torch.float16), (96, torch.float16), (128, torch.float16), (256, torch.float16), (256, torch.bfloat16)])
def test_coordinates_on_a_boundary(cuda_lib, golden, d, dtype):
    """Vectors with a coordinate whose two sums, the tensor cores' and the FMA chain's, lie 1.6e-7 - 2.4e-7 apart on either side of
    a boundary (found among 2.5e12 coordinates of vectors that few coordinates dominate): the bytes are the FMA kernels'."""
    from turboquant_vllm.kernels import ops

    pr = Prims(d)
    p = pr.cuda()
    hard = torch.from_numpy(golden("near_boundary.npz")[f"d{d}_{str(dtype)[6:]}"]).view(dtype).cuda()
    few, few_norms = ops.tq4_compress(hard[:, None].contiguous(), p["even"], p["odd"], p["kb"])
    n = {64: 6601, 96: 3101, 128: 4801, 256: 1101}[d]  # the tensor-core kernel's turn
    x = torch.randn(n, d, generator=torch.Generator().manual_seed(d)).to(dtype).cuda()
    at = torch.arange(0, n, 5, device="cuda")  # (six rows of a warp: its list runs full)
    x[at] = hard[at // 5 % len(hard)]
    packed, norms = ops.tq4_compress(x[:, None].contiguous(), p["even"], p["odd"], p["kb"])
    assert torch.equal(packed[at], few[at // 5 % len(hard)]) and torch.equal(norms[at], few_norms[at // 5 % len(hard)])
