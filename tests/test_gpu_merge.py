"""The merge kernel at the edges of its splits: vectors per block, partials per warp, column blocks."""

import pytest
import torch

from tests.helpers import Prims, cosine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [64, 96, 128, 256])
@pytest.mark.parametrize("rows,hq,world", [(1, 1, 1), (1, 28, 65), (37, 2, 8), (74, 4, 9), (149, 8, 33), (300, 5, 7)])
def test_merge_matches_fp32(d, rows, hq, world):
    from turboquant_vllm.kernels import ops

    g = torch.Generator().manual_seed(d + rows)
    o = torch.randn(world, rows, hq, d, generator=g)
    lse = 4 * torch.randn(world, rows, hq, generator=g)
    lse[0, 0, 0] = float("-inf")  # an empty part
    rot = Prims(d).rot
    w = torch.exp(lse - lse.max(dim=0, keepdim=True).values.clamp_min(-1e30))
    den = w.sum(0)
    want = torch.where(den[..., None] > 0, (w[..., None] * o).sum(0) / den.clamp_min(1e-30)[..., None], 0.0) @ rot
    for dtype in (torch.float32, torch.bfloat16):
        got = ops.combine_partials(o.cuda(), lse.cuda(), rot.cuda(), out_dtype=dtype).cpu()
        tol = 2e-5 if dtype == torch.float32 else 2e-2
        assert (got.float() - want).abs().max() <= tol
        assert world == 1 or cosine(got.float(), want) >= 0.9999
