"""The prologue kernel (query rotation + cache write of a step) at the edges of its column blocks."""

import pytest
import torch

from oracle import tq4_oracle as O
from tests.helpers import Prims, build_paged_case, cosine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 3, 100, 260])  # a block per vector; 32-column blocks; past one wave of them
@pytest.mark.parametrize("d", [64, 96, 128, 256])
def test_step_writes_and_rotates(cuda_lib, d, rows):
    from turboquant_vllm.kernels import ops

    hq, hkv, bs = 8, 4, 16
    pr = Prims(d)
    p = pr.cuda()
    lens = [1 + (7 * i) % 37 for i in range(rows)]
    case = build_paged_case(lens, hkv, d, bs, pr, seed=d, padded=True)
    bt = case["block_table"]
    slots = torch.tensor([int(bt[i, (s - 1) // bs]) * bs + (s - 1) % bs for i, s in enumerate(lens)])
    k, v = (x.cuda() for x in O.synthetic_kv(rows, hkv, d, seed=3, dtype=torch.bfloat16))
    q = torch.randn(rows, hq, d, generator=torch.Generator().manual_seed(1)).bfloat16()
    want = case["cache"].cuda()
    ops.tq4_write_paged(k, v, want, slots.cuda(), p["even"], p["odd"], p["kb"], p["vb"])
    cache = case["cache"].cuda()
    out = ops.paged_tq4_attention(
        q.cuda(), cache, bt.cuda(), case["seq_lens"].cuda(), p["kc"], p["vc"], p["rot"], hkv, bs,
        out_dtype=torch.float32, write=(k, v, slots.cuda(), p["even"], p["odd"], p["kb"], p["vb"]))
    assert torch.equal(cache, want)
    alone = ops.paged_tq4_attention(  # without a write: the queries of few rows are rotated from Pi itself
        q.cuda(), want, bt.cuda(), case["seq_lens"].cuda(), p["kc"], p["vc"], p["rot"], hkv, bs, out_dtype=torch.float32)
    assert torch.equal(alone, out)
    pick = sorted({0, rows // 2, rows - 1})
    ref = O.paged_decode_fp32(q[pick], want.cpu(), bt[pick], [lens[i] for i in pick], pr.kc, pr.vc, pr.rot, hkv)
    got = out.cpu()[pick]
    assert cosine(got, ref) >= 0.9999 and (got - ref).abs().max() <= 2e-3
    assert ops.read_and_clear_errors(torch.device("cuda")) == 0
