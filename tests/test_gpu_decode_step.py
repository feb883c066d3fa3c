"""The kernel of small decode steps (a cluster of CTAs per row and KV head) next to the streaming kernel."""

import pytest
import torch

from tests.helpers import Prims, build_paged_case

pytestmark = pytest.mark.gpu

LENS = [1, 15, 17, 129, 300, 0]  # one tile and less, a tile's edge, fewer tiles than a cluster's warps, more, none
CASES = [  # head_dim, q heads, KV heads, lengths, page, padded rows, window
    (128, 28, 4, [1024], 16, True, None),         # two column blocks of heads; clusters of eight
    (128, 32, 8, [700, 33], 16, True, None),
    (128, 32, 8, LENS, 16, True, None),           # clusters of four
    (128, 32, 8, LENS * 2, 32, True, None),       # clusters of two
    (128, 4, 1, LENS, 48, False, None),           # 136-byte rows: 4-byte loads; pages that are no power of two
    (128, 20, 2, [300, 17], 16, True, 100),       # groups of ten: two sets of heads
    (96, 8, 8, LENS, 16, True, None),
    (64, 14, 2, LENS, 16, True, 64),
    (256, 8, 4, LENS, 16, True, None),
    (256, 12, 2, [90, 300], 16, False, None),     # groups of six at head_dim 256
]


def _run(ops, nv, args, **kw):
    nv.profile_start(8)
    out = ops.paged_tq4_attention(*args, **kw)
    merges = len(nv.profile_read(nv.PROF_COMBINE, 8))
    nv.profile_stop()
    return out, merges


@pytest.mark.parametrize("d,hq,hkv,lens,page,padded,window", CASES)
@pytest.mark.parametrize("rotated", [False, True])
def test_against_the_streaming_kernel(cuda_lib, d, hq, hkv, lens, page, padded, window, rotated):
    """Same tables and sums of the same terms; queries and weights as two fp16 terms (2^-22 of a score of about ten: 2^-18 of
    a weight), partials in another order."""
    from turboquant_vllm import _native as nv
    from turboquant_vllm.kernels import ops

    pr = Prims(d, v_bits=3 if page == 32 else 4)
    p = pr.cuda()
    case = build_paged_case(lens, hkv, d, page, pr, seed=5, padded=padded)
    q = torch.randn(len(lens), hq, d, generator=torch.Generator().manual_seed(1)).cuda()
    args = (q, case["cache"].cuda(), case["block_table"].cuda(), case["seq_lens"].cuda(), p["kc"], p["vc"], p["rot"], hkv, page)
    got = []
    for mode in (0, 2):
        lse = torch.empty(len(lens), hq, device="cuda")
        out, merges = _run(ops, nv, args, sliding_window=window, mode=mode, lse_out=lse, out_rotated=rotated)
        assert merges == (mode == 2)
        got.append((out.double(), lse))
    (a, la), (b, lb) = got
    assert (a - b).norm() / b.norm() <= 2.0**-18
    assert torch.equal(torch.isinf(la), torch.isinf(lb)) and torch.allclose(la, lb, atol=1e-4, rtol=0)
    for i, n in enumerate(lens):
        assert n > 0 or (a[i] == 0).all()
    half = torch.empty(len(lens), hq, d + 2, dtype=torch.float16, device="cuda")[..., :d]
    ops.paged_tq4_attention(*args, sliding_window=window, out=half, out_rotated=rotated)
    assert torch.equal(half, a.float().half())
    assert ops.read_and_clear_errors(torch.device("cuda")) == 0


@pytest.mark.parametrize("power", [-100, -20, 20, 100])
def test_large_and_small_queries(cuda_lib, power):
    from turboquant_vllm import _native as nv
    from turboquant_vllm.kernels import ops

    p = Prims(128).cuda()
    case = build_paged_case([200, 90], 8, 128, 16, Prims(128), seed=5, padded=True)
    q = torch.randn(2, 32, 128, generator=torch.Generator().manual_seed(1)).cuda()
    rest = (case["cache"].cuda(), case["block_table"].cuda(), case["seq_lens"].cuda(), p["kc"], p["vc"], p["rot"], 8, 16)
    want, _ = _run(ops, nv, (q, *rest), sm_scale=0.1, mode=2)
    out, merges = _run(ops, nv, (q * 2.0**power, *rest), sm_scale=0.1 * 2.0**-power)
    assert merges == 0 and (out - want).double().norm() / want.double().norm() <= 2.0**-18


def test_rows_of_several_queries_and_bad_pages(cuda_lib):
    """A call with query_start_loc of few rows takes the kernel, too; a page out of range is masked and reported, a length
    beyond the table's row is cut and reported."""
    from turboquant_vllm import _native as nv
    from turboquant_vllm.kernels import ops

    pr = Prims(128)
    p = pr.cuda()
    case = build_paged_case([100, 40, 60], 4, 128, 16, pr, seed=5, padded=True)
    q = torch.randn(9, 8, 128, generator=torch.Generator().manual_seed(1)).cuda()  # (the last row: of no sequence)
    qsl = torch.tensor([0, 5, 5, 8], dtype=torch.int32).cuda()
    bt, lens = case["block_table"].clone(), case["seq_lens"].clone()
    for broken in (False, True):
        if broken:
            bt[0, 2] = 10_000
            lens[2] = 10_000
        args = (q, case["cache"].cuda(), bt.cuda(), lens.cuda(), p["kc"], p["vc"], p["rot"], 4, 16)
        for causal in (True, False):
            (a, ma), (b, mb) = (_run(ops, nv, args, query_start_loc=qsl, causal=causal, mode=m) for m in (0, 2))
            assert (ma, mb) == (0, 1) and (a[8] == 0).all()
            assert (a - b).double().norm() / b.double().norm() <= 2.0**-18
        assert ops.read_and_clear_errors(torch.device("cuda")) == (nv.DEV_BAD_BLOCK if broken else 0)


@pytest.mark.parametrize("d,rows,keys,steps", [
    (128, 1, 8192, 1), (128, 1, 8208, 0),      # 8 units
    (128, 2, 5120, 1), (128, 2, 5136, 0),
    (128, 8, 2560, 1), (128, 8, 2576, 0), (128, 9, 2560, 0),
    (128, 18, 1024, 1), (128, 18, 1040, 0), (128, 19, 1024, 0),
])
def test_which_calls_take_it(cuda_lib, d, rows, keys, steps):
    """The longest context that the table (or the caller) allows decides, whatever the lengths are."""
    from turboquant_vllm import _native as nv
    from turboquant_vllm.kernels import ops

    p = Prims(d).cuda()
    case = build_paged_case([40] * rows, 8, d, 16, Prims(d), seed=5, padded=True)
    table = torch.zeros(rows, 1024, dtype=torch.int32)
    table[:, : case["block_table"].shape[1]] = case["block_table"]
    q = torch.randn(rows, 32, d, generator=torch.Generator().manual_seed(1)).cuda()
    rest = (case["seq_lens"].cuda(), p["kc"], p["vc"], p["rot"], 8, 16)
    a, ma = _run(ops, nv, (q, case["cache"].cuda(), table[:, : keys // 16].contiguous().cuda(), *rest))
    b, mb = _run(ops, nv, (q, case["cache"].cuda(), table.cuda(), *rest), max_seq_len=keys)
    assert ma == mb == 1 - steps and torch.equal(a, b)
