"""The tcgen05 prefill kernel at the edges of its row blocks, tiles, key splits and row layouts."""

import numpy as np
import pytest
import torch

from oracle import tq4_oracle as O
from tests.helpers import Prims, build_paged_case, cosine

pytestmark = pytest.mark.gpu

CASES = [  # head_dim, q heads, KV heads, lengths, new rows, mode, window, causal, padded rows
    (128, 4, 4, [64], [16], 3, None, True, True),            # one row block, one full tile
    (128, 8, 2, [300, 90], [120, 90], 3, None, True, True),  # a last CTA with one of its two blocks in use
    (128, 28, 4, [150], [150], 3, None, True, True),         # groups of 7: 126 of 128 lanes
    (128, 8, 4, [65], [65], 3, None, True, True),            # one key in the second tile
    (128, 32, 8, [3000], [40], 3, None, True, True),         # cut along the keys
    (128, 32, 8, [3000, 0, 20], [8, 8, 8], 3, None, True, True),  # ... parts without keys, a sequence without any
    (256, 8, 4, [2000, 0, 20], [8, 8, 8], 3, None, True, True),
    (128, 4, 1, [700], [333], 3, None, False, False),        # 136-byte rows: 4-byte loads; not causal
    (64, 14, 2, [333], [200], 3, None, True, True),
    (96, 4, 4, [300, 41], [100, 9], 3, None, True, False),
    (256, 8, 4, [300, 90], [120, 90], 3, 64, True, True),
    (256, 2, 2, [700], [9], 3, None, True, True),
    (128, 32, 8, [300, 90, 50, 77], [120, 1, 7, 77], 0, None, True, True),  # long and short sequences
    (256, 8, 4, [900, 90, 8], [300, 1, 8], 0, None, True, True),
    (128, 8, 2, [300, 90, 50, 77], [120, 1, 7, 77], 0, None, True, True),   # few rows: the streaming kernel alone
    (256, 8, 4, [900, 90, 8], [12, 1, 8], 0, None, True, True),
]


@pytest.mark.parametrize("d,hq,hkv,lens,new,mode,window,causal,padded", CASES)
def test_prefill_edges(cuda_lib, d, hq, hkv, lens, new, mode, window, causal, padded):
    from turboquant_vllm.kernels import ops

    pr = Prims(d)
    p = pr.cuda()
    case = build_paged_case(lens, hkv, d, 16, pr, seed=5, padded=padded)
    q = torch.randn(sum(new), hq, d, generator=torch.Generator().manual_seed(1)).bfloat16()
    qsl = torch.tensor(np.concatenate([[0], np.cumsum(new)]), dtype=torch.int32)
    lse = torch.empty(sum(new), hq, device="cuda")
    out = ops.paged_tq4_attention(
        q.cuda(), case["cache"].cuda(), case["block_table"].cuda(), case["seq_lens"].cuda(), p["kc"], p["vc"], p["rot"],
        hkv, 16, query_start_loc=qsl.cuda(), causal=causal, sliding_window=window, out_dtype=torch.float32, mode=mode,
        lse_out=lse).cpu()
    ref, ref_lse = O.paged_attention_fp32(q, case["cache"], case["block_table"], lens, qsl, pr.kc, pr.vc, pr.rot, hkv, None,
                                          causal, window, return_lse=True)
    assert cosine(out, ref) >= 0.9999 and (out - ref).abs().max() <= 2e-3
    assert torch.allclose(lse.cpu(), ref_lse.reshape(lse.shape), atol=1e-3, rtol=1e-4)
    assert ops.read_and_clear_errors(torch.device("cuda")) == 0


@pytest.mark.parametrize("d,hq,hkv,lens,new,rows,mode", [
    (128, 8, 2, [300, 90], [120, 90], 211, 3),     # one row past the last offset
    (128, 32, 8, [3000, 50], [40, 9], 300, 3),     # many, the call cut along the keys
    (256, 8, 4, [300], [20], 300, 3),
    (64, 14, 2, [400], [400], 600, 0),             # one long sequence: the prefill kernel alone
    (128, 32, 8, [300, 90], [120, 1], 300, 0),     # both kernels
    (128, 32, 8, [300, 90], [120, 1], 300, 2),
])
def test_rows_of_no_sequence_are_zero(cuda_lib, d, hq, hkv, lens, new, rows, mode):
    """Rows past the last offset of query_start_loc: zeros and an LSE of -inf, whichever kernel the call takes."""
    from turboquant_vllm.kernels import ops

    pr = Prims(d)
    p = pr.cuda()
    case = build_paged_case(lens, hkv, d, 16, pr, seed=5, padded=True)
    q = torch.randn(rows, hq, d, generator=torch.Generator().manual_seed(1)).bfloat16().cuda()
    qsl = torch.tensor(np.concatenate([[0], np.cumsum(new)]), dtype=torch.int32).cuda()
    n = sum(new)
    args = (case["cache"].cuda(), case["block_table"].cuda(), case["seq_lens"].cuda(), p["kc"], p["vc"], p["rot"], hkv, 16)
    ws = torch.full((ops.attention_workspace_bytes(rows, hq, hkv, d),), 0x7f, dtype=torch.uint8, device="cuda")
    for rotated in (False, True):
        out, lse = torch.full((rows, hq, d), 7.0, device="cuda"), torch.full((rows, hq), 7.0, device="cuda")
        ops.paged_tq4_attention(q, *args, query_start_loc=qsl, mode=mode, out=out, lse_out=lse, out_rotated=rotated, workspace=ws)
        assert (out[n:] == 0).all() and (lse[n:] == float("-inf")).all()
        want = ops.paged_tq4_attention(q[:n], *args, query_start_loc=qsl, mode=2, out_dtype=torch.float32, out_rotated=rotated)
        assert (out[:n] - want).abs().max() <= 2e-3 and torch.isfinite(lse[:n]).all()


def test_prefill_hides_and_reports_bad_pages(cuda_lib):
    from turboquant_vllm import _native as nv
    from turboquant_vllm.kernels import ops

    pr = Prims(128)
    p = pr.cuda()
    case = build_paged_case([100], 4, 128, 16, pr, seed=5, padded=True)
    q = torch.randn(30, 8, 128, generator=torch.Generator().manual_seed(1)).bfloat16()
    qsl = torch.tensor([0, 30], dtype=torch.int32)
    bt = case["block_table"].clone()
    bt[0, 1] = 10_000  # keys 16 .. 31 are not there
    args = (case["seq_lens"].cuda(), p["kc"], p["vc"], p["rot"], 4, 16)
    out = [ops.paged_tq4_attention(q.cuda(), case["cache"].cuda(), bt.cuda(), *args, query_start_loc=qsl.cuda(),
                                   out_dtype=torch.float32, mode=m) for m in (2, 3)]
    torch.cuda.synchronize()
    assert ops.read_and_clear_errors(torch.device("cuda")) == nv.DEV_BAD_BLOCK
    assert (out[0] - out[1]).abs().max() <= 2e-3


@pytest.mark.parametrize("d,hq,hkv,lens,new,cut", [
    (128, 32, 8, [3000], [40], True),
    (128, 32, 8, [1200, 1200, 900], [200, 40, 1], True),   # behind the plan of the streaming part
    (64, 14, 2, [1200], [200], True),
    (256, 8, 4, [1200], [100], True),
    (128, 28, 4, [1200], [1200], False),                   # the row blocks fill the GPU
])
def test_announced_scratch_is_room_for_the_key_parts(cuda_lib, d, hq, hkv, lens, new, cut):
    """A workspace of exactly the announced bytes: calls of few row blocks are cut along the keys (a merge follows
    the prefill kernel), and nothing is written past its end."""
    from turboquant_vllm import _native as nv
    from turboquant_vllm.kernels import ops

    pr = Prims(d)
    p = pr.cuda()
    case = build_paged_case(lens, hkv, d, 16, pr, seed=5, padded=True)
    rows = sum(new)
    q = torch.randn(rows, hq, d, generator=torch.Generator().manual_seed(1)).bfloat16().cuda()
    qsl = torch.tensor(np.concatenate([[0], np.cumsum(new)]), dtype=torch.int32).cuda()
    args = (q, case["cache"].cuda(), case["block_table"].cuda(), case["seq_lens"].cuda(), p["kc"], p["vc"], p["rot"], hkv, 16)
    need = ops.attention_workspace_bytes(rows, hq, hkv, d)
    ws = torch.full((need + 4096,), 0x55, dtype=torch.uint8, device="cuda")
    nv.profile_start(8)
    out = ops.paged_tq4_attention(*args, query_start_loc=qsl, out_dtype=torch.float32, workspace=ws[:need])
    merges, passes = (len(nv.profile_read(k, 8)) for k in (nv.PROF_COMBINE, nv.PROF_ATTENTION))
    nv.profile_stop()
    assert merges == passes - 1 + cut and (ws[need:] == 0x55).all()
    want = ops.paged_tq4_attention(*args, query_start_loc=qsl, out_dtype=torch.float32, mode=2)
    assert (out - want).abs().max() <= 2e-3


@pytest.mark.parametrize("hq,hkv,lens,new,bound,launches", [
    # 19 rows whose table would let every one read 65 536 keys: one streaming pass (attention, merge), or two passes
    (32, 8, [60, 40, 90], [17, 1, 1], 90, (1, 1)),
    (32, 8, [60, 40, 90], [17, 1, 1], None, (2, 2)),
    (32, 8, [60, 40, 90], [17, 1, 1], 10**9, (2, 2)),
    (32, 8, [300], [300], 300, (1, 0)),    # five tiles: not cut (36 us against 52 in three parts, B200)
    (32, 8, [300], [300], None, (1, 1)),
])
def test_known_length_decides_instead_of_the_table_width(cuda_lib, hq, hkv, lens, new, bound, launches):
    """max_seq_len: the kernels chosen on a table as wide as the model allows, and no other results."""
    from turboquant_vllm import _native as nv
    from turboquant_vllm.kernels import ops

    pr = Prims(128)
    p = pr.cuda()
    case = build_paged_case(lens, hkv, 128, 16, pr, seed=5, padded=True)
    rows = sum(new)
    q = torch.randn(rows, hq, 128, generator=torch.Generator().manual_seed(1)).bfloat16().cuda()
    qsl = torch.tensor(np.concatenate([[0], np.cumsum(new)]), dtype=torch.int32).cuda()
    table = torch.zeros(len(lens), 4096, dtype=torch.int32)
    table[:, : case["block_table"].shape[1]] = case["block_table"]
    args = (q, case["cache"].cuda(), table.cuda(), case["seq_lens"].cuda(), p["kc"], p["vc"], p["rot"], hkv, 16)
    nv.profile_start(8)
    out = ops.paged_tq4_attention(*args, query_start_loc=qsl, out_dtype=torch.float32, max_seq_len=bound)
    assert tuple(len(nv.profile_read(k, 8)) for k in (nv.PROF_ATTENTION, nv.PROF_COMBINE)) == launches
    nv.profile_stop()
    # (too small a value is only a worse choice)
    wrong = ops.paged_tq4_attention(*args, query_start_loc=qsl, out_dtype=torch.float32, max_seq_len=1)
    want = ops.paged_tq4_attention(*args, query_start_loc=qsl, out_dtype=torch.float32, mode=2)
    assert (out - want).abs().max() <= 2e-3 and (wrong - want).abs().max() <= 2e-3


@pytest.mark.parametrize("d,hq,hkv,lens,new", [
    (128, 32, 8, [2900, 1500, 700], [400, 300, 700]),
    (128, 28, 4, [700], [333]),                # cut along the keys
    (64, 14, 2, [2900, 300], [500, 300]),
    (96, 8, 8, [2900, 300], [300, 300]),
    (256, 8, 4, [2900, 300], [300, 300]),
])
@pytest.mark.parametrize("q_dtype", [torch.bfloat16, torch.float32])
def test_prefill_kernel_next_to_the_streaming_kernel(cuda_lib, d, hq, hkv, lens, new, q_dtype):
    """Both read keys and values through the same fp16 tables, so what separates them is the prefill kernel's own:
    the sum O in tensor memory, truncated by every MMA (eight a tile of 64 keys, at most 2^-23 of the sum each), and
    two-term fp16 operands (2^-22 of a row's largest coordinate: with scores of about ten, 2^-18 of a weight)."""
    from turboquant_vllm.kernels import ops

    p, gen = Prims(d).cuda(), torch.Generator(device="cuda").manual_seed(1)
    rand = lambda *shape: torch.randn(*shape, device="cuda", generator=gen)  # noqa: E731
    pages = [-(-n // 16) for n in lens]
    cache = torch.zeros(sum(pages), 16, hkv * O.padded_slot_bytes(d), dtype=torch.uint8, device="cuda")
    k, v = rand(2, cache.shape[0] * 16, hkv, d)
    k[..., 5] *= 8
    ops.tq4_write_paged(k, v, cache, torch.arange(k.shape[0], device="cuda"), p["even"], p["odd"], p["kb"], p["vb"])
    table = torch.zeros(len(lens), max(pages), dtype=torch.int32, device="cuda")
    for i, n in enumerate(pages):
        table[i, :n] = torch.arange(n) + sum(pages[:i])
    q = rand(sum(new), hq, d).to(q_dtype)
    qsl = torch.tensor(np.concatenate([[0], np.cumsum(new)]), dtype=torch.int32).cuda()
    args = (q, cache, table, torch.tensor(lens, dtype=torch.int32).cuda(), p["kc"], p["vc"], p["rot"], hkv, 16)
    a, b = (ops.paged_tq4_attention(*args, query_start_loc=qsl, out_dtype=torch.float32, mode=m).double() for m in (3, 2))
    tiles = -(-max(lens) // 64)
    assert (a - b).norm() / b.norm() <= 8 * tiles * 2.0**-23 + 2.0**-18


@pytest.mark.parametrize("d,hq,hkv,v_bits", [(64, 14, 2, 4), (96, 4, 4, 4), (128, 28, 4, 3), (256, 8, 4, 4), (256, 8, 4, 3)])
@pytest.mark.parametrize("power", [-14, -4, 0, 4, 14])
def test_prefill_large_and_small_queries(cuda_lib, d, hq, hkv, v_bits, power):
    """Queries times 2^power over keys times 2^-power: the scores are the same, the factor that makes them is inside the
    range of the queries' fp16 terms, or partly outside.  Against the streaming kernel, bound as above."""
    from turboquant_vllm.kernels import ops

    pk, pv, gen = Prims(d).cuda(), Prims(d, v_bits=v_bits).cuda(), torch.Generator(device="cuda").manual_seed(1)
    rand = lambda *shape: torch.randn(*shape, device="cuda", generator=gen)  # noqa: E731
    n, new = 300, 150
    cache = torch.zeros(19, 16, hkv * O.padded_slot_bytes(d), dtype=torch.uint8, device="cuda")
    ops.tq4_write_paged(rand(n, hkv, d) * 2.0**-power, rand(n, hkv, d), cache, torch.arange(n, device="cuda"), pk["even"],
                        pk["odd"], pk["kb"], pv["vb"])
    table = torch.arange(19, dtype=torch.int32, device="cuda")[None]
    q = (rand(new, hq, d) * 2.0**power).bfloat16()
    args = (q, cache, table, torch.tensor([n], dtype=torch.int32).cuda(), pk["kc"], pv["vc"], pk["rot"], hkv, 16)
    qsl = torch.tensor([0, new], dtype=torch.int32).cuda()
    a, b = (ops.paged_tq4_attention(*args, query_start_loc=qsl, out_dtype=torch.float32, mode=m).double() for m in (3, 2))
    assert (a - b).norm() / b.norm() <= 8 * 5 * 2.0**-23 + 2.0**-18


@pytest.mark.parametrize("d,hq,hkv", [(64, 14, 2), (96, 4, 4), (128, 28, 4), (256, 8, 4)])
@pytest.mark.parametrize("power", [-9, 9])
def test_prefill_some_rows_large_or_small(cuda_lib, d, hq, hkv, power):
    """Some rows of a warp outside the range of the queries' terms, some inside; tiles that all rows see whole, and others.
    Bound as above (the scores of the rows that are not scaled are 2^9 times smaller or larger: of the smaller of the two)."""
    from turboquant_vllm.kernels import ops

    p, gen = Prims(d).cuda(), torch.Generator(device="cuda").manual_seed(1)
    rand = lambda *shape: torch.randn(*shape, device="cuda", generator=gen)  # noqa: E731
    n, new = 300, 150
    cache = torch.zeros(19, 16, hkv * O.padded_slot_bytes(d), dtype=torch.uint8, device="cuda")
    ops.tq4_write_paged(rand(n, hkv, d) * min(1.0, 2.0**-power), rand(n, hkv, d), cache, torch.arange(n, device="cuda"), p["even"],
                        p["odd"], p["kb"], p["vb"])
    table = torch.arange(19, dtype=torch.int32, device="cuda")[None]
    q = rand(new, hq, d)
    q[::5] *= 2.0**power
    args = (q, cache, table, torch.tensor([n], dtype=torch.int32).cuda(), p["kc"], p["vc"], p["rot"], hkv, 16)
    qsl = torch.tensor([0, new], dtype=torch.int32).cuda()
    a, b = (ops.paged_tq4_attention(*args, query_start_loc=qsl, out_dtype=torch.float32, mode=m).double() for m in (3, 2))
    for rows in (slice(0, None, 5), slice(1, None, 5)):
        assert (a[rows] - b[rows]).norm() / b[rows].norm() <= 8 * 5 * 2.0**-23 + 2.0**-18

@pytest.mark.parametrize("d,hq,hkv", [(64, 14, 2), (96, 4, 4), (128, 28, 4), (256, 8, 4)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("pad", [0, 8, 2])
def test_prefill_16bit_rows_are_the_rounded_fp32_ones(cuda_lib, d, hq, hkv, dtype, pad):
    """Outputs that leave through shared memory (rows on 16 bytes) or not: each the rounded fp32 result, nothing beside it."""
    from turboquant_vllm.kernels import ops

    pr = Prims(d)
    p = pr.cuda()
    case = build_paged_case([170, 40], hkv, d, 16, pr, seed=5, padded=True)
    new = [99, 9]
    q = torch.randn(sum(new), hq, d, generator=torch.Generator().manual_seed(1)).to(dtype).cuda()
    qsl = torch.tensor([0, 99, 108], dtype=torch.int32).cuda()
    args = (q, case["cache"].cuda(), case["block_table"].cuda(), case["seq_lens"].cuda(), p["kc"], p["vc"], p["rot"], hkv, 16)
    want = ops.paged_tq4_attention(*args, query_start_loc=qsl, out_dtype=torch.float32, mode=3).to(dtype)
    wide = torch.full((sum(new), hq, d + pad), 7.0, dtype=dtype, device="cuda")
    ops.paged_tq4_attention(*args, query_start_loc=qsl, out=wide[..., :d], mode=3)
    assert torch.equal(wide[..., :d], want) and (wide[..., d:] == 7).all()


@pytest.mark.parametrize("d,hq,hkv", [(128, 40, 40), (64, 66, 33), (256, 32, 32)])
def test_more_row_blocks_and_heads_than_sms(cuda_lib, d, hq, hkv):
    """More CTAs than fit at once, spare ones and rows of no sequence among them: every (row, head) by its own CTA."""
    from turboquant_vllm.kernels import ops

    pr, lens, new, rows = Prims(d), [90, 300, 20], [70, 261, 20], 400
    p = pr.cuda()
    case = build_paged_case(lens, hkv, d, 16, pr, seed=6, padded=True)
    q = torch.randn(rows, hq, d, generator=torch.Generator().manual_seed(2)).bfloat16()
    qsl = torch.tensor(np.concatenate([[0], np.cumsum(new)]), dtype=torch.int32)
    args = (case["cache"].cuda(), case["block_table"].cuda(), case["seq_lens"].cuda(), p["kc"], p["vc"], p["rot"], hkv, 16)
    outs, lses = zip(*((torch.full((rows, hq, d), 7.0, device="cuda"), torch.full((rows, hq), 7.0, device="cuda")) for _ in range(2)))
    for mode, out, lse in zip((3, 2), outs, lses):
        ops.paged_tq4_attention(q.cuda(), *args, query_start_loc=qsl.cuda(), mode=mode, out=out, lse_out=lse)
    n = sum(new)
    (got, want), (lse, want_lse) = outs, lses
    # the two kernels share their tables; the sums of at most five 64-key tiles, their order, and the split terms are what differs
    assert (got[:n] - want[:n]).norm() <= (8 * 5 * 2.0**-23 + 2.0**-18) * want[:n].norm()
    assert ((got[:n] - want[:n]).norm(dim=-1) <= 2.0**-10 * want[:n].norm(dim=-1)).all()  # (a vector from elsewhere would be 1 away)
    assert torch.allclose(lse[:n], want_lse[:n], atol=1e-3, rtol=1e-4)
    assert (got[n:] == 0).all() and (lse[n:] == -torch.inf).all()
    assert ops.read_and_clear_errors(torch.device("cuda")) == 0
