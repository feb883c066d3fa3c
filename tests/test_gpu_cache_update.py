"""The one-launch cache updates (default mode's buffers, fused mode's token rows) against the tensor-by-tensor path."""

import pytest
import torch

from oracle import tq4_oracle as O

pytestmark = pytest.mark.gpu


def _states(b, h, n, d, dtype, seed):
    """As a projection hands them over: [B, H, N, D] views of [B, N, H, D]."""
    k, v = O.synthetic_kv(b * n, h, d, seed=seed, dtype=dtype)
    return [x.cuda().view(b, n, h, d).transpose(1, 2) for x in (k, v)]


@pytest.mark.parametrize("d", [64, 96, 128, 256])
@pytest.mark.parametrize("b,h,dtype,bits", [
    (1, 1, torch.bfloat16, (4, 4)), (2, 3, torch.float16, (4, 3)), (3, 2, torch.float32, (3, 2)),
    (4, 40, torch.bfloat16, (4, 4))])  # the last: eight vectors a warp, compressed ahead at head_dim 128
def test_default_mode(cuda_lib, d, b, h, dtype, bits):
    from transformers import DynamicCache
    from turboquant_vllm import CompressedDynamicCache

    cc = CompressedDynamicCache(DynamicCache(), d, k_bits=bits[0], v_bits=bits[1])
    want = [[], [], []], [[], [], []]
    for step, n in enumerate((33, 1, 1, 60)):  # a remainder of a block's vectors; single tokens; growth
        kv = _states(b, h, n, d, dtype, seed=d + step)
        got = cc.cache.update(*kv, 0)
        for x, comp, nib, w in zip(kv, (cc.key_compressor, cc.value_compressor), (bits[0] == 4, bits[1] == 4), want):
            # few vectors a call: the kernels that agree bit for bit; what the tensor cores write at 128 whole
            for part in x.split(n if d == 128 and b * h * n > 8192 else 3, dim=2):
                layer = cc._compress_tensor(comp, part, nibble_packed=nib)
                for held, y in zip(w, (layer.indices, layer.norms, cc._dequantize_layer(comp, layer))):
                    held.append(y)
    k_idx, k_n, v_idx, v_n = cc.get_compressed(0)
    for w, idx, norm, dec in zip(want, (k_idx, v_idx), (k_n, v_n), got):
        assert torch.equal(idx, torch.cat(w[0], 2)) and torch.equal(norm, torch.cat(w[1], 2))
        ref = torch.cat(w[2], 2)
        torch.testing.assert_close(dec, ref, **(dict(rtol=0, atol=5e-5) if dtype == torch.float32 else dict(rtol=1e-2, atol=2e-2)))


@pytest.mark.parametrize("d", [64, 96, 128, 256])
@pytest.mark.parametrize("b,h", [(1, 2), (3, 4)])
def test_token_rows(cuda_lib, d, b, h):
    from turboquant_vllm.quantizer import TurboQuantMSE
    from turboquant_vllm.token_rows import TokenRowStore

    kq, vq = TurboQuantMSE(d, 4), TurboQuantMSE(d, 4)
    store = TokenRowStore(b, h, d, torch.device("cuda"))
    steps = [_states(b, h, n, d, torch.bfloat16, seed=d + n) for n in (1, 250, 7, 900)]  # pages crossed; each write kernel
    for k, v in steps:
        store.append(k, v, kq, vq)
    k_all, v_all = (torch.cat([s[i] for s in steps], 2) for i in (0, 1))
    for x, idx, norm in ((k_all, *store.views()[:2]), (v_all, *store.views()[2:])):
        packed, norms = O.compress_rows(x.cpu().reshape(-1, 1, d), kq.rotation, kq.codebook.boundaries)
        got = idx.contiguous().cpu().reshape(-1, d // 2)
        assert (O.nibble_unpack(got) != O.nibble_unpack(packed.reshape(-1, d // 2))).float().mean() <= 1e-4
        assert torch.allclose(norm.cpu().reshape(-1), norms.reshape(-1), rtol=1e-6)


@pytest.mark.parametrize("d", [64, 96, 128])
@pytest.mark.parametrize("b,h,n,dtype", [
    (1, 1, 2369, torch.bfloat16),   # one vector past the line, 19 tiles a tensor, 65 vectors in the last
    (1, 4, 640, torch.float16),     # whole tiles
    (3, 5, 171, torch.bfloat16),    # batch and head change inside a tile
    (5, 32, 120, torch.bfloat16),   # 300 tiles: three a CTA for some; at 128 above the line of the tensor cores' own bytes
])
@pytest.mark.parametrize("aligned", [True, False])
def test_prompt_restored_by_the_tensor_cores(cuda_lib, d, b, h, n, dtype, aligned):
    """Indices and norms of the compression by itself; the reconstruction against 64 bits: half a unit of the 16-bit type and
    2^-19 of a vector's norm for the sums (128 terms of 22 bits, fp32); nothing beside the update's own rows."""
    from turboquant_vllm import TurboQuantMSE
    from turboquant_vllm import _native as nv
    from turboquant_vllm.kernels import ops

    kq, vq = TurboQuantMSE(d, 4, seed=42), TurboQuantMSE(d, 3, seed=42)
    rot = kq.rotation.contiguous().cuda()
    even, odd = rot.T[:, 0::2].contiguous(), rot.T[:, 1::2].contiguous()
    kb, vb, kc, vc = (x.cuda() for x in (kq.codebook.boundaries, vq.codebook.boundaries, kq.codebook.centroids, vq.codebook.centroids))
    k, v = _states(b, h, n, d, dtype, seed=d)
    cap, off = n + 7, 3

    def dec():  # (misaligned: the FMA kernels' turn)
        return torch.zeros(b * h * cap * d + 1, dtype=dtype, device="cuda")[0 if aligned else 1:][: b * h * cap * d].view(b, h, cap, d)

    ki, vi = (torch.zeros(b, h, cap, w, dtype=torch.uint8, device="cuda") for w in (d // 2, d))
    kn, vn = (torch.zeros(b, h, cap, 1, device="cuda") for _ in range(2))
    kd, vd = dec(), dec()
    nv.host().cache_update(k, v, rot, even, odd, kb, vb, kc, vc, True, False, ki, kn, vi, vn, off, kd, vd, off)
    for x, bounds, cents, idx, norm, out in ((k, kb, kc, torch.stack([ki >> 4, ki & 15], -1).flatten(-2), kn, kd), (v, vb, vc, vi, vn, vd)):
        whole = d == 128 and b * h * n > 8192
        parts = [ops.tq4_compress(p.transpose(1, 2).reshape(-1, h, d), even, odd, bounds) for p in x.split(n if whole else 5, dim=2)]
        packed, norms = (torch.cat([p[i].view(b, -1, h, p[i].shape[-1]) for p in parts], 1).transpose(1, 2) for i in (0, 1))
        live = slice(off, off + n)
        assert torch.equal(idx[:, :, live], torch.stack([packed >> 4, packed & 15], -1).flatten(-2)) and torch.equal(norm[:, :, live], norms)
        want = (cents.double()[idx[:, :, live].long()] * norms.double()) @ rot.double()
        half = 2.0**-8 if dtype == torch.bfloat16 else 2.0**-11  # (significands of 8 and 11 bits)
        assert ((out[:, :, live].double() - want).abs() <= half * want.abs() * (1 + 2.0**-7) + 2.0**-19 * norms.double()).all()
        for t in (idx, norm, out):
            assert (t[:, :, :off] == 0).all() and (t[:, :, off + n:] == 0).all()


def test_prompt_without_tensor_cores(cuda_lib):
    """TQ4_NO_TC (read once a process): a prompt past the line is neither compressed nor restored by a tcgen05 kernel."""
    import os
    import subprocess
    import sys

    prog = """
import sys
sys.path.insert(0, {pkg!r})
import torch
from torch.profiler import ProfilerActivity, profile
from transformers import DynamicCache
from turboquant_vllm import CompressedDynamicCache

cc = CompressedDynamicCache(DynamicCache(), 128, k_bits=4, v_bits=4)
k, v = (torch.randn(1, 8, 700, 128, generator=torch.Generator().manual_seed(i)).cuda().bfloat16() for i in range(2))
with profile(activities=[ProfilerActivity.CUDA]) as p:
    cc.cache.update(k, v, 0)
    torch.cuda.synchronize()
print([e.key for e in p.key_averages() if "tq4::" in e.key])
"""
    pkg = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "turboquant-vllm_b200")
    for env, tensor_cores in (({}, True), ({"TQ4_NO_TC": "1"}, False)):
        done = subprocess.run([sys.executable, "-c", prog.format(pkg=pkg)], capture_output=True, text=True, timeout=300,
                              env={**{k: v for k, v in os.environ.items() if k != "TQ4_NO_TC"}, **env})
        assert done.returncode == 0, done.stderr[-2000:]
        assert "tq4::" in done.stdout and ("_tc" in done.stdout) == tensor_cores, done.stdout


@pytest.mark.parametrize("fused", [False, True])
def test_a_copied_cache_goes_its_own_way(cuda_lib, fused):
    """A copy made in the middle of a generation (a shared prompt, a file): takes its next update, and neither sees the other's."""
    import copy
    import pickle

    from transformers import DynamicCache
    from turboquant_vllm import CompressedDynamicCache

    d, b, h = 128, 2, 2
    cc = CompressedDynamicCache(DynamicCache(), d, k_bits=4, v_bits=4)
    cc.fused_mode = fused
    steps = [_states(b, h, n, d, torch.bfloat16, seed=i) for i, n in enumerate((20, 1, 1, 1, 1))]
    for kv in steps[:3]:
        cc.cache.update(*kv, 0)
    twins = [copy.deepcopy(cc), pickle.loads(pickle.dumps(cc))]
    for w, kv in zip([*twins, cc], (steps[3], steps[4], steps[4])):
        w.cache.update(*kv, 0)
    got = [w.get_compressed(0) for w in (*twins, cc)]
    assert all(t.shape[2] == 23 for g in got for t in g)
    assert all(torch.equal(x, y) for x, y in zip(got[1], got[2]))
    assert all(torch.equal(x[:, :, :22], y[:, :, :22]) and not torch.equal(x, y) for x, y in zip(got[0], got[2]))
