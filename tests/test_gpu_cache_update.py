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
