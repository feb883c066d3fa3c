"""What a user has this package do, as cases that can be prepared, run and compared.

Every case goes through the package's public entry points, with the tensors that a serving engine or
a HuggingFace program has in hand at that moment:

* ``decode``  -- one decode step of a layer: ``tq4_write_and_attention`` (one new token a sequence).
* ``prefill`` -- a prefill or mixed step of a layer: ``tq4_write_paged`` of the new tokens, then
  ``fused_paged_tq4_prefill`` (what the vLLM backend's forward does).
* ``write``   -- the cache write of a long prompt alone: ``tq4_write_paged``.
* ``hf``      -- one short generation through ``CompressedDynamicCache``: a fresh cache, the prompt,
  then single tokens; with the fused attention backend or in the cache's default mode.

Model shapes are the ones of this repository's benchmark configurations and tests.  Keys and values
are N(0, 1) with four outlier channels scaled by 8, queries N(0, 1); block tables are shuffled; the
cache has vLLM's padded rows (heads x next power of two of head_dim + 8 bytes).
"""

from __future__ import annotations

import math
import os
import random
import sys

import torch

_PKG = os.path.join(os.getcwd(), "turboquant-vllm_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from turboquant_vllm import CompressedDynamicCache, TurboQuantMSE  # noqa: E402
from turboquant_vllm.kernels import fused_paged_tq4_prefill, tq4_write_and_attention, tq4_write_paged  # noqa: E402
from turboquant_vllm.triton.attention_interface import triton_fa_tq4_kv_forward  # noqa: E402

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
OUTLIERS = (3, 17, 41, 52)
POOL = 16384  # distinct cached token rows; a cache draws its tokens from them
BLOCK = 16    # tokens per page (vLLM's default)


# --------------------------------------------------------------------------------------------------
# cases
# --------------------------------------------------------------------------------------------------
def _decode(batch, lo, hi, hq, hkv, dim, dtype, v_bits=4, window=0):
    """A decode step: ``batch`` sequences whose lengths are spread over [lo, hi]."""
    return {"op": "decode", "batch": batch, "ctx_lo": lo, "ctx_hi": hi, "hq": hq, "hkv": hkv, "dim": dim,
            "dtype": dtype, "v_bits": v_bits, "window": window}


def _prefill(chunks, new_lo, new_hi, prefix_lo, prefix_hi, decodes, hq, hkv, dim, dtype, v_bits=4, window=0):
    """``chunks`` sequences with new tokens spread over [new_lo, new_hi] behind cached prefixes spread over
    [prefix_lo, prefix_hi], beside ``decodes`` sequences of those prefixes with one new token each."""
    return {"op": "prefill", "chunks": chunks, "new_lo": new_lo, "new_hi": new_hi, "prefix_lo": prefix_lo,
            "prefix_hi": prefix_hi, "decodes": decodes, "hq": hq, "hkv": hkv, "dim": dim, "dtype": dtype,
            "v_bits": v_bits, "window": window}


def _write(tokens, hkv, dim, dtype, v_bits=4):
    return {"op": "write", "tokens": tokens, "hkv": hkv, "dim": dim, "dtype": dtype, "v_bits": v_bits}


def _hf(batch, prompt, steps, layers, hq, hkv, dim, dtype, fused, v_bits=4):
    return {"op": "hf", "batch": batch, "prompt": prompt, "steps": steps, "layers": layers, "hq": hq, "hkv": hkv,
            "dim": dim, "dtype": dtype, "fused": fused, "v_bits": v_bits}


def listed():
    return [
        # a single user's chat: one short sequence, where latency and launches are everything
        dict(_decode(1, 1024, 1024, 28, 4, 128, "bf16"), name="decode-1"),
        # an ordinary moment of a server: a few sequences of ragged lengths, fp16 model
        dict(_decode(16, 300, 8100, 32, 8, 128, "fp16"), name="decode-16-ragged"),
        # the benchmark's headline step
        dict(_decode(64, 4096, 4096, 32, 8, 128, "bf16"), name="decode-64x4096"),
        # a loaded server: mixed lengths, asymmetric bit widths (the largest case)
        dict(_decode(256, 512, 32768, 32, 8, 128, "bf16", v_bits=3), name="decode-256-mix"),
        # long documents on a model without grouped queries and an odd head dimension
        dict(_decode(8, 131072, 131072, 32, 32, 96, "bf16"), name="decode-8x131072-d96"),
        # chunked prefill of several long prompts behind cached prefixes, a full scheduler step
        dict(_prefill(8, 2048, 2048, 8192, 8192, 0, 32, 8, 128, "bf16"), name="prefill-8x2048"),
        # the first prompt of a chat: one sequence, nothing cached, an odd length, groups of 7 heads
        dict(_prefill(1, 1531, 1531, 0, 0, 0, 28, 4, 128, "bf16"), name="prefill-1x1531"),
        # a mixed step of continuous batching: one chunk of a prompt beside running sequences
        dict(_prefill(1, 480, 480, 1024, 6000, 32, 32, 8, 128, "bf16"), name="prefill-mixed-32"),
        # sliding-window layers of a model with head_dim 256
        dict(_prefill(8, 2048, 2048, 8192, 8192, 0, 8, 4, 256, "bf16", window=4096), name="prefill-d256-window"),
        # the cache write of a full prefill step
        dict(_write(16384, 8, 128, "bf16"), name="write-16384"),
        # a HuggingFace generation with the fused attention backend
        dict(_hf(1, 700, 8, 4, 32, 8, 128, "bf16", True), name="hf-fused"),
        # the same cache in its default mode, which hands dequantised keys and values back
        dict(_hf(4, 1100, 8, 2, 32, 8, 128, "bf16", False, v_bits=3), name="hf-default"),
    ]


# query heads, KV heads, head_dim, sliding window: the shapes of the benchmark configurations and the tests
# (32/8/128 whole and as one of eight ranks; 28/4/128; 32/32/96; 14/2/64; 8/4/256)
SHAPES = ((32, 8, 128, 0), (32, 8, 128, 0), (28, 4, 128, 0), (4, 1, 128, 0), (32, 32, 96, 0), (14, 2, 64, 0),
          (8, 4, 256, 4096))


def _log_int(rng: random.Random, lo: int, hi: int) -> int:
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng: random.Random):
    hq, hkv, dim, window = rng.choice(SHAPES)
    dtype = rng.choice(("bf16", "bf16", "fp16"))
    v_bits = rng.choice((4, 4, 3))
    op = rng.choice(("decode", "decode", "decode", "prefill", "prefill", "write", "hf"))
    if op == "decode":
        batch = _log_int(rng, 1, 256)
        # tokens held so that the packed bytes stay below those of the largest listed case
        most = min(131072, int(6e9 / (batch * hkv * (dim + 8))))
        hi = _log_int(rng, 100, most)
        return _decode(batch, rng.choice((hi, max(1, hi // 20))), hi, hq, hkv, dim, dtype, v_bits, window)
    if op == "prefill":
        chunks, new = _log_int(rng, 1, 8), _log_int(rng, 17, 2048)
        prefix = rng.choice((0, _log_int(rng, 50, 8192)))
        decodes = rng.choice((0, _log_int(rng, 1, 64)))
        return _prefill(chunks, max(1, new // rng.choice((1, 4))), new, prefix // 4, prefix, decodes, hq, hkv, dim,
                        dtype, v_bits, window)
    if op == "write":
        return _write(_log_int(rng, 33, 16384), hkv, dim, dtype, v_bits)
    return _hf(_log_int(rng, 1, 4), _log_int(rng, 30, 2000), rng.randint(4, 10), rng.randint(1, 4), hq, hkv, dim, dtype,
               rng.random() < 0.5, v_bits if dim != 96 else 4)


# --------------------------------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------------------------------
_quantizers: dict = {}  # rotation and codebooks of a model shape: made once by a program, like its weights


def _quantizer(dim: int, bits: int) -> TurboQuantMSE:
    if (dim, bits) not in _quantizers:
        _quantizers[dim, bits] = TurboQuantMSE(dim, bits, seed=42)
    return _quantizers[dim, bits]


def _spread(n: int, lo: int, hi: int) -> list[int]:
    """``n`` lengths spread evenly over [lo, hi] (a case holds the same number of tokens for every seed)."""
    return [lo + round((hi - lo) * (i + 0.5) / n) for i in range(n)]


def _shuffled(items: list, seed: int) -> list:
    items = list(items)
    random.Random(seed).shuffle(items)
    return items


def _kv(shape, dtype, gen):
    x = torch.randn(shape, device="cuda", generator=gen)
    x[..., list(OUTLIERS)] *= 8.0
    return x.to(dtype)


def _packed(x: torch.Tensor, q: TurboQuantMSE):
    """Plain PyTorch packing of ``[N, D]`` rows: nibble bytes and fp32 norms (for the tokens already cached)."""
    norm = x.norm(dim=1, keepdim=True)
    y = (x / (norm + 1e-10)) @ q.rotation.T.to(x)
    idx = torch.bucketize(y, q.codebook.boundaries.to(x)).to(torch.uint8)
    return (idx[:, 0::2] << 4) | idx[:, 1::2], norm


def _row_width(hkv: int, dim: int) -> int:
    return hkv * (1 << (dim + 7).bit_length())


def _cached_rows(n: int, hkv: int, dim: int, kq, vq, gen) -> torch.Tensor:
    """``n`` padded token rows [K indices | K norms | V indices | V norms | padding]."""
    pool = min(n, max(64, POOL // hkv))
    parts = []
    for q in (kq, vq):
        idx, norm = _packed(_kv((pool * hkv, dim), torch.float32, gen), q)
        parts += [idx.reshape(pool, -1), norm.reshape(pool, hkv).view(torch.uint8)]
    rows = torch.zeros(pool, _row_width(hkv, dim), dtype=torch.uint8, device="cuda")
    data = torch.cat(parts, dim=1)
    rows[:, : data.shape[1]] = data
    pick = torch.randint(pool, (n,), device="cuda", generator=gen)
    return rows.view(torch.int64)[pick].view(torch.uint8)


def _paged(lens: list[int], hkv: int, dim: int, kq, vq, gen):
    """Cache ``[blocks, 16, width]`` full of cached tokens, a shuffled block table, int32 lengths."""
    need = [-(-n // BLOCK) for n in lens]
    blocks = sum(need) + 2
    cache = _cached_rows(blocks * BLOCK, hkv, dim, kq, vq, gen).view(blocks, BLOCK, -1)
    order = torch.randperm(blocks, device="cuda", generator=gen).to(torch.int32)
    table = torch.zeros(len(lens), max(need), dtype=torch.int32, device="cuda")
    at = torch.arange(max(need), device="cuda")[None, :] < torch.tensor(need, device="cuda")[:, None]
    table[at] = order[: sum(need)]
    return cache, table, torch.tensor(lens, dtype=torch.int32, device="cuda")


def _slots(table: torch.Tensor, first: list[int], count: list[int]) -> torch.Tensor:
    """Flat slots of positions first[i] .. first[i] + count[i] - 1 of every sequence i."""
    seq = torch.repeat_interleave(torch.arange(len(first)), torch.tensor(count))
    start = torch.tensor(first) - (torch.cumsum(torch.tensor(count), 0) - torch.tensor(count))
    pos = (torch.arange(sum(count)) + start[seq]).cuda()
    return table[seq.cuda(), pos // BLOCK].long() * BLOCK + pos % BLOCK


def _primitives(dim: int, v_bits: int):
    kq, vq = _quantizer(dim, 4), _quantizer(dim, v_bits)
    rot_t = kq.rotation.T
    return dict(
        kq=kq, vq=vq, rotation=kq.rotation.contiguous().cuda(), even=rot_t[:, 0::2].contiguous().cuda(),
        odd=rot_t[:, 1::2].contiguous().cuda(), kc=kq.codebook.centroids.cuda(), kb=kq.codebook.boundaries.cuda(),
        vc=vq.codebook.centroids.cuda(), vb=vq.codebook.boundaries.cuda())


class _HostLayer:
    is_initialized = True
    keys = values = None


class _HostCache:
    """The face of a HuggingFace ``DynamicCache`` that the wrapper uses."""

    layer_class_to_replicate = _HostLayer

    def __init__(self):
        self.layers = []

    def update(self, key_states, value_states, layer_idx, cache_kwargs=None):
        raise NotImplementedError

    def get_seq_length(self, layer_idx=0):
        return 0


class _Attention(torch.nn.Module):
    """An attention module of a HuggingFace model, as the attention backend sees it."""

    is_causal = True

    def __init__(self, layer_idx):
        super().__init__()
        self.layer_idx = layer_idx


def prepare(case, seed):
    c = case
    gen = torch.Generator(device="cuda").manual_seed(seed)
    dtype = DTYPES[c["dtype"]]
    if c["op"] == "hf":
        total = c["prompt"] + c["steps"]
        q = torch.randn(c["layers"], c["batch"], c["hq"], total, c["dim"], device="cuda", generator=gen).to(dtype)
        k = _kv((c["layers"], c["batch"], c["hkv"], total, c["dim"]), dtype, gen)
        v = _kv((c["layers"], c["batch"], c["hkv"], total, c["dim"]), dtype, gen)
        # as a model's projections hand them over: the prompt, then one token at a time
        cuts = [(0, c["prompt"])] + [(c["prompt"] + i, c["prompt"] + i + 1) for i in range(c["steps"])]
        steps = [[tuple(x[layer, :, :, a:b].transpose(1, 2).contiguous().transpose(1, 2) for x in (q, k, v))
                  for layer in range(c["layers"])] for a, b in cuts]
        return dict(case=c, steps=steps, modules=[_Attention(i) for i in range(c["layers"])])
    s = _primitives(c["dim"], c["v_bits"])
    s["case"] = c
    hkv, dim = c["hkv"], c["dim"]
    if c["op"] == "write":
        n = c["tokens"]
        s["cache"], table, _ = _paged([n], hkv, dim, s["kq"], s["vq"], gen)
        s["slots"] = _slots(table, [0], [n])
    elif c["op"] == "decode":
        lens = _shuffled(_spread(c["batch"], c["ctx_lo"], c["ctx_hi"]), seed)
        n = c["batch"]
        s["cache"], s["table"], s["lens"] = _paged(lens, hkv, dim, s["kq"], s["vq"], gen)
        s["slots"] = _slots(s["table"], [x - 1 for x in lens], [1] * n)
    else:
        new, prefix = _prefill_lens(c, seed)
        n = sum(new)
        lens = [a + b for a, b in zip(new, prefix)]
        s["cache"], s["table"], s["lens"] = _paged(lens, hkv, dim, s["kq"], s["vq"], gen)
        s["slots"] = _slots(s["table"], prefix, new)
        s["starts"] = torch.tensor([0] + [sum(new[: i + 1]) for i in range(len(new))], dtype=torch.int32, device="cuda")
    s["key"], s["value"] = _kv((n, hkv, dim), dtype, gen), _kv((n, hkv, dim), dtype, gen)
    if c["op"] != "write":
        s["q"] = torch.randn(n, c["hq"], dim, device="cuda", generator=gen).to(dtype)
        s["out"] = torch.empty_like(s["q"])
    return s


def _prefill_lens(c, seed):
    """New tokens and cached tokens of every sequence: running sequences first, as the scheduler orders them."""
    seqs = []
    for n, lo, hi in ((c["decodes"], 1, 1), (c["chunks"], c["new_lo"], c["new_hi"])):
        prefix = _shuffled(_spread(n, c["prefix_lo"], c["prefix_hi"]), 0)
        seqs += _shuffled(list(zip(_spread(n, lo, hi), prefix)), seed)
    return [a for a, _ in seqs], [b for _, b in seqs]


# --------------------------------------------------------------------------------------------------
# one pass
# --------------------------------------------------------------------------------------------------
def run(state):
    s, c = state, state["case"]
    if c["op"] == "decode":
        tq4_write_and_attention(
            s["key"], s["value"], s["slots"], s["even"], s["odd"], s["kb"], s["vb"], s["q"], s["cache"], s["table"],
            s["lens"], s["kc"], s["vc"], s["rotation"], c["hkv"], BLOCK, sliding_window=c["window"] or None, out=s["out"])
        return s["out"], s["cache"]
    if c["op"] == "hf":
        return _generate(s, c)
    tq4_write_paged(s["key"], s["value"], s["cache"], s["slots"], s["even"], s["odd"], s["kb"], s["vb"])
    if c["op"] == "write":
        return s["cache"]
    fused_paged_tq4_prefill(
        s["q"], s["cache"], s["table"], s["lens"], s["starts"], s["kc"], s["rotation"], c["hkv"], c["dim"], BLOCK,
        out=s["out"], v_centroids=s["vc"], sliding_window=c["window"] or None)
    return s["out"], s["cache"]


def _generate(s, c):
    cache = CompressedDynamicCache(_HostCache(), c["dim"], k_bits=4, v_bits=c["v_bits"])
    cache.fused_mode = c["fused"]
    outs = []
    for module in s["modules"]:
        module._tq4_cache = cache
    for layers in s["steps"]:
        for module, (q, k, v) in zip(s["modules"], layers):
            k, v = cache.cache.update(k, v, module.layer_idx)
            if c["fused"]:
                outs.append(triton_fa_tq4_kv_forward(module, q, k, v, None)[0])
    if c["fused"]:
        return outs
    return [(layer.keys, layer.values) for layer in cache.cache.layers]


# --------------------------------------------------------------------------------------------------
# what a pass cannot do without, and how far correct results may lie apart
# --------------------------------------------------------------------------------------------------
def _pairs(new: int, prefix: int, window: int) -> int:
    """Visible (query, key) pairs of ``new`` causal queries behind ``prefix`` keys."""
    if not window:
        return new * prefix + new * (new + 1) // 2
    return sum(min(window, prefix + i + 1) for i in range(new))


def work(case):
    c = case
    hkv, dim, es = c["hkv"], c["dim"], 2
    token = hkv * (dim + 8)                   # packed bytes of a token
    rotate = 2 * dim * dim                    # operations that rotate one vector
    if c["op"] == "write":
        n = c["tokens"]
        return {"bytes": n * (2 * hkv * dim * es + token), "flops": 2 * n * hkv * rotate}
    hq = c["hq"]
    if c["op"] == "hf":
        b, total = c["batch"], c["prompt"] + c["steps"]
        n = c["layers"] * b * total
        kv, flops = n * 2 * hkv * dim * es, 2 * n * hkv * rotate
        if not c["fused"]:  # keys and values in, dequantised keys and values out
            return {"bytes": 2 * kv, "flops": 2 * flops}
        read = c["layers"] * b * token * sum(c["prompt"] + i for i in range(c["steps"] + 1))
        pairs = c["layers"] * b * total * (total + 1) // 2
        return {"bytes": kv + n * token + read + 2 * n * hq * dim * es,
                "flops": flops + 2 * n * hq * rotate + 4 * dim * hq * pairs}
    if c["op"] == "decode":
        new, lens = [1] * c["batch"], _spread(c["batch"], c["ctx_lo"], c["ctx_hi"])
        prefix = [x - 1 for x in lens]
    else:
        new, prefix = _prefill_lens(c, 0)
    n, window = sum(new), c["window"]
    keys = sum(min(a + b, window + a) if window else a + b for a, b in zip(new, prefix))
    pairs = sum(_pairs(a, b, window) for a, b in zip(new, prefix))
    return {"bytes": keys * token + n * (2 * hkv * dim + 2 * hq * dim) * es,
            "flops": 4 * dim * hq * pairs + 2 * n * (hq + hkv) * rotate}


def tolerance(case):
    # Outputs have 16 bits (a rounding is 2^-9 of a value for bf16); packed bytes may differ where a
    # rotated coordinate lies on a bucket boundary to within fp32 rounding (at most 1e-4 of the indices),
    # and such a key or value moves by one bucket.
    if case["op"] == "hf" and not case["fused"]:
        return {"rel": 5e-3, "max": 0.2}
    return {"rel": 5e-3, "max": 0.1, "differ": 2e-4}
