"""HuggingFace ``DynamicCache`` wrapper that stores TQ-compressed K/V (GPU only).

Same public surface as the reference's ``CompressedDynamicCache``
(src/turboquant_vllm/kv_cache.py:275-1044): it replaces ``update`` / ``get_seq_length`` of the
wrapped cache, keeps uint8 centroid indices (nibble-packed at 4 bits) plus fp32 norms per layer,
hands the fused attention path the packed tensors through ``get_compressed``, and otherwise
returns incrementally dequantised K/V.  Differences under the surface:

* an update is one launch (norm + rotate + bucketize + pack into the layer's buffers, and in the default
  mode the reconstructed K/V behind the ones held), not a chain of PyTorch ops;
* storage grows by capacity doubling, so appending a token does not re-copy the whole layer
  (the reference ``torch.cat``s every step);
* in fused mode a 4-bit layer is kept as token rows in the paged kernels' own format
  (:class:`turboquant_vllm.token_rows.TokenRowStore`): an update is one launch of the paged write
  kernel and the fused attention reads the rows in place; ``get_compressed`` then returns strided
  views of that buffer;
* tensors must live on a CUDA device — there is no CPU compute path.
"""

from __future__ import annotations

import sys
import threading
import types
import warnings
import weakref
from dataclasses import dataclass
from typing import Any

import torch

from turboquant_vllm import _native as nv
from turboquant_vllm.compressors import CompressedValues, TurboQuantCompressorMSE
from turboquant_vllm.quantizer import nibble_pack, nibble_unpack
from turboquant_vllm.token_rows import TokenRowStore


def _packed_size(bits: int, head_dim: int) -> int:
    """Index bytes per token per head: nibble-packed at 4 bits, one byte per index otherwise."""
    return head_dim // 2 if bits == 4 else head_dim


_UPDATE_DIMS, _UPDATE_DTYPES = (64, 96, 128, 256), (torch.float16, torch.bfloat16, torch.float32)
_STORE_DTYPES = (torch.uint8, torch.float32, torch.uint8, torch.float32)


@dataclass
class _CompressedLayer:
    """Indices (uint8, ``[B, H, S, D]`` or ``[B, H, S, D/2]`` when ``packed``) + fp32 norms ``[B, H, S, 1]``."""

    indices: torch.Tensor
    norms: torch.Tensor
    packed: bool = False


class _GrowBuffer:
    """A ``[B, H, capacity, W]`` tensor that is appended to along dim 2 with amortised O(1) copies."""

    fit = None  # (first buffer of a layer) plan of the last in-place update, see CompressedDynamicCache._step

    def __init__(self) -> None:
        self.buf: torch.Tensor | None = None
        self.len = 0

    def __getstate__(self) -> dict:
        """What a copy or a file takes along: not the plan, which is of these buffers."""
        return {k: v for k, v in self.__dict__.items() if k != "fit"}

    def reserve(self, b: int, h: int, n: int, w: int, dtype: torch.dtype, device: torch.device) -> torch.Tensor:
        """The buffer with room for ``n`` more tokens of ``[b, h, ., w]``; a new one if it held another shape."""
        buf = self.buf
        if buf is None or buf.shape[:2] != (b, h) or buf.shape[3] != w:
            cap = max(64, 1 << (max(n, 1) - 1).bit_length())
            self.buf = torch.empty(b, h, cap, w, dtype=dtype, device=device)
            self.len = 0
            self.fit = None
        elif self.len + n > buf.shape[2]:
            cap = max(2 * buf.shape[2], 1 << (self.len + n - 1).bit_length())
            grown = torch.empty(b, h, cap, w, dtype=dtype, device=device)
            grown[:, :, : self.len] = buf[:, :, : self.len]
            self.buf = grown
            self.fit = None
        return self.buf

    def append(self, x: torch.Tensor) -> torch.Tensor:
        n = x.shape[2]
        buf = self.reserve(x.shape[0], x.shape[1], n, x.shape[3], x.dtype, x.device)
        buf[:, :, self.len : self.len + n] = x
        self.len += n
        return self.view()

    def view(self) -> torch.Tensor:
        assert self.buf is not None
        return self.buf.narrow(2, 0, self.len)


class _RowsField:
    """One of the four reference tensors of a row-format layer, with the ``len`` / ``view()`` face of
    :class:`_GrowBuffer` (0 = K indices, 1 = K norms, 2 = V indices, 3 = V norms)."""

    def __init__(self, store: TokenRowStore, which: int) -> None:
        self.store, self.which = store, which

    @property
    def len(self) -> int:
        return self.store.len

    def view(self) -> torch.Tensor:
        return self.store.views()[self.which]


# Wrappers alive.  A wrapped cache and its wrapper hold one another (either alone has to keep both), so dropping both
# leaves their device memory to Python's cycle collector, which counts objects, not bytes: a program that makes a cache
# per generation piled up dead ones and spent half of a short generation in cudaMalloc.  Each new wrapper
# therefore cuts those pairs that only their own cycle holds.
_wrappers: set = set()
_wrappers_lock = threading.RLock()


def _only_cycle_holds(w: "CompressedDynamicCache") -> bool:
    """Whether every reference to the wrapper ``w``, its cache and the four methods between them is one of theirs."""
    probe = object()
    base = sys.getrefcount(probe)  # what this frame adds to an object that it names
    c = w.cache
    held = getattr(c, "__dict__", {})
    own = [held.get("update"), held.get("get_seq_length")]
    if any(getattr(m, "__self__", None) is not w for m in own):
        return False
    originals = [w._original_update, w._original_get_seq_length]
    for methods in (own, originals):
        while methods:
            m = methods.pop()
            if sys.getrefcount(m) != base + 1:
                return False
    m = None
    bound = sum(getattr(x, "__self__", None) is c for x in (w._original_update, w._original_get_seq_length))
    # w: its two methods in the cache, the caller's name for it; c: w.cache and the original methods bound to it
    return sys.getrefcount(w) == base + 3 and sys.getrefcount(c) == base + 1 + bound


def _counts_tell() -> bool:
    """Whether this interpreter's reference counts tell a dead pair from a live one, tried on stand-ins.

    The arithmetic of :func:`_only_cycle_holds` rests on how names and arguments are counted, which is the
    interpreter's own affair; where any of these pairs is judged wrongly, nothing is released by it."""
    if not getattr(sys, "_is_gil_enabled", lambda: True)():
        return False  # (free threading: the counts are not exact)

    class Cache:
        def update(self): ...
        def get_seq_length(self): ...

    def pair():
        c, w = Cache(), object.__new__(CompressedDynamicCache)
        w.cache, w._original_update, w._original_get_seq_length = c, c.update, c.get_seq_length
        c.update, c.get_seq_length = w._compressed_update, w._compressed_get_seq_length
        return w

    def judged_dead(ref):
        w = ref()
        return _only_cycle_holds(w)

    def with_held(part):
        w = pair()
        ref, held = weakref.ref(w), part(w)
        w = None
        return judged_dead(ref), held

    def as_argument(w):
        return judged_dead(weakref.ref(w))

    def suspended(w):
        yield
        yield w

    def held_by_generator(w):
        g = suspended(w)
        next(g)
        return g

    live = (lambda w: w, lambda w: w.cache, lambda w: w.cache.update, lambda w: w.cache.get_seq_length,
            lambda w: w._original_update, lambda w: w._original_get_seq_length, lambda w: w.restore,
            lambda w: types.MethodType(Cache.update, w.cache), lambda w: [w], lambda w: lambda: w, held_by_generator)
    try:
        return (with_held(lambda w: None)[0] and not as_argument(pair()) and not as_argument(w=pair())
                and not any(with_held(part)[0] for part in live))
    except Exception:  # noqa: BLE001  (an interpreter without getrefcount, say)
        return False


def _release_unreachable() -> None:
    if not _counts_are_exact:
        return
    with _wrappers_lock:
        for ref in list(_wrappers):
            w = ref()
            if w is None:
                _wrappers.discard(ref)
            elif _only_cycle_holds(w):
                _wrappers.discard(ref)
                del w.cache.update, w.cache.get_seq_length
            w = None


class CompressedDynamicCache:
    """KV cache wrapper with real memory savings (uint8 indices + fp32 norms).

    Args:
        cache: a HuggingFace ``DynamicCache``.
        head_dim: primary head dimension; even when any component uses 4 bits.
        bits: shorthand for ``k_bits = v_bits = bits``.
        k_bits, v_bits: per-component bit widths (2-4).
        seed: rotation seed.
        model_config: optional model config; when its ``layer_types`` mixes sliding and full
            attention, FULL-attention layers bypass compression (they are the only retrieval path
            for tokens beyond the window) and sliding layers are compressed.

    Raises:
        ValueError: no bit width given, or a 4-bit component with odd ``head_dim``.
    """

    def __init__(
        self,
        cache: Any,
        head_dim: int,
        bits: int | None = 3,
        *,
        k_bits: int | None = None,
        v_bits: int | None = None,
        seed: int = 42,
        model_config: Any = None,
    ) -> None:
        kb = k_bits if k_bits is not None else bits
        vb = v_bits if v_bits is not None else bits
        if kb is None or vb is None:
            raise ValueError(
                "No bit-width specified. Provide `bits` as shorthand, or `k_bits` and `v_bits` individually."
            )
        for name, b in (("k_bits", kb), ("v_bits", vb)):
            if b == 4 and head_dim % 2:
                raise ValueError(f"{name}=4 requires even head_dim for nibble packing, got {head_dim}")
        self.cache = cache
        self.head_dim = head_dim
        self.bits = kb  # kept for callers that read a single width
        self.k_bits, self.v_bits = kb, vb
        self._k_nibble_packed, self._v_nibble_packed = kb == 4, vb == 4
        self._seed = seed
        self.enabled = True
        self.fused_mode = False
        self._original_dtype: torch.dtype = torch.bfloat16
        self._key_compressors: dict[int, TurboQuantCompressorMSE] = {
            head_dim: TurboQuantCompressorMSE(head_dim, kb, seed=seed)
        }
        self._value_compressors: dict[int, TurboQuantCompressorMSE] = {
            head_dim: TurboQuantCompressorMSE(head_dim, vb, seed=seed)
        }
        # per layer: growable storage; None = layer not compressed (bypassed)
        self._k_store: list[tuple[_GrowBuffer, _GrowBuffer] | None] = []
        self._v_store: list[tuple[_GrowBuffer, _GrowBuffer] | None] = []
        self._dec_k: list[_GrowBuffer | None] = []
        self._dec_v: list[_GrowBuffer | None] = []
        # per layer: token-row storage while the layer is in fused mode (then _k_store/_v_store
        # hold _RowsField views of it)
        self._rows: list[TokenRowStore | None] = []

        if hasattr(cache.update, "__self__") and isinstance(cache.update.__self__, CompressedDynamicCache):
            warnings.warn(
                "Cache is already wrapped by TurboQuant. Call restore() on the existing wrapper first.",
                UserWarning, stacklevel=2,
            )
        layer_types = getattr(model_config, "layer_types", None)
        mixed = bool(layer_types) and any("sliding" in t for t in layer_types)
        self._full_attn_bypass: set[int] = (
            {i for i, t in enumerate(layer_types) if "full" in t} if mixed else set()
        )
        if model_config is not None and mixed and not any(
            getattr(layer, "is_sliding", False) for layer in cache.layers
        ):
            warnings.warn(
                "Cache appears to lack sliding window layer metadata. Create cache with "
                "`DynamicCache(config=model.config)` for correct Gemma support.",
                UserWarning, stacklevel=2,
            )
        _release_unreachable()
        self._original_update = cache.update
        self._original_get_seq_length = cache.get_seq_length
        cache.update = self._compressed_update
        cache.get_seq_length = self._compressed_get_seq_length
        with _wrappers_lock:
            _wrappers.add(weakref.ref(self))

    # ----- compressors ------------------------------------------------------------------------
    def _get_compressors(self, dim: int):
        """Compressors for ``dim`` (created on first use: heterogeneous head dims)."""
        if dim not in self._key_compressors:
            for name, packed in (("k_bits", self._k_nibble_packed), ("v_bits", self._v_nibble_packed)):
                if packed and dim % 2:
                    raise ValueError(
                        f"{name}=4 requires even head_dim for nibble packing, got layer head_dim={dim}"
                    )
            self._key_compressors[dim] = TurboQuantCompressorMSE(dim, self.k_bits, seed=self._seed)
            self._value_compressors[dim] = TurboQuantCompressorMSE(dim, self.v_bits, seed=self._seed)
        return self._key_compressors[dim], self._value_compressors[dim]

    @property
    def key_compressor(self) -> TurboQuantCompressorMSE:
        return self._key_compressors[self.head_dim]

    @property
    def value_compressor(self) -> TurboQuantCompressorMSE:
        return self._value_compressors[self.head_dim]

    @property
    def rotation(self) -> torch.Tensor:
        """Shared rotation ``[head_dim, head_dim]`` fp32 (K and V use the same seed)."""
        return self.key_compressor.quantizer.rotation

    @property
    def centroids(self) -> torch.Tensor:
        """Key codebook ``[2^k_bits]`` fp32."""
        return self.key_compressor.quantizer.codebook.centroids

    _nibble_pack = staticmethod(nibble_pack)
    _nibble_unpack = staticmethod(nibble_unpack)

    # ----- compress / dequantise one tensor ------------------------------------------------------
    def _compress_tensor(self, compressor: TurboQuantCompressorMSE, tensor: torch.Tensor, *,
                         nibble_packed: bool) -> _CompressedLayer:
        """``[B, H, S, D]`` -> indices + fp32 norms; one fused kernel launch."""
        packed, norms = compressor.quantizer.quantize_packed(tensor)
        if nibble_packed:
            return _CompressedLayer(packed, norms, True)
        return _CompressedLayer(nibble_unpack(packed).to(torch.uint8), norms, False)

    def _dequantize_layer(self, compressor: TurboQuantCompressorMSE, layer: _CompressedLayer) -> torch.Tensor:
        """Indices + norms -> reconstructed tensor in the dtype of the last update."""
        packed = layer.indices if layer.packed else nibble_pack(layer.indices)
        return compressor.quantizer.dequantize_packed(packed, layer.norms, self._original_dtype)

    @staticmethod
    def _cat_layers(existing: _CompressedLayer, new: _CompressedLayer) -> _CompressedLayer:
        return _CompressedLayer(
            torch.cat([existing.indices, new.indices], dim=-2),
            torch.cat([existing.norms, new.norms], dim=-2),
            existing.packed,
        )

    def _ensure_layer_initialized(self, layer: Any, key_states, value_states) -> None:
        if not layer.is_initialized:
            try:
                layer.lazy_initialization(key_states, value_states)
            except TypeError:  # transformers 4.x signature
                layer.lazy_initialization(key_states)

    def _pad_to(self, layer_idx: int) -> None:
        while len(self._k_store) <= layer_idx:
            self._k_store.append(None)
            self._v_store.append(None)
            self._dec_k.append(None)
            self._dec_v.append(None)
            self._rows.append(None)

    # ----- the patched cache methods ----------------------------------------------------------------
    def _compressed_update(self, key_states, value_states, layer_idx: int, cache_kwargs=None):
        """Compress the new tokens, append, return K/V for attention (or placeholders in fused mode)."""
        kv = self._step(key_states, value_states, layer_idx)
        if kv is not None:
            return kv
        if not self.enabled:
            return self._original_update(key_states, value_states, layer_idx, cache_kwargs)
        if layer_idx in self._full_attn_bypass:
            self._pad_to(layer_idx)
            return self._original_update(key_states, value_states, layer_idx, cache_kwargs)
        self._original_dtype = key_states.dtype
        if self.cache.layer_class_to_replicate is not None:
            while len(self.cache.layers) <= layer_idx:
                self.cache.layers.append(self.cache.layer_class_to_replicate())
        dim = key_states.shape[-1]
        if self.fused_mode and dim != self.head_dim:
            raise RuntimeError(
                f"Fused TQ4 mode only supports the primary head_dim={self.head_dim}, but layer "
                f"{layer_idx} has head_dim={dim}. Disable fused mode for heterogeneous architectures."
            )
        k_comp, v_comp = self._get_compressors(dim)
        self._pad_to(layer_idx)
        if self.fused_mode and self._k_nibble_packed and self._v_nibble_packed:
            self._append_rows(layer_idx, key_states, value_states, k_comp, v_comp)
            layer = self.cache.layers[layer_idx]
            self._ensure_layer_initialized(layer, key_states, value_states)
            layer.keys, layer.values = key_states, value_states  # placeholders; attention reads the rows
            return key_states, value_states
        if self._rows[layer_idx] is not None:
            self._rows_to_buffers(layer_idx, k_comp, v_comp)
        ks = self._k_store[layer_idx] or (_GrowBuffer(), _GrowBuffer())
        vs = self._v_store[layer_idx] or (_GrowBuffer(), _GrowBuffer())
        dec = ()
        if not self.fused_mode:  # (in fused mode the kernel reads get_compressed(); no K/V is reconstructed)
            dec = (self._dec_k[layer_idx] or _GrowBuffer(), self._dec_v[layer_idx] or _GrowBuffer())
        if not self._update_in_place(key_states, value_states, ks + vs, dec, k_comp.quantizer, v_comp.quantizer):
            new_k = self._compress_tensor(k_comp, key_states, nibble_packed=self._k_nibble_packed)
            new_v = self._compress_tensor(v_comp, value_states, nibble_packed=self._v_nibble_packed)
            ks[0].append(new_k.indices)
            ks[1].append(new_k.norms)
            vs[0].append(new_v.indices)
            vs[1].append(new_v.norms)
            if dec:
                dec[0].append(self._dequantize_layer(k_comp, new_k))
                dec[1].append(self._dequantize_layer(v_comp, new_v))
        self._k_store[layer_idx], self._v_store[layer_idx] = ks, vs
        if dec:
            self._dec_k[layer_idx], self._dec_v[layer_idx] = dec

        layer = self.cache.layers[layer_idx]
        self._ensure_layer_initialized(layer, key_states, value_states)
        if self.fused_mode:  # placeholders
            layer.keys, layer.values = key_states, value_states
            return key_states, value_states
        layer.keys, layer.values = dec[0].view(), dec[1].view()
        return layer.keys, layer.values

    def _step(self, key_states, value_states, layer_idx: int):
        """An update like the one before of its layer, which is most of a generation: what it returns, or ``None`` (nothing
        changed) for the whole way round.  The native part compares what the earlier update found with what is there now."""
        if not self.enabled or layer_idx >= len(self._k_store) or layer_idx >= len(self.cache.layers):
            return None
        ks = self._k_store[layer_idx]
        layer = self.cache.layers[layer_idx]
        if ks is None or layer_idx in self._full_attn_bypass or not layer.is_initialized:
            return None
        dim = key_states.shape[-1]
        k_comp, v_comp = self._key_compressors.get(dim), self._value_compressors.get(dim)
        if k_comp is None or v_comp is None:
            return None
        rows, kv = self._rows[layer_idx], True
        if self.fused_mode and self._k_nibble_packed and self._v_nibble_packed:
            if rows is None or dim != self.head_dim or not rows.append_like(
                    key_states, value_states, k_comp.quantizer, v_comp.quantizer):
                return None
        else:
            dec = () if self.fused_mode else (self._dec_k[layer_idx], self._dec_v[layer_idx])
            if rows is not None or ks[0].fit is None or None in dec or self.fused_mode and dim != self.head_dim:
                return None
            kv = nv.host().cache_step(ks[0].fit, (*ks, *self._v_store[layer_idx], *dec), key_states, value_states,
                                      k_comp.quantizer, v_comp.quantizer)
            if kv is None:
                return None
        layer.keys, layer.values = (key_states, value_states) if kv is True else kv  # (fused mode: placeholders)
        self._original_dtype = key_states.dtype
        return layer.keys, layer.values

    def _update_in_place(self, key_states, value_states, store, dec, k_quant, v_quant) -> bool:
        """Compress, store and (``dec``) reconstruct the new tokens in one launch behind the tokens held.

        False, with nothing changed, for shapes and types the kernel does not take, K and V that are not
        alike, or buffers that hold something else: the caller then goes tensor by tensor.
        """
        dev, dtype = key_states.device, key_states.dtype
        if (key_states.dim() != 4 or key_states.shape != value_states.shape or dtype != value_states.dtype
                or dev != value_states.device or not key_states.is_cuda or dtype not in _UPDATE_DTYPES):
            return False
        b, h, n, d = key_states.shape
        if n == 0 or d not in _UPDATE_DIMS or k_quant.bits > 4 or v_quant.bits > 4:
            return False
        rot, even, odd, k_cents, k_bounds = k_quant.device_primitives(dev)
        v_rot, _, _, v_cents, v_bounds = v_quant.device_primitives(dev)
        if rot is not v_rot:
            return False
        bufs = []
        for group, widths, types in (
            (store, (_packed_size(self.k_bits, d), 1, _packed_size(self.v_bits, d), 1), _STORE_DTYPES),
            (dec, (d, d), (dtype, dtype)),
        ):
            for g, w, t in zip(group, widths, types):
                first, buf = group[0], g.buf
                if g.len != first.len or (buf is None) != (first.buf is None) or buf is not None and (
                        buf.shape != (b, h, first.buf.shape[2], w) or buf.dtype != t or buf.device != dev):
                    return False
                bufs.append((g, w, t))
        # nothing here may hold the old buffers: each goes when its copy is made, not when all six have grown
        store[0].fit = out = buf = t = None
        out = [g.reserve(b, h, n, w, t, dev) for g, w, t in bufs]
        prims = (rot, even, odd, k_bounds, v_bounds, k_cents, v_cents)
        store[0].fit = nv.host().cache_update(
            key_states, value_states, *prims, self._k_nibble_packed, self._v_nibble_packed, *out[:4], store[0].len,
            *(out[4:] or (None, None)), dec[0].len if dec else 0, k_quant, v_quant)
        for g, _, _ in bufs:
            g.len += n
        return True

    # ----- token-row storage (fused mode) -------------------------------------------------------------
    def _append_rows(self, layer_idx: int, key_states, value_states, k_comp, v_comp) -> None:
        """Fused-mode update: compress and store the new tokens as token rows, one kernel launch."""
        b, h, n, d = key_states.shape
        store = self._rows[layer_idx]
        if store is None or not store.matches(b, h, d, key_states.device):
            held = self._k_store[layer_idx]
            if store is None and held is not None and held[0].len and held[0].view().shape[:2] == (b, h):
                # tokens stored before fused mode was switched on: carry them over
                ks, vs = held, self._v_store[layer_idx]
                store = TokenRowStore.from_tensors(ks[0].view(), ks[1].view(), vs[0].view(), vs[1].view())
            else:
                store = TokenRowStore(b, h, d, key_states.device, n)  # (with room for these at once: no second buffer and table)
            self._rows[layer_idx] = store
            self._k_store[layer_idx] = (_RowsField(store, 0), _RowsField(store, 1))
            self._v_store[layer_idx] = (_RowsField(store, 2), _RowsField(store, 3))
            self._dec_k[layer_idx] = self._dec_v[layer_idx] = None
        store.append(key_states, value_states, k_comp.quantizer, v_comp.quantizer)

    def _rows_to_buffers(self, layer_idx: int, k_comp, v_comp) -> None:
        """Leave fused mode for one layer: four growable tensors again, plus the dequantised K/V of
        the tokens held so far (what the non-fused ``update`` returns)."""
        store = self._rows[layer_idx]
        assert store is not None
        k_idx, k_n, v_idx, v_n = (x.contiguous() for x in store.views())
        self._rows[layer_idx] = None
        for slot, idx, norm, comp, dec in ((self._k_store, k_idx, k_n, k_comp, self._dec_k),
                                           (self._v_store, v_idx, v_n, v_comp, self._dec_v)):
            pair = (_GrowBuffer(), _GrowBuffer())
            pair[0].append(idx)
            pair[1].append(norm)
            slot[layer_idx] = pair
            dec[layer_idx] = _GrowBuffer()
            dec[layer_idx].append(self._dequantize_layer(comp, _CompressedLayer(idx, norm, True)))

    def get_token_rows(self, layer_idx: int) -> TokenRowStore | None:
        """The layer's token-row storage, or ``None`` when the layer is not held in that format
        (not in fused mode, a bit width other than 4, bypassed, or never updated)."""
        return self._rows[layer_idx] if layer_idx < len(self._rows) else None

    def _compressed_get_seq_length(self, layer_idx: int = 0) -> int:
        if not self.enabled or layer_idx in self._full_attn_bypass:
            return self._original_get_seq_length(layer_idx)
        if layer_idx >= len(self._k_store):
            return 0
        entry = self._k_store[layer_idx]
        if entry is None:
            return self._original_get_seq_length(layer_idx)
        return int(entry[0].len)

    # ----- views used by callers / tests of the reference ----------------------------------------------
    @property
    def _compressed_keys(self) -> list[_CompressedLayer | None]:
        return [None if e is None else _CompressedLayer(e[0].view(), e[1].view(), self._k_nibble_packed)
                for e in self._k_store]

    @property
    def _compressed_values(self) -> list[_CompressedLayer | None]:
        return [None if e is None else _CompressedLayer(e[0].view(), e[1].view(), self._v_nibble_packed)
                for e in self._v_store]

    def get_compressed(self, layer_idx: int):
        """``(k_indices, k_norms, v_indices, v_norms)`` of a layer, no dequantisation.

        Raises:
            ValueError: the layer has no compressed data (never updated, or bypassed).
        """
        if layer_idx >= len(self._k_store):
            raise ValueError(f"Layer {layer_idx} has no compressed data (not yet updated)")
        if self._k_store[layer_idx] is None:
            raise ValueError(f"Layer {layer_idx} has no compressed data (SWA-bypassed layer)")
        ks, vs = self._k_store[layer_idx], self._v_store[layer_idx]
        return ks[0].view(), ks[1].view(), vs[0].view(), vs[1].view()

    # ----- lifecycle --------------------------------------------------------------------------------------
    def disable(self) -> None:
        self.enabled = False

    def enable(self) -> None:
        self.enabled = True

    def restore(self) -> None:
        """Put the wrapped cache's original ``update`` / ``get_seq_length`` back."""
        self.cache.update = self._original_update
        self.cache.get_seq_length = self._original_get_seq_length

    def __enter__(self) -> "CompressedDynamicCache":
        return self

    def __exit__(self, *exc: object) -> bool:
        self.restore()
        return False

    # ----- statistics (keys as in the reference, kv_cache.py:953-1044) -----------------------------------------
    def vram_bytes(self) -> int:
        """Bytes of compressed storage in use (keys + values, bypassed layers excluded)."""
        total = 0
        for store in (self._k_store, self._v_store):
            for e in store:
                if e is not None:
                    for gb in e:
                        v = gb.view()
                        total += v.numel() * v.element_size()
        return total

    def baseline_vram_bytes(self) -> int:
        """Bytes the same tokens would take as fp16 tensors."""
        total = 0
        for store, packed in ((self._k_store, self._k_nibble_packed), (self._v_store, self._v_nibble_packed)):
            for e in store:
                if e is not None:
                    b, h, s, d = e[0].view().shape
                    total += b * h * s * (2 * d if packed else d) * 2
        return total

    def compression_stats(self) -> dict[str, Any]:
        layers = [e for e in self._k_store if e is not None]
        if not layers:
            return {}
        comp, base = self.vram_bytes(), self.baseline_vram_bytes()
        b, h, s, _ = layers[0][0].view().shape
        per_token = len(layers) * h * (
            _packed_size(self.k_bits, self.head_dim) + 4 + _packed_size(self.v_bits, self.head_dim) + 4
        )
        return {
            "num_layers": len(layers), "seq_len": s, "batch_size": b, "num_heads": h,
            "head_dim": self.head_dim, "bits": self.bits, "k_bits": self.k_bits, "v_bits": self.v_bits,
            "k_nibble_packed": self._k_nibble_packed, "v_nibble_packed": self._v_nibble_packed,
            "compressed_mib": comp / 2**20, "baseline_mib": base / 2**20,
            "compression_ratio": round(base / comp, 2) if comp else 0.0,
            "savings_mib": (base - comp) / 2**20,
            "vram_estimate": {n: round(per_token * n / 2**20, 2) for n in (4096, 16384, 32768)},
        }


_counts_are_exact = _counts_tell()

__all__ = ["CompressedDynamicCache", "CompressedValues"]
