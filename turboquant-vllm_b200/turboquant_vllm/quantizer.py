"""Rotation + Lloyd-Max quantiser (host-side holder of the TQ4 primitives).

Mirrors ``TurboQuantMSE`` and ``_generate_rotation_matrix`` of the reference
(src/turboquant_vllm/quantizer.py:46-191).  Construction is CPU-side and deterministic from
``(dim, bits, seed)``; ``quantize`` / ``dequantize`` on CUDA tensors run the fused sm_100a
kernels (norm + normalise + rotate + bucketize in one launch).  CPU tensors are rejected:
this package has no CPU compute path.
"""

from __future__ import annotations

import threading
from collections import OrderedDict

import torch

from turboquant_vllm.lloyd_max import LloydMaxCodebook, solve_lloyd_max


def _generate_rotation_matrix(dim: int, seed: int = 42) -> torch.Tensor:
    """Haar-distributed orthogonal ``[dim, dim]`` fp32 matrix on CPU.

    QR of a seeded CPU Gaussian; each column is multiplied by the sign of the matching
    diagonal entry of R so the distribution is uniform over O(d).  Uses the same torch CPU
    generator + LAPACK calls as the reference (src/turboquant_vllm/quantizer.py:46-69), so the
    matrix is bit-identical for a given torch build.
    """
    rng = torch.Generator(device="cpu")
    rng.manual_seed(seed)
    g = torch.randn(dim, dim, generator=rng, device="cpu", dtype=torch.float32)
    q, r = torch.linalg.qr(g)
    signs = torch.sign(torch.diagonal(r))
    signs = torch.where(signs == 0, torch.ones_like(signs), signs)
    return q * signs.unsqueeze(0)


class _Recent:
    """The last ``size`` results of pure functions of their key: safe with several threads, older ones dropped.

    A cache object is made per generation, and its rotation (a QR on the host, about a millisecond at
    head_dim 128) and device tensors (ten small copies) depend only on ``(dim, bits, seed)``: a
    generation of some tokens spent half its time on them."""

    def __init__(self, size: int) -> None:
        self._size, self._lock, self._held = size, threading.Lock(), OrderedDict()

    def get(self, key, make):
        with self._lock:
            hit = self._held.get(key)
            if hit is not None:
                self._held.move_to_end(key)
                return hit
        made = make()
        with self._lock:
            made = self._held.setdefault(key, made)
            self._held.move_to_end(key)
            while len(self._held) > self._size:
                self._held.popitem(last=False)
        return made


_rotations = _Recent(8)
_device_rotations = _Recent(8)   # at most 8 x 768 KB (head_dim 256)
_device_codebooks = _Recent(16)


def nibble_unpack(packed: torch.Tensor) -> torch.Tensor:
    """u8 ``[..., D/2]`` -> int64 ``[..., D]`` (high nibble first)."""
    hi = (packed >> 4).long()
    lo = (packed & 0x0F).long()
    return torch.stack([hi, lo], dim=-1).flatten(-2)


def nibble_pack(indices: torch.Tensor) -> torch.Tensor:
    """uint8 ``[..., D]`` with values < 16 -> u8 ``[..., D/2]``."""
    u = indices.to(torch.uint8)
    return (u[..., 0::2] << 4) | u[..., 1::2]


class TurboQuantMSE:
    """Rotation + per-coordinate Lloyd-Max quantiser.

    Attributes:
        dim, bits: vector dimension and bits per coordinate.
        codebook: :class:`LloydMaxCodebook` (fp32 CPU tensors).
        rotation: orthogonal ``[dim, dim]`` fp32 CPU tensor (``Pi``).
    """

    def __init__(self, dim: int, bits: int, *, seed: int = 42) -> None:
        self.dim = dim
        self.bits = bits
        cents, bounds = solve_lloyd_max(dim, bits)
        self.codebook = LloydMaxCodebook(centroids=cents, boundaries=bounds, bits=bits, dim=dim)
        self.rotation = _rotations.get((dim, seed), lambda: _generate_rotation_matrix(dim, seed=seed)).clone()
        self._seed = seed
        # the tensors as made here, to tell whether a caller has changed or replaced one since
        self._made = [(x, x._version) for x in (self.rotation, cents, bounds)]
        self._dev: dict[torch.device, tuple[torch.Tensor, ...]] = {}

    def device_primitives(self, device: torch.device):
        """(rotation, rot_T_even, rot_T_odd, centroids, boundaries) resident on ``device``."""
        prim = self._dev.get(device)
        if prim is None:
            device = torch.device(device)
            prim = self._dev.get(device)
        if prim is None:
            def rotation():
                rot_t = self.rotation.T.contiguous()
                return (self.rotation.to(device).contiguous(), rot_t[:, 0::2].contiguous().to(device),
                        rot_t[:, 1::2].contiguous().to(device))

            def codebook():
                return self.codebook.centroids.to(device), self.codebook.boundaries.to(device)

            now = (self.rotation, self.codebook.centroids, self.codebook.boundaries)
            if device.type == "cuda" and all(x is y and x._version == n for x, (y, n) in zip(now, self._made)):
                # shared by the quantisers first used on one stream (the allocator's unit of reuse)
                where = (device, torch.cuda.current_stream(device).cuda_stream)
                prim = (_device_rotations.get((self.dim, self._seed, *where), rotation)
                        + _device_codebooks.get((self.dim, self.bits, *(n for _, n in self._made[1:]), *where), codebook))
            else:
                prim = rotation() + codebook()
            self._dev[device] = prim
        return prim

    def quantize_packed(self, x: torch.Tensor) -> tuple[torch.Tensor, torch.Tensor]:
        """``[..., dim]`` -> (nibble-packed u8 ``[..., dim/2]``, norms f32 ``[..., 1]``)."""
        from turboquant_vllm.kernels.ops import tq4_compress

        if x.shape[-1] != self.dim:
            raise ValueError(
                f"Input last dimension {x.shape[-1]} does not match quantizer dim {self.dim}. "
                "Ensure the compressor's head_dim matches the model's actual head dimension."
            )
        if self.bits > 4:
            raise NotImplementedError("nibble-packed storage holds at most 4 bits per coordinate")
        _, even, odd, _, bounds = self.device_primitives(x.device)
        lead = x.shape[:-1]
        flat = x.reshape(-1, 1, self.dim)
        packed, norms = tq4_compress(flat, even, odd, bounds)
        return packed.reshape(*lead, self.dim // 2), norms.reshape(*lead, 1)

    def quantize(self, x: torch.Tensor) -> tuple[torch.Tensor, torch.Tensor]:
        """``[..., dim]`` -> (indices int64 ``[..., dim]``, norms f32 ``[..., 1]``)."""
        packed, norms = self.quantize_packed(x)
        return nibble_unpack(packed), norms

    def dequantize_packed(self, packed: torch.Tensor, norms: torch.Tensor,
                          dtype: torch.dtype = torch.float32) -> torch.Tensor:
        """Nibble-packed indices + norms -> reconstructed ``[..., dim]`` in original space."""
        from turboquant_vllm.kernels.ops import tq4_decompress

        rot, _, _, cents, _ = self.device_primitives(packed.device)
        lead = packed.shape[:-1]
        rows = tq4_decompress(
            packed.reshape(-1, 1, self.dim // 2), norms.reshape(-1, 1, 1), cents, torch.float32
        )
        return (rows.reshape(-1, self.dim) @ rot).reshape(*lead, self.dim).to(dtype)

    def dequantize(self, indices: torch.Tensor, norms: torch.Tensor) -> torch.Tensor:
        """``centroids[indices] @ Pi * norm`` (fp32)."""
        if indices.shape[-1] != self.dim:
            raise ValueError(
                f"Indices last dimension {indices.shape[-1]} does not match quantizer dim "
                f"{self.dim}. Check that the same quantizer instance is used for quantize and "
                "dequantize."
            )
        return self.dequantize_packed(nibble_pack(indices), norms)
