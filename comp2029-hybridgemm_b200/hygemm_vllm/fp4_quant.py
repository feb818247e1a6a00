"""Offline MXFP4 quantisation with a per-group exponent search, and the E2M1 helpers around it.

Counterpart of the reference's `integrations/vllm/allocation/fp4_quant.py`: same
function names, arguments and return values (`unpack`, `codes_rne`, `pack_codes`,
`decode_logical`, `quantize`).  The search itself is one CUDA kernel
(`hg_clip_pack`) instead of a chain of full-tensor torch ops; the helpers are
plain torch and run on any device, which is what the CPU tests use.  Online
quantisation and the GEMM are untouched: the result only replaces the stored
MXFP4 rows of a layer (`offline_weights.replace_low_weight`).
"""
from __future__ import annotations

import ctypes as C

import torch

from . import native

# Midpoints between neighbouring E2M1 magnitudes 0, .5, 1, 1.5, 2, 3, 4, 6.
_MIDPOINTS = (0.25, 0.75, 1.25, 1.75, 2.5, 3.5, 5.0)
_MAGNITUDES = (0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0)


def unpack(q: torch.Tensor) -> torch.Tensor:
    """`[rows, k/2]` bytes -> `[rows, k]` 4-bit codes (even k in the low nibble)."""
    return torch.stack((q & 15, q >> 4), dim=-1).reshape(q.shape[0], -1)


def pack_codes(code: torch.Tensor) -> torch.Tensor:
    """`[rows, k]` 4-bit codes -> `[rows, k/2]` bytes."""
    return (code[:, 0::2] | (code[:, 1::2] << 4)).contiguous()


def codes_rne(x: torch.Tensor) -> torch.Tensor:
    """E2M1 code of every element: nearest magnitude, ties to the even code, saturating at 6, sign kept for -0."""
    mids = torch.tensor(_MIDPOINTS, dtype=x.dtype, device=x.device)
    mag = x.abs().contiguous()
    code = torch.bucketize(mag, mids, right=False)                  # first midpoint >= |x|
    on_midpoint = (code < 7) & (mag == mids[code.clamp(max=6)])
    code = code + (on_midpoint & (code % 2 == 1)).long()             # an odd code on a midpoint yields to its even neighbour
    return code.to(torch.uint8) | (torch.signbit(x).to(torch.uint8) << 3)


def decode_logical(q: torch.Tensor, scales: torch.Tensor, k: int) -> torch.Tensor:
    """fp32 values of packed codes `[rows, k/2]` under logical scale bytes `[rows, k/32]`."""
    table = torch.tensor(_MAGNITUDES + tuple(-m for m in _MAGNITUDES), dtype=torch.float32, device=q.device)
    table[8] = 0.0
    values = table[unpack(q).long()].reshape(q.shape[0], k // 32, 32)
    return (values * torch.exp2(scales.float() - 127).unsqueeze(-1)).reshape(q.shape[0], k)


def quantize(w: torch.Tensor, importance: torch.Tensor | None = None, offsets=(0, -1, -2)):
    """Search the E8M0 exponent of every K32 group of `w` `[rows, k]` (reference: fp4_quant.py:28-58).

    Returns `(q4 [rows, k/2], scales [rows, k/32], stats)`: codes and logical scale bytes that never have a
    larger importance-weighted squared error than round-to-nearest, and the same statistics dictionary as the
    reference (`groups`, `shift_groups`, `weighted_error_before/after`, `weight_error_before/after`).
    """
    if w.ndim != 2 or w.dtype not in native.DTYPES or not w.is_cuda or w.shape[1] % 128:
        raise ValueError("quantize needs a CUDA FP16/BF16 [rows, K] matrix with K % 128 == 0")
    rows, k = w.shape
    w = w.contiguous()
    weight = None
    if importance is not None:
        weight = importance.to(device=w.device, dtype=torch.float32).contiguous()
        if weight.shape != (k,):
            raise ValueError("importance must be k finite non-negative values")
    q4 = torch.empty((rows, k // 2), dtype=torch.uint8, device=w.device)
    scales = q4.new_empty((rows, k // 32))
    shifts, found = (C.c_int * len(offsets))(*[int(o) for o in offsets]), (C.c_double * 16)()
    native.check(native.library().hg_clip_pack_stats(
        w.data_ptr(), weight.data_ptr() if weight is not None else None, q4.data_ptr(), scales.data_ptr(), rows, k, shifts,
        len(offsets), native.DTYPES[w.dtype], found, native._stream(w.device)))
    # One read of sixteen numbers tells whether the inputs were valid and what the search did.
    weighted_before, weighted_after, before, after, not_finite, bad_importance, grew, _, *moved = found
    if not_finite:
        raise ValueError("weights must be finite")
    if bad_importance:
        raise ValueError("importance must be k finite non-negative values")
    if grew:
        raise AssertionError("exponent search increased a group's weighted error")
    stats = {"groups": rows * (k // 32),
             "shift_groups": {str(-s): int(count) for s, count in zip(offsets, moved)},
             "weighted_error_before": weighted_before,
             "weighted_error_after": weighted_after,
             "weight_error_before": before,
             "weight_error_after": after}
    return q4, scales, stats
