"""Drop-in ``rmsnorm_fp4quant`` / ``add_rmsnorm_fp4quant``.

Same call signatures as the flashinfer CuTe-DSL operators the reference loads
and runs (call sites tests/python/test_flashinfer_norm_verbatim.py:134 and
:155-164; tools/perf/bench_flashinfer_norm.py:53-60).  The work is one CUDA
kernel launch on the current stream through ``b200fp4_rmsnorm_fp4quant`` /
``b200fp4_add_rmsnorm_fp4quant``; nothing is computed or checked in Python and
there is no CPU path.

``global_scale`` MULTIPLIES before quantisation (sf = amax * gs / 6), the
convention of the reference's golden (same file, lines 58-68).
"""
from __future__ import annotations

from typing import Optional, Tuple

import torch

from . import _lib
from .layout import ceil_div

_norm = _lib.native.norm           # checks, allocations and the launch: csrc/torch_binding.cpp
_ONES = {}


def _unit_scale(device) -> torch.Tensor:
    key = (device.type, device.index)
    if key not in _ONES:
        _ONES[key] = torch.ones(1, dtype=torch.float32, device=device)
    return _ONES[key]


def rmsnorm_fp4quant(
    input: torch.Tensor,
    weight: torch.Tensor,
    y_fp4: Optional[torch.Tensor] = None,
    block_scale: Optional[torch.Tensor] = None,
    global_scale: Optional[torch.Tensor] = None,
    eps: float = 1e-6,
    block_size: int = 16,
    scale_format: Optional[str] = None,
    is_sf_swizzled_layout: bool = False,
    enable_pdl: Optional[bool] = None,
) -> Tuple[torch.Tensor, torch.Tensor]:
    """y = RMSNorm(input) * weight, quantised to NVFP4.

    Returns ``(y_fp4, block_scale)``: packed e2m1 codes ``[..., H/2]`` (uint8,
    even element in the low nibble) and e4m3 scale factors, row-major
    ``[..., H/16]`` or, with ``is_sf_swizzled_layout``, in 128x4 tiles.
    ``enable_pdl`` is accepted for signature compatibility and ignored.
    """
    return _norm(input, None, weight, y_fp4, block_scale, None,
                 _unit_scale(input.device) if global_scale is None else global_scale, eps, block_size, scale_format,
                 is_sf_swizzled_layout, False)


def add_rmsnorm_fp4quant(
    input: torch.Tensor,
    residual: torch.Tensor,
    weight: torch.Tensor,
    y_fp4: Optional[torch.Tensor] = None,
    block_scale: Optional[torch.Tensor] = None,
    global_scale: Optional[torch.Tensor] = None,
    eps: float = 1e-6,
    block_size: int = 16,
    scale_format: Optional[str] = None,
    is_sf_swizzled_layout: bool = False,
    output_both_sf_layouts: bool = False,
    block_scale_unswizzled: Optional[torch.Tensor] = None,
    enable_pdl: Optional[bool] = None,
):
    """residual <- input + residual (in place); y = RMSNorm(residual) * weight -> NVFP4.

    Returns ``(y_fp4, block_scale)`` or, with ``output_both_sf_layouts``,
    ``(y_fp4, block_scale, block_scale_unswizzled)`` where ``block_scale`` is
    tiled and the third tensor row-major.
    """
    if residual is None:
        raise ValueError("residual is required")
    return _norm(input, residual, weight, y_fp4, block_scale, block_scale_unswizzled,
                 _unit_scale(input.device) if global_scale is None else global_scale, eps, block_size, scale_format,
                 is_sf_swizzled_layout, output_both_sf_layouts)


__all__ = ["rmsnorm_fp4quant", "add_rmsnorm_fp4quant", "ceil_div"]
