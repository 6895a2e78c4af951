"""Orthorhombic periodic geometry on [..., 3] tensors; ``cell`` [3] holds the edge lengths in nm.

The same functions and arithmetic as src/nabladyn/space.py:11-64. The MD engine does its own
wrapping inside its kernels; these serve the host-side API (allocation, checks, export).
"""

import torch
from torch import Tensor

from . import _native


def _displacement_wrapped(left: Tensor, right: Tensor, cell: Tensor) -> Tensor:
    """The minimum-image vector ``left - right`` for coordinates already in [0, L).

    The coordinate on the far side moves by L first, which is exact, so the vector is rounded
    once (src/nabladyn/space.py:11-19).
    """
    raw = left - right
    half = 0.5 * cell
    left_shift = torch.where(raw > half, cell, 0.0)
    right_shift = torch.where(raw < -half, cell, 0.0)
    return (left - left_shift) - (right - right_shift)


def wrap(positions: Tensor, cell: Tensor) -> tuple[Tensor, Tensor]:
    """Wrap positions [..., 3] into [0, L); return (wrapped, crossings int64).

    The floor of the quotient, then two fix-ups in this order keep every result in [0, L)
    (src/nabladyn/space.py:22-38).
    """
    crossings = torch.floor(positions / cell)
    wrapped = positions - crossings * cell
    below = wrapped < 0
    wrapped = torch.where(below, wrapped + cell, wrapped)
    crossings = torch.where(below, crossings - 1, crossings)
    above = wrapped >= cell
    wrapped = torch.where(above, wrapped - cell, wrapped)
    crossings = torch.where(above, crossings + 1, crossings)
    return wrapped, crossings.to(torch.int64)


def wrapped_only(positions: Tensor, cell: Tensor) -> Tensor:
    """``wrap(positions, cell)[0]`` of a frame [N, 3] and cell [3], or of frames [F, N, 3] and
    their cells [F, 3], without autograd and contiguous. CUDA frames take one kernel (nd_wrap,
    the same rounding) instead of ``wrap``'s dozen elementwise ones."""
    positions, cell = positions.detach(), cell.detach()
    if not (positions.is_cuda and positions.dtype in (torch.float32, torch.float64)
            and cell.dtype == positions.dtype and cell.device == positions.device
            and positions.shape[-1:] == (3,) and positions.ndim in (2, 3)
            and cell.shape == (*positions.shape[:-2], 3)):
        return wrap(positions, cell if cell.ndim == 1 else cell[:, None])[0].contiguous()
    positions, cell = positions.contiguous(), cell.contiguous()
    out = torch.empty_like(positions)
    frames = 1 if positions.ndim == 2 else positions.shape[0]
    with _native.on_device(positions.device):
        _native.call("nd_wrap", _native.dtype_code(positions.dtype), positions.data_ptr(),
                     cell.data_ptr(), frames, positions.shape[-2], out.data_ptr(),
                     _native.stream_handle(positions.device))
    return out


def shift(positions: Tensor, delta: Tensor, cell: Tensor) -> tuple[Tensor, Tensor]:
    """``positions + delta`` wrapped into the cell, with ``wrap``'s crossings."""
    return wrap(positions + delta, cell)


def displacement(left: Tensor, right: Tensor, cell: Tensor) -> Tensor:
    """The minimum-image vector ``left - right`` [..., 3], for positions anywhere."""
    return _displacement_wrapped(wrap(left, cell)[0], wrap(right, cell)[0], cell)


def strained(vectors: Tensor, strain: Tensor | None) -> Tensor:
    """Deform ``vectors`` [..., 3] by (I + strain); None returns ``vectors`` itself."""
    if strain is None:
        return vectors
    return (
        vectors
        + vectors[..., 0:1] * strain[:, 0]
        + vectors[..., 1:2] * strain[:, 1]
        + vectors[..., 2:3] * strain[:, 2]
    )


__all__ = ("wrap", "shift", "displacement", "strained")
