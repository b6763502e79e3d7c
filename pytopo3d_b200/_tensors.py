"""Conversions between the reference's (nely, nelx, nelz) arrays and the flat
Fortran-ordered device vectors the kernels use (e = y + nely*(x + nelx*z))."""

from __future__ import annotations

import numpy as np
import torch


_cuda_seen = False


def device() -> torch.device:
    global _cuda_seen
    if not _cuda_seen:  # a device that was there stays; the query costs microseconds per call
        if not torch.cuda.is_available():
            raise RuntimeError("pytopo3d_b200 needs a CUDA device (B200, sm_100a); no CPU fallback")
        _cuda_seen = True
    return torch.device("cuda", torch.cuda.current_device())


def _on_device(t: torch.Tensor, dtype) -> bool:
    return t.is_cuda and t.dtype == dtype and t.get_device() == torch.cuda.current_device()


def to_flat(a, dtype=torch.float64) -> torch.Tensor:
    """(nely, nelx, nelz) array/tensor -> contiguous flat device vector in Fortran order."""
    t = a if isinstance(a, torch.Tensor) else torch.as_tensor(a)
    if t.dim() == 3:
        t = t.permute(2, 1, 0)
    if not _on_device(t, dtype):
        t = t.to(device=device(), dtype=dtype)
    return t.contiguous().reshape(-1)


def to_flat_mask(m) -> torch.Tensor | None:
    if m is None:
        return None
    return to_flat(m, torch.uint8)


def to_flat_mask_view(m) -> torch.Tensor | None:
    """``to_flat_mask`` for a call that only reads the mask before it returns control
    of the stream: a boolean device mask is taken as its own bytes (0 / 1), with no
    conversion kernel and no copy where it already lies in Fortran order."""
    if isinstance(m, torch.Tensor) and m.dtype == torch.bool and m.is_cuda:
        m = m.view(torch.uint8)
    return to_flat_mask(m)


def from_flat(v: torch.Tensor, shape) -> torch.Tensor:
    """Flat Fortran-ordered vector -> (nely, nelx, nelz) view."""
    nely, nelx, nelz = shape
    return v.reshape(nelz, nelx, nely).permute(2, 1, 0)


def like_input(v: torch.Tensor, shape, template):
    """Return a result shaped like the reference (numpy in -> numpy out)."""
    out = from_flat(v, shape)
    if isinstance(template, np.ndarray):
        return out.cpu().numpy()
    return out


def vec(a, dtype=torch.float64) -> torch.Tensor:
    """1-D array/tensor -> contiguous device vector."""
    t = a if isinstance(a, torch.Tensor) else torch.as_tensor(a)
    if not _on_device(t, dtype):
        t = t.to(device=device(), dtype=dtype)
    return t.contiguous().reshape(-1)
