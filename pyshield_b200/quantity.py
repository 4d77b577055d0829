"""Quantity-like containers and the strided-pointer view the C-ABI takes.

pySHiELD passes NDSL ``Quantity`` objects: ``.data`` is the full storage
(compute domain plus halo), ``.origin`` / ``.extent`` locate the compute
domain. Any object with those three attributes works here, as long as
``.data`` is a float64 CUDA array: a ``torch.Tensor`` or anything exposing
``__cuda_array_interface__`` (CuPy, Numba, ...). The layout is free: the
element strides are passed to the kernels.
"""

import struct
from operator import index

import numpy as np

try:
    import torch

    _Tensor, _F64 = torch.Tensor, torch.float64
except ImportError:  # pragma: no cover
    _Tensor, _F64 = (), None

from ._lib import ShieldField2D, ShieldField3D


class Quantity:
    """Minimal NDSL-style quantity: storage + compute-domain origin/extent."""

    def __init__(self, data, dims, units, origin=None, extent=None):
        self.data = data
        self.dims = tuple(dims)
        self.units = units
        nd = len(tuple(data.shape))
        self.origin = tuple(origin) if origin is not None else (0,) * nd
        self.extent = tuple(extent) if extent is not None else tuple(data.shape)

    @property
    def view(self):
        """The compute-domain view of ``data`` (torch tensors only)."""
        sl = tuple(slice(o, o + e) for o, e in zip(self.origin, self.extent))
        return self.data[sl]


def _array_info(a):
    """(device pointer, element strides, shape) of a float64 CUDA array."""
    if isinstance(a, _Tensor):
        if a.dtype != _F64:
            raise TypeError(f"expected float64 data, got {a.dtype}")
        if not a.is_cuda:
            raise TypeError("the microphysics kernels need device (CUDA) arrays")
        return a.data_ptr(), tuple(a.stride()), tuple(a.shape)
    cai = getattr(a, "__cuda_array_interface__", None)
    if cai is None:
        raise TypeError(f"{type(a).__name__} is not a CUDA array (no __cuda_array_interface__)")
    if np.dtype(cai["typestr"]) != np.float64:
        raise TypeError(f"expected float64 data, got {cai['typestr']}")
    shape = tuple(cai["shape"])
    if cai.get("strides") is None:
        st = [1] * len(shape)
        for d in range(len(shape) - 2, -1, -1):
            st[d] = st[d + 1] * shape[d + 1]
        strides = tuple(st)
    else:
        if any(s % 8 for s in cai["strides"]):
            raise ValueError("strides must be whole elements")
        strides = tuple(s // 8 for s in cai["strides"])
    return cai["data"][0], strides, shape


def _unpack(q):
    data = getattr(q, "data", q)
    origin = getattr(q, "origin", None)
    ptr, strides, shape = _array_info(data)
    if origin is None:
        origin = (0,) * len(shape)
    return ptr, strides, shape, tuple(origin)


def field3d(q, extent=None):
    """ShieldField3D for a 3-D quantity: pointer at the compute-domain origin."""
    ptr, st, shape, org = _unpack(q)
    if len(shape) != 3:
        raise ValueError(f"expected a 3-D field, got shape {shape}")
    ext = tuple(extent) if extent is not None else tuple(getattr(q, "extent", shape))
    for d in range(3):
        if org[d] < 0 or org[d] + ext[d] > shape[d]:
            raise ValueError(f"domain origin {org} extent {ext} exceeds storage {shape}")
    off = index(org[0] * st[0] + org[1] * st[1] + org[2] * st[2])
    return ShieldField3D(ptr + 8 * off, st[0], st[1], st[2])


def field2d(q, extent=None):
    ptr, st, shape, org = _unpack(q)
    if len(shape) != 2:
        raise ValueError(f"expected a 2-D field, got shape {shape}")
    ext = tuple(extent) if extent is not None else tuple(getattr(q, "extent", shape))
    for d in range(2):
        if org[d] < 0 or org[d] + ext[d] > shape[d]:
            raise ValueError(f"domain origin {org} extent {ext} exceeds storage {shape}")
    off = index(org[0] * st[0] + org[1] * st[1])
    return ShieldField2D(ptr + 8 * off, st[0], st[1])


def _words3d(qs, ext):
    """field3d(q, ext) of every quantity in ``qs`` as a flat list of words.
    A call names 24 to 60 fields, and one ctypes structure per field was much
    of a small call's time (one C12 tile's step: 51 us of host time for 33 us
    on the GPU; 39 us with the words packed at once)."""
    nx, ny, nz = ext
    out = []
    for q in qs:
        data = q if isinstance(q, _Tensor) else getattr(q, "data", q)
        if not (isinstance(data, _Tensor) and data.dtype == _F64 and data.is_cuda and data.dim() == 3):
            f = field3d(q, ext)
            out += (f.ptr or 0, f.si, f.sj, f.sk)
            continue
        si, sj, sk = data.stride()
        ni, nj, nk = data.shape
        org = getattr(q, "origin", None)
        if org is None:
            oi = oj = ok = 0
        else:
            try:
                oi, oj, ok = org
            except ValueError:
                oi, oj, ok = tuple(org)[:3]
        if oi < 0 or oj < 0 or ok < 0 or oi + nx > ni or oj + ny > nj or ok + nz > nk:
            raise ValueError(f"domain origin {(oi, oj, ok)} extent {tuple(ext)} exceeds storage {(ni, nj, nk)}")
        out += (data.data_ptr() + 8 * (oi * si + oj * sj + ok * sk), si, sj, sk)
    return out


def fields3d(qs, ext):
    """An array of ShieldField3D: field3d(q, ext) of every quantity."""
    words = _words3d(qs, ext)
    arr = (ShieldField3D * (len(words) // 4))()
    struct.pack_into(f"{len(words)}q", arr, 0, *words)
    return arr


def set_fields3d(struct_, qs, ext, first=0):
    """field3d(q, ext) of every quantity into the ShieldField3D members of a
    structure, from member ``first`` on (they stand one after another)."""
    words = _words3d(qs, ext)
    struct.pack_into(f"{len(words)}q", struct_, 32 * first, *words)
