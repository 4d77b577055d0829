"""The packed field table against one field3d per field, for every form of a
quantity: the same words where field3d accepts it, a refusal where it refuses."""
import struct

import numpy as np
import pytest

from pyshield_b200 import quantity
from pyshield_b200.quantity import field3d, fields3d


class Storage:
    """What the packing reads of a CUDA tensor, on the host."""

    def __init__(self, shape, stride, dtype="f64", is_cuda=True):
        self.shape, self._stride, self.dtype, self.is_cuda = shape, stride, dtype, is_cuda

    def dim(self):
        return len(self.shape)

    def stride(self):
        return self._stride

    def data_ptr(self):
        return 1 << 40


class Q:
    def __init__(self, data, origin):
        self.data, self.origin = data, origin


@pytest.fixture(autouse=True)
def storages_are_tensors(monkeypatch):
    monkeypatch.setattr(quantity, "_Tensor", Storage)
    monkeypatch.setattr(quantity, "_F64", "f64")


IFIRST = ((13, 11, 80), (1, 13, 143))
KFIRST = ((13, 11, 80), (880, 80, 1))


@pytest.mark.parametrize("layout", [IFIRST, KFIRST])
@pytest.mark.parametrize("origin", [
    None, (3, 3, 0), [3, 3, 0], np.array([3, 3, 0]), np.array([0, 0, 0]), (np.int64(3), 2, np.int32(1)), (3, 3, 0, 7),
    range(3),
])
def test_same_words(layout, origin):
    q = Q(Storage(*layout), origin)
    want, got = field3d(q, (6, 4, 78)), fields3d([q], (6, 4, 78))[0]
    assert (got.ptr, got.si, got.sj, got.sk) == (want.ptr, want.si, want.sj, want.sk)


@pytest.mark.parametrize("q", [
    Q(Storage(*IFIRST), (3, 3)), Q(Storage(*IFIRST), ()), Q(Storage(*IFIRST), (8, 3, 0)), Q(Storage(*IFIRST), np.array([-1, 0, 0])),
    Q(Storage(*IFIRST, dtype="f32"), (0, 0, 0)), Q(Storage(*IFIRST, is_cuda=False), (0, 0, 0)),
    Q(Storage((13, 11), (1, 13)), (0, 0)), Q(Storage(*IFIRST), (3.0, 3.0, 0.0)),
])
def test_refused_by_both(q):
    for pack in (lambda: field3d(q, (6, 4, 79)), lambda: fields3d([q], (6, 4, 79))):
        with pytest.raises((TypeError, ValueError, IndexError, struct.error)):
            pack()
