"""The packed call records equal the general ones: scalar slots against numpy's
conversion, array views against the fields of the C struct."""
import numpy as np
import pytest

from ncarray_gb300 import _lib
from ncarray_gb300.dtype import DType, scalar_slot, to_numpy

INTS = [DType.uint8, DType.uint16, DType.uint32, DType.uint64, DType.int8, DType.int16, DType.int32, DType.int64]


def _numpy_slot(value, dt):
    raw = np.array([value]).astype(to_numpy(dt)).tobytes()
    return int.from_bytes(raw + b"\0" * (8 - len(raw)), "little")


@pytest.mark.parametrize("dt", INTS)
def test_int_slots(dt):
    info = np.iinfo(to_numpy(dt))
    for v in (int(info.min), int(info.max), 0, 1, int(info.max) // 3):
        assert scalar_slot(v, dt) == _numpy_slot(v, dt)
    for v in (-1, 255, 256, 1 << 20):   # also out of the type's range
        assert scalar_slot(v, dt) == _numpy_slot(v, dt)


@pytest.mark.parametrize("dt", [DType.float32, DType.float64])
@pytest.mark.parametrize("v", [0.0, -0.0, 0.1, 1e-46, 3.4028234e38, 3.5e38, 1e300, float("inf"), float("-inf"), float("nan"), 3])
@pytest.mark.filterwarnings("ignore:overflow")
def test_float_slots(dt, v):
    assert scalar_slot(v, dt) == _numpy_slot(v, dt)


@pytest.mark.parametrize("shape,strides", [((), ()), ((5,), (-8,)), ((2, 3, 4), (96, 0, 8)), (tuple(range(1, 9)), (8,) * 8)])
def test_view_fields(shape, strides):
    v = _lib.make_view(0x1000, DType.float64, shape, strides, 16)
    assert (v.data, v.dtype, v.ndim, v.pointer_axis, v.flags) == (0x1010, int(DType.float64), len(shape), -1, 0)
    n = _lib.MAX_NDIM - len(shape)
    assert tuple(v.shape) == shape + (0,) * n and tuple(v.strides) == strides + (0,) * n and not any(v.offsets)


def test_view_refuses_too_many_dims():
    with pytest.raises(ValueError):
        _lib.make_view(0x1000, DType.float64, (1,) * (_lib.MAX_NDIM + 1), (8,) * (_lib.MAX_NDIM + 1))
    assert _lib.make_view(0, DType.float64, (0,), (8,), 64).data is None
