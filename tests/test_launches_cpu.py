"""What the host side of a call launches, without a GPU (tests/fake_cuda)."""
import pytest

from tests import fake_cuda


def test_short_vectors(built_lib, tmp_path):
    """1-D and 0-d expressions of fewer elements than a 16-byte vector: one launch each, no division by the zero whole
    groups (a process on an x86-64 host dies of one)."""
    code = """
result = []
for dt in (DType.float32, DType.int8, DType.float64, DType.bfloat16):
    for shape in ((), (1,), (2,), (3,), (5,), (15,), (16,), (17,)):
        x = array(shape, dt)
        e = nca.DevExpr.leaf(x) + nca.DevExpr.leaf(x)
        e.evaluate(out=array(shape, e.dtype))
        ls = launches()
        result.append([str(dt), shape, len(ls), ls[0]["grid"], ls[0]["consts"]["NCA_VEC"]])
"""
    for dt, shape, n, grid, _ in fake_cuda.run(code, tmp_path):
        assert n == 1 and grid == [1, 1, 1], (dt, shape)
