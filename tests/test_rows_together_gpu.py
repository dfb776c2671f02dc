"""Outer reductions whose rows are loaded several at a time: row counts around
the trips of 32 rows and their splits, odd kept extents, few and many sets of
columns, strided operands; against numpy and the thread-per-column form."""
import numpy as np
import pytest

import ncarray_gb300 as nca
from ncarray_gb300.dtype import DType, to_numpy
from tests.helpers import SEED

pytestmark = pytest.mark.gpu

SHAPES = [(1, 64), (31, 300), (32, 4096), (33, 257), (63, 1024), (65, 40000), (128, 16), (700, 33), (1000, 4), (257, 130000),
          (40, 700000), (97, 160000)]


def _run(a, red):
    return [r.to_host() for r in nca.DevExpr.leaf(a).evaluate(None, red)]


@pytest.mark.parametrize("dt", [DType.float32, DType.float64, DType.int32, DType.uint16])
@pytest.mark.parametrize("shape", SHAPES)
def test_rows_together(cuda, monkeypatch, dt, shape):
    rng = np.random.default_rng(SEED + 611)
    h = (rng.standard_normal(shape) * 100).astype(to_numpy(dt)) if dt in (DType.float32, DType.float64) else \
        rng.integers(0, 1000, shape).astype(to_numpy(dt))
    a = nca.NCDevArray.from_host(h)
    sets = [[(nca.RedOp.SUM, 0)], [(nca.RedOp.MAX, 0)], [(nca.RedOp.SUM, 0), (nca.RedOp.ARGMIN, 0)]]
    got = [_run(a, r) for r in sets]
    monkeypatch.setenv("NCA_K4_ROWS", "0")
    ref = [_run(a, r) for r in sets]
    wide = h.astype(np.float64)
    # float64: shape[0] roundings of at most 2^-53 of the sum of magnitudes; float32 sums are compensated; integers exact
    ulp = {DType.float64: shape[0] * 2.0 ** -53, DType.float32: 2.0 ** -23}.get(dt, 0.0)
    bound = ulp * np.abs(wide).sum(axis=0)
    for g, r in ((got[0][0], ref[0][0]), (got[2][0], ref[2][0])):
        assert np.all(np.abs(g.astype(np.float64) - wide.sum(axis=0)) <= bound)
        assert np.all(np.abs(g.astype(np.float64) - r.astype(np.float64)) <= 2 * bound)
    np.testing.assert_array_equal(got[1][0], h.max(axis=0))
    np.testing.assert_array_equal(got[1][0], ref[1][0])
    np.testing.assert_array_equal(got[2][1], h.argmin(axis=0))
    np.testing.assert_array_equal(got[2][1], ref[2][1])


@pytest.mark.parametrize("axis", [0, 1])
def test_crops_and_strides(cuda, axis):
    h = np.random.default_rng(SEED + 612).integers(-99, 99, (130, 70, 531)).astype(np.int32)
    a = nca.NCDevArray.from_host(h)
    for sl in ((slice(3, 120), slice(1, 68), slice(5, 517)), (slice(None, None, 2), slice(None), slice(0, 528, 3)),
               (slice(None), slice(None), slice(0, 528))):
        got = _run(a[sl], [(nca.RedOp.SUM, axis), (nca.RedOp.ARGMAX, axis)])
        np.testing.assert_array_equal(got[0], h[sl].sum(axis=axis))
        np.testing.assert_array_equal(got[1], h[sl].argmax(axis=axis))
