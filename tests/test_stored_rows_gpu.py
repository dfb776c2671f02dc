"""Expressions stored while an outer axis is reduced (rows taken several at a time, splits chosen by fill): row counts around
the batches and splits, odd kept extents, an in-place store. Stored values and maxima bit for bit against the oracle, sums
within the rounding of a float64 sum."""
import numpy as np
import pytest

import ncarray_gb300 as nca
from ncarray_gb300.dtype import DType
from tests.helpers import SEED, assert_bits_equal, oracle_eval, rand

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", [DType.float64, DType.float32])
@pytest.mark.parametrize("shape", [(1, 40), (3, 1000), (31, 257), (33, 64), (65, 4096), (256, 20000), (700, 33)])
def test_stored_outer_reduction(cuda, orc, dt, shape):
    rng = np.random.default_rng(SEED + 510)
    a, b, c = (rand(rng, shape, dt) for _ in range(3))
    d = [nca.NCDevArray.from_host(v) for v in (a, b, c)]
    with nca.lazy_mode():
        e = d[0] * d[1] + nca.sqrt(abs(d[2])) - 0.5 * d[0]
    want = oracle_eval(orc, e, [{id(x): h for x, h in zip(d, (a, b, c))}[id(v)] for v in e.arrays])
    out = nca.NCDevArray(shape, dt)
    s, m = e.evaluate(out=out, reductions=[(nca.RedOp.SUM, 0), (nca.RedOp.MAX, 0)])
    assert_bits_equal(out.to_host(), want, "stored")
    assert_bits_equal(m.to_host(), want.max(axis=0), "max")
    exact = want.astype(np.float64).sum(axis=0)
    # float64 sums: shape[0] roundings of at most 2^-53 of the sum of magnitudes; float32 ones are compensated
    bound = (shape[0] * 2.0 ** -53 if dt == DType.float64 else 2.0 ** -23) * np.abs(want).astype(np.float64).sum(axis=0)
    assert np.all(np.abs(s.to_host().astype(np.float64) - exact) <= bound)
    e.evaluate(out=d[0], reductions=[(nca.RedOp.MAX, 0)])   # stored over an operand
    assert_bits_equal(d[0].to_host(), want, "in place")
