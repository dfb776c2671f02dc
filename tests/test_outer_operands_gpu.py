"""Outer reductions of expressions over many operands and few rows, where the rows of a lane are loaded together or one by
one: stored values and integer results bit for bit against numpy."""
import numpy as np
import pytest

import ncarray_gb300 as nca
from ncarray_gb300 import RedOp
from tests.helpers import SEED

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nops", [1, 6, 7, 12, 13, 25])
@pytest.mark.parametrize("rows,cols", [(5, 2048), (19, 517), (20, 2048), (33, 260), (64, 517), (300, 64)])
@pytest.mark.parametrize("dt", [np.int32, np.float64])
def test_many_operands(cuda, nops, rows, cols, dt):
    rng = np.random.default_rng(SEED + 450)
    host = [rng.integers(-99, 99, (rows, cols)).astype(dt) for _ in range(nops)]   # sums exact in float64 too
    with nca.lazy_mode():
        e = nca.DevExpr.leaf(nca.NCDevArray.from_host(host[0]))
        for h in host[1:]:
            e = e + nca.NCDevArray.from_host(h)
    want = np.sum(host, axis=0, dtype=dt)
    red = [(RedOp.SUM, 0), (RedOp.MAX, 0), (RedOp.ARGMIN, 0)]
    out = nca.NCDevArray((rows, cols), e.expr_dtype)
    for got in (e.evaluate(out, red), e.evaluate(None, red)):
        np.testing.assert_array_equal(got[0].to_host(), want.sum(axis=0, dtype=got[0].to_host().dtype))
        np.testing.assert_array_equal(got[1].to_host(), want.max(axis=0))
        np.testing.assert_array_equal(got[2].to_host(), want.argmin(axis=0))
    np.testing.assert_array_equal(out.to_host(), want)
    (s,) = e.evaluate(None, red[:1])
    np.testing.assert_array_equal(s.to_host(), want.sum(axis=0, dtype=s.to_host().dtype))
