"""Several Jacobi steps in one call: the three-steps-per-pass kernel against single steps.

Both forms add the same terms in the same order, so the two grids afterwards (the last two iterates) are bit-identical to
those of one apply() per step. Extents sit at the tile's edges: 120 columns and 26 rows of outputs a tile, one plane, fewer
planes than steps, several z chunks."""
import numpy as np
import pytest

import ncarray_gb300 as nca
from ncarray_gb300.stencil import Stencil3D, device_status, laplacian7, laplacian27
from tests.helpers import SEED

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 1, 4), (2, 26, 120), (5, 27, 124), (7, 25, 128), (40, 53, 244), (90, 130, 364)])
@pytest.mark.parametrize("kind", ["7", "27", "star"])
def test_iterate_equals_single_steps(cuda, shape, kind):
    rng = np.random.default_rng(SEED + 31)
    u = rng.normal(size=shape).astype(np.float32)
    w = {"7": laplacian7(), "27": laplacian27(), "star": laplacian7()}[kind].copy()
    if kind == "star":   # seven different weights
        w[w != 0.0] = rng.normal(size=7) / 4
    st = Stencil3D(w, 0.1)
    for steps in (3, 4, 5, 7, 11):
        a, b = nca.NCDevArray.from_host(u), nca.NCDevArray(shape, nca.DType.float32).fill(7.0)
        res = st.iterate(a, b, steps)
        assert res is (a if steps % 2 == 0 else b)
        c, d = nca.NCDevArray.from_host(u), nca.NCDevArray(shape, nca.DType.float32)
        for _ in range(steps):
            st.apply(c, d)
            c, d = d, c
        last, before = c.to_host(), d.to_host()
        assert device_status() == 0
        assert np.array_equal(res.to_host(), last), (shape, kind, steps)
        assert np.array_equal((b if res is a else a).to_host(), before), (shape, kind, steps)
