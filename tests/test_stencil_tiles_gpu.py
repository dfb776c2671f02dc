"""The three-steps-per-pass stencil at the edges of its tiles: 120 columns, 36 rows (star weights) or 18 (isotropic), chunks
of planes; bit for bit against single steps. The grids are ones that take the pass (two launches for four steps)."""
import numpy as np
import pytest

import ncarray_gb300 as nca
from ncarray_gb300 import _lib
from ncarray_gb300.stencil import Stencil3D, device_status, laplacian7, laplacian27
from tests.helpers import SEED

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("points", [7, 27])
@pytest.mark.parametrize("ny", [1, 17, 18, 19, 35, 36, 37, 54, 72, 73])
@pytest.mark.parametrize("nz,nx", [(8, 4), (8, 116), (9, 120), (8, 124), (37, 240), (20, 364)])
def test_tile_edges(cuda, points, ny, nz, nx):
    shape = (nz, ny, nx)
    u = np.random.default_rng(SEED + 32).normal(size=shape).astype(np.float32)
    st = Stencil3D(laplacian7() if points == 7 else laplacian27(), 0.1)
    a, b = nca.NCDevArray.from_host(u), nca.NCDevArray(shape, nca.DType.float32).fill(7.0)
    before = _lib.lib().nca_launch_count()
    res = st.iterate(a, b, 4)
    assert _lib.lib().nca_launch_count() - before == 2
    c, d = nca.NCDevArray.from_host(u), nca.NCDevArray(shape, nca.DType.float32)
    for _ in range(4):
        st.apply(c, d)
        c, d = d, c
    assert device_status() == 0
    assert np.array_equal(res.to_host(), c.to_host())
    assert np.array_equal((b if res is a else a).to_host(), d.to_host())
