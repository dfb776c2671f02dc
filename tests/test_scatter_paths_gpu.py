"""scatter_add where its form changes: destinations from one entry to past the private copies' 200 KB, element counts around
the choice, skewed, sorted and out-of-range indices; integer sums bit for bit against numpy, float64 sums to the rounding of
their order."""
import numpy as np
import pytest

import ncarray_gb300 as nca
from ncarray_gb300.dtype import DType
from tests.helpers import SEED

pytestmark = pytest.mark.gpu

KINDS = {
    "uniform": lambda rng, n, m: rng.integers(0, m, n),
    "sorted": lambda rng, n, m: np.sort(rng.integers(0, m, n)),
    "hot": lambda rng, n, m: np.where(rng.random(n) < 0.3, m // 2, rng.integers(0, m, n)),
    "outside": lambda rng, n, m: rng.integers(-m, 2 * m, n),
}


@pytest.mark.parametrize("m", [1, 33, 6000, 12289, 25601, 51200, 51201, 300007])
@pytest.mark.parametrize("kind", sorted(KINDS))
def test_forms(cuda, m, kind):
    rng = np.random.default_rng(SEED + 410 + m)
    n = 2_000_003
    idx = KINDS[kind](rng, n, m).astype(np.int32)
    ok = (idx >= 0) & (idx < m)
    src = rng.integers(-50, 50, n)
    want = np.bincount(idx[ok], weights=src[ok], minlength=m) + np.arange(m)
    for dt in (DType.int32, DType.float64):
        d = nca.NCDevArray.from_host(np.arange(m).astype(np.int32 if dt == DType.int32 else np.float64))
        d.scatter_add(idx, src.astype(np.int32 if dt == DType.int32 else np.float64))   # small integers: exact in float64 too
        assert np.array_equal(d.to_host(), want), (m, kind, dt)
