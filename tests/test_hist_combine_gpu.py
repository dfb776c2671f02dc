"""Weight sums of the partitioned histogram where large weights cancel.

Every bin gets the weights 2^50, 2^26, 1, -2^50 and -2^26, far apart in the input, so that they come to the combine pass in
different pieces, and zeros. Their sum, 1, needs 51 bits of the partial sums: float64 has them. (Pieces that hold 2^50,
2^26 and 1 together cannot keep the 1; a piece is about a hundredth of the input, so few bins have one.)"""
import numpy as np
import pytest

import ncarray_gb300 as nca
from ncarray_gb300.dtype import DType
from ncarray_gb300.hist import hist2d_into
from tests.helpers import SEED

pytestmark = pytest.mark.gpu

NBX, NBY = 37, 61   # 2257 bins: the last 256 that a block combines are cut short, and its last group of four too


def _sum(x, y, w, nbx, nby):
    c = nca.NCDevArray((nby, nbx), DType.uint64).fill(0)
    s = nca.NCDevArray((nby, nbx), DType.float32).fill(0.0)
    hist2d_into(*(nca.NCDevArray.from_host(v) for v in (x, y)), c, (0.0, 1.0), (0.0, 1.0), nca.NCDevArray.from_host(w), s)
    return c.to_host().reshape(-1), s.to_host().reshape(-1)


def _points():
    rng = np.random.default_rng(SEED + 940)
    nb = NBX * NBY
    special = np.array([2.0**50, 2.0**26, 1.0, -(2.0**50), -(2.0**26)], np.float32)
    n = 1 << 20
    bins = rng.integers(0, nb, n)
    w = np.zeros(n, np.float32)
    for k, v in enumerate(special):   # a fifth of the input each, in a random order of the five
        at = rng.permutation(n // 5)[:nb] + k * (n // 5)
        bins[at], w[at] = np.arange(nb), v
    x = ((bins % NBX) + 0.5) / NBX
    y = ((bins // NBX) + 0.5) / NBY
    return x.astype(np.float32), y.astype(np.float32), w, np.bincount(bins, minlength=nb)


def _poison():
    """NaN weights in every bin of the largest grid of as many tiles: NaN in the pieces that the pool gives out next."""
    n = 1 << 21
    rng = np.random.default_rng(SEED + 941)
    _sum(rng.random(n, dtype=np.float32), rng.random(n, dtype=np.float32), np.full(n, np.nan, np.float32), 128, 128)


def test_scratch_contents_choose_nothing(cuda):
    """The bins beside the end of the grid are summed as the others are, whatever the scratch held."""
    x, y, w, want = _points()
    _poison()
    c, s = _sum(x, y, w, NBX, NBY)
    assert np.array_equal(c, want)
    last = NBX * NBY // 256 * 256
    ones = s == 1.0
    # 201 bins against 2056: shares of equal chance differ by 0.2 with a probability below 1e-7
    assert abs(ones[last:].mean() - ones[:last].mean()) < 0.2
