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


def test_cancelling_weights_keep_float64_precision(cuda):
    """Nine bins in ten and more sum to exactly 1; a sum held in 48 bits loses the 1 under 2^50 in most orders."""
    x, y, w, want = _points()
    c, s = _sum(x, y, w, NBX, NBY)
    assert np.array_equal(c, want)
    # three of the weights together in one of the 152 pieces (at most three chunks of the input in a piece of the
    # 256 chunks): about (1/85)^2; four in five would already show a lost bit in most bins
    assert (s == 1.0).mean() > 0.97
    # the same into an output that is not empty
    c2 = nca.NCDevArray((NBY, NBX), DType.uint64).fill(0)
    s2 = nca.NCDevArray((NBY, NBX), DType.float32).fill(3.0)
    hist2d_into(*(nca.NCDevArray.from_host(v) for v in (x, y)), c2, (0.0, 1.0), (0.0, 1.0), nca.NCDevArray.from_host(w), s2)
    assert (s2.to_host() == 4.0).mean() > 0.97


@pytest.mark.parametrize("nbx,nby,n", [(37, 61, 1 << 20), (1024, 1024, 1 << 21), (100, 100, (1 << 22) + 5)])
def test_signed_weights_against_float64(cuda, nbx, nby, n):
    """Signed lognormal weights over a wide range: no further from the exact sums than float32 records allow. A bin of m
    records: TwoSum keeps every addition's error but the compensation's own roundings, m additions of size below
    u M each losing u of it, and the last rounding."""
    rng = np.random.default_rng(SEED + 942)
    bx, by = rng.integers(0, nbx, n), rng.integers(0, nby, n)
    x, y = ((bx + 0.5) / nbx).astype(np.float32), ((by + 0.5) / nby).astype(np.float32)
    w = (np.exp(rng.normal(size=n) * 4) * rng.choice([-1.0, 1.0], n)).astype(np.float32)
    b = by * nbx + bx
    c, s = _sum(x, y, w, nbx, nby)
    assert np.array_equal(c, np.bincount(b, minlength=nbx * nby))
    want = np.bincount(b, weights=w.astype(np.float64), minlength=nbx * nby)
    size = np.bincount(b, weights=np.abs(w).astype(np.float64), minlength=nbx * nby)   # bounds every partial sum
    m = np.bincount(b, minlength=nbx * nby)
    u = 2.0**-24
    assert np.all(np.abs(s - want) <= u * np.abs(want) * 1.001 + 2 * m * m * u * u * size + 1e-30)
