"""scatter_add where a warp changes its mind: hot indices that come and go over many trips of one warp, several of them,
runs, one index only, none; integer sums bit for bit against numpy, float64 sums of small integers exactly."""
import numpy as np
import pytest

import ncarray_gb300 as nca
from ncarray_gb300.dtype import DType
from tests.helpers import SEED

pytestmark = pytest.mark.gpu


def _phases(rng, n, m):
    """An eighth of the input each: uniform, one hot index, another one, three of them, runs of 16, one index alone, runs of
    512, indices outside the destination between uniform ones."""
    idx = rng.integers(0, m, n)
    e = n // 8
    r = rng.random(n)

    def part(k):
        return slice(k * e, (k + 1) * e)

    idx[part(1)] = np.where(r[part(1)] < 0.05, m // 3, idx[part(1)])
    idx[part(2)] = np.where(r[part(2)] < 0.3, m // 2, idx[part(2)])
    idx[part(3)] = np.where(r[part(3)] < 0.3, (r[part(3)] * 10).astype(np.int64) % m, idx[part(3)])
    idx[part(4)] = np.arange(e) // 16 % m
    idx[part(5)] = m - 1
    idx[part(6)] = rng.integers(0, m, e // 512 + 1)[np.arange(e) // 512]
    idx[part(7)] = np.where(r[part(7)] < 0.5, idx[part(7)], rng.integers(-5, 0, e))
    return idx


# 24 M elements: some twenty trips a warp through L2 atomics, so that hot entries are found, lost and replaced; 3000 and
# 12000 entries through private copies, with and without runs to global memory; 50 M elements into 40 entries
@pytest.mark.parametrize("dt", [DType.int32, DType.float64, DType.float32, DType.int64])
@pytest.mark.parametrize("n,m", [(24_000_003, 300_007), (24_000_003, 12_000), (24_000_003, 3_000), (24_000_003, 40), (1_244_160, 99_991),
                                 (1_245_185, 99_991), (1, 70_000), (33, 70_000)])
@pytest.mark.parametrize("shuffle", [False, True])
def test_phases(cuda, n, m, dt, shuffle):
    rng = np.random.default_rng(SEED + 440 + m)
    idx = _phases(rng, n, m) if n > 100 else rng.integers(0, 3, n)
    if shuffle:   # blocks of 128 elements, a trip of a warp, in another order
        idx[:n // 128 * 128] = idx[:n // 128 * 128].reshape(-1, 128)[rng.permutation(n // 128)].reshape(-1)
    src = rng.integers(-3, 5, n)
    ok = (idx >= 0) & (idx < m)
    want = np.bincount(idx[ok], weights=src[ok], minlength=m) + np.arange(m)
    host = {DType.int32: np.int32, DType.int64: np.int64, DType.float32: np.float32, DType.float64: np.float64}[dt]
    d = nca.NCDevArray.from_host(np.arange(m).astype(host))
    d.scatter_add(idx.astype(np.int64 if dt == DType.int64 else np.int32), src.astype(host))
    # every partial sum is an integer below 2^24 in float32 too: 12 M elements of at most 4 around a mean of 0.5
    assert np.abs(want).max() < 2**24
    assert np.array_equal(d.to_host(), want)
