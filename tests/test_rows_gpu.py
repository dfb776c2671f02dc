"""Elementwise expressions whose rows defeat 16-byte vectors: odd row lengths, crops that start anywhere, operands that stay
put along an outer axis (loaded once for several of its indices), rows shorter and longer than a warp's segment. Bit for bit
against the oracle, in every layout the row-segment kernel takes and at its edges."""
import numpy as np
import pytest

import ncarray_gb300 as nca
from ncarray_gb300.dtype import DType
from tests.helpers import SEED, assert_bits_equal, oracle_eval, rand

pytestmark = pytest.mark.gpu


def check(orc, expr, pairs, out, what):
    host = {id(d): h for d, h in pairs}
    want = oracle_eval(orc, expr, [host[id(a)] for a in expr.arrays])
    expr.evaluate(out=out)
    assert_bits_equal(out.to_host(), want, what)


@pytest.mark.parametrize("shape", [(70, 90, 255), (40, 130, 1015), (9, 600, 33), (3, 1700, 64), (5, 7, 31), (37, 41, 129),
                                   (2, 3, 70001)])
@pytest.mark.parametrize("dt", [DType.uint16, DType.float32, DType.float64])
def test_frames(cuda, orc, shape, dt):
    """(raw - dark) * gain + row offset over a crop: dark and gain stay put along axis 0, the offset along axes 0 and 2."""
    rng = np.random.default_rng(SEED + 210)
    n, h, w = shape
    raw, dark, gain = rand(rng, (n, h + 3, w + 5), dt), rand(rng, (h + 1, w + 2), DType.float32), rand(rng, (h, w), DType.float32)
    off = rand(rng, (h, 1), DType.float32)
    d = [nca.NCDevArray.from_host(a) for a in (raw, dark, gain, off)]
    v = [d[0][:, 2:2 + h, 3:3 + w], d[1][1:, 1:1 + w], d[2], d[3]]
    hv = [raw[:, 2:2 + h, 3:3 + w], dark[1:, 1:1 + w], gain, off]
    with nca.lazy_mode():
        e = (v[0] - v[1]) * v[2] + v[3]
    check(orc, e, list(zip(v, hv)), nca.NCDevArray(e.shape, e.dtype), f"{shape} {dt.name}")


@pytest.mark.parametrize("n", [1, 3, 31, 4095, 100001, 1 << 20])
@pytest.mark.parametrize("dt", [DType.float32, DType.bfloat16, DType.int8])
def test_one_dim_tails(cuda, orc, n, dt):
    """Contiguous 1-D operands of any length (a last group of fewer elements), and the same off the 16-byte grid."""
    rng = np.random.default_rng(SEED + 211)
    a, b = rand(rng, (n + 1,), dt), rand(rng, (n + 1,), dt)
    da, db = nca.NCDevArray.from_host(a, dt), nca.NCDevArray.from_host(b, dt)
    for lo in (0, 1):
        u, v = da[lo:lo + n], db[lo:lo + n]
        with nca.lazy_mode():
            e = u * v + u
        check(orc, e, [(u, a[lo:lo + n]), (v, b[lo:lo + n])], nca.NCDevArray(e.shape, e.dtype), f"{n} {dt.name} {lo}")


def test_strides_orders_and_index(cuda, orc):
    """Reversed and stepped inner axes, a permuted output, the IDX tape, and an in-place update, on odd rows."""
    rng = np.random.default_rng(SEED + 212)
    a, b = rand(rng, (60, 130, 303), DType.float32), rand(rng, (60, 130, 303), DType.int32)
    da, db = nca.NCDevArray.from_host(a), nca.NCDevArray.from_host(b)
    u, hu = da[:, ::-1, 1:302:3], a[:, ::-1, 1:302:3]
    v, hv = db[:, :, 302:201:-1], b[:, :, 302:201:-1]
    with nca.lazy_mode():
        e = u * 2.0 + v
    check(orc, e, [(u, hu), (v, hv)], nca.NCDevArray(e.shape, e.dtype), "stepped and reversed")
    out = nca.NCDevArray((130, 60, 101), e.dtype).transpose(1, 0, 2)
    check(orc, e, [(u, hu), (v, hv)], out, "permuted output")
    with nca.lazy_mode():
        i = da[:, :, 1:302] + nca.iota((60, 130, 301))
    got = i.materialize().to_host()
    want = a[:, :, 1:302].astype(np.float64) + np.arange(60 * 130 * 301).reshape(60, 130, 301)
    assert np.array_equal(got, want.astype(got.dtype)) if got.dtype == np.float64 else np.allclose(got, want, rtol=2e-7)
    w = da[:, 1:, 1:302]
    w += db[:, 1:, 1:302]
    h = a.copy()
    h[:, 1:, 1:302] += b[:, 1:, 1:302].astype(np.float32)
    assert_bits_equal(da.to_host(), h, "in place")
