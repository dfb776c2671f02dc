"""Reductions whose last CTA merges the partials: the counters a stream keeps
are left zero by every kernel, whatever ran on the stream before."""
import numpy as np
import pytest
import torch

import ncarray_gb300 as nca
from ncarray_gb300 import RedOp

pytestmark = pytest.mark.gpu

# (shape, axes): a full reduction (one counter), few kept positions, columns
# (counters per set of columns), and more sets of columns than a stream's block
# of 16384 counters (16385 * 256 columns of float32: beyond any block)
CASES = [((64, 4096), None), ((3, 70000), [1]), ((600, 1000), [0]), ((3000, 256), [0])]


def _array(shape, seed):
    h = np.random.default_rng(seed).integers(-9, 9, shape).astype(np.int32)
    return h, nca.NCDevArray.from_host(h)


def _sum(a, axes):
    return nca.DevExpr.leaf(a).evaluate(None, [(RedOp.SUM, axes)])[0]


def _want(h, axes):
    return h.sum(axis=None if axes is None else tuple(axes), dtype=np.int64)


@pytest.mark.parametrize("shape,axes", CASES)
def test_repeats_and_streams(cuda, shape, axes):
    h, a = _array(shape, 1)
    want = _want(h, axes)
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(40)]
    outs = []
    for s in streams * 2 + [torch.cuda.default_stream()]:
        with torch.cuda.stream(s):
            outs += [_sum(a, axes) for _ in range(2)]
    torch.cuda.synchronize()
    for o in outs:
        np.testing.assert_array_equal(o.to_host().reshape(want.shape), want)


def test_capture_beside_plain_calls(cuda):
    h, a = _array((600, 1000), 2)
    want = _want(h, [0])
    e = nca.DevExpr.leaf(a)
    out = e.evaluate(None, [(RedOp.SUM, [0])])[0]
    full = e.evaluate(None, [(RedOp.SUM, None)])[0]
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        e.evaluate(None, [(RedOp.SUM, [0])], [out])
        e.evaluate(None, [(RedOp.SUM, None)], [full])
    side = torch.cuda.Stream()
    for _ in range(5):
        out._buf.zero_()
        full._buf.zero_()
        torch.cuda.synchronize()
        g.replay()
        with torch.cuda.stream(side):
            other = e.evaluate(None, [(RedOp.SUM, [0])])[0]
        torch.cuda.synchronize()
        np.testing.assert_array_equal(out.to_host(), want)
        np.testing.assert_array_equal(other.to_host(), want)
        assert int(full.to_host()) == int(want.sum())


def test_staged_units(cuda):
    """Transposed 4-byte operands stored and reduced: pieces of a unit split
    between CTAs, on several streams, repeated, and in a graph beside them."""
    rng = np.random.default_rng(4)
    h = rng.integers(-9, 9, (64, 64, 128, 8)).astype(np.int32)    # (p, b, r, q)
    t = nca.NCDevArray.from_host(h).transpose(3, 1, 2, 0)
    want = h.transpose(3, 1, 2, 0) * 3
    with nca.lazy_mode():
        e = t * np.int32(3)
    red = [(RedOp.SUM, 2), (RedOp.MAX, 2)]
    out = nca.NCDevArray(want.shape, e.dtype)
    ref = e.evaluate(out, red)
    g = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(g):
        e.evaluate(out, red, ref)
    sides = []
    for s in [torch.cuda.Stream() for _ in range(3)]:
        with torch.cuda.stream(s):
            o = nca.NCDevArray(want.shape, e.dtype)
            sides += [(o, e.evaluate(o, red)) for _ in range(3)]
    g.replay()
    g.replay()
    torch.cuda.synchronize()
    for o, (sm, mx) in sides + [(out, ref)]:
        np.testing.assert_array_equal(o.to_host(), want)
        np.testing.assert_array_equal(sm.to_host(), want.sum(axis=2))
        np.testing.assert_array_equal(mx.to_host(), want.max(axis=2))


def test_more_sets_than_counters(cuda):
    # (16, 16385 * 256) has more sets of 256 columns than a stream has counters
    n = 16385 * 256
    h = np.random.default_rng(3).integers(-9, 9, (16, n)).astype(np.int32)
    a = nca.NCDevArray.from_host(h)
    got = nca.DevExpr.leaf(a).evaluate(None, [(RedOp.SUM, [0])])[0]
    np.testing.assert_array_equal(got.to_host(), h.sum(axis=0, dtype=np.int64))
