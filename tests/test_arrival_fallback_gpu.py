"""Reductions whose last CTA merges, beyond the counters that a stream keeps: more sets of columns than 4096, more staged
units than 16384, and more streams than there are blocks (64). Those zero counters of their own."""
import os
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

import ncarray_gb300 as nca
from ncarray_gb300 import RedOp
from tests.helpers import SEED

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parent.parent


def test_more_sets_than_counters(cuda, monkeypatch):
    """The persistent form splits every set of 256 columns between CTAs somewhere: 4100 sets."""
    monkeypatch.setenv("NCA_K4_ROWS", "3")
    h = np.random.default_rng(SEED + 460).integers(-9, 9, (32, 4100 * 256)).astype(np.int32)
    e = nca.DevExpr.leaf(nca.NCDevArray.from_host(h))
    for _ in range(2):
        s, m = e.evaluate(None, [(RedOp.SUM, 0), (RedOp.ARGMAX, 0)])
        np.testing.assert_array_equal(s.to_host(), h.sum(axis=0, dtype=np.int32))
        np.testing.assert_array_equal(m.to_host(), h.argmax(axis=0))


def test_more_staged_units_than_counters(cuda):
    h = np.random.default_rng(SEED + 461).integers(-9, 9, (64, 8200, 24, 8)).astype(np.int32)   # (p, b, r, q)
    t = nca.NCDevArray.from_host(h).transpose(3, 1, 2, 0)
    with nca.lazy_mode():
        e = t * np.int32(3)
    out = nca.NCDevArray(t.shape, e.dtype)
    for _ in range(2):
        s, m = e.evaluate(out, [(RedOp.SUM, 2), (RedOp.MAX, 2)])
        want = h.transpose(3, 1, 2, 0) * 3
        np.testing.assert_array_equal(s.to_host(), want.sum(axis=2, dtype=s.to_host().dtype))
        np.testing.assert_array_equal(m.to_host(), want.max(axis=2))


CHILD = r"""
import ctypes
import numpy as np
import torch
import ncarray_gb300 as nca
from ncarray_gb300 import RedOp
h = np.random.default_rng(7).integers(-9, 9, (600, 1000)).astype(np.int32)
a = nca.NCDevArray.from_host(h)
p = np.random.default_rng(8).integers(-9, 9, (64, 16, 40, 8)).astype(np.int32)
t = nca.NCDevArray.from_host(p).transpose(3, 1, 2, 0)
with nca.lazy_mode():
    e = t * np.int32(3)
torch.cuda.synchronize()
cu = ctypes.CDLL("libcuda.so.1")
raw = [ctypes.c_void_p() for _ in range(70)]
for r in raw:   # torch hands out the streams of a pool again; these are all different
    assert cu.cuStreamCreate(ctypes.byref(r), 1) == 0
outs = []
for _ in range(2):
    for r in raw:
        with torch.cuda.stream(torch.cuda.ExternalStream(r.value)):
            o = nca.NCDevArray(t.shape, e.dtype)
            outs.append((nca.DevExpr.leaf(a).evaluate(None, [(RedOp.SUM, [0])])[0], e.evaluate(o, [(RedOp.MAX, 2)])[0], o))
torch.cuda.synchronize()
want = h.sum(axis=0, dtype=np.int32), p.transpose(3, 1, 2, 0).max(axis=2) * 3
for s, m, _ in outs:
    assert np.array_equal(s.to_host(), want[0]) and np.array_equal(m.to_host(), want[1])
print("ok", len(outs))
"""


def test_more_streams_than_blocks(cuda):
    """In a process of its own: the blocks stay with the first 64 streams of a process."""
    env = dict(os.environ, PYTHONPATH=str(ROOT) + os.pathsep + os.environ.get("PYTHONPATH", ""))
    r = subprocess.run([sys.executable, "-c", CHILD], env=env, cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.split() == ["ok", "140"], r.stderr[-2000:]
