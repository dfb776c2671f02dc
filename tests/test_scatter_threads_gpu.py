"""scatter_add from two threads on two streams, with private copies of different sizes: each launch finds the
shared-memory limit that it needs."""
import threading

import numpy as np
import pytest

import ncarray_gb300 as nca
from tests.helpers import SEED

pytestmark = pytest.mark.gpu


def test_two_threads_two_sizes(cuda):
    n, rounds = 1 << 23, 150
    rng = np.random.default_rng(SEED + 430)
    cases = []
    for m in (13000, 50000):
        idx = rng.integers(0, m, n).astype(np.int32)
        cases.append((nca.NCDevArray.from_host(idx), nca.NCDevArray.from_host(np.ones(n, np.int32)),
                      nca.NCDevArray.from_host(np.zeros(m, np.int32)), np.bincount(idx, minlength=m)))
    cuda.cuda.synchronize()
    errors = []

    def work(idx, ones, dest, _):
        try:
            with cuda.cuda.stream(cuda.cuda.Stream()):
                for _ in range(rounds):
                    dest.scatter_add(idx, ones)
                cuda.cuda.current_stream().synchronize()
        except Exception as e:   # noqa: BLE001 - reported below
            errors.append(e)

    threads = [threading.Thread(target=work, args=c) for c in cases]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for _, _, dest, want in cases:
        assert np.array_equal(dest.to_host(), rounds * want)
