"""Results of large lattices on their way to the caller: arrays above 2 MB pass through the context's pinned
buffers, above 16 MB converted by several threads.  What was imported comes back exactly (in the
type that the lattice keeps), also for lengths that no buffer divides, repeatedly, and from two contexts
in two threads.
"""
from __future__ import annotations

import threading
import time

import numpy as np
import pytest

from nonnewlbm_b200 import CaseSpec, Lattice, capi
from nonnewlbm_b200 import geometry as G

pytestmark = pytest.mark.gpu
SMALL, LARGE = (97, 89, 83), (163, 167, 171)   # a single-precision field: 2.9 MB, 18.6 MB


def _fields(lat, seed):
    return np.random.default_rng(seed).standard_normal((capi.M_N,) + lat.shape())


@pytest.mark.parametrize("dtype", ["f32", "f64", "f16"])
@pytest.mark.parametrize("shape", [SMALL, LARGE])
def test_fields_come_back(shape, dtype):
    kept = np.float64 if dtype == "f64" else np.float32
    with Lattice(CaseSpec(shape, collision="CUM", dtype=dtype)) as lat:
        for seed in (1, 2):
            f = _fields(lat, seed)
            lat.import_macro(f)
            for k in (0, 3, f.shape[0] - 1):
                assert np.array_equal(lat.macro(k), f[k].astype(kept).astype(np.float64)), (seed, k)


@pytest.mark.parametrize("stats_f64", [True, False])
def test_sums_come_back(stats_f64):
    with Lattice(CaseSpec(SMALL, collision="CUM", dtype="f32", stats_f64=stats_f64)) as lat:
        s = np.random.default_rng(3).standard_normal((6,) + SMALL[::-1])
        lat.import_stats(s, 7)
        got, n = lat.stats()
        assert n == 7
        assert np.array_equal(got, s if stats_f64 else s.astype(np.float32).astype(np.float64))


def test_two_contexts_in_two_threads():
    lats = [Lattice(CaseSpec(LARGE, collision="CUM", dtype="f32")) for _ in range(2)]
    fields = [_fields(lat, 5 + k) for k, lat in enumerate(lats)]
    bad = []

    def read(k):
        lats[k].import_macro(fields[k])
        for _ in range(3):
            for j in range(4):
                if not np.array_equal(lats[k].macro(j), fields[k][j].astype(np.float32).astype(np.float64)):
                    bad.append((k, j))

    threads = [threading.Thread(target=read, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for lat in lats:
        lat.close()
    assert not bad


def test_converting_threads_start_with_the_first_data():
    """A large field is asked for while steps are queued: nothing but the calling thread's own wait
    takes processor time until they have run (five threads convert this field)."""
    with Lattice(CaseSpec(LARGE, collision="CUM", dtype="f64")) as lat:
        lat.set_map(np.full(LARGE[::-1], G.MAP_PERIODIC, dtype=np.uint8))
        lat.init_equilibrium()
        lat.step(2, macro=True)
        lat.macro(0)
        lat.step(1500, macro=True, wait=False)
        wall, cpu = time.perf_counter(), time.process_time()
        lat.macro(0)
        wall, cpu = time.perf_counter() - wall, time.process_time() - cpu
        assert wall > 0.2              # the steps were still queued
        assert cpu <= 2.0 * wall
