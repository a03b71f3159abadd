"""Builds from host arrays: their particles come back in windows where that pays (from 2^24 particles),
in one copy an array below, whatever the subtree kernel takes. Bit for bit against the oracle, with
windows asked for as well."""
import time

import numpy as np
import pytest

from test_gpu_staged import check_host_build, context_with_windows

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("windows", [None, 2, 16])
@pytest.mark.parametrize("kind,seed,n,d,use_pinned", [
    ("uniform", 310, 500, 16, False),
    ("uniform", 310, 70_001, 1000, True),
    ("plummer", 315, 1 << 20, 1 << 10, True),
    ("uniform", 310, (1 << 22) + 12345, 1 << 12, False),
    ("plummer", 311, 1 << 22, 1 << 14, True),
    ("uniform", 312, (1 << 24) + 1, 1 << 13, True),
    ("plummer", 313, (1 << 24) + 3, 1 << 13, False),
])
def test_host_builds_match_oracle(engine, oracle, kind, seed, n, d, use_pinned, windows):
    x, y, z = (oracle.gen_uniform if kind == "uniform" else oracle.gen_plummer)(seed, n)
    c = engine.Context(0) if windows is None else context_with_windows(engine, windows)
    try:
        check_host_build(c, oracle, x, y, z, d, use_pinned)
    finally:
        c.close()


@pytest.mark.parametrize("n,d", [(30_000, 64), (1 << 19, 256)])
def test_small_host_builds_are_not_cut_into_windows(engine, oracle, n, d):
    """From ordinary memory, against a context that copies everything after the build: sixteen copies
    an array made 2^19 particles 1.8 times as slow."""
    src = oracle.gen_uniform(4, n)

    def ms(c):
        times = []
        for _ in range(15):
            h = [a.copy() for a in src]
            t = time.perf_counter()
            c.build(*h, d)
            times.append(time.perf_counter() - t)
        c.close()
        return np.median(times[3:])

    assert ms(engine.Context(0)) < 1.25 * ms(context_with_windows(engine, 0))
