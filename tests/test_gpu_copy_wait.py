"""The subtree kernel's bounded wait for its own copies of keys, run out on purpose: the copies are
left out (nothing is under way when the wait ends), the polls few. The kernel leaves the cells it
has not finished, the build returns ORB_ERR_TIMEOUT in a bounded time, whatever the cells' size
(groups of 32, 16, 8 and 2 warps) and the entry point, and the same context then builds the
oracle's tree bit for bit."""
import time

import numpy as np
import pytest

from test_gpu_parity import assert_same

pytestmark = pytest.mark.gpu

ORB_ERR_TIMEOUT = 6


@pytest.fixture
def fresh(engine):
    c = engine.Context(0)
    yield c
    c.close()


def times_out(engine, call):
    with pytest.raises(engine.OrbError) as e:
        call()
    assert e.value.status == ORB_ERR_TIMEOUT


@pytest.mark.parametrize("polls", [64, 0])
def test_build_gives_up_and_context_recovers(fresh, engine, oracle, polls):
    n, d = 30011, 64
    x, y, z = oracle.gen_uniform(11, n)
    fresh.test_set_scan_wait(polls, 0)
    fresh.test_drop_copies(True)
    t = time.monotonic()
    times_out(engine, lambda: fresh.build(x.copy(), y.copy(), z.copy(), d))
    assert time.monotonic() - t < 20.0  # about a second at the default number of polls
    fresh.test_set_scan_wait(0, 0)
    fresh.test_drop_copies(False)
    gx, gy, gz = x.copy(), y.copy(), z.copy()
    assert_same(fresh.build(gx, gy, gz, d), oracle.build_tree(x, y, z, d), gx, gy, gz)


@pytest.mark.parametrize("n", [500, 5000, 15000, 30000])
def test_every_group_size_gives_up(fresh, engine, oracle, n):
    """200 instances, more cells than SMs: each class of cells has groups of its own size."""
    k = 200
    x, y, z = oracle.gen_uniform(n, k * n)
    inst = [{"offset": i * n, "n": n, "d": 16} for i in range(k)]
    fresh.test_set_scan_wait(64, 0)
    fresh.test_drop_copies(True)
    times_out(engine, lambda: fresh.build_batch(x.copy(), y.copy(), z.copy(), inst))
    fresh.test_drop_copies(False)
    fresh.test_set_scan_wait(0, 0)
    gx, gy, gz = x.copy(), y.copy(), z.copy()
    parts, perm, _ = fresh.build_batch(gx, gy, gz, inst)
    for i in (0, 77, k - 1):
        s = slice(i * n, (i + 1) * n)
        ref = oracle.build_tree(x[s], y[s], z[s], 16)
        assert parts[i][0].tobytes() == ref.heap.tobytes() and np.array_equal(parts[i][1], ref.ranges[0])
        assert np.array_equal(perm[s], ref.perm)
