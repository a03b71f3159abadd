"""Boxes with an end past 2^127, whose midpoints overflow: the cut is then infinite, outside its
bracket, and the reference's count is over all the cell's keys, those outside the box too. Keys
beyond either end of the box, infinite and NaN ones among them, on every bisection path (level
kernels, one CTA a cell, subtrees, weighted passes). Bit for bit against the oracle."""
import numpy as np
import pytest

from test_gpu_parity import run_both

pytestmark = pytest.mark.gpu

BOXES = {
    "high": (1.5e38, 3.2e38),  # the first midpoint is +inf
    "low": (-3.2e38, -1.5e38),  # ... -inf
    "wide": (-3.2e38, 3.2e38),
    "half": (-1.0, 3.3e38),
}


def keys(n, seed):
    """Keys over the whole range of floats, half of them at 1.5e38 to 3.4e38 on either side."""
    rng = np.random.default_rng(seed)
    u = (rng.random((3, n)) * 2 - 1) * 3.4e38
    near = rng.random((3, n)) < 0.5
    u[near] = (np.sign(u) * (1.5e38 + rng.random((3, n)) * 1.9e38))[near]
    u = u.astype(np.float32)
    pick = rng.random((3, n))
    u[pick < 0.02] = np.inf
    u[(pick >= 0.02) & (pick < 0.03)] = -np.inf
    u[(pick >= 0.03) & (pick < 0.04)] = np.nan
    return tuple(np.ascontiguousarray(a) for a in u)


@pytest.fixture
def fresh(engine):
    c = engine.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("tune", [dict(subtree_levels=0), dict(subtree_levels=0, cta_min_cells=1), dict(subtree_levels=6)],
                         ids=["levels", "cta", "subtree"])
@pytest.mark.parametrize("n", [3, 900, 3001, 70_001, 300_001])
@pytest.mark.parametrize("box", BOXES)
def test_keys_outside_a_box_past_2_127(fresh, oracle, box, n, tune):
    lo, hi = BOXES[box]
    fresh.set_tuning(**tune)
    run_both(fresh, oracle, *keys(n, n), 16, lower=(lo,) * 3, upper=(hi,) * 3)


@pytest.mark.parametrize("n", [3, 900, 3001, 16_000, 70_001, 300_001])
@pytest.mark.parametrize("box", BOXES)
def test_weighted_keys_outside_a_box_past_2_127(fresh, oracle, box, n):
    lo, hi = BOXES[box]
    x, y, z = keys(n, n + 1)
    w = np.random.default_rng(n).integers(0, 1 << 20, n).astype(np.uint32)
    kw = dict(lower=(lo,) * 3, upper=(hi,) * 3)
    ref, wref = oracle.build_tree_weighted(x, y, z, w, 16, **kw)
    g = [a.copy() for a in (x, y, z, w)]
    res = fresh.build_weighted(*g, 16, **kw)
    assert res.heap.tobytes() == ref.heap.tobytes() and np.array_equal(res.ranges, ref.ranges[0])
    assert np.array_equal(res.perm, ref.perm) and np.array_equal(g[3], wref)
    for a, b in zip(g, (ref.x, ref.y, ref.z)):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))


def test_instances_outside_a_box_past_2_127(fresh, oracle):
    """One wide box in a batch, and sampled first passes (cells of at least 2^18 particles)."""
    fresh.set_tuning(subtree_levels=0, predict_sigmas=4)
    boxes = [(-0.5, 0.5), BOXES["high"], BOXES["half"]]
    parts = [keys(600_000, i) if i else oracle.gen_uniform(5, 600_000) for i in range(3)]
    inst = [{"offset": i * 600_000, "n": 600_000, "d": 16, "lower": (b[0],) * 3, "upper": (b[1],) * 3}
            for i, b in enumerate(boxes)]
    trees, perm, _ = fresh.build_batch(*(np.concatenate([p[a] for p in parts]) for a in range(3)), inst)
    for (heap, ranges), ins, p in zip(trees, inst, parts):
        ref = oracle.build_tree(*p, 16, lower=ins["lower"], upper=ins["upper"])
        assert heap.tobytes() == ref.heap.tobytes() and np.array_equal(ranges, ref.ranges[0])
        assert np.array_equal(perm[ins["offset"]:ins["offset"] + ins["n"]], ref.perm)
