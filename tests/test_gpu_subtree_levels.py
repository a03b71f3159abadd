"""tune.subtree_levels bounds the levels one CTA per cell finishes, each value as it says, and a
context whose tuning was never set takes as many as fit (six). Trees bit for bit against the
oracle either way, at every cell size where the groups of warps change."""
import numpy as np
import pytest

from test_gpu_levels import keys
from test_gpu_parity import run_both

pytestmark = pytest.mark.gpu


@pytest.fixture
def fresh(engine):
    c = engine.Context(0)
    yield c
    c.close()


def level_passes(ctx, x, y, z, d):
    ctx.profile_reset()
    gx, gy, gz = x.copy(), y.copy(), z.copy()
    ctx.build_batch(gx, gy, gz, [{"offset": 0, "n": x.size, "d": d}])
    return ctx.profile().get("part_classify", {"launches": 0})["launches"]


def test_each_value_bounds_the_levels(fresh, oracle):
    x, y, z = oracle.gen_uniform(6, 30_000)
    assert level_passes(fresh, x, y, z, 64) == 0
    for most in (4, 5, 6, 3, 2, 1, 0):
        fresh.set_tuning(subtree_levels=most)
        assert level_passes(fresh, x, y, z, 64) == 6 - most
        run_both(fresh, oracle, x, y, z, 64)


def test_the_autotuner_tells_four_levels_from_six(fresh, oracle):
    x, y, z = oracle.gen_uniform(7, 30_000)
    best, _ = fresh.autotune_batch(x, y, z, [{"offset": 0, "n": x.size, "d": 64}], reps=3)
    assert best == fresh.get_tuning()
    assert level_passes(fresh, x, y, z, 64) == 6 - best["subtree_levels"]


@pytest.mark.parametrize("kind", ["uniform", "narrow", "ends"])
@pytest.mark.parametrize("n", [33, 257, 769, 1089, 6657, 16_400, 16_401, 33_024])
def test_six_levels_match_oracle(fresh, oracle, kind, n):
    x, y, z = keys(kind, n, n + 2)
    for d in (16, 64, 50):
        run_both(fresh, oracle, x, y, z, d)


@pytest.mark.parametrize("kind", ["uniform", "narrow", "ends"])
def test_class_edges_match_oracle(fresh, oracle, kind):
    """Instances of 16400 and 16401 particles (two cells of an SM or one), 1088/1089 and 6656/6657,
    and ones whose descendants have about 768 keys (one warp's registers), more of them than SMs."""
    sizes = [16_400, 16_401, 1088, 1089, 6656, 6657, 12_288 - 17, 12_288 + 40, 6144 + 9, 16_399] * 20
    parts = [keys(kind, n, i) for i, n in enumerate(sizes)]
    inst, off = [], 0
    for n in sizes:
        inst.append({"offset": off, "n": n, "d": 64})
        off += n
    b = [np.concatenate([p[a] for p in parts]) for a in range(3)]
    trees, perm, _ = fresh.build_batch(*b, inst)
    for i, ((heap, ranges), ins, p) in enumerate(zip(trees, inst, parts)):
        ref = oracle.build_tree(*p, 64)
        assert heap.tobytes() == ref.heap.tobytes() and np.array_equal(ranges, ref.ranges[0]), i
        assert np.array_equal(perm[ins["offset"]:ins["offset"] + ins["n"]], ref.perm), i
