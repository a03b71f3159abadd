"""Warm builds: which levels start from hints is decided where the cells are expected to fit the
former subtree kernel (34816 particles), by the largest cell found there, also for sizes that
today's subtree kernel does not take at that level (33024)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
f32 = np.float32


@pytest.fixture
def fresh(engine):
    c = engine.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("lump", [0, 60_000])
def test_a_cell_above_the_line_keeps_every_hint(fresh, lump):
    """512 cells of about 34000 at the line. With 60000 particles on one point a cell is larger, and
    every level starts from its hints, as in a context without subtree levels; without them the
    levels below the line start from their extents."""
    n, d = 34_000 * 512, 1 << 13
    rng = np.random.default_rng(4)
    x, y, z = (rng.random(n, dtype=f32) - f32(0.5) for _ in range(3))
    for a in (x, y, z):
        a[:lump] = 0.123
    prev = fresh.build(x.copy(), y.copy(), z.copy(), d, perm=None).heap
    for a in (x, y, z):
        a[lump:] = np.clip(a[lump:] + f32(1e-3) * rng.standard_normal(n - lump, dtype=f32), f32(-0.5), np.nextafter(f32(0.5), f32(0)))
    trees = {}
    for name, tune in (("default", {}), ("hinted", dict(subtree_levels=0))):
        if tune:
            fresh.set_tuning(**tune)
        r = fresh.build_warm(x.copy(), y.copy(), z.copy(), d, prev, 8.0, perm=None)
        trees[name] = (r.heap.tobytes(), r.ranges.tobytes(), r.info["warm_cells"])
    if lump:
        assert trees["default"] == trees["hinted"]
    else:
        assert trees["default"][2] < trees["hinted"][2] // 8
