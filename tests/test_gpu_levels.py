"""The level kernels at the sizes and keys where their steps change: partition and count tile
edges (4096 and 16384 positions), cells a warp or a CTA finishes, brackets a few floats wide
(whose cut can come out as the bracket's upper end), keys at the box ends, NaN, and lists of
bracket keys from almost none to every key. Bit for bit against the oracle."""
import numpy as np
import pytest

from test_gpu_parity import run_both

pytestmark = pytest.mark.gpu


@pytest.fixture()
def tuned(ctx):
    saved = ctx.get_tuning()
    yield ctx
    ctx.set_tuning(**saved)


def keys(kind, n, seed):
    rng = np.random.default_rng(seed)
    u = rng.random((3, n), dtype=np.float32) - np.float32(0.5)
    if kind == "narrow":  # a few neighbouring floats: every bracket ends a few ulps wide
        base = np.float32(0.25).view(np.int32)
        u = (base + rng.integers(0, 5, (3, n)).astype(np.int32)).view(np.float32)
    elif kind == "ends":  # many keys on the box ends and on the first cuts, some NaN
        pick = rng.integers(0, 6, (3, n))
        u[pick == 0] = -0.5
        u[pick == 1] = 0.5
        u[pick == 2] = 0.0
        u[(pick == 3) & (rng.random((3, n)) < 0.05)] = np.nan
    return tuple(np.ascontiguousarray(a) for a in u)


@pytest.mark.parametrize("kind", ["uniform", "narrow", "ends"])
@pytest.mark.parametrize("n", [1023, 4095, 4097, 16384, 16385, 65537, (1 << 18) + 1, (1 << 20) + 4097])
def test_level_kernels_match_oracle(tuned, oracle, kind, n):
    x, y, z = keys(kind, n, n)
    for sparse in (64, 1, 16384):
        tuned.set_tuning(sparse_keys_per_tile=sparse, subtree_levels=4 if sparse == 64 else 0)
        run_both(tuned, oracle, x, y, z, 16)
        run_both(tuned, oracle, x, y, z, 11)


def test_many_listed_keys_in_one_cell(tuned, oracle):
    """A root whose bracket holds tens of thousands of keys for the list (several CTAs on one
    cell) and one whose list a single warp takes."""
    tuned.set_tuning(sparse_keys_per_tile=16384)
    for n in ((1 << 22) + 3, 300001):
        x, y, z = keys("uniform", n, n)
        run_both(tuned, oracle, x, y, z, 8)


@pytest.mark.parametrize("n", [256 * 1024 - 7, 256 * 1024 + 300, 256 * 4096 + 5, 256 * 16384 + 300])
def test_many_cells_about_a_warp_and_a_tile(tuned, oracle, n):
    """256 cells of 1024 keys (the most a warp bisects) and of 16384 (a count tile), and a few
    more or less."""
    x, y, z = keys("narrow", n, n)
    tuned.set_tuning(subtree_levels=0)
    run_both(tuned, oracle, x, y, z, 512)


@pytest.mark.parametrize("n", [1_240_003, 1_250_001, 2_480_001, 2_500_003, 7_450_001])
def test_sizes_where_launch_shapes_change(tuned, oracle, n):
    """A swap tile's pairs go to 4, 2 or 1 CTAs, a count tile to 1024, 512 or 256 threads."""
    x, y, z = keys("ends", n, n)
    tuned.set_tuning(subtree_levels=0)
    run_both(tuned, oracle, x, y, z, 6)


@pytest.mark.parametrize("width", [2.0**-6, 2.0**-9, 2.0**-10, 2.0**-14])
@pytest.mark.parametrize("n", [70_001, 1 << 20])
def test_thin_box_far_from_the_origin(tuned, oracle, n, width):
    """Boxes whose bins are a few floats wide, with keys on their ends, outside them and NaN: a
    warp's keys binned by guess alone, by guess and edges (margins below half a bin), by search."""
    rng = np.random.default_rng(n)
    x, y, z = (np.float32(0.3) + np.float32(width) * (rng.random((3, n), dtype=np.float32) - np.float32(0.01))).astype(np.float32)
    hi = np.float32(0.3) + np.float32(width)
    pick = rng.integers(0, 12, (3, n))
    for a, p in zip((x, y, z), pick):
        a[p == 0] = np.float32(0.3)
        a[p == 1] = hi
        a[(p == 2) & (rng.random(n) < 0.01)] = np.nan
    tuned.set_tuning(subtree_levels=0)
    run_both(tuned, oracle, x, y, z, 8, lower=(np.float32(0.3),) * 3, upper=(hi,) * 3)


@pytest.mark.parametrize("subtree", [0, 4])
@pytest.mark.parametrize("n", [3001, 70_001, 300_001])
@pytest.mark.parametrize("box,spread", [(1.8e38, 1e38), (3.2e38, 3.2e38)])
def test_box_wider_than_the_largest_float(tuned, oracle, box, spread, n, subtree):
    """Extents whose difference overflows, and cells whose midpoints do: no guess of a bin holds,
    and a cut can leave its bracket."""
    rng = np.random.default_rng(n)
    x, y, z = ((rng.random((3, n)) * 2 - 1) * spread).astype(np.float32)
    tuned.set_tuning(subtree_levels=subtree)
    run_both(tuned, oracle, x, y, z, 16, lower=(-box,) * 3, upper=(box,) * 3)
