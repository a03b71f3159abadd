"""Cells whose cut comes out as their bracket's upper end, or whose bracket narrows towards the box's
end (keys on and beyond it): few different values in many keys. Such cells' masks are corrected by
all warps of a CTA, or their loop ended without further counts; bit for bit against the oracle, and
not many times slower than spread keys."""
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


def grid(n, values, seed):
    """Coordinates of `values` different values, spread over the box."""
    rng = np.random.default_rng(seed)
    return tuple((np.floor(rng.random(n, dtype=np.float32) * values) / np.float32(values) - np.float32(0.5)) for _ in range(3))


@pytest.mark.parametrize("d", [4, 16, 512, 2048])
@pytest.mark.parametrize("n", [4096 * 31 + 1, 655_360, 655_361, 1 << 20, (1 << 21) + 77])
@pytest.mark.parametrize("kind", ["narrow", "grid3", "grid300", "grid40000"])
def test_few_values_match_oracle(fresh, oracle, kind, n, d):
    x, y, z = grid(n, int(kind[4:]), n) if kind.startswith("grid") else keys(kind, n, n)
    fresh.set_tuning(subtree_levels=0, sparse_keys_per_tile=1000)
    run_both(fresh, oracle, x, y, z, d)


@pytest.mark.parametrize("box", [((0, 0, 0), (0, 0, 0)), ((0.25, -0.5, 0.1), (0.25, 0.0, 0.1)), ((-0.5, -0.5, -0.5), (-0.4, -0.4, -0.4))])
def test_keys_beyond_the_box_match_oracle(fresh, oracle, box):
    for n, d in ((70_001, 16), (700_001, 512)):
        run_both(fresh, oracle, *keys("uniform", n, n), d, lower=box[0], upper=box[1])


def test_a_box_without_extent_is_not_slow(fresh, oracle):
    """Nearly every cut is the box's end: each level read its cells again with one warp a cell
    (30 times the time of spread keys)."""
    torch = pytest.importorskip("torch")
    n, d = 1 << 20, 1 << 10
    src = [torch.from_numpy(a).cuda() for a in oracle.gen_uniform(9, n)]

    def ms(**box):
        times = []
        for _ in range(4):
            dev = [s.clone() for s in src]
            torch.cuda.synchronize()
            times.append(fresh.build(*dev, d, perm=None, device_pointers=True, **box).info["device_ms"])
        return min(times[1:])

    assert ms(lower=(0, 0, 0), upper=(0, 0, 0)) < 10 * ms()


@pytest.mark.parametrize("value", [0.123, 0.0, -0.5, 0.49999997])
@pytest.mark.parametrize("n", [900, 5000, 15_000, 32_768])
def test_equal_keys_in_a_subtree_match_oracle(fresh, oracle, n, value):
    """Every cut is counted over all the keys, until the bracket is two neighbouring floats."""
    x, y, z = (np.full(n, value, np.float32) for _ in range(3))
    run_both(fresh, oracle, x, y, z, 64)
    z = np.where(np.arange(n) % 3 == 0, np.nextafter(np.float32(value), np.float32(1)), z).astype(np.float32)
    run_both(fresh, oracle, x, z, y, 64)
    run_both(fresh, oracle, x, y, z, 64, lower=(-1.0, -2.0, -3.0), upper=(1.0, 2.0, 3.0))
