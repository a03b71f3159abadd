"""Weighted levels where most cells have one tile and a few have many (particles on a few points).
Bit for bit against the oracle, and not slower by the number of small cells."""
import numpy as np
import pytest

from test_gpu_weighted import check

pytestmark = pytest.mark.gpu


def lump(n, share, points, seed):
    rng = np.random.default_rng(seed)
    a = [rng.random(n, dtype=np.float32) - np.float32(0.5) for _ in range(3)]
    p = rng.random((3, points), dtype=np.float32) - np.float32(0.5)
    p[:, 0] = 0.123  # (below the grid of the other keys: no cut comes to lie on it)
    at, on = rng.integers(0, points, n), rng.random(n) < share
    return [np.where(on, q[at], x).astype(np.float32) for x, q in zip(a, p)]


@pytest.mark.parametrize("share,points", [(0.5, 1), (0.9, 1), (0.3, 7), (1.0, 3)])
@pytest.mark.parametrize("n,d", [(300_001, 1 << 9), (1 << 20, 1 << 12), (700_001, 3000), (300_001, 1 << 13), (200_000, 1 << 16)])
def test_few_large_cells_match_oracle(ctx, oracle, n, d, share, points):
    x, y, z = lump(n, share, points, n + points)
    w = np.random.default_rng(n).integers(0, 1 << 18, n, dtype=np.uint64).astype(np.uint32)
    check(ctx, oracle, x, y, z, w, d)


def test_many_small_cells_beside_a_large_one_are_not_slow(engine):
    """6.4 million particles, half of them on one point, into 2^9 and into 2^14 leaves: five levels more,
    whose small cells held the large one's CTAs up (3.5 times the time)."""
    torch = pytest.importorskip("torch")
    n = 6_400_000
    src = [torch.from_numpy(a).cuda() for a in lump(n, 0.5, 1, 3)]
    w0 = torch.randint(1, 5000, (n,), device="cuda", dtype=torch.int32)
    with engine.Context(0) as c:
        def ms(d):
            times = []
            for _ in range(5):
                dev, w = [s.clone() for s in src], w0.clone()
                torch.cuda.synchronize()
                times.append(c.build_weighted(*dev, w, d, perm=None, device_pointers=True).info["device_ms"])
            return min(times[1:])

        fine, coarse = ms(1 << 14), ms(1 << 9)
        assert fine < 2.6 * coarse, (fine, coarse)


@pytest.mark.parametrize("n,d", [(256, 2), (257, 2), (512 * 256, 512), (512 * 256 + 900, 512), (60_000, 1 << 13), (60_000, 1 << 16)])
def test_cells_a_warp_holds_match_oracle(ctx, oracle, n, d):
    """Cells of at most 256 keys (every warp holds all of them) and of a few more, many equal keys,
    weights whose 16-bit halves fill."""
    for share, points, wmax in ((0.0, 1, 50), (0.8, 500, 1 << 32), (1.0, 37, 65_537)):
        x, y, z = lump(n, share, points, n)
        w = np.random.default_rng(n).integers(0, wmax, n, dtype=np.uint64).astype(np.uint32)
        check(ctx, oracle, x, y, z, w, d)
