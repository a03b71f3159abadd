"""The weighted pass where its ways of bisecting a cell change: cells one CTA holds in registers
(up to 4096 keys), in shared bins (one tile), in several tiles and in pieces dealt to several
CTAs, weights on both sides of what their 16-bit halves and 32-bit sums take, and totals on both
sides of 2^32 (the 64-bit and the 128-bit form of the test). Bit for bit against the oracle."""
import numpy as np
import pytest

from test_gpu_levels import keys
from test_gpu_weighted import check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("wmax", [1, 65535, 65537, (1 << 29) + 5, (1 << 32) - 1])
@pytest.mark.parametrize("n,d", [(2047, 4), (2049, 4), (16385, 3), (70001, 32), (300001, 1 << 9), (1 << 20, 1 << 8)])
def test_weighted_pass_matches_oracle(ctx, oracle, n, d, wmax):
    rng = np.random.default_rng(n + wmax)
    w = rng.integers(0, wmax + 1, n, dtype=np.uint64).astype(np.uint32)
    w[rng.random(n) < 0.1] = 0
    for kind in ("uniform", "ends"):
        check(ctx, oracle, *keys(kind, n, n), w, d)


def test_weighted_many_small_cells(ctx, oracle):
    n = 1 << 20
    x, y, z = oracle.gen_plummer(5, n)
    w = np.random.default_rng(3).integers(1, 100, n).astype(np.uint32)
    check(ctx, oracle, x, y, z, w, 1 << 13)


@pytest.mark.parametrize("n", [256 * 2048 + 99, 256 * 4096 - 99, 256 * 4096 + 99])
def test_cells_a_cta_holds_match_oracle(ctx, oracle, n):
    """256 cells about the most keys a CTA holds at 8 and at 16 a thread."""
    rng = np.random.default_rng(n)
    w = rng.integers(0, 1 << 17, n, dtype=np.uint64).astype(np.uint32)
    for kind in ("uniform", "ends", "narrow"):
        check(ctx, oracle, *keys(kind, n, n), w, 1 << 9)
