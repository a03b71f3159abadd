"""The subtree kernel at the cell sizes where its groups of warps change (1088, 6656 and 33024
particles; the fourth edge, 16400, is in test_gpu_subtree_levels.py), one to six levels deep, on keys that its key windows settle and on keys that
they do not (a few neighbouring floats, many keys on the box ends and on cuts, NaN, a box far
wider than its keys). Alone and with every size in one batch. Bit for bit against the oracle."""
import numpy as np
import pytest

from test_gpu_levels import keys
from test_gpu_parity import assert_same, run_both

pytestmark = pytest.mark.gpu

SIZES = [33, 255, 257, 1088, 1089, 6656, 6657, 14848, 14849, 33023, 33024]


def build_on_device(ctx, oracle, x, y, z, d, levels=0):
    torch = pytest.importorskip("torch")
    ref = oracle.build_tree(x, y, z, d, levels=levels or None)
    dev = [torch.from_numpy(a.copy()).cuda() for a in (x, y, z)]
    perm = torch.empty(x.size, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    res = ctx.build(*dev, d, levels=levels, perm=perm, device_pointers=True)
    res.perm = perm.cpu().numpy().view(np.uint32)
    assert_same(res, ref, *(a.cpu().numpy() for a in dev))


@pytest.mark.parametrize("kind", ["uniform", "narrow", "ends"])
@pytest.mark.parametrize("n", SIZES)
def test_one_cell_trees_match_oracle(ctx, oracle, kind, n):
    x, y, z = keys(kind, n, n + 1)
    for d in (2, 16, 64, 5, 50, 100):
        build_on_device(ctx, oracle, x, y, z, d)


@pytest.mark.parametrize("d,levels", [(3, 0), (7, 0), (11, 0), (100, 3), (1000, 0), (1 << 10, 7), (96, 0)])
def test_leaf_counts_and_level_bounds_match_oracle(ctx, oracle, d, levels):
    """Leaf counts that are not powers of two (odd ratios in the test, partial slices that keep
    the level kernels) and trees not built to their leaves."""
    for n in (100, 30001, 200003):
        x, y, z = oracle.gen_plummer(d + n, n)
        build_on_device(ctx, oracle, x, y, z, d, levels)


@pytest.mark.parametrize("cell", [300, 1087, 6650, 14840])
def test_many_cells_match_oracle(ctx, oracle, cell):
    """Levels of 512 cells of about `cell` particles above the subtree levels (3 of them)."""
    x, y, z = keys("uniform", 512 * cell + 77, cell)
    saved = ctx.get_tuning()
    try:
        ctx.set_tuning(subtree_levels=3)
        run_both(ctx, oracle, x, y, z, 1 << 12)
    finally:
        ctx.set_tuning(**saved)


def test_wide_box_matches_oracle(ctx, oracle):
    x, y, z = keys("uniform", 20000, 5)
    run_both(ctx, oracle, x, y, z, 32, lower=(-1e30, -1e30, -1e30), upper=(1e30, 1e30, 1e30))
    run_both(ctx, oracle, x, y, z, 32, lower=(-3.0, -0.4, -0.5), upper=(0.1, 5.0, 0.5))


@pytest.mark.parametrize("kind", ["uniform", "plummer", "narrow", "ends"])
def test_batch_of_every_class_matches_oracle(ctx, oracle, kind):
    sizes = [n + i % 3 - 1 for i, n in enumerate(SIZES[:-1] * 16)]
    parts = [oracle.gen_plummer(i, n) if kind == "plummer" else keys(kind, n, i) for i, n in enumerate(sizes)]
    inst, off = [], 0
    for i, n in enumerate(sizes):
        inst.append({"offset": off, "n": n, "d": 1 << (1 + i % 6)})
        off += n
    b = [np.concatenate([p[a] for p in parts]) for a in range(3)]
    trees, perm, _ = ctx.build_batch(*b, inst)
    for (heap, ranges), ins, (x, y, z) in zip(trees, inst, parts):
        ref = oracle.build_tree(x, y, z, ins["d"])
        o, e = ins["offset"], ins["offset"] + ins["n"]
        assert heap.tobytes() == ref.heap.tobytes() and np.array_equal(ranges, ref.ranges[0])
        assert np.array_equal(perm[o:e], ref.perm)
        for got, want in zip(b, (ref.x, ref.y, ref.z)):
            assert np.array_equal(got[o:e].view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("kind", ["uniform", "plummer", "narrow", "ends"])
def test_two_cells_of_an_sm_match_oracle(ctx, oracle, kind):
    """256 cells of about 16396 particles, on both sides of the most two cells of an SM can have,
    six levels each (their descendants of 512 end in one warp's registers, those of 1025 do not)."""
    n = 256 * 16396
    x, y, z = oracle.gen_plummer(3, n) if kind == "plummer" else keys(kind, n, 3)
    run_both(ctx, oracle, x, y, z, 256 * 64)
