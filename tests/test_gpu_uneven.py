"""Trees whose cells are uneven, so that the subtree kernel refuses the level it was planned for:
it is tried again further down, where the largest cell fits, and the levels between go to the level
kernels. Bit for bit against the oracle, alone and batched, from device and host arrays; and the
kernel does take the tree that it took when it was planned four levels above the leaves."""
import numpy as np
import pytest

from test_gpu_parity import assert_same, run_both

pytestmark = pytest.mark.gpu


@pytest.fixture
def fresh(engine):
    c = engine.Context(0)
    yield c
    c.close()


def sites(n, k, seed, lump=0.0):
    """Particles on k points, `lump` of them on the first one."""
    rng = np.random.default_rng(seed)
    p = (rng.random((3, k), dtype=np.float32) - np.float32(0.5))
    i = rng.integers(0, k, n)
    i[rng.random(n) < lump] = 0
    return tuple(np.ascontiguousarray(p[a][i]) for a in range(3))


def subtree_launches(ctx, x, y, z, d):
    """Launches of the subtree kernel and of the levels' classify pass in one build."""
    torch = pytest.importorskip("torch")
    dev = [torch.from_numpy(a.copy()).cuda() for a in (x, y, z)]
    torch.cuda.synchronize()
    ctx.profile_reset()
    ctx.build(*dev, d, perm=None, device_pointers=True)
    p = ctx.profile()
    return p["subtree"]["launches"], p["part_classify"]["launches"]


@pytest.mark.parametrize("n,k,lump,d", [(1 << 21, 130, 0.0, 1 << 13), (1 << 21, 1000, 0.02, 1 << 13), (700_001, 300, 0.2, 1 << 10),
                                        (1 << 20, 3, 0.0, 1 << 10), (500_003, 64, 0.0, 192)])
def test_uneven_trees_match_oracle(fresh, oracle, n, k, lump, d):
    x, y, z = sites(n, k, n + k, lump)
    run_both(fresh, oracle, x, y, z, d)  # from the host (windows planned, then refused)
    torch = pytest.importorskip("torch")
    ref = oracle.build_tree(x, y, z, d)
    for _ in range(2):  # captured, replayed
        dev = [torch.from_numpy(a.copy()).cuda() for a in (x, y, z)]
        perm = torch.empty(n, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        res = fresh.build(*dev, d, perm=perm, device_pointers=True)
        res.perm = perm.cpu().numpy().view(np.uint32)
        assert_same(res, ref, *(a.cpu().numpy() for a in dev))


def test_batch_with_one_uneven_instance_matches_oracle(fresh, oracle):
    parts = [oracle.gen_uniform(1, 200_000), sites(300_000, 12, 2), oracle.gen_plummer(3, 100_000)]
    inst, off = [], 0
    for p in parts:
        inst.append({"offset": off, "n": p[0].size, "d": 256})
        off += p[0].size
    b = [np.concatenate([p[a] for p in parts]) for a in range(3)]
    trees, perm, _ = fresh.build_batch(*b, inst)
    for (heap, ranges), ins, p in zip(trees, inst, parts):
        ref = oracle.build_tree(*p, ins["d"])
        assert heap.tobytes() == ref.heap.tobytes() and np.array_equal(ranges, ref.ranges[0])
        assert np.array_equal(perm[ins["offset"]:ins["offset"] + ins["n"]], ref.perm)


def test_the_subtree_kernel_is_tried_again(fresh):
    """2^21 particles on 130 points: cells of about 32768 six levels above the leaves hold up to a
    few of the points, more than a CTA takes; two levels down they fit."""
    x, y, z = sites(1 << 21, 130, (1 << 21) + 130)
    launches, levels = subtree_launches(fresh, x, y, z, 1 << 12)
    assert launches >= 2 and levels < 12


@pytest.mark.parametrize("n,d", [(57_700, 7), (57_900, 7), (66_000, 7), (120_000, 13), (130_000, 9), (33_024 * 2 - 40, 3), (1 << 20, 65), (264_000, 33)])
def test_odd_leaf_counts_are_not_refused(fresh, oracle, n, d):
    """The larger children of odd leaf counts have more than half of the particles (4/7, 7/13, ...):
    the level planned for the subtree kernel is one whose largest cell fits, so spread particles are
    never refused (one check, one subtree launch, and no second graph)."""
    x, y, z = oracle.gen_uniform(d, n)
    run_both(fresh, oracle, x, y, z, d)
    fresh.profile_reset()
    gx, gy, gz = x.copy(), y.copy(), z.copy()
    fresh.build(gx, gy, gz, d)
    p = fresh.profile()
    assert "plan" not in p  # launched by a second graph alone
    assert p.get("subtree", {"launches": 0})["launches"] <= 1


def test_a_refused_tree_is_copied_once(fresh):
    """A tree of more than 1 MiB whose subtree level is refused: its cells are copied to the host when
    the tree is done, not before as well (with 10 of 20 levels built, the copy was half of the
    build's time)."""
    torch = pytest.importorskip("torch")
    n, d = 1 << 22, 1_407_823
    src = [torch.from_numpy(a).cuda() for a in sites(n, 400, 5)]

    def ms(most):
        fresh.set_tuning(subtree_levels=most)
        times = []
        for _ in range(6):
            dev = [s.clone() for s in src]
            torch.cuda.synchronize()
            times.append(fresh.build(*dev, d, levels=9, perm=None, device_pointers=True).info["device_ms"])
        return min(times[2:])

    refused, without = ms(6), ms(0)
    assert refused < without + 0.4
