"""Builds without particles, the coordinate arrays empty device tensors (null addresses): a tree
of empty cells, as from host arrays, and no wait of the subtree kernel runs out."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [1, 2, 64, 100, 1 << 10])
@pytest.mark.parametrize("call", ["build", "weighted", "batch"])
def test_no_particles_on_the_device(ctx, oracle, call, d):
    torch = pytest.importorskip("torch")
    x, y, z = (np.zeros(0, np.float32) for _ in range(3))
    ref = oracle.build_tree(x, y, z, d)
    dev = [torch.empty(0, device="cuda") for _ in range(3)]
    perm = torch.empty(1, dtype=torch.int32, device="cuda")
    if call == "batch":
        parts, _, _ = ctx.build_batch(*dev, [{"offset": 0, "n": 0, "d": d}] * 3, perm=perm, device_pointers=True)
    elif call == "weighted":
        w = torch.empty(0, dtype=torch.int32, device="cuda")
        r = ctx.build_weighted(*dev, w, d, perm=perm, device_pointers=True)
        parts = [(r.heap, r.ranges)]
    else:
        r = ctx.build(*dev, d, perm=perm, device_pointers=True)
        parts = [(r.heap, r.ranges)]
    for heap, ranges in parts:
        assert heap.tobytes() == ref.heap.tobytes()
        assert np.array_equal(ranges, ref.ranges[0])
