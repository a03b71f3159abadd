"""The work this framework is measured on: ORB builds and services through their public
entry points, from a few thousand particles to 2^27.

A case names an entry point (`call`) and its sizes and options; prepare() makes its inputs
and the context a program keeps, run() is one pass. A build partitions its particle arrays
in place, so a pass starts as a simulation's step does: the particles are copied into the
arrays the build may reorder, then the build is called.

Every output is a whole number or moved bytes: the cell heap (bytes of the 52-byte cells),
the ranges, counts and permutation, and the reordered coordinates and weights, which are
the inputs' own bit patterns. They are the same bit for bit under any correct
implementation, so coordinates are returned as their bits and there is nothing to compute
again in 64 bits: exact() has no value for any of them.
"""
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "gpu-load-balance_gb300"))
import orb_gb300 as orb  # noqa: E402


def _build(name, kind, n, d, perm=True, levels=0):
    return {"name": name, "call": "build", "kind": kind, "n": n, "d": d, "perm": perm, "levels": levels}


def listed():
    return [
        # the smallest instance of the batched and served workloads: latency
        _build("build_2e14_d64", "uniform", 1 << 14, 1 << 6),
        # an odd size and a leaf count that is not a power of two (ranks of a job of 100 processes)
        _build("build_100003_d100", "uniform", 100003, 100),
        # the reference's own quick run, `orbit 20 10 0`; no permutation asked for
        _build("build_2e20_d1024", "uniform", 1 << 20, 1 << 10, perm=False),
        # the largest instance of the served workload, clustered as cosmological particles are
        _build("build_plummer_4100001_d4096", "plummer", 4100001, 1 << 12),
        # clustered production run, fine leaves
        _build("build_plummer_2e26_d2e18", "plummer", 1 << 26, 1 << 18),
        # the headline workload: 2^27 particles into 2^16 leaves, coordinates only
        _build("build_2e27_d2e16", "uniform", 1 << 27, 1 << 16, perm=False),
        # 128 uneven instances in one call, half of them clustered
        {"name": "batch_128", "call": "batch", "k": 128, "lo": 14.0, "hi": 22.0, "dlo": 6, "dhi": 12,
         "sizes": 1},
        # per-particle work weights (individual time steps), clustered
        {"name": "weighted_16000003_d16384", "call": "weighted", "kind": "plummer", "n": 16000003,
         "d": 1 << 14, "wmax": 64},
        # rebuild after a small displacement, from the previous tree
        {"name": "warm_2e24_d8192", "call": "warm", "kind": "uniform", "n": 1 << 24, "d": 1 << 13,
         "sigma": 1e-3, "width": 8.0},
        # particles in (pinned) host memory, in and out, as the reference's driver holds them
        {"name": "host_2e24_d8192", "call": "host", "kind": "uniform", "n": 1 << 24, "d": 1 << 13},
        # the per-rank services under a driver of the caller's own: load, then count-left and
        # partition level by level, then the particles back
        {"name": "services_2e22_l6", "call": "services", "kind": "uniform", "n": 1 << 22, "levels": 6},
        # count-left of a level's cells that allocates nothing, on the caller's stream
        {"name": "count_left_static_2e24_1024", "call": "static", "kind": "plummer", "n": 1 << 24,
         "cells": 1 << 10},
    ]


def draw(rng):
    call = rng.choice(["build", "build", "build", "batch", "weighted", "warm", "host", "services", "static"])
    kind = rng.choice(["uniform", "plummer"])

    def size(lo, hi):
        return int(2.0 ** rng.uniform(lo, hi)) | 1

    def leaves(n, power=False):  # 2^7 .. 2^12 particles a leaf, at least two leaves
        d = max(2, int(n / 2.0 ** rng.uniform(7, 12)))
        return d if not power and rng.random() < 0.3 else 1 << (d.bit_length() - 1)

    if call == "build":
        n = size(12, 26.5)
        d = leaves(n)
        return {"call": call, "kind": kind, "n": n, "d": d, "perm": rng.random() < 0.5, "levels": 0}
    if call == "batch":
        lo = rng.uniform(10, 17)
        return {"call": call, "k": int(2.0 ** rng.uniform(1, 7)), "lo": lo, "hi": lo + rng.uniform(1, 5),
                "dlo": 3, "dhi": rng.choice([6, 8, 10]), "sizes": rng.randint(0, 1 << 30)}
    if call == "weighted":
        n = size(14, 24)
        return {"call": call, "kind": kind, "n": n, "d": leaves(n), "wmax": rng.choice([2, 64, 100000])}
    if call == "warm":
        n = size(14, 25)
        return {"call": call, "kind": kind, "n": n, "d": leaves(n, power=True),
                "sigma": rng.choice([1e-4, 1e-3, 1e-2]), "width": rng.choice([4.0, 8.0, 16.0])}
    if call == "host":
        n = size(14, 24)
        return {"call": call, "kind": kind, "n": n, "d": leaves(n)}
    if call == "services":
        return {"call": call, "kind": kind, "n": size(14, 22), "levels": rng.randint(2, 7)}
    return {"call": call, "kind": kind, "n": size(12, 25), "cells": 1 << rng.randint(0, 12)}


# Inputs -----------------------------------------------------------------------------------

def _particles(kind, n, gen):
    """Three coordinates in [-0.5, 0.5): uniform on the 2^-24 grid, or 90% in 64 Plummer
    spheres (scale radii log-uniform in [0.005, 0.05)) on a uniform background."""
    dev = "cuda"
    box = [torch.rand(n, generator=gen, device=dev) - 0.5 for _ in range(3)]
    if kind == "uniform":
        return box
    centre = torch.rand(64, 3, generator=gen, device=dev) - 0.5
    scale = 0.005 * 10.0 ** torch.rand(64, generator=gen, device=dev)
    which = torch.randint(0, 64, (n,), generator=gen, device=dev)
    w = torch.rand(n, generator=gen, device=dev).pow_(1.0 / 3.0).clamp_(max=1.0 - 2.0 ** -20)
    r = w / torch.sqrt(1.0 - w * w) * scale[which]
    del w
    v = [torch.randn(n, generator=gen, device=dev) for _ in range(3)]
    r /= torch.sqrt(v[0] ** 2 + v[1] ** 2 + v[2] ** 2).clamp_(min=1e-20)
    field = torch.rand(n, generator=gen, device=dev) < 0.1
    top = float(np.nextafter(np.float32(0.5), np.float32(-1)))
    for a in range(3):
        v[a].mul_(r).add_(centre[which, a]).clamp_(-0.5, top)
        torch.where(field, box[a], v[a], out=box[a])
    return box


def _pinned(count, dtype):
    """A page-locked host array of `count` elements (a program's own result buffers)."""
    dtype = np.dtype(dtype)
    t = torch.zeros(count * dtype.itemsize, dtype=torch.uint8, pin_memory=True)
    return t.numpy().view(dtype)


def _sizes(case):
    """The batch's uneven instances: particles log-uniform, leaves 2^k, packed back to back."""
    rng = random.Random(case["sizes"])
    inst, off = [], 0
    for _ in range(case["k"]):
        n = int(2.0 ** rng.uniform(case["lo"], case["hi"]))
        d = 1 << max(1, min(rng.randint(case["dlo"], case["dhi"]), int(math.log2(n)) - 2))
        inst.append({"offset": off, "n": n, "d": d})
        off += n
    return inst, off


def _level_cells(heap, level):
    """The cells of one level of a finished tree, their cuts as the bisection left them."""
    return np.ascontiguousarray(heap[(1 << level) - 1:(2 << level) - 1])


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    call = case["call"]
    st = {"case": case}
    if call == "batch":
        st["inst"], _ = _sizes(case)
        parts = [_particles("uniform" if i % 2 == 0 else "plummer", ins["n"], gen)
                 for i, ins in enumerate(st["inst"])]  # every second one clustered
        src = [torch.cat([p[a] for p in parts]) for a in range(3)]
        del parts
    else:
        src = _particles(case["kind"], case["n"], gen)
    n = src[0].numel()
    st["src"] = src
    if call != "static":
        st["ctx"] = orb.Context(0)
    if call in ("build", "batch", "weighted", "warm"):
        st["work"] = [torch.empty_like(s) for s in src]
    if call in ("batch", "weighted", "warm") or case.get("perm"):
        st["perm"] = torch.empty(n, dtype=torch.int32, device="cuda")
    if call in ("build", "host"):
        cells = 2 * case["d"] - 1
        st["heap"] = _pinned(cells, orb.CELL_DTYPE)
        st["ranges"] = _pinned(2 * cells, np.uint32).reshape(cells, 2)
    if call == "weighted":
        st["wsrc"] = torch.randint(1, case["wmax"] + 1, (n,), generator=gen, device="cuda", dtype=torch.int32)
        st["w"] = torch.empty_like(st["wsrc"])
    if call == "host":
        st["hsrc"] = [s.cpu() for s in src]
        st["hwork"] = [torch.empty(n, pin_memory=True) for _ in range(3)]
        st["hperm"] = _pinned(n, np.uint32)
        del st["src"]
    if call in ("warm", "services", "static"):
        # the tree of the step before (warm), or the cells the services are called with
        d = {"warm": case.get("d"), "services": 2 << case.get("levels", 0), "static": 2 * case.get("cells", 0)}[call]
        arr = [s.clone() for s in src]
        torch.cuda.synchronize()
        with orb.Context(0) as c:
            tree = c.build(*arr, d, perm=None, device_pointers=True)
        if call == "warm":
            st["prev"] = tree.heap
            top = float(np.nextafter(np.float32(0.5), np.float32(-1)))
            for s in src:
                s.add_(torch.randn(n, generator=gen, device="cuda"), alpha=case["sigma"]).clamp_(-0.5, top)
        elif call == "services":
            st["cells"] = [_level_cells(tree.heap, l) for l in range(case["levels"])]
            for c in st["cells"]:
                c["foundCut"] = 0
        else:
            cells = _level_cells(tree.heap, int(math.log2(case["cells"])))
            cells["foundCut"] = 0  # a bisection under way: first cuts, some cells found
            cells["foundCut"][1::4] = 1
            axis = np.maximum(cells["cutAxis"], 0)
            pick = np.arange(len(cells))
            cells["cutMarginLeft"] = cells["lower"][pick, axis]
            cells["cutMarginRight"] = cells["upper"][pick, axis]
            st["src"] = arr
            st["cells"] = torch.from_numpy(cells.view(np.uint8).copy()).cuda()
            st["map"] = torch.from_numpy(tree.ranges.reshape(-1).view(np.int32).copy()).cuda()
            st["out"] = torch.zeros(case["cells"], dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    return st


# One pass ---------------------------------------------------------------------------------

def _restore(st):
    for w, s in zip(st["work"], st["src"]):
        w.copy_(s)
    if "w" in st:
        st["w"].copy_(st["wsrc"])
    torch.cuda.current_stream().synchronize()  # the context runs on its own stream


def _bits(ts):
    return [t.view(torch.int32) for t in ts]


def _tree(heap, ranges):
    return {"heap": heap.view(np.uint8), "ranges": ranges.view(np.int32)}


def run(st):
    case = st["case"]
    call = case["call"]
    if call == "static":
        n, k = case["n"], case["cells"]
        orb.count_left_static(*st["src"], n, st["cells"], k, st["map"], st["map"].numel() // 2, st["out"],
                              torch.cuda.current_stream().cuda_stream)
        return st["out"]
    ctx = st["ctx"]
    if call == "services":
        torch.cuda.current_stream().synchronize()
        ids = 2 << case["levels"]
        ctx.load_particles(*st["src"], ids, device_pointers=True)
        counts = []
        for cells in st["cells"]:
            counts.append(ctx.count(cells))
            counts.append(ctx.count_left(cells))
            ctx.partition(cells)
        out = [*counts, ctx.get_ranges(ids - 1), *ctx.store_particles()]
        return [a.view(np.int32) for a in out]
    if call == "host":
        for w, s in zip(st["hwork"], st["hsrc"]):
            w.copy_(s)
        ctx.build(*(w.numpy() for w in st["hwork"]), case["d"], perm=st["hperm"], heap_out=st["heap"],
                  ranges_out=st["ranges"])
        return [_bits(st["hwork"]), st["hperm"].view(np.int32), _tree(st["heap"], st["ranges"])]
    _restore(st)
    out = [_bits(st["work"])]
    if call == "build":
        ctx.build(*st["work"], case["d"], levels=case["levels"], perm=st.get("perm"), device_pointers=True,
                  heap_out=st["heap"], ranges_out=st["ranges"])
        out.append(_tree(st["heap"], st["ranges"]))
    elif call == "batch":
        parts, _, _ = ctx.build_batch(*st["work"], st["inst"], perm=st["perm"], device_pointers=True)
        out.append(_tree(parts[0][0].base, parts[0][1].base))  # the instances' trees back to back
    elif call == "weighted":
        res = ctx.build_weighted(*st["work"], st["w"], case["d"], perm=st["perm"], device_pointers=True)
        out += [st["w"], _tree(res.heap, res.ranges)]
    else:
        res = ctx.build_warm(*st["work"], case["d"], st["prev"], case["width"], perm=st["perm"],
                             device_pointers=True)
        out.append(_tree(res.heap, res.ranges))
    if "perm" in st:
        out.append(st["perm"])
    return out


def work(case):
    """Bytes: the particles (and weights) read once and written once, the permutation, heap
    and ranges written. Flops: one comparison of a particle's key per level."""
    call = case["call"]
    if call == "static":
        # a quarter of the cells (one at least of four) is found and not counted
        n, k = case["n"], case["cells"]
        live = k - len(range(1, k, 4))
        return {"bytes": 4 * n * live // k + 64 * k, "flops": n * live // k}
    if call == "batch":
        inst, n = _sizes(case)
        return {"bytes": 28 * n + sum(60 * (2 * i["d"] - 1) for i in inst),
                "flops": sum(i["n"] * (i["d"].bit_length() - 1) for i in inst)}
    n = case["n"]
    if call == "services":
        return {"bytes": 28 * n + 8 * (2 << case["levels"]), "flops": 2 * n * case["levels"]}
    d = case["d"]
    per = 24 + (4 if call != "build" or case["perm"] else 0) + (8 if call == "weighted" else 0)
    return {"bytes": per * n + 60 * (2 * d - 1), "flops": n * max(1, d.bit_length() - 1)}


def exact(case, seed):
    return None
