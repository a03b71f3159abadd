// ORB engine kernels for sm_103a.
//
// Per level of the tree (all cells of the level in every launch):
//   hist       count-left: every key of an active cell is binned into a midpoint tree of
//              depth 11 over the cell's bracket [cutMarginLeft, cutMarginRight); keys below
//              the bracket are counted. The CTA that finishes a cell's last tile replays up
//              to 11 iterations of the reference's bisection (src/orbit.cpp:146-232) on the
//              histogram: the same cuts, the same integer counts, the same float32 test.
//   classify   masks of the keys >= cut and <= cut; a cell whose bracket holds few keys is
//              classified against the bracket, and the bracket's keys are listed
//   cells      the rest of the bisection on the cell's list, the listed keys' mask bits, and
//              the Hoare partition of src/services/partition.cpp:30-52 characterised: with
//              L_k the k-th key >= cut from the left and R_k the k-th key <= cut from the
//              right, Hoare swaps exactly (L_k, R_k) for k <= s where
//              s = max_x min(#{>= cut in [0,x)}, #{<= cut in [x,n)}), stops at
//              i = min(L_{s+1}, R_s) and swaps (i, n-1).
//   swap       the pairs; whoever finishes a cell's last tile does the final swap and the split
//              (src/cell.h:78-126, src/orbit.cpp:235-250) and plans the children for the
//              next level.
// Beside them: the bisection of small cells in one launch (a warp per cell), the subtree kernel
// (a group of warps finishes a cell's last levels in shared memory), the
// optional sampled first pass, the service count-left, seeded generators and the batched
// and served forms' helpers.
#include <type_traits>
#include <cuda_runtime.h>
#include <stdint.h>

#include "orb_internal.cuh"

namespace orb {

const char *const kKernelNames[kNumKernels] = {
    "init", "plan", "count_left_hist", "part_classify", "part_cells", "part_swap", "part_finish",
    "count_left",
    "generate", "bisect_cta", "bisect_tile", "subtree_check", "subtree", "count_left_sample",
    "count_left_sample_pick", "count_left_weighted", "stage_gather"};

namespace {

__device__ __forceinline__ void add_bytes(const Level &v, Kernel k, unsigned long long b) {
    atomicAdd(&v.counters->bytes[k], b);
}

// Programmatic dependent launch (level kernels are launched with it): wait until the
// previous kernel of the stream has finished and its writes are visible, then let the next
// kernel's CTAs be scheduled as this kernel's CTAs retire (its launch and ramp-up overlap
// this kernel's tail). Every level kernel calls this before it reads anything a previous
// kernel wrote; without a programmatic dependency both instructions do nothing.
__device__ __forceinline__ void pdl_enter() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" :::);
}

// A level may not start when a cell of the level above was never finished (its arrivals
// never completed) or an earlier step flagged an error: the build is flagged and its
// remaining kernels do nothing (ORB_ERR_TIMEOUT). The threads of a CTA decide alike without a vote
// (one in every kernel cost a level 0.5 us): nothing counted in done[] changes below its level, and
// the one kernel that can flag an error while its other CTAs start, k_part_classify, looks at
// level_late() alone; a warp that left there without the others would leave them at a barrier.
__device__ __forceinline__ bool level_late(const Level &v) {
    if (v.prev_C && *(volatile const uint32_t *)&v.counters->done[v.depth - 1] != v.prev_C) {
        if (threadIdx.x == 0) atomicExch(&v.counters->error, 1u);
        return true;
    }
    return false;
}
__device__ __forceinline__ bool level_failed(const Level &v) {
    return *(volatile const uint32_t *)&v.counters->error || level_late(v);
}

// Arrival at a counter, by one thread after a barrier of its CTA: the CTA's writes before the
// barrier are visible to whoever sees the count. Returns the count before. Release only: a
// __threadfence() also drops the SM's L1 lines, and one of those per tile (and thread) made
// the swap 30% slower. Whoever finds itself last calls acquire() before it reads the others'
// writes.
__device__ __forceinline__ uint32_t arrive_release(uint32_t *counter, uint32_t k) {
    uint32_t old;
    asm volatile("atom.add.release.gpu.global.u32 %0, [%1], %2;" : "=r"(old) : "l"(counter), "r"(k) : "memory");
    return old;
}
__device__ __forceinline__ void acquire() { __threadfence(); }

// ------------------------------------------------------------------------------------
// Block helpers
// ------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t warp_sum(uint32_t v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ uint32_t warp_max(uint32_t v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// Exclusive scan over the warp (lane order); every lane gets the total.
__device__ __forceinline__ uint32_t warp_excl_scan(uint32_t v, uint32_t *total) {
    const int lane = threadIdx.x & 31;
    uint32_t inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += t;
    }
    *total = __shfl_sync(0xffffffffu, inc, 31);
    return inc - v;
}

// Sum over the block; every thread gets the total. `sh` holds >= 32 words.
__device__ __forceinline__ uint32_t block_sum(uint32_t v, uint32_t *sh) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    v = warp_sum(v);
    __syncthreads();
    if (lane == 0) sh[warp] = v;
    __syncthreads();
    uint32_t t = lane < nw ? sh[lane] : 0u;
    return warp_sum(t);
}

__device__ __forceinline__ uint32_t block_max(uint32_t v, uint32_t *sh) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    v = warp_max(v);
    __syncthreads();
    if (lane == 0) sh[warp] = v;
    __syncthreads();
    uint32_t t = lane < nw ? sh[lane] : 0u;
    return warp_max(t);
}

// Exclusive scan of two counters over the block (thread order). Returns the exclusive
// prefix; *ta, *tb receive the block totals. `sh` holds >= 64 words.
__device__ __forceinline__ uint2 block_excl_scan2(uint32_t a, uint32_t b, uint32_t *sh,
                                                  uint32_t *ta, uint32_t *tb) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    uint32_t ia = a, ib = b;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t xa = __shfl_up_sync(0xffffffffu, ia, o);
        uint32_t xb = __shfl_up_sync(0xffffffffu, ib, o);
        if (lane >= o) {
            ia += xa;
            ib += xb;
        }
    }
    __syncthreads();
    if (lane == 31) {
        sh[warp] = ia;
        sh[32 + warp] = ib;
    }
    __syncthreads();
    if (warp == 0) {
        uint32_t wa = lane < nw ? sh[lane] : 0u, wb = lane < nw ? sh[32 + lane] : 0u;
        uint32_t sa = wa, sb = wb;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t xa = __shfl_up_sync(0xffffffffu, sa, o);
            uint32_t xb = __shfl_up_sync(0xffffffffu, sb, o);
            if (lane >= o) {
                sa += xa;
                sb += xb;
            }
        }
        sh[lane] = sa - wa;  // exclusive warp offsets
        sh[32 + lane] = sb - wb;
        if (lane == 31) {
            sh[64] = sa;
            sh[65] = sb;
        }
    }
    __syncthreads();
    uint2 r = make_uint2(sh[warp] + ia - a, sh[32 + warp] + ib - b);
    *ta = sh[64];
    *tb = sh[65];
    __syncthreads();
    return r;
}

// Visits every key of [e0, e1) once, float4 loads over the 16-byte aligned body.
template <class F>
__device__ __forceinline__ void for_keys(const float *__restrict__ keys, uint32_t e0, uint32_t e1,
                                         F &&f) {
    const uint32_t tid = threadIdx.x, nt = blockDim.x;
    const uintptr_t addr = reinterpret_cast<uintptr_t>(keys + e0);
    const uint32_t mis = (uint32_t)(((16u - (addr & 15u)) & 15u) >> 2);
    const uint32_t a0 = min(e1, e0 + mis);
    for (uint32_t i = e0 + tid; i < a0; i += nt) f(__ldg(keys + i));
    const uint32_t n4 = (e1 - a0) >> 2;
    const float4 *k4 = reinterpret_cast<const float4 *>(keys + a0);
#pragma unroll 4
    for (uint32_t j = tid; j < n4; j += nt) {
        float4 q = __ldg(k4 + j);
        f(q.x);
        f(q.y);
        f(q.z);
        f(q.w);
    }
    for (uint32_t i = a0 + (n4 << 2) + tid; i < e1; i += nt) f(__ldg(keys + i));
}

// Tile t of the level -> (cell, slot, key range). Block-uniform.
struct TileRef {
    int c;
    int slot;
    uint32_t e0, e1;   // absolute key range of the tile
    uint32_t local;    // tile index within the cell
};

__device__ __forceinline__ TileRef tile_ref(const Level &v, uint32_t t) {
    TileRef r;
    r.c = (int)v.htile_cell[t];
    r.slot = level_slot(v, r.c);
    r.local = t - v.tile_off[r.c];
    const uint2 rg = v.ranges[r.slot];
    r.e0 = rg.x + r.local * (uint32_t)kTile;
    r.e1 = min(rg.y, r.e0 + (uint32_t)kTile);
    return r;
}

// Slots of a cell's list: a cell whose bracket holds at most that many keys is finished on
// the list (sparse_per_tile a count tile, at most an eighth of a one-tile cell's keys and
// max(2048, n/64) of a larger one's, so that a level's lists have a bound: ensure_level_buffers).
__device__ __forceinline__ uint32_t list_capacity(const Level &v, uint32_t n) {
    const unsigned long long want =
        (unsigned long long)v.sparse_per_tile * ((n + (uint32_t)kTile - 1) / (uint32_t)kTile);
    return (uint32_t)min(want, (unsigned long long)(n <= (uint32_t)kTile ? n / 8 : max(2048u, n / 64)));
}

static_assert(kColdHistPasses * kMaxBinsLog2 >= kMaxIterations, "3 cold passes reach the cap");

// ------------------------------------------------------------------------------------
// Plan: a cell's tiles, histogram bins, list and state, set when the cell becomes known
// (the root by init, a child when its parent is finished, service cells by k_plan). Tiles
// and pool slots are taken from the level's totals with one or two atomics a cell, so no
// scan over the level's cells and no launch of its own is needed; the order of the
// allocations changes where scratch lies, never a result.
// ------------------------------------------------------------------------------------
struct PlanCell {
    int c;           // the cell's index in its level (-1: not planned)
    uint32_t t0, T;  // partition tiles
    uint32_t h0, H;  // count tiles
};

// Warm builds: a cell whose previous tree cut on the same axis starts from the hinted bracket
// (clipped to its extent) when that narrows it.
__device__ __forceinline__ void warm_start_cell(const Level &v, int c, int slot, uint32_t n) {
    orb_cell_t &cell = v.heap[slot];
    const float2 h = v.hint[slot];
    uint8_t w = 0;
    if (n > 1 && !isnan(h.x) && v.hint_axis[slot] == cell.cutAxis && cell.cutAxis >= 0) {
        // half-width w x extent / sqrt(n): about w sqrt(n) keys each side if evenly spread,
        // the scale by which a median drifts when the particles move a little
        const float L = cell.cutMarginLeft, R = cell.cutMarginRight;
        const float half = __fdiv_rn(h.y, sqrtf((float)n));
        const float Lw = fmaxf(L, __fsub_rn(h.x, half)), Rw = fminf(R, __fadd_rn(h.x, half));
        if (Lw < Rw && (Lw > L || Rw < R)) {
            cell.cutMarginLeft = Lw;
            cell.cutMarginRight = Rw;
            w = 1;
            v.inb[c] = n - 1;  // the first pass counts the keys below the bracket
            atomicAdd(&v.counters->warm_cells, 1u);
        }
    }
    v.warm[c] = w;
}

// The tiles of cell c of n particles (c < 0: none); cells of at most `small` particles get no
// count tiles.
__device__ __forceinline__ PlanCell plan_sizes(uint32_t small, int c, uint32_t n) {
    PlanCell p;
    p.c = c;
    p.T = c < 0 ? 0u : (n + (uint32_t)kPTile - 1) / (uint32_t)kPTile;
    p.H = c >= 0 && n > small ? (n + (uint32_t)kTile - 1) / (uint32_t)kTile : 0u;
    p.t0 = p.h0 = 0;
    return p;
}
// Its share of the level's tiles (count << 32 | partition), and of the pools (bins << 32 | list):
// bins for cells of several tiles (one CTA reads a one-tile cell and keeps its bins in shared
// memory), for all where a tile is dealt in pieces; a list unless weighted.
__device__ __forceinline__ unsigned long long plan_tiles(const PlanCell &p) {
    return ((unsigned long long)p.H << 32) | (unsigned long long)p.T;
}
__device__ __forceinline__ unsigned long long plan_pools(const Level &v, const PlanCell &p, uint32_t n) {
    if (!p.H || !v.plan_bins) return 0ull;
    const unsigned long long bins = p.H > 1 || v.plan_bins > 1 ? 1ull : 0ull;
    return (bins << 32) | (v.wt ? 0ull : (unsigned long long)list_capacity(v, n));
}

// The plan of a cell (heap slot `slot`) of n particles whose shares start at `tiles` and `pools`.
__device__ __forceinline__ void plan_store(const Level &v, PlanCell &p, unsigned long long tiles,
                                           unsigned long long pools, uint32_t small, int slot, uint32_t n) {
    const int c = p.c;
    if (p.T) {
        p.t0 = (uint32_t)tiles;
        p.h0 = (uint32_t)(tiles >> 32);
    }
    v.ptile_off[c] = p.t0;
    v.tile_off[c] = p.h0;
    v.hist_off[c] = (uint32_t)(pools >> 32) << kMaxBinsLog2;
    v.cmp_off[c] = (uint32_t)pools;
    uint8_t st = kActive;
    uint32_t it = 0;
    if (n <= small && small) {
        st = kSmall;
    } else if (n == 0) {
        // no key: the first cut is found (src/orbit.cpp:204-213 with count 0)
        st = kFound;
        it = 1;
        v.heap[slot].foundCut = 1;
        atomicMax(&v.counters->max_iters, 1u);
    }
    v.state[c] = st;
    v.iters[c] = (uint8_t)it;
    v.hdone[c] = 0;
    v.below[c] = 0;
    v.inb[c] = n;
    v.cmp_cnt[c] = 0;
    v.pred[c] = 0u;  // no sampled bracket unless k_sample_pick sets one
    if (v.wt) {
        v.wbelow[c] = 0ull;
        v.wtot[c] = 0ull;
    }
    if (v.warm) {
        v.warm[c] = 0;
        if (v.plan_hint) warm_start_cell(v, c, slot, n);
    }
}

// One thread: plans cell c (heap slot `slot`, n particles) with the totals `tot`.
__device__ PlanCell plan_cell(const Level &v, PlanTotals *tot, uint32_t small, int c, int slot, uint32_t n) {
    PlanCell p = plan_sizes(small, c, n);
    const unsigned long long ti = plan_tiles(p), po = plan_pools(v, p, n);
    const unsigned long long a = ti ? atomicAdd(&tot->tiles, ti) : 0ull, b = po ? atomicAdd(&tot->pools, po) : 0ull;
    plan_store(v, p, a, b, small, slot, n);
    return p;
}

// The tile maps of a planned cell, by nt threads.
__device__ __forceinline__ void plan_fill(const Level &v, const PlanCell &p, uint32_t ti, uint32_t nt) {
    if (p.c < 0) return;
    for (uint32_t t = ti; t < p.T; t += nt) v.ptile_cell[p.t0 + t] = (uint32_t)p.c;
    for (uint32_t t = ti; t < p.H; t += nt) v.htile_cell[p.h0 + t] = (uint32_t)p.c;
}

// Plans every cell of the level, a warp per cell (service calls, and the levels a refused
// subtree path leaves). The totals are zero.
__global__ void __launch_bounds__(kThreads) k_plan(const __grid_constant__ Level v) {
    pdl_enter();
    const int c = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    const uint32_t lane = threadIdx.x & 31;
    if (c >= v.C) return;
    PlanCell p = {};
    const int slot = level_slot(v, c);
    if (v.cells_in) {
        if (lane < 13)
            reinterpret_cast<uint32_t *>(v.heap + slot)[lane] = reinterpret_cast<const uint32_t *>(v.cells_in + c)[lane];
        __syncwarp();
    }
    if (lane == 0) {
        const uint2 rg = v.ranges[slot];
        p = plan_cell(v, v.tot, v.small, c, slot, rg.y - rg.x);
    }
    p.c = c;
    p.t0 = __shfl_sync(0xffffffffu, p.t0, 0);
    p.T = __shfl_sync(0xffffffffu, p.T, 0);
    p.h0 = __shfl_sync(0xffffffffu, p.h0, 0);
    p.H = __shfl_sync(0xffffffffu, p.H, 0);
    plan_fill(v, p, lane, 32);
}

// ------------------------------------------------------------------------------------
// Init: identity permutation, zeroed heap/ranges, root cell (src/orbit.cpp:74-81)
// ------------------------------------------------------------------------------------
__global__ void k_init(const __grid_constant__ Level v, uint32_t n, float lo0, float lo1, float lo2, float hi0,
                       float hi1, float hi2, uint32_t d, int heap_cells) {
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    const uint64_t g = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (v.idx)
        for (uint64_t i = g; i < n; i += stride) v.idx[i] = (uint32_t)i;
    uint32_t *hw = reinterpret_cast<uint32_t *>(v.heap);
    const uint64_t words = (uint64_t)heap_cells * 13;
    for (uint64_t i = g + 13; i < words; i += stride) hw[i] = 0u;
    for (uint64_t i = g + 1; i < (uint64_t)heap_cells; i += stride) v.ranges[i] = make_uint2(0u, 0u);
    // the root's tile maps (its index in level 1 is 0)
    for (uint64_t i = g; i * kPTile < n; i += stride) v.ptile_cell[i] = 0u;
    for (uint64_t i = g; i * kTile < n; i += stride) v.htile_cell[i] = 0u;
    if (g == 0) {
        orb_cell_t r;
        r.id = 0;
        r.nLeafCells = (int32_t)d;
        r.prevCutAxis = -1;
        r.cutAxis = 0;  // orbit.cpp:75
        r.foundCut = 0;
        r.pad_[0] = r.pad_[1] = r.pad_[2] = 0;
        r.lower[0] = lo0;
        r.lower[1] = lo1;
        r.lower[2] = lo2;
        r.upper[0] = hi0;
        r.upper[1] = hi1;
        r.upper[2] = hi2;
        r.cutMarginLeft = lo0;  // setCutMargin, orbit.cpp:76
        r.cutMarginRight = hi0;
        v.heap[0] = r;
        v.ranges[0] = make_uint2(0u, n);
        BuildCounters z = {};
        *v.counters = z;
        if (v.C) plan_cell(v, v.tot, v.small, 0, 0, n);
    }
}

// Batched init: every instance's root cell and root range (heap and ranges are zeroed by
// the host before) and idx = position relative to the instance. blockIdx.y walks the
// instances, blockIdx.x their particles.
__global__ void k_init_batch(const __grid_constant__ Level v, const BatchRoot *roots, int k) {
    __shared__ PlanCell s_plan;
    for (int i = blockIdx.y; i < k; i += gridDim.y) {
        const BatchRoot r = roots[i];
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            orb_cell_t c;
            c.id = 0;
            c.nLeafCells = (int32_t)r.d;
            c.prevCutAxis = -1;
            c.cutAxis = 0;  // orbit.cpp:75
            c.foundCut = 0;
            c.pad_[0] = c.pad_[1] = c.pad_[2] = 0;
            for (int a = 0; a < 3; ++a) {
                c.lower[a] = r.lower[a];
                c.upper[a] = r.upper[a];
            }
            c.cutMarginLeft = r.lower[0];  // setCutMargin, orbit.cpp:76
            c.cutMarginRight = r.upper[0];
            v.heap[r.heap_base] = c;
            const uint2 rg = make_uint2(r.offset, r.offset + r.n);
            v.ranges[r.heap_base] = rg;
            s_plan.c = -1;
            if (r.cell >= 0) s_plan = plan_cell(v, v.tot, v.small, r.cell, (int)r.heap_base, r.n);
        }
        if (blockIdx.x == 0) {
            __syncthreads();
            plan_fill(v, s_plan, threadIdx.x, blockDim.x);
            __syncthreads();
        }
        if (v.idx)
            for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < r.n; p += gridDim.x * blockDim.x)
                v.idx[r.offset + p] = p;
    }
}

// Warm builds: whether a hinted bracket [L, R) can hold the cut the bisection looks for,
// given the counts of keys below L and below R. Outside it every tested cut would keep
// moving the same margin: count(< L) already too high, or count(< R) still too low.
__device__ __forceinline__ bool warm_bracket_holds(uint32_t below_L, uint32_t below_R, uint32_t n,
                                                   float ratio) {
    return convergence(below_L, n, ratio) <= 0 && convergence(below_R, n, ratio) >= 0;
}

// Restart of a cell whose hinted bracket missed: the reference's own start, the cell's extent
// along its cut axis (setCutMargin, src/cell.h:123-126).
__device__ __forceinline__ void warm_reset(orb_cell_t &cell, float &L, float &R, BuildCounters *ctr) {
    const int a = eff_axis(cell.cutAxis);
    L = cell.lower[a];
    R = cell.upper[a];
    cell.cutMarginLeft = L;
    cell.cutMarginRight = R;
    atomicAdd(&ctr->warm_resets, 1u);
}

// ------------------------------------------------------------------------------------
// Count-left histogram pass
// ------------------------------------------------------------------------------------
// The midpoint tree over [L, R] with nb = 2^K leaves: edge e(0) = L, e(nb) = R, and the
// inner node j is the midpoint of its two nearest ancestors, i.e. exactly the cut the
// reference's bisection computes at that node (src/cell.h:74-76).
// Inner edges of the subtree of S leaves over [lo, hi] = [e(base), e(base + S)], written to
// e[base .. base + S): each the midpoint of its two nearest ancestors, as in the full tree.
template <int S>
__device__ __forceinline__ void fill_sub(float *e, uint32_t base, float lo, float hi) {
    float loc[S + 1];
    loc[0] = lo;
    loc[S] = hi;
#pragma unroll
    for (int st = S / 2; st >= 1; st /= 2) {
#pragma unroll
        for (int j = st; j < S; j += 2 * st) loc[j] = mid_cut(loc[j - st], loc[j + st]);
    }
#pragma unroll
    for (int j = 0; j < S; ++j) e[base + j] = loc[j];
}

// Edge table e[0 .. 2^K] of the midpoint tree over [L, R], filled by nt threads (ti = this
// thread's index, 2^K <= 16 nt): each descends once to the subtree of 2^K / nt leaves it
// owns, then fills that subtree. The caller synchronises.
__device__ void fill_edges(float *e, float L, float R, int K, uint32_t ti, uint32_t nt) {
    const uint32_t nb = 1u << K;
    int ks = 0;
    while ((nt << ks) < nb) ++ks;
    const uint32_t S = 1u << ks, base = ti * S;
    if (base < nb) {
        float lo = L, hi = R;
        for (int d = K - 1; d >= ks; --d) {
            const float mm = mid_cut(lo, hi);
            if (base & (1u << d))
                lo = mm;
            else
                hi = mm;
        }
        switch (ks) {
            case 0: e[base] = lo; break;
            case 1: fill_sub<2>(e, base, lo, hi); break;
            case 2: fill_sub<4>(e, base, lo, hi); break;
            case 3: fill_sub<8>(e, base, lo, hi); break;
            default: fill_sub<16>(e, base, lo, hi); break;
        }
    }
    if (ti == 0) e[nb] = R;
}

// Leaf of key k (L <= k < R) in that tree: the reference's descent itself (k below the
// midpoint: left half, else right half), K midpoints.
__device__ __forceinline__ int tree_bin(float k, float L, float R, int K) {
    float lo = L, hi = R;
    int b = 0;
    for (int d = K - 1; d >= 0; --d) {
        const float mm = mid_cut(lo, hi);
        if (k < mm) {
            hi = mm;
        } else {
            lo = mm;
            b += 1 << d;
        }
    }
    return b;
}

// Edge e(j) of that tree (e(0) = L, e(2^K) = R): the lower end of leaf j, reached by the same
// midpoints as tree_bin. The edges are non-decreasing (a midpoint of [lo, hi] rounds into
// [lo, hi]), so tree_bin(k) >= j exactly when k >= e(j), for L <= k < R.
__device__ __forceinline__ float tree_edge(float L, float R, int K, uint32_t j) {
    if (j >= (1u << K)) return R;
    float lo = L, hi = R;
    for (int d = K - 1; d >= 0; --d) {
        const float mm = mid_cut(lo, hi);
        if (j & (1u << d))
            lo = mm;
        else
            hi = mm;
    }
    return lo;
}

// Bin of key k (L <= k < R) in the edge table e[0..nb]: the largest b with e[b] <= k, i.e.
// the leaf the bisection's descent reaches. The spacing of the edges is uniform to a few
// ulps, so the scaled guess is off by at most one except in brackets only a few ulps
// wide, which fall back to a binary search over the table.
template <class EdgeAt>
__device__ __forceinline__ int edge_bin(float k, float L, float scale, int top, EdgeAt e) {
    int g = __float2int_rz((k - L) * scale);
    g = min(max(g, 0), top);
    if (k < e(g)) {
        --g;
        if (g >= 0 && !(k < e(g))) return g;
    } else if (!(k < e(g + 1))) {
        ++g;
        if (g <= top && k < e(g + 1)) return g;
    } else {
        return g;
    }
    int lo = 0, hi = top;  // largest b in [0, top] with e(b) <= k (e(0) = L <= k)
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (e(mid) <= k)
            lo = mid;
        else
            hi = mid - 1;
    }
    return lo;
}

// Margin of the scaled guess, in bins. The tree's edges deviate from the linear edges
// L + j (R-L)/2^K by at most K u/2 <= 5.5u (every midpoint rounds once, to within u/2 of the
// mean of its two endpoints; u = spacing of floats at max(|L|, |R|)). The guess
// t = fl(fl(k-L) * scale), scale = fl(2^K / fl(R-L)), is within 1.01 u S + 2^K 2^-22 of the
// exact (k-L) S, S = 2^K/(R-L). A fractional part of t farther than
// m = 8 u scale + 2^K 2^-21 from 0 and 1 therefore puts k strictly between the edges of
// bin floor(t). Returns 1 (guess never trusted) for tiny brackets and where an end lies at or past
// 2^127: midpoints can overflow there (edges are then infinite, not linear), and R - L.
__device__ __forceinline__ float bin_margin(float L, float R, float scale, uint32_t nb) {
    const float M = fmaxf(fabsf(L), fabsf(R));
    const int e = (__float_as_int(M) >> 23) & 0xff;
    if (e < 24 || e >= 0xfe) return 1.0f;
    const float u = __int_as_float((e - 23) << 23);
    return __fadd_ru(__fmul_ru(__fmul_ru(8.0f, u), scale), __fmul_ru((float)nb, 0x1p-21f));
}

// edge_bin() over a table in shared memory, out of line: it runs for a few keys only, and
// the streaming loops that call it stay small enough for the instruction cache.
__device__ __noinline__ int edge_bin_slow(float k, float L, float scale, int top, const float *e) {
    return edge_bin(k, L, scale, top, [&](int j) { return e[j]; });
}

// The scaled guess with no float<->int conversion. For a key whose guess t = (k-L) scale lies
// in [0, 2^11), y = fl(fl(k-L) scale + 2^11) is 2^11 + t rounded to 12 fraction bits, so the
// encoding of y minus that of 2^11 holds the bin above bit 12 and the fraction below it. Its
// error is that of fl(fl(k-L) scale) except the last rounding, 2^-13 bins instead of
// t 2^-24, which the margin taken at 2^11 bins or more (2^-10) covers. The guess is exact
// when its fraction f = i/4096 lies in (m, 1 - m), i.e. i in [mi+1, 4095-mi] with
// mi = floor(4096 m) (4096 m is exact). `base` is the encoding of 2^11 plus mi+1, so the test
// is a subtraction and two unsigned comparisons; a key below L (y under 2^11 or negative),
// at or past R (a bin past the table) or NaN fails it.
static_assert(kMaxBinsLog2 <= 11, "guess_bin holds bins below 2^11");
struct Guess {
    float L, scale;
    uint32_t base, lim, span;
};

__device__ __forceinline__ Guess make_guess(float L, float R, float scale, uint32_t nb) {
    Guess g;
    g.L = L;
    g.scale = scale;
    const float M = __fmul_rn(bin_margin(L, R, scale, max(nb, 2048u)), 4096.0f);
    const uint32_t mi = M < 2048.0f ? (uint32_t)M : 0u;  // M >= 2048 or NaN: accept nothing
    g.base = __float_as_uint(2048.0f) + mi + 1u;
    g.lim = nb << 12;
    g.span = M < 2048.0f ? 4095u - 2u * mi : 0u;
    return g;
}

// The guessed bin of k in *b; true when it is the exact bin (edge_bin's answer).
__device__ __forceinline__ bool guess_bin(const Guess &g, float k, uint32_t *b) {
    const uint32_t e = __float_as_uint(__fmaf_rn(__fsub_rn(k, g.L), g.scale, 2048.0f)) - g.base;
    *b = e >> 12;
    return e < g.lim && (e & 0xfffu) < g.span;
}

// Exact bin of L <= k < R by the edge table e[0..top+1] (in shared memory) for a key the
// scaled guess did not settle: floor(t) of the same guess, then its neighbours (the guess is
// off by at most one bin when the margin lets it be trusted at all: bins are then more than
// 16 ulps wide); a search over the table otherwise (out of line: brackets a few ulps wide).
__device__ __forceinline__ uint32_t near_bin(float k, const Guess &gs, const float *e, uint32_t top) {
    const uint32_t t = __float_as_uint(__fmaf_rn(__fsub_rn(k, gs.L), gs.scale, 2048.0f)) - 0x45000000u;
    const uint32_t g = min(t >> 12, top);  // 0x45000000: the encoding of 2048.0f (t >= 0 for k >= L)
    if (k < e[g]) {
        if (g > 0 && !(k < e[g - 1])) return g - 1;
    } else if (!(k < e[g + 1])) {
        if (g < top && k < e[g + 2]) return g + 1;
    } else {
        return g;
    }
    return (uint32_t)edge_bin_slow(k, gs.L, gs.scale, (int)top, e);
}

// The cell a count pass's CTA is working on, in shared memory (thread 0 fills it when the
// CTA's tiles move to a new cell): the rare paths read it there, so the streaming loop keeps
// only what it needs in registers.
constexpr uint32_t kHDense = 1, kHBracket = 2, kHPred = 4;
struct HistCell {
    const float *keys;  // the cut axis
    uint32_t *gh;       // the cell's global bins
    float L, R;
    uint32_t mode;      // kHDense (first pass over the extent: nearly every key inside
                        // [L, R)), kHBracket (many keys outside) or kHPred (sampled bracket)
    uint32_t base, end; // the cell's key range [base, end)
    uint32_t t0;        // its first tile
    uint32_t below;     // dense: keys below L met by the exact path
    float pa, pb;       // kHPred: the sampled bracket [e(lo), e(hi)) of the tree over [L, R)
    Guess gs;           // the scaled guess
    uint32_t whole;     // the CTA read every tile of the cell: its bins and count are complete
    uint32_t last;      // the CTA finished the cell's last tile
};
constexpr int kHistK = kMaxBinsLog2;  // depth of the count passes' midpoint trees
constexpr uint32_t kHistBins = 1u << kHistK;

// A dense pass's key the scaled guess did not settle: below L counted, inside [L, R) binned
// by the edge table (near_bin), at or past R (or NaN) ignored.
__device__ __forceinline__ void dense_exact(float k, HistCell *hc, uint32_t *s_hist, const float *s_edge) {
    const float L = hc->L, R = hc->R;
    if (k < L)
        atomicAdd(&hc->below, 1u);
    else if (k < R)
        atomicAdd(&s_hist[near_bin(k, hc->gs, s_edge, kHistBins - 1u)], 1u);
}

// A sampled pass's bracket key (e(lo) <= k < e(hi), inside [L, R)): its bin by the scaled
// guess (the edge table when the guess is not proven) into the shared bins.
__device__ __noinline__ void pred_key(float k, const HistCell *hc, uint32_t *s_hist, const float *s_edge) {
    uint32_t g;
    if (!guess_bin(hc->gs, k, &g)) g = near_bin(k, hc->gs, s_edge, kHistBins - 1u);
    atomicAdd(&s_hist[g], 1u);
}

// A compile-time flag passed to a generic lambda.
template <bool B>
struct Flag {
    static constexpr bool value = B;
};

// Keys per thread per round of the histogram pass (float4 loads issued together).
constexpr int kHistVec = 4;

// The keys [e0, e1) of one tile (at most kTile keys), visited by the CTA's threads, for a
// pass that leaves a few percent of its keys (the sampled pass). The 16-byte aligned body is
// read in rounds of kHistVec float4 loads a thread (all issued before any key is used); each
// key goes through settle(k), branch-free code for the common case that returns false for a
// key it leaves; a round's left keys are visited right after it through rest(k) (reloaded
// while its lines are still in L1). The unaligned head and tail go through visit(k). `pad`
// fills the missing lanes of the last round: settle(pad) must count nothing (a pad it leaves
// is skipped).
template <uint32_t NT, class Settle, class Rest, class Visit>
__device__ __forceinline__ void scan_tile(const float *keys, uint32_t e0, uint32_t e1, float pad,
                                          Settle settle, Rest rest, Visit visit) {
    const uint32_t ti = threadIdx.x;  // NT = blockDim.x
    const uintptr_t addr = reinterpret_cast<uintptr_t>(keys + e0);
    const uint32_t a0 = min(e1, e0 + (uint32_t)(((16u - (addr & 15u)) & 15u) >> 2));
    for (uint32_t i = e0 + ti; i < a0; i += NT) visit(__ldg(keys + i));
    const uint32_t n4 = (e1 - a0) >> 2;
    const float4 *k4 = reinterpret_cast<const float4 *>(keys + a0);
    const float *kb = keys + a0;
    uint32_t j0 = 0;
    auto round = [&](auto full) {
        float4 q[kHistVec];
#pragma unroll
        for (int u = 0; u < kHistVec; ++u) {
            const uint32_t j = j0 + u * NT + ti;
            if (decltype(full)::value)
                q[u] = __ldg(k4 + j);
            else
                q[u] = j < n4 ? __ldg(k4 + j) : make_float4(pad, pad, pad, pad);
        }
        uint32_t miss = 0;  // bit 4u + c: component c of load u left
#pragma unroll
        for (int u = 0; u < kHistVec; ++u) {
            const float kk[4] = {q[u].x, q[u].y, q[u].z, q[u].w};
#pragma unroll
            for (int c = 0; c < 4; ++c) miss |= (uint32_t)!settle(kk[c]) << (4 * u + c);
        }
        while (miss) {
            const uint32_t b = (uint32_t)__ffs(miss) - 1u;
            miss &= miss - 1u;
            const uint32_t j = j0 + (b >> 2) * NT + ti;
            if (j < n4) rest(__ldg(kb + 4 * j + (b & 3u)));  // else a pad lane
        }
    };
    for (; j0 + kHistVec * NT <= n4; j0 += kHistVec * NT) round(Flag<true>());
    if (j0 < n4) round(Flag<false>());
    for (uint32_t i = a0 + (n4 << 2) + ti; i < e1; i += NT) visit(__ldg(keys + i));
}

// A dense pass's key, its guess corrected by the edges either side of it: exact while the guess
// errs by less than a bin (bin_margin below 1; see make_guess for the form of the guess). Returns 1
// for a key below L, which it does not bin.
__device__ __forceinline__ uint32_t edges_key(float k, const Guess &gs, float R, uint32_t *s_hist, const float *s_edge) {
    const uint32_t t = __float_as_uint(__fmaf_rn(__fsub_rn(k, gs.L), gs.scale, 2048.0f)) - 0x45000000u;
    const uint32_t g = min(t >> 12, kHistBins - 1u);  // (a key outside [L, R): not used)
    const float a = s_edge[g], b = s_edge[g + 1];
    if (k >= gs.L && k < R) atomicAdd(&s_hist[g + (k >= b ? 1u : 0u) - (k < a ? 1u : 0u)], 1u);
    return k < gs.L ? 1u : 0u;
}

// The dense pass's tile [e0, e1) in the first pass of a cold level: every key binned by the
// scaled guess into the CTA's shared bins (a key the guess does not settle counted in the
// lane's spare bin and binned exactly right after its round). Where a round leaves a warp many
// keys (many equal ones on an edge, or a cell thin for its distance from the origin) the warp
// bins every key of the cell's later rounds by its guess and two edges (by_edges): 1.4 times a
// clean round's time, where key by key a pass over 2^26 clustered particles took 160-300 us on
// levels with such cells, 80 on the others. Rounds of kHistVec float4 loads a thread; the
// unaligned head and tail and a last partial round key by key.
constexpr uint32_t kByEdges = 32;  // many: more of a warp's 512
constexpr int kEdgeVec = 2;        // float4 loads of a round by edges
template <uint32_t NT>
__device__ __forceinline__ void dense_tile(const float *keys, uint32_t e0, uint32_t e1, const Guess gs,
                                           uint32_t *s_hist, HistCell *hc, const float *s_edge, uint32_t &below,
                                           bool &by_edges) {
    const uint32_t ti = threadIdx.x;
    const uint32_t spare = (gs.lim >> 12) + (ti & 31u);
    auto one = [&](float k) {
        uint32_t g;
        if (guess_bin(gs, k, &g))
            atomicAdd(&s_hist[g], 1u);
        else
            dense_exact(k, hc, s_hist, s_edge);
    };
    const uintptr_t addr = reinterpret_cast<uintptr_t>(keys + e0);
    const uint32_t a0 = min(e1, e0 + (uint32_t)(((16u - (addr & 15u)) & 15u) >> 2));
    for (uint32_t i = e0 + ti; i < a0; i += NT) one(__ldg(keys + i));
    const uint32_t n4 = (e1 - a0) >> 2;
    const float4 *k4 = reinterpret_cast<const float4 *>(keys + a0);
    const float *kb = keys + a0;
    uint32_t j0 = 0;
#pragma unroll 1
    for (; !by_edges && j0 + kHistVec * NT <= n4; j0 += kHistVec * NT) {
        float4 q[kHistVec];
#pragma unroll
        for (int u = 0; u < kHistVec; ++u) q[u] = __ldg(k4 + j0 + u * NT + ti);
        uint32_t miss = 0;
#pragma unroll
        for (int u = 0; u < kHistVec; ++u) {
            const float kk[4] = {q[u].x, q[u].y, q[u].z, q[u].w};
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                uint32_t g;
                const bool ok = guess_bin(gs, kk[c], &g);
                atomicAdd(&s_hist[ok ? g : spare], 1u);
                if (!ok) miss |= 1u << (4 * u + c);
            }
        }
        if (__reduce_add_sync(0xffffffffu, (uint32_t)__popc(miss)) > kByEdges) by_edges = gs.span != 0u;
        while (miss) {
            const uint32_t b = (uint32_t)__ffs(miss) - 1u;
            miss &= miss - 1u;
            dense_exact(__ldg(kb + 4 * (j0 + (b >> 2) * NT + ti) + (b & 3u)), hc, s_hist, s_edge);
        }
    }
#pragma unroll 1
    for (; by_edges && j0 + kEdgeVec * NT <= n4; j0 += kEdgeVec * NT) {
        const float R = hc->R;
        float4 q[kEdgeVec];
#pragma unroll
        for (int u = 0; u < kEdgeVec; ++u) q[u] = __ldg(k4 + j0 + u * NT + ti);
#pragma unroll
        for (int u = 0; u < kEdgeVec; ++u) {
            const float kk[4] = {q[u].x, q[u].y, q[u].z, q[u].w};
#pragma unroll
            for (int c = 0; c < 4; ++c) below += edges_key(kk[c], gs, R, s_hist, s_edge);
        }
    }
    for (uint32_t j = j0 + ti; j < n4; j += NT) {
        const float4 q = __ldg(k4 + j);
        one(q.x);
        one(q.y);
        one(q.z);
        one(q.w);
    }
    for (uint32_t i = a0 + (n4 << 2) + ti; i < e1; i += NT) one(__ldg(keys + i));
}

// A later pass's tile [e0, e1): keys below L counted in `below`, keys inside [L, R) binned by
// the scaled guess (a key the guess does not settle exactly right after its round), keys at
// or above R and NaN ignored. Same rounds as dense_tile; a key outside the bracket costs its
// comparisons only (the dense loop would send each one through the exact path: clustered
// cells' second passes ran at 1.7 TB/s that way). Where a round leaves a warp many keys they are
// mostly equal ones, which kept their cell's bracket full (its bins are a few floats wide by then):
// 32 at a time, the first one's bin is found once and takes all its equals in one addition. (Half
// of 2^24 particles on one point, 2^13 leaves: passes two and three of a level 135 and 240 us with a
// search and an addition a key.)
constexpr uint32_t kTies = 64;  // many: more of a warp's 512
template <uint32_t NT>
__device__ __forceinline__ void bracket_tile(const float *keys, uint32_t e0, uint32_t e1, const Guess gs, float L,
                                             float R, uint32_t &below, uint32_t *s_hist, const float *s_edge) {
    const uint32_t ti = threadIdx.x;
    auto one = [&](float k) {
        if (k < L) {
            ++below;
        } else if (k < R) {
            uint32_t g;
            if (!guess_bin(gs, k, &g)) g = near_bin(k, gs, s_edge, kHistBins - 1u);
            atomicAdd(&s_hist[g], 1u);
        }
    };
    const uintptr_t addr = reinterpret_cast<uintptr_t>(keys + e0);
    const uint32_t a0 = min(e1, e0 + (uint32_t)(((16u - (addr & 15u)) & 15u) >> 2));
    for (uint32_t i = e0 + ti; i < a0; i += NT) one(__ldg(keys + i));
    const uint32_t n4 = (e1 - a0) >> 2;
    const float4 *k4 = reinterpret_cast<const float4 *>(keys + a0);
    const float *kb = keys + a0;
    uint32_t j0 = 0;
#pragma unroll 1
    for (; j0 + kHistVec * NT <= n4; j0 += kHistVec * NT) {
        float4 q[kHistVec];
#pragma unroll
        for (int u = 0; u < kHistVec; ++u) q[u] = __ldg(k4 + j0 + u * NT + ti);
        uint32_t miss = 0;
#pragma unroll
        for (int u = 0; u < kHistVec; ++u) {
            const float kk[4] = {q[u].x, q[u].y, q[u].z, q[u].w};
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                if (kk[c] < L) ++below;
                uint32_t g;
                const bool ok = guess_bin(gs, kk[c], &g);
                if (ok) atomicAdd(&s_hist[g], 1u);
                if (!ok && kk[c] >= L && kk[c] < R) miss |= 1u << (4 * u + c);
            }
        }
        if (__reduce_add_sync(0xffffffffu, (uint32_t)__popc(miss)) > kTies) {
            const uint32_t lane = ti & 31u;
            float tie = __int_as_float(0x7fc00000);
            uint32_t bin = 0;
#pragma unroll 1
            for (uint32_t b = 0; b < 4u * kHistVec; ++b) {
                const bool in = (miss >> b) & 1u;
                const uint32_t m = __ballot_sync(0xffffffffu, in);
                if (!m) continue;
                const float k = in ? __ldg(kb + 4 * (j0 + (b >> 2) * NT + ti) + (b & 3u)) : 0.0f;
                const uint32_t first = (uint32_t)__ffs(m) - 1u;
                const float t = __shfl_sync(0xffffffffu, k, (int)first);
                if (t != tie) bin = near_bin(t, gs, s_edge, kHistBins - 1u);
                tie = t;
                const uint32_t same = __ballot_sync(0xffffffffu, in && k == t);
                if (lane == first)
                    atomicAdd(&s_hist[bin], (uint32_t)__popc(same));
                else if (in && k != t)
                    atomicAdd(&s_hist[near_bin(k, gs, s_edge, kHistBins - 1u)], 1u);
            }
            continue;
        }
        while (miss) {
            const uint32_t b = (uint32_t)__ffs(miss) - 1u;
            miss &= miss - 1u;
            const float k = __ldg(kb + 4 * (j0 + (b >> 2) * NT + ti) + (b & 3u));
            atomicAdd(&s_hist[near_bin(k, gs, s_edge, kHistBins - 1u)], 1u);
        }
    }
    for (uint32_t j = j0 + ti; j < n4; j += NT) {
        const float4 q = __ldg(k4 + j);
        one(q.x);
        one(q.y);
        one(q.z);
        one(q.w);
    }
    for (uint32_t i = a0 + (n4 << 2) + ti; i < e1; i += NT) one(__ldg(keys + i));
}

// ------------------------------------------------------------------------------------
// Sampled first pass. The first count pass of a cold level bins every key of a cell into
// the 2^K leaves of its midpoint tree. k_sample_bin and k_sample_pick predict from a strided
// sample of the cell
// (one key per 2^kSampleShift) a run of leaves [lo, hi) holding the cut: the sample's
// median +- pred_sigmas standard errors (sqrt(s)/2 sample keys), widened to leaf edges
// a = e(lo), b = e(hi). That pass then counts the keys below a and bins only the keys of
// [a, b). Its replay in resolve_cell is the reference loop unchanged once the exact counts
// show count(< a) with difference <= -3 and count(< b) with difference >= 3: every tested
// cut below a then has a count <= count(< a) and moves L, every cut above b has one
// >= count(< b) and moves R (the float test is monotone in the count), and cuts inside
// [a, b] get their exact counts from the bins. Otherwise the pass is discarded and the
// next one bins every key. Same cuts, same integer counts, same iterations either way.
// (resolve_cell checks the counts; sample sizes and widths only change the speed.)
// ------------------------------------------------------------------------------------
constexpr uint32_t kPredValid = 1u << 25;
__device__ __forceinline__ uint32_t pred_lo(uint32_t p) { return p & 0xfffu; }
__device__ __forceinline__ uint32_t pred_hi(uint32_t p) { return (p >> 12) & 0xfffu; }
constexpr int kSampleThreads = 256;
constexpr int kSampleShift = 8;              // one sample key per 256 keys of the cell
constexpr uint32_t kSampleMax = 16384;       // sample keys per cell at most
constexpr uint32_t kSampleMin = 1024;        // fewer: no prediction (a dense first pass)
constexpr uint32_t kSamplePerCta = 4 * kSampleThreads;
__device__ __forceinline__ uint32_t sample_count(uint32_t n) {
    const uint32_t ns = min(n >> kSampleShift, kSampleMax);
    return ns >= kSampleMin ? ns : 0u;
}

// Sample binning: CTA (x, y) takes samples [x kSamplePerCta, (x+1) kSamplePerCta) of the
// cells y, y + gridDim.y, ...; sample j of a cell of n keys is the key at position
// ((2j+1) n / (2 ns)) (fixed point), binned into the cell's histogram bins (all zero
// between passes) by the scaled guess or the descent; samples below L are counted in
// pred[c], which k_sample_pick then replaces by the prediction.
__global__ void __launch_bounds__(kSampleThreads) k_sample_bin(const __grid_constant__ Level v) {
    pdl_enter();
    if (level_failed(v)) return;
    const uint32_t ti = threadIdx.x;
    for (int c = blockIdx.y; c < v.C; c += gridDim.y) {
        if (v.state[c] != kActive) continue;
        const int slot = level_slot(v, c);
        const uint2 rg = v.ranges[slot];
        const uint32_t n = rg.y - rg.x;
        const uint32_t ns = sample_count(n);
        const uint32_t j0 = blockIdx.x * kSamplePerCta;
        if (j0 >= ns) continue;
        const orb_cell_t &cell = v.heap[slot];
        const float L = cell.cutMarginLeft, R = cell.cutMarginRight;
        constexpr int K = kHistK;
        constexpr uint32_t nb = kHistBins;
        const float *keys = axis_keys(v, eff_axis(cell.cutAxis)) + rg.x;
        uint32_t *gh = v.hist + v.hist_off[c];
        // (2j+1) step >> 17 < n for j < ns: step = floor(n 2^16 / ns) < 2^37, products < 2^52
        const uint64_t step = ((uint64_t)n << 16) / ns;
        float k[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const uint32_t j = j0 + u * kSampleThreads + ti;
            k[u] = j < ns ? __ldg(keys + (uint32_t)(((2ull * j + 1ull) * step) >> 17)) : R;
        }
        const float scale = __fdiv_rn((float)nb, __fsub_rn(R, L));
        const Guess gs = make_guess(L, R, scale, nb);
        uint32_t below = 0;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            if (k[u] < L) {
                ++below;
            } else if (k[u] < R) {
                uint32_t g;
                if (!guess_bin(gs, k[u], &g)) g = (uint32_t)tree_bin(k[u], L, R, K);
                atomicAdd(&gh[g], 1u);
            }
        }
        below = warp_sum(below);
        if ((ti & 31u) == 0 && below) atomicAdd(&v.pred[c], below);
        if (ti == 0) add_bytes(v, kKSample, 4ull * min(kSamplePerCta, ns - j0));
    }
}

// One CTA per sampled cell (cells y, y + gridDim.x, ...): the leaves [lo, hi) around the
// sample median (+- pred_sigmas standard errors), packed into pred[c]; the bins are cleared
// again. Each thread holds 8 consecutive bins in registers.
constexpr int kPickThreads = 256;
static_assert((1 << kMaxBinsLog2) == 8 * kPickThreads, "8 bins a thread");
__global__ void __launch_bounds__(kPickThreads) k_sample_pick(const __grid_constant__ Level v) {
    pdl_enter();
    if (level_failed(v)) return;
    __shared__ uint32_t s_red[72];
    const uint32_t ti = threadIdx.x;
    for (int c = blockIdx.x; c < v.C; c += gridDim.x) {
        if (v.state[c] != kActive) continue;
        const uint2 rg = v.ranges[level_slot(v, c)];
        const uint32_t ns = sample_count(rg.y - rg.x);
        if (!ns) continue;
        constexpr uint32_t nb = kHistBins;
        uint4 *gh4 = reinterpret_cast<uint4 *>(v.hist + v.hist_off[c]);
        const uint32_t below = v.pred[c];  // samples below L
        // thread t owns leaves [8t, 8t + 8) (none past nb)
        uint32_t h[8];
        if (8 * ti < nb) {
            const uint4 a = gh4[2 * ti], b = gh4[2 * ti + 1];
            h[0] = a.x; h[1] = a.y; h[2] = a.z; h[3] = a.w;
            h[4] = b.x; h[5] = b.y; h[6] = b.z; h[7] = b.w;
            gh4[2 * ti] = make_uint4(0u, 0u, 0u, 0u);
            gh4[2 * ti + 1] = make_uint4(0u, 0u, 0u, 0u);
        } else {
#pragma unroll
            for (int i = 0; i < 8; ++i) h[i] = 0u;
        }
        uint32_t run = 0;
#pragma unroll
        for (int i = 0; i < 8; ++i) run += h[i];
        uint32_t total, unused;
        const uint32_t pre = block_excl_scan2(run, 0u, s_red, &total, &unused).x;
        const float half = 0.5f * (float)ns, w = v.pred_sigmas * 0.5f * sqrtf((float)ns);
        const float r_lo = half - w, r_hi = half + w;
        // cum(j) = samples below edge e(j) = below + bins [0, j); count the edges j in [0, nb]
        // with cum(j) <= r_lo and with cum(j) < r_hi
        uint32_t n_le = 0, n_lt = 0, cum = below + pre;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const bool own = 8 * ti + i < nb;
            n_le += own && (float)cum <= r_lo;
            n_lt += own && (float)cum < r_hi;
            cum += h[i];
        }
        if (ti == 0) {
            n_le += (float)(below + total) <= r_lo;
            n_lt += (float)(below + total) < r_hi;
        }
        n_le = block_sum(n_le, s_red);
        n_lt = block_sum(n_lt, s_red);
        // lo: the last edge with at most r_lo samples below it; hi: the first with at least r_hi
        const uint32_t lo = n_le ? n_le - 1u : 0u, hi = min(n_lt, nb);
        if (ti == 0) {
            uint32_t p = 0u;
            if (n_le > 0 && lo < hi && (lo > 0 || hi < nb)) {
                p = lo | (hi << 12) | kPredValid;
                atomicAdd(&v.counters->pred_cells, 1u);
            }
            v.pred[c] = p;
        }
        __syncthreads();  // s_red reused by the next cell
    }
}

// Midpoints overflow in brackets with an end at or past 2^127: the cut is then infinite and not in
// its bracket, and its count is over all the cell's keys (none below -inf, those below +inf), which
// the bins do not hold.
__device__ __forceinline__ bool may_overflow(float L, float R) { return !(fmaxf(fabsf(L), fabsf(R)) < 0x1p127f); }
__device__ __forceinline__ bool overflowed(float cut) { return fabsf(cut) == __int_as_float(0x7f800000); }
// Keys (of [e0, e1)) below +inf, by the CTA. `sh` holds >= 32 words.
__device__ __noinline__ uint32_t finite_keys(const float *keys, uint32_t e0, uint32_t e1, uint32_t *sh) {
    uint32_t cnt = 0;
    for_keys(keys, e0, e1, [&](float k) { cnt += k < __int_as_float(0x7f800000); });
    return block_sum(cnt, sh);
}

// Up to K iterations of the reference loop (src/orbit.cpp:146-232) on the prefix counts pre[] of a
// midpoint tree's leaves over [L, R): leaf `pos` starts the new bracket. kWide: cuts can be infinite;
// `finite` is then the cell's keys below +inf, and the result false if one comes up while that is
// not known (~0).
template <bool kWide>
__device__ __forceinline__ bool replay(const uint32_t *pre, int K, uint32_t below, uint32_t n, float ratio,
                                       uint32_t finite, float &L, float &R, uint32_t &it, uint32_t &pos, uint8_t &st) {
    uint32_t width = 1u << K;
    for (int step = 0; step < K; ++step) {
        if (it >= (uint32_t)kMaxIterations) break;
        const uint32_t half = width >> 1;
        uint32_t cl = below + pre[pos + half];
        if (kWide && overflowed(mid_cut(L, R))) {
            if (finite == 0xffffffffu) return false;
            cl = mid_cut(L, R) > 0.f ? finite : 0u;
        }
        ++it;
        const int dir = convergence(cl, n, ratio);
        if (dir == 0) {
            st = kFound;
            break;
        }
        const float cut = mid_cut(L, R);
        if (dir > 0) {
            R = cut;
        } else {
            L = cut;
            pos += half;
        }
        width = half;
    }
    if (st == kActive && it >= (uint32_t)kMaxIterations) st = kCapped;
    return true;
}

// `finite` for the replay of cell c (described by hc; pre: its prefix counts), by the CTA, if a trial
// run by every thread meets an infinite cut.
__device__ __noinline__ uint32_t infinite_cut_count(const Level &v, int c, const HistCell *hc, const uint32_t *pre,
                                                    uint32_t *sh) {
    uint32_t finite = 0xffffffffu;
    const float ratio = leaf_ratio(v.heap[level_slot(v, c)].nLeafCells);
    float L = hc->L, R = hc->R;
    uint32_t it = v.iters[c], pos = 0;
    uint8_t st = kActive;
    if (!replay<true>(pre, kHistK, hc->whole ? hc->below : __ldcg(&v.below[c]), hc->end - hc->base, ratio, finite, L, R, it, pos, st))
        finite = finite_keys(hc->keys, hc->base, hc->end, sh);
    __syncthreads();  // every thread has read the cell
    return finite;
}

// Replay of up to 11 iterations of the reference loop (src/orbit.cpp:146-232) on the finished
// histogram of cell c, by the CTA that finished its last tile (every thread; hc describes the
// cell). The bins are read, cleared and turned into prefix counts in shared memory, so a step
// is one shared load and the float test. The cell then is found, capped, ready (its bracket's
// keys fit a list: the classify pass lists them, k_part_cells goes on) or active for the next
// pass. Fused here: as a kernel of its own behind every pass it took 9-10 us a launch, three
// times a level, most of it launch and load latency.
// kWide: midpoints can overflow (builds whose box reaches 2^127 have their own instances of the
// passes: the registers this takes made the others 0.7% slower).
template <uint32_t NT, bool kWide>
__device__ __noinline__ void resolve_cell(const Level &v, int c, const HistCell *hc, uint32_t *s_hist, uint32_t *s_red) {
    constexpr uint32_t kPer = kHistBins / NT;  // bins a thread
    static_assert(kPer == 2 || kPer == 4 || kPer == 8, "vector loads");
    const uint32_t tid = threadIdx.x;
    uint32_t h[kPer];
    using Vec = typename std::conditional<kPer == 2, uint2, uint4>::type;
    constexpr uint32_t kVecs = kPer * sizeof(uint32_t) / sizeof(Vec);
#pragma unroll
    for (uint32_t q = 0; q < kVecs; ++q) {
        Vec a;
        if (hc->whole) {
            a = reinterpret_cast<const Vec *>(s_hist)[kVecs * tid + q];
        } else {
            Vec *g = reinterpret_cast<Vec *>(hc->gh) + kVecs * tid + q;
            a = __ldcg(g);  // other CTAs' atomics: from L2
            *g = Vec{};
        }
        h[q * kPer / kVecs] = a.x;
        h[q * kPer / kVecs + 1] = a.y;
        if constexpr (kPer > 2) {
            h[q * 4 + 2] = a.z;
            h[q * 4 + 3] = a.w;
        }
    }
    uint32_t loc = 0;
#pragma unroll
    for (uint32_t j = 0; j < kPer; ++j) loc += h[j];
    uint32_t tot, unused;
    uint32_t run = block_excl_scan2(loc, 0u, s_red, &tot, &unused).x;
#pragma unroll
    for (uint32_t j = 0; j < kPer; ++j) {
        s_hist[kPer * tid + j] = run;
        run += h[j];
    }
    __syncthreads();
    const uint32_t finite = kWide ? infinite_cut_count(v, c, hc, s_hist, s_red) : 0xffffffffu;
    if (tid >= 32) return;  // one warp replays (identically in every lane)
    const int slot = level_slot(v, c);
    orb_cell_t &cell = v.heap[slot];
    const uint32_t n = hc->end - hc->base;
    const float ratio = leaf_ratio(cell.nLeafCells);  // src/orbit.cpp:204
    float L = hc->L, R = hc->R;
    uint32_t it = v.iters[c];
    const uint32_t below = hc->whole ? hc->below : __ldcg(&v.below[c]);
    const uint32_t pr = v.pass == 0 ? v.pred[c] : 0u;
    const bool warm = v.warm && v.warm[c];
    // a sampled or hinted bracket must hold the cut (see k_sample_bin, warm_bracket_holds);
    // else the pass is discarded and the next one bins the whole extent
    const bool pred_miss = (pr & kPredValid) && !(convergence(below, n, ratio) < 0 && convergence(below + tot, n, ratio) > 0);
    const bool warm_miss = warm && !warm_bracket_holds(below, below + tot, n, ratio);
    __syncwarp();
    if (pred_miss || warm_miss) {
        if (tid == 0) {
            if (pred_miss) atomicAdd(&v.counters->pred_misses, 1u);
            if (warm_miss) {
                warm_reset(cell, L, R, v.counters);
                v.warm[c] = 0;
            }
            v.inb[c] = n;
            v.below[c] = 0;
            v.hdone[c] = 0;
            v.counters->any_active[v.pass] = 1u;
        }
        return;
    }
    uint32_t pos = 0;
    uint8_t st = kActive;
    replay<kWide>(s_hist, kHistK, below, n, ratio, finite, L, R, it, pos, st);
    if (tid != 0) return;
    uint32_t inb = 0;
    bool inside = false;  // the later cuts lie in the bracket (where no midpoint can overflow)
    if (st == kActive) {
        // keys in the bracket the next step looks at, and keys below it
        inb = (pos + 1 < kHistBins ? s_hist[pos + 1] : tot) - s_hist[pos];
        inside = !(kWide && may_overflow(L, R));
        // Where the bracket's lowest and highest counts give the same answer, so does every cut in
        // it (the test is monotone in the count) and the loop ends without another count: many keys
        // on or beyond the box's end, whose bracket narrows towards that end.
        const int dir = convergence(below + s_hist[pos], n, ratio);
        if (inside && dir == convergence(below + s_hist[pos] + inb, n, ratio)) {
            while (st == kActive) {
                if (it >= (uint32_t)kMaxIterations) {
                    st = kCapped;
                    break;
                }
                ++it;
                if (dir == 0)
                    st = kFound;
                else if (dir > 0)
                    R = mid_cut(L, R);
                else
                    L = mid_cut(L, R);
            }
        }
    }
    cell.cutMarginLeft = L;
    cell.cutMarginRight = R;
    cell.foundCut = st == kFound ? 1 : 0;
    v.iters[c] = (uint8_t)it;
    v.hdone[c] = 0;
    if (warm) v.warm[c] = 0;
    if (st == kActive) {
        v.inb[c] = inb;
        if (inb <= list_capacity(v, n) && inside) {
            st = kReady;
            v.below[c] = below + s_hist[pos];
        } else {
            v.below[c] = 0;
            v.counters->any_active[v.pass] = 1u;
            // the last pass leaves no cell active (tree depth 11): flag it if one does
            if (v.pass == v.last_pass) atomicExch(&v.counters->error, 1u);
        }
    } else {
        atomicMax(&v.counters->max_iters, it);
        if (st == kCapped) atomicAdd(&v.counters->unfound, 1u);
    }
    v.state[c] = st;
}

// One count-left pass over the tiles of the level's active cells, a tile loop over all CTAs.
// A cell's keys are binned into a shared-memory histogram added to the cell's global bins.
// Each CTA takes a run of consecutive tiles (runs of equal length to one tile); a cell's
// shared bins and count below stay with the CTA while its tiles follow one another and are
// added to the global ones once per run; the CTA that brings a cell's last tile resolves it.
// Allowed: the modes this instance handles (the other paths are compiled out, which keeps
// each instance's streaming loop within its registers): kHFirstDense, the first pass of a
// cold level without sampled brackets (every cell dense); kHFirstSampled, the first pass of
// a sampled level (sampled or dense cells); kHRest, every other pass.
constexpr uint32_t kHFirstDense = kHDense;
constexpr uint32_t kHFirstSampled = kHDense | kHPred;
constexpr uint32_t kHRest = kHDense | kHBracket;
template <uint32_t Allowed, uint32_t NT, bool kWide = false>
__global__ void __launch_bounds__(NT, NT == kThreads ? kHistBlocksPerSm : (NT == 512 ? kHistBlocks512 : 1)) k_hist(const __grid_constant__ Level v) {
    pdl_enter();
    __shared__ __align__(16) uint32_t s_hist[kHistBins + 32];  // + the dense loop's spare bins
    __shared__ float s_edge[kHistBins + 1];                    // the tree's edges
    __shared__ uint32_t s_red[72];
    __shared__ HistCell s_hc;
    __shared__ uint32_t s_run[2];           // the CTA's tiles [first, end)
    __shared__ unsigned long long s_bytes;  // thread 0's count of bytes read
    if (v.pass == 0 && level_failed(v)) return;
    // every cell of the level finished in an earlier pass: nothing to bin
    if (v.pass > 0 && *(volatile uint32_t *)&v.counters->any_active[v.pass - 1] == 0u) return;
    if (threadIdx.x == 0) {
        const uint64_t total = v.tot->tiles >> 32;
        s_run[0] = (uint32_t)(total * blockIdx.x / gridDim.x);
        s_run[1] = (uint32_t)(total * (blockIdx.x + 1) / gridDim.x);
        s_bytes = 0;
    }
    __syncthreads();
    int cur = -1;         // the cell s_hc describes (every thread follows it)
    uint32_t ntiles = 0;  // the CTA's tiles of it so far
    uint32_t below = 0;   // this thread's keys below L in them
    bool by_edges = false;  // (dense) the warp's keys by their edges, see dense_tile
    // the current cell's count below L and its shared bins to the global ones; then, with the
    // cell's last tile, its replay
    auto end_cell = [&]() {
        below = block_sum(below, s_red);
        const uint32_t tiles = (s_hc.end - s_hc.base + (uint32_t)kTile - 1) / (uint32_t)kTile;
        const bool whole = ntiles == tiles;  // CTA-uniform: nothing to add up with other CTAs
        if (threadIdx.x == 0) {
            const uint32_t tot = below + s_hc.below;
            s_hc.whole = s_hc.last = whole ? 1u : 0u;
            s_hc.below = tot;
            if (tot && !whole) atomicAdd(&v.below[cur], tot);
        }
        if (!whole) {
            uint32_t *gh = s_hc.gh;
            for (uint32_t b = threadIdx.x; b < kHistBins; b += NT) {
                const uint32_t h = s_hist[b];
                if (h) atomicAdd(&gh[b], h);
            }
            __syncthreads();
            if (threadIdx.x == 0) {
                s_hc.last = arrive_release(&v.hdone[cur], ntiles) + ntiles == tiles;
                if (s_hc.last) acquire();
            }
        }
        __syncthreads();
        if (s_hc.last) resolve_cell<NT, kWide>(v, cur, &s_hc, s_hist, s_red);
        __syncthreads();  // s_hc and s_hist free for the next cell
        below = 0;
        ntiles = 0;
    };
    const uint32_t t_end = s_run[1];
    auto tile_cell = [&](uint32_t t) { return t < t_end ? (int)v.htile_cell[t] : -1; };
    int c_next = tile_cell(s_run[0]);
    int skip_c = -1;  // an inactive cell whose tiles are being passed over
    for (uint32_t t = s_run[0]; t < t_end; ++t) {
        const int c = c_next;
        c_next = tile_cell(t + 1);  // the next tile's cell, loaded while this tile is read
        if (c == skip_c) continue;
        if (c != cur) {
            // a cell with a tile still to come is not resolved in this pass, so its state
            // stands while this CTA reads it
            if (v.state[c] != kActive) {  // the run's tiles of a cell are consecutive
                skip_c = c;
                continue;
            }
            if (cur >= 0) end_cell();
            cur = c;
            by_edges = false;
            if (threadIdx.x == 0) {
                const int slot = level_slot(v, c);
                const orb_cell_t &cell = v.heap[slot];
                const uint2 rg = v.ranges[slot];
                const float L = cell.cutMarginLeft, R = cell.cutMarginRight;
                const uint32_t pr = (Allowed & kHPred) ? v.pred[c] : 0u;
                uint32_t mode = kHDense;
                if (pr & kPredValid)
                    mode = kHPred;
                else if ((Allowed & kHBracket) && v.inb[c] != rg.y - rg.x)
                    mode = kHBracket;
                s_hc.keys = axis_keys(v, eff_axis(cell.cutAxis));
                s_hc.gh = v.hist + v.hist_off[c];
                s_hc.L = L;
                s_hc.R = R;
                s_hc.mode = mode;
                s_hc.base = rg.x;
                s_hc.end = rg.y;
                s_hc.t0 = v.tile_off[c];
                s_hc.below = 0;
                s_hc.pa = pr & kPredValid ? tree_edge(L, R, kHistK, pred_lo(pr)) : L;
                s_hc.pb = pr & kPredValid ? tree_edge(L, R, kHistK, pred_hi(pr)) : R;
                s_hc.gs = make_guess(L, R, __fdiv_rn((float)kHistBins, __fsub_rn(R, L)), kHistBins);
            }
            __syncthreads();
            for (uint32_t j = threadIdx.x; j < kHistBins; j += NT) s_hist[j] = 0u;
            fill_edges(s_edge, s_hc.L, s_hc.R, kHistK, threadIdx.x, NT);
            __syncthreads();
        }
        ++ntiles;
        const uint32_t mode = s_hc.mode;
        const uint32_t e0 = s_hc.base + (t - s_hc.t0) * (uint32_t)kTile;
        const uint32_t e1 = min(s_hc.end, e0 + (uint32_t)kTile);
        const float *keys = s_hc.keys;
        if ((Allowed & kHPred) && (mode & kHPred)) {
            // sampled bracket [pa, pb): keys below it counted, keys inside it (a few percent)
            // binned afterwards, keys above it and NaN ignored
            const float pa = s_hc.pa, pb = s_hc.pb;
            auto key = [&](float k) { pred_key(k, &s_hc, s_hist, s_edge); };
            scan_tile<NT>(
                keys, e0, e1, s_hc.R,
                [&](float k) {
                    below += k < pa;
                    return !(k >= pa && k < pb);
                },
                key,
                [&](float k) {
                    if (k < pa)
                        ++below;
                    else if (k < pb)
                        key(k);
                });
        } else if ((Allowed & kHBracket) && (mode & kHBracket)) {
            bracket_tile<NT>(keys, e0, e1, s_hc.gs, s_hc.L, s_hc.R, below, s_hist, s_edge);
        } else {
            // every key by the scaled guess (no range test: guess_bin fails keys outside
            // [L, R) and NaN, which dense_exact then counts or ignores)
            dense_tile<NT>(keys, e0, e1, s_hc.gs, s_hist, &s_hc, s_edge, below, by_edges);
        }
        if (threadIdx.x == 0) s_bytes += 4ull * (e1 - e0);
    }
    if (cur >= 0) end_cell();
    if (threadIdx.x == 0 && s_bytes) add_bytes(v, kKHist, s_bytes);
}

// ------------------------------------------------------------------------------------
// Bisection of small cells (at most kWarpKeys keys): one warp per cell, the whole reference
// loop (src/orbit.cpp:146-232) in one launch.
// ------------------------------------------------------------------------------------
constexpr int kWarpKeysPerLane = kWarpKeys / 32;

// Bisection of a small cell (at most kWarpKeys keys) by one warp: the keys held in registers,
// every iteration of the reference loop (src/orbit.cpp:146-232) a register count plus a
// warp reduction.
__device__ __forceinline__ void bisect_small(const Level &v, int c, uint32_t lane) {
    const int slot = level_slot(v, c);
    orb_cell_t &cell = v.heap[slot];
    const uint2 rg = v.ranges[slot];
    const uint32_t n = rg.y - rg.x;
    const float ratio = leaf_ratio(cell.nLeafCells);  // src/orbit.cpp:204
    const float *keys = axis_keys(v, eff_axis(cell.cutAxis));
    float k[kWarpKeysPerLane];
#pragma unroll
    for (int j = 0; j < kWarpKeysPerLane; ++j) {
        const uint32_t i = (uint32_t)(j * 32 + lane);
        k[j] = i < n ? __ldg(keys + rg.x + i) : __int_as_float(0x7fc00000);  // NaN: never below
    }
    float L = cell.cutMarginLeft, R = cell.cutMarginRight;
    if (v.warm && v.warm[c]) {
        // hinted bracket: keep it only if it holds the target
        uint32_t bl = 0, br = 0;
#pragma unroll
        for (int j = 0; j < kWarpKeysPerLane; ++j) {
            bl += k[j] < L;
            br += k[j] < R;
        }
        if (!warm_bracket_holds(warp_sum(bl), warp_sum(br), n, ratio)) {
            const int a = eff_axis(cell.cutAxis);
            L = cell.lower[a];
            R = cell.upper[a];
            if (lane == 0) atomicAdd(&v.counters->warm_resets, 1u);
        }
        if (lane == 0) v.warm[c] = 0;
    }
    uint32_t it = 0;
    uint8_t st = kActive;
    while (st == kActive) {
        if (it >= (uint32_t)kMaxIterations) {
            st = kCapped;
            break;
        }
        const float cut = mid_cut(L, R);
        uint32_t cnt = 0;
#pragma unroll
        for (int j = 0; j < kWarpKeysPerLane; ++j) cnt += k[j] < cut;
        cnt = warp_sum(cnt);
        ++it;
        const int dir = convergence(cnt, n, ratio);
        if (dir == 0)
            st = kFound;
        else if (dir > 0)
            R = cut;
        else
            L = cut;
    }
    if (lane == 0) {
        cell.cutMarginLeft = L;
        cell.cutMarginRight = R;
        cell.foundCut = st == kFound ? 1 : 0;
        v.iters[c] = (uint8_t)it;
        v.state[c] = st;
        atomicMax(&v.counters->max_iters, it);
        if (st == kCapped) atomicAdd(&v.counters->unfound, 1u);
        add_bytes(v, kKBisectTile, 4ull * n);  // the launch that bisects it
    }
}

// A warp a cell. (Cells of up to a whole tile took this kernel before, in histogram rounds of a
// warp: 36-42 us a cell of 2^14 keys, 1.3 of the 11 ms of a batch of 128 instances; a CTA of the
// count passes takes about 7.)
__global__ void __launch_bounds__(kThreads, kTileBlocksPerSm) k_bisect_tile(const __grid_constant__ Level v) {
    pdl_enter();
    if (level_failed(v)) return;
    const uint32_t lane = threadIdx.x & 31;
    const int nwarps = (int)(gridDim.x * (blockDim.x >> 5));
    for (int c = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5); c < v.C; c += nwarps)
        if (v.state[c] == kSmall) bisect_small(v, c, lane);
}

// ------------------------------------------------------------------------------------
// Bisection with one CTA per cell, for levels with many cells (no multi-CTA passes, no
// global histograms, no host round trip). Every round bins the candidate keys of the cell
// into a shared-memory midpoint tree and replays up to K iterations of the reference loop
// (src/orbit.cpp:146-232) on it; then the keys of the remaining bracket become the
// candidates of the next round. Candidates start as the cell's keys in global memory, or
// in the shared list when they fit; as soon as the bracket fits the list it is compacted
// into it. `base` counts the keys already known to lie below L. Same cuts, same integer
// counts, same float test as the reference.
// ------------------------------------------------------------------------------------
constexpr int kCtaThreads = 512;
constexpr uint32_t kListCap = 8192;                     // shared list of candidate keys
constexpr uint32_t kListPerThread = kListCap / kCtaThreads;
constexpr size_t kCtaSmemBytes = kListCap * sizeof(float) +
                                 (1u << kMaxBinsLog2) * sizeof(uint32_t) +
                                 ((1u << kMaxBinsLog2) + 1) * sizeof(float);

__global__ void __launch_bounds__(kCtaThreads) k_bisect_cta(const __grid_constant__ Level v) {
    pdl_enter();
    if (level_failed(v)) return;
    extern __shared__ __align__(16) unsigned char cta_smem[];
    float *list = reinterpret_cast<float *>(cta_smem);
    uint32_t *s_hist = reinterpret_cast<uint32_t *>(list + kListCap);
    float *s_edge = reinterpret_cast<float *>(s_hist + (1u << kMaxBinsLog2));
    __shared__ uint32_t sh[96];
    __shared__ uint32_t s_fill;
    const uint32_t tid = threadIdx.x;
    constexpr uint32_t kBins = 1u << kMaxBinsLog2;
    for (int c = blockIdx.x; c < v.C; c += gridDim.x) {
        const int slot = level_slot(v, c);
        orb_cell_t &cell = v.heap[slot];
        const uint2 rg = v.ranges[slot];
        const uint32_t n = rg.y - rg.x;
        const float ratio = leaf_ratio(cell.nLeafCells);  // src/orbit.cpp:204
        const float *keys = axis_keys(v, eff_axis(cell.cutAxis));
        float L = cell.cutMarginLeft, R = cell.cutMarginRight;
        uint32_t it = 0, base = 0, m = n, inb = n, finite = 0xffffffffu;
        uint8_t st = kActive;
        bool in_list = n <= kListCap;
        unsigned long long bytes = 0;
        if (in_list) {
            for (uint32_t i = tid; i < n; i += blockDim.x) list[i] = __ldg(keys + rg.x + i);
            bytes += 4ull * n;
        }
        for (;;) {
            // ---- histogram round over the candidates, tree depth from their count
            const uint32_t cand = in_list ? m : inb;
            const int K = max(1, min(kMaxBinsLog2, 32 - __clz(max(cand, 1u))));
            const uint32_t nb = 1u << K;
            for (uint32_t j = tid; j < kBins; j += blockDim.x) s_hist[j] = 0u;
            fill_edges(s_edge, L, R, K, tid, blockDim.x);
            __syncthreads();
            const float scale = __fdividef((float)nb, R - L);
            uint32_t below = 0;
            auto visit = [&](float k) {
                if (k < L) {
                    ++below;
                } else if (k < R) {
                    const int g = edge_bin(k, L, scale, (int)nb - 1, [&](int j) { return s_edge[j]; });
                    atomicAdd(&s_hist[g], 1u);
                }
            };
            if (in_list) {
                for (uint32_t i = tid; i < m; i += blockDim.x) visit(list[i]);
            } else {
                for_keys(keys, rg.x, rg.y, visit);
                bytes += 4ull * n;
            }
            below = base + block_sum(below, sh);
            // exclusive prefix of the bins in place (4 bins per thread)
            uint32_t h4[4], loc = 0;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                h4[q] = s_hist[tid * 4 + q];
                loc += h4[q];
            }
            uint32_t tot_a, tot_b;
            const uint2 ex = block_excl_scan2(loc, 0u, sh, &tot_a, &tot_b);
            uint32_t run = ex.x;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                s_hist[tid * 4 + q] = run;
                run += h4[q];
            }
            __syncthreads();
            // ---- replay up to K iterations (identically in every thread)
            uint32_t pos = 0;
            float l = L, r = R;
            uint32_t i0 = it;
            if (!replay<true>(s_hist, K, below, n, ratio, finite, l, r, i0, pos, st)) {
                finite = finite_keys(keys, rg.x, rg.y, sh);
                bytes += 4ull * n;
                l = L, r = R, i0 = it, pos = 0, st = kActive;
                replay<true>(s_hist, K, below, n, ratio, finite, l, r, i0, pos, st);
            }
            L = l;
            R = r;
            it = i0;
            if (st != kActive) break;
            // keys in the new bracket [L, R) (entry nb of the prefix is the round's total)
            inb = (pos + 1 < nb ? s_hist[pos + 1] : tot_a) - s_hist[pos];
            __syncthreads();
            // ---- the new bracket's keys become the candidates
            if (in_list) {
                // every thread reads its keys, then (after the barrier in block_sum) the
                // keys of the new bracket are appended, one warp-aggregated slot per round
                float kq[kListPerThread];
                uint32_t blw = 0;
#pragma unroll
                for (uint32_t q = 0; q < kListPerThread; ++q) {
                    const uint32_t i = tid + q * kCtaThreads;
                    kq[q] = i < m ? list[i] : R;  // R: neither below L nor kept
                    blw += kq[q] < L;
                }
                if (tid == 0) s_fill = 0;
                base += block_sum(blw, sh);
                const uint32_t lane = tid & 31;
#pragma unroll
                for (uint32_t q = 0; q < kListPerThread; ++q) {
                    const bool keep = !(kq[q] < L) && kq[q] < R;
                    const uint32_t bal = __ballot_sync(0xffffffffu, keep);
                    uint32_t wb = 0;
                    if (lane == 0 && bal) wb = atomicAdd(&s_fill, (uint32_t)__popc(bal));
                    wb = __shfl_sync(0xffffffffu, wb, 0);
                    if (keep) list[wb + __popc(bal & ((1u << lane) - 1u))] = kq[q];
                }
                __syncthreads();
                m = s_fill;
            } else if (inb <= kListCap) {
                if (tid == 0) s_fill = 0;
                __syncthreads();
                uint32_t blw = 0;
                for_keys(keys, rg.x, rg.y, [&](float k) {
                    if (k < L)
                        ++blw;
                    else if (k < R) {
                        const uint32_t q = atomicAdd(&s_fill, 1u);
                        if (q < kListCap) list[q] = k;
                    }
                });
                bytes += 4ull * n;
                base = block_sum(blw, sh);
                m = min(s_fill, kListCap);
                in_list = true;
            }
            __syncthreads();
        }
        if (tid == 0) {
            cell.cutMarginLeft = L;
            cell.cutMarginRight = R;
            cell.foundCut = st == kFound ? 1 : 0;
            v.iters[c] = (uint8_t)it;
            v.state[c] = st;
            atomicMax(&v.counters->max_iters, it);
            if (st == kCapped) atomicAdd(&v.counters->unfound, 1u);
            add_bytes(v, kKBisectCta, bytes);
        }
        __syncthreads();
    }
}

// ------------------------------------------------------------------------------------
// Partition
//
// Partition tiles are kPTile consecutive positions of one cell. Per tile, the classify
// pass stores two bitmasks (key >= cut, key <= cut) and their counts; k_part_cells turns the
// counts into prefixes within the cell and finds s and the split index i, and a CTA per tile
// performs the swaps of the pairs whose left element lies in that tile.
// ------------------------------------------------------------------------------------
__device__ __forceinline__ float cell_cut(const orb_cell_t &c) {
    return mid_cut(c.cutMarginLeft, c.cutMarginRight);
}

// The next float above c (NaN for NaN and +inf, above which no key lies): k >= next_above(c)
// exactly when k > c.
__device__ __forceinline__ float next_above(float c) {
    const int32_t b = __float_as_int(c);
    if (!(c < __int_as_float(0x7f800000))) return __int_as_float(0x7fc00000);
    if (c == 0.0f) return __int_as_float(1);
    return __int_as_float(b > 0 ? b + 1 : b - 1);
}

// P1: bitmasks of keys >= cut and keys <= cut per partition tile, and their counts.
// One warp per tile: the metadata chains (tile -> cell -> range, cut) of the CTA's warps
// overlap, and each lane keeps kClassifyLoads loads in flight. The mask words are staged in
// shared memory and stored coalesced.
// A cell with a final cut is classified against it. A kReady cell's cut lies in its bracket
// [L, R): keys below L are <= cut, keys at or above R are >= cut (and not <=, unless the cut
// comes out as R itself: k_part_cells then classifies the cell again), NaN is both, and the
// keys in between (a few in a thousand) go to the cell's list. So the pass that would only
// count the bracket's keys and the pass over the final cut are one read of the keys. With
// a = k >= lo and b = k < hi, both kinds are le = !a, ge = !b, listed = a and b: a final cut
// takes hi = cut and lo = the next float above it, which leaves no listed key.
constexpr int kClassifyLoads = 16;
constexpr uint32_t kListStage = 128;  // listed keys a warp stages before it appends them

// kParts: warps a tile (consecutive ones of a CTA, each a run of its words). 4 on levels of few
// tiles, where one warp's eight rounds of loads are all the launch lasts.
template <int kParts>
__global__ void __launch_bounds__(kThreads) k_part_classify(const __grid_constant__ Level v) {
    pdl_enter();
    if (blockIdx.x == 0 && threadIdx.x < 4) {
        // the next level's plan and count passes start from zero (neither is in use now)
        v.counters->any_active[threadIdx.x] = 0u;
        if (threadIdx.x == 0 && v.tot_next) {
            v.tot_next->tiles = 0ull;
            v.tot_next->pools = 0ull;
            v.tot_next->swaps = 0u;
        }
    }
    if (level_late(v)) return;  // (an error found meanwhile stops the next kernel)
    __shared__ uint32_t s_words[kThreads / 32][2][kPWords];
    __shared__ float s_lkey[kThreads / 32][kListStage];
    __shared__ uint32_t s_lpos[kThreads / 32][kListStage];
    const uint64_t total = (uint32_t)v.tot->tiles;
    const int lane = threadIdx.x & 31;
    uint32_t(*sw)[kPWords] = s_words[threadIdx.x >> 5];
    float *lkey = s_lkey[threadIdx.x >> 5];
    uint32_t *lpos = s_lpos[threadIdx.x >> 5];
    constexpr int kWords = kPWords / kParts;  // mask words of a warp's part of a tile
    const int part = kParts > 1 ? (int)(threadIdx.x >> 5) % kParts : 0, w_at = part * kWords;
    __shared__ uint32_t s_cnt[kThreads / 32][2];
    const uint32_t nwarps = gridDim.x * (kThreads / 32 / kParts), warp = (blockIdx.x * kThreads + threadIdx.x) / (32 * kParts);
    unsigned long long bytes = 0;
    // a run of consecutive tiles a warp: a cell's bracket and its staged keys stay with it
    const uint32_t t_end = (uint32_t)(total * (warp + 1) / nwarps);
    int c = -1;
    uint32_t t0 = 0, nl = 0;  // nl: staged listed keys of cell c
    float lo = 0.f, hi = 0.f;
    const float *keys = nullptr;
    uint2 rg = make_uint2(0u, 0u);
    auto flush = [&]() {
        __syncwarp();
        uint32_t base = 0;
        if (lane == 0) base = atomicAdd(&v.cmp_cnt[c], nl);
        base = __shfl_sync(0xffffffffu, base, 0);
        // (the count pass saw to it that they fit)
        if (base + nl > list_capacity(v, rg.y - rg.x)) {
            if (lane == 0) atomicExch(&v.counters->error, 1u);
        } else {
            base += v.cmp_off[c];
            for (uint32_t j = lane; j < nl; j += 32) {
                v.cmp_keys[base + j] = lkey[j];
                v.cmp_pos[base + j] = lpos[j];
            }
        }
        __syncwarp();
        nl = 0;
    };
    for (uint32_t t = (uint32_t)(total * warp / nwarps); t < t_end; ++t) {
        const int ct = (int)v.ptile_cell[t];
        if (ct != c) {
            if (nl) flush();
            c = ct;
            t0 = v.ptile_off[c];
            const int slot = level_slot(v, c);
            const orb_cell_t &cell = v.heap[slot];
            const bool ready = v.state[c] == kReady;
            const float cut = cell_cut(cell);
            lo = ready ? cell.cutMarginLeft : next_above(cut);
            hi = ready ? cell.cutMarginRight : cut;
            keys = axis_keys(v, eff_axis(cell.cutAxis));
            rg = v.ranges[slot];
        }
        const uint32_t p0 = rg.x + (t - t0) * (uint32_t)kPTile;
        const uint32_t m = min((uint32_t)kPTile, rg.y - p0);
        uint32_t cg = 0, cl = 0;
        // the words of kClassifyLoads loads a lane; a full tile needs no bounds
        auto round = [&](int r, auto full) {
            constexpr bool kFull = decltype(full)::value;
            float k[kClassifyLoads];
#pragma unroll
            for (int u = 0; u < kClassifyLoads; ++u) {
                const uint32_t i = (uint32_t)(r + u) * 32u + lane;
                k[u] = kFull || i < m ? __ldg(keys + p0 + i) : 0.0f;
            }
            uint32_t listed = 0;  // words of this round with listed keys
#pragma unroll
            for (int u = 0; u < kClassifyLoads; ++u) {
                const uint32_t w0 = (uint32_t)(r + u) * 32u;  // the word's first position
                uint32_t vm = 0xffffffffu;
                if (!kFull) vm = w0 + 32u <= m ? vm : (w0 < m ? (1u << (m - w0)) - 1u : 0u);
                const uint32_t gb = __ballot_sync(0xffffffffu, !(k[u] < hi)) & vm;
                const uint32_t lb = __ballot_sync(0xffffffffu, !(k[u] >= lo)) & vm;
                if (lane == u) {
                    sw[0][r + u] = gb;
                    sw[1][r + u] = lb;
                }
                cg += __popc(gb);
                cl += __popc(lb);
                if ((gb | lb) != vm) listed |= 1u << u;
            }
            while (listed) {  // warp-uniform
                const int u = __ffs(listed) - 1;
                listed &= listed - 1;
                const uint32_t i = (uint32_t)(r + u) * 32u + lane;
                const float kk = i < m ? __ldg(keys + p0 + i) : hi;
                const bool in = kk >= lo && kk < hi;
                const uint32_t ib = __ballot_sync(0xffffffffu, in);
                if (nl + 32 > kListStage) flush();
                if (in) {
                    const uint32_t q = nl + __popc(ib & ((1u << lane) - 1u));
                    lkey[q] = kk;
                    lpos[q] = p0 + i;
                }
                nl += __popc(ib);
            }
        };
        if (m == (uint32_t)kPTile) {
#pragma unroll 1
            for (int r = w_at; r < w_at + kWords; r += kClassifyLoads) round(r, Flag<true>());
        } else {
#pragma unroll 1
            for (int r = w_at; r < w_at + kWords; r += kClassifyLoads) round(r, Flag<false>());
        }
        uint32_t *gw = v.ge_bits + (size_t)t * kPWords;
        uint32_t *lw = v.le_bits + (size_t)t * kPWords;
        __syncwarp();
#pragma unroll
        for (int q = 0; q < kWords / 32; ++q) {
            gw[w_at + q * 32 + lane] = sw[0][w_at + q * 32 + lane];
            lw[w_at + q * 32 + lane] = sw[1][w_at + q * 32 + lane];
        }
        __syncwarp();
        if constexpr (kParts > 1) {
            // the parts' counts (the tile's warps walk the same tiles)
            const int bar = 1 + (int)(threadIdx.x / (32 * kParts)), w0 = (int)(threadIdx.x >> 5) - part;
            if (lane == 0) {
                s_cnt[threadIdx.x >> 5][0] = cg;
                s_cnt[threadIdx.x >> 5][1] = cl;
            }
            asm volatile("bar.sync %0, %1;" ::"r"(bar), "n"(32 * kParts) : "memory");
            cg = cl = 0;
            for (int q = 0; q < kParts; ++q) {
                cg += s_cnt[w0 + q][0];
                cl += s_cnt[w0 + q][1];
            }
            asm volatile("bar.sync %0, %1;" ::"r"(bar), "n"(32 * kParts) : "memory");
        }
        if (lane == 0 && part == 0) {
            v.pt_ge[t] = cg;
            v.pt_le[t] = cl;
            bytes += 4ull * m + 8ull * kPWords + 8ull;
        }
    }
    if (nl) flush();
    if (lane == 0 && bytes) add_bytes(v, kKPartClassify, bytes);
}

// Position of the bit of rank r (0-based) in w (r < popc(w)).
__device__ __forceinline__ uint32_t select_in_word(uint32_t w, uint32_t r) {
    uint32_t pos = 0;
#pragma unroll
    for (int step = 16; step >= 1; step >>= 1) {
        const uint32_t c = (uint32_t)__popc(w & ((1u << step) - 1u));
        if (r >= c) {
            r -= c;
            w >>= step;
            pos += (uint32_t)step;
        }
    }
    return pos;
}

// Largest u in [lo, hi] with pre[u] <= r, for a nondecreasing pre with pre[lo] <= r: a 32-way
// search (every lane probes one point per round, the passing probes are a prefix of the
// lanes), three rounds for 2^15 candidates. Warp-uniform result.
__device__ __forceinline__ uint32_t warp_last_at_most(const uint32_t *pre, uint32_t lo, uint32_t hi,
                                                      uint32_t r) {
    const uint32_t lane = threadIdx.x & 31;
    while (lo < hi) {
        const uint32_t step = (hi - lo + 31) / 32;
        const uint32_t u = lo + (lane + 1) * step;
        const bool ok = u <= hi && pre[u] <= r;
        const uint32_t cnt = (uint32_t)__popc(__ballot_sync(0xffffffffu, ok));
        lo += cnt * step;
        hi = min(hi, lo + step - 1);
    }
    return lo;
}

// Largest u in [lo, hi] with pre[u] <= r for two arrays at once, each as in warp_last_at_most:
// the loads of a round are in flight together.
__device__ __forceinline__ uint2 warp_last_at_most2(const uint32_t *pa, const uint32_t *pb, uint32_t lo, uint32_t hi,
                                                    uint32_t ra, uint32_t rb) {
    const uint32_t lane = threadIdx.x & 31;
    uint2 l = make_uint2(lo, lo), h = make_uint2(hi, hi);
    while (l.x < h.x || l.y < h.y) {
        const uint32_t sa = (h.x - l.x + 31) / 32, sb = (h.y - l.y + 31) / 32;
        const uint32_t ua = l.x + (lane + 1) * sa, ub = l.y + (lane + 1) * sb;
        const uint32_t va = sa && ua <= h.x ? pa[ua] : 0xffffffffu, vb = sb && ub <= h.y ? pb[ub] : 0xffffffffu;
        const bool oka = sa && ua <= h.x && va <= ra, okb = sb && ub <= h.y && vb <= rb;
        l.x += (uint32_t)__popc(__ballot_sync(0xffffffffu, oka)) * sa;
        l.y += (uint32_t)__popc(__ballot_sync(0xffffffffu, okb)) * sb;
        if (sa) h.x = min(h.x, l.x + sa - 1);
        if (sb) h.y = min(h.y, l.y + sb - 1);
    }
    return l;
}

// The smaller position (cell-relative; ~0: none) of two set bits among the masks of tiles
// [t0, t1): the one of in-cell rank rg of the >= masks (if g), of rank rl of the <= masks (if l).
// Warp-cooperative; every lane returns the answer. The masks are read from L2 (atomics may have
// set bits). Both searches step by step together: one after the other they were a quarter of
// k_part_cells' chain on levels of few cells.
__device__ uint32_t warp_select2(const Level &v, uint32_t t0, uint32_t t1, bool g, uint32_t rg, bool l, uint32_t rl) {
    const uint32_t lane = threadIdx.x & 31;
    const uint2 at = warp_last_at_most2(v.pt_ge_pre, v.pt_le_pre, t0, t1 - 1, g ? rg : 0u, l ? rl : 0u);
    static_assert(kPWords == 128, "four mask words a lane");
    const uint4 qg = __ldcg(reinterpret_cast<const uint4 *>(v.ge_bits + (size_t)at.x * kPWords) + lane);
    const uint4 ql = __ldcg(reinterpret_cast<const uint4 *>(v.le_bits + (size_t)at.y * kPWords) + lane);
    const uint32_t r[2] = {rg - v.pt_ge_pre[at.x], rl - v.pt_le_pre[at.y]}, tile[2] = {at.x, at.y};
    const uint32_t words[2][4] = {{qg.x, qg.y, qg.z, qg.w}, {ql.x, ql.y, ql.z, ql.w}};
    uint32_t pos = 0xffffffffu;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        uint32_t cnt = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) cnt += __popc(words[k][j]);
        uint32_t tot;
        const uint32_t ex = warp_excl_scan(cnt, &tot);
        if ((k ? l : g) && r[k] >= ex && r[k] < ex + cnt) {
            uint32_t rr = r[k] - ex;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint32_t pc = __popc(words[k][j]);
                if (rr < pc) {
                    pos = min(pos, (tile[k] - t0) * (uint32_t)kPTile + (lane * 4 + (uint32_t)j) * 32u +
                                       select_in_word(words[k][j], rr));
                    break;
                }
                rr -= pc;
            }
        }
    }
    return __reduce_min_sync(0xffffffffu, pos);
}

// By a warp, a lane an array (y or z null: that array is not moved at this level; builds from host
// memory reorder it later through the permutation, see orb_build). Read from L2: in the swap
// kernel other CTAs wrote these particles.
__device__ __forceinline__ void swap_particles(const Level &v, uint32_t a, uint32_t b, uint32_t lane) {
    uint32_t *p = nullptr;
    if (lane == 0) p = reinterpret_cast<uint32_t *>(v.x);
    if (lane == 1) p = reinterpret_cast<uint32_t *>(v.y);
    if (lane == 2) p = reinterpret_cast<uint32_t *>(v.z);
    if (lane == 3) p = v.idx;
    if (lane == 4) p = v.wt;
    if (!p) return;
    const uint32_t xa = __ldcg(p + a), xb = __ldcg(p + b);
    p[a] = xb;
    p[b] = xa;
}

__device__ void set_axis_and_margin(orb_cell_t &c, BuildCounters *ctr) {
    // setCutAxis (src/cell.h:102-121) then setCutMargin (src/cell.h:123-126)
    int max_d = -1;
    float max_size = 0.0f;
    for (int k = 0; k < 3; ++k) {
        const float size = __fsub_rn(c.upper[k], c.lower[k]);
        if (size > max_size) {
            max_size = size;
            max_d = k;
        }
    }
    c.cutAxis = max_d;
    if (max_d < 0) atomicAdd(&ctr->zero_volume, 1u);
    const int a = eff_axis(max_d);
    c.cutMarginLeft = c.lower[a];
    c.cutMarginRight = c.upper[a];
}

// Child q of a cell at its cut: Cell::cut (src/cell.h:78-100) and src/orbit.cpp:238-246.
__device__ __forceinline__ void split_child(const orb_cell_t &cell, int q, orb_cell_t &kid, BuildCounters *ctr) {
    const float cut = cell_cut(cell);
    const int a = eff_axis(cell.cutAxis);
    const int n_left = (cell.nLeafCells + 1) / 2;
    kid.id = 2 * cell.id + 1 + q;
    kid.nLeafCells = q ? cell.nLeafCells - n_left : n_left;
    kid.prevCutAxis = cell.cutAxis;
    kid.foundCut = 0;
    kid.pad_[0] = kid.pad_[1] = kid.pad_[2] = 0;
    for (int k = 0; k < 3; ++k) {
        kid.lower[k] = k == a && q ? cut : cell.lower[k];
        kid.upper[k] = k == a && !q ? cut : cell.upper[k];
    }
    set_axis_and_margin(kid, ctr);
}

// What finishing cell c reads besides its split point; the swap's CTAs load it before their
// last arrival (it does not change while the level's particles move).
struct FinishIn {
    orb_cell_t cell;
    int slot;
    int map;  // where the children stand in the next level (see Level::child_map)
};
__device__ __forceinline__ FinishIn finish_in(const Level &v, int c) {
    FinishIn f;
    f.slot = level_slot(v, c);
    f.cell = v.heap[f.slot];
    f.map = !v.next_C ? 0
            : v.child_map ? v.child_map[c]
                          : 8 * c + (2 * c < v.next_C ? 1 : 0) + (2 * c + 1 < v.next_C ? 2 : 0);
    return f;
}

// One warp: the final swap(i, n-1) of partitioned cell c of the level
// (src/services/partition.cpp:52), its children's ranges, (optionally) their cells, and their
// plan for the next level, lane q for child q. One chain of dependent accesses, which a level of
// few cells waits for: both children's shares of the level's totals in one atomic each, issued
// ahead of the swap's loads (one thread doing all of it, an access after the other, took 6 us).
struct Kids {
    PlanCell p[2];
};
__device__ __noinline__ void finish_and_plan(const Level &v, const FinishIn &f, const CellPart &P, bool do_split, Kids &out) {
    const uint32_t lane = threadIdx.x & 31u, n = P.n, i = P.i;
    const int q = (int)(lane & 1u);
    const uint32_t nq = q ? n - i : i;
    PlanCell p = plan_sizes(v.small_next, (f.map >> q) & 1 ? (f.map >> 2) + q : -1, nq);
    const unsigned long long ti = plan_tiles(p), po = plan_pools(v, p, nq);
    const unsigned long long t0 = __shfl_sync(0xffffffffu, ti, 0), p0 = __shfl_sync(0xffffffffu, po, 0);
    const unsigned long long ts = t0 + __shfl_sync(0xffffffffu, ti, 1), ps = p0 + __shfl_sync(0xffffffffu, po, 1);
    unsigned long long at = 0;
    if (lane == 0 && ts) at = atomicAdd(&v.tot_next->tiles, ts);
    if (lane == 1 && ps) at = atomicAdd(&v.tot_next->pools, ps);
    if (i < n) {
        if (i != n - 1) swap_particles(v, P.b + i, P.b + n - 1, lane);
    } else if (lane == 0) {
        atomicAdd(&v.counters->degenerate, 1u);
    }
    // children slots: slot - id is the instance's heap base
    const int slot = f.slot + f.cell.id + 1 + q;
    if (lane < 2) {
        v.ranges[slot] = make_uint2(P.b + (q ? i : 0u), P.b + (q ? n : i));
        if (do_split) {
            orb_cell_t kid;
            split_child(f.cell, q, kid, v.counters);
            v.heap[slot] = kid;
        }
    }
    const unsigned long long a = __shfl_sync(0xffffffffu, at, 0) + (q ? t0 : 0ull);
    const unsigned long long b = __shfl_sync(0xffffffffu, at, 1) + (q ? p0 : 0ull);
    if (lane < 2) {
        if (p.c >= 0) plan_store(v, p, a, b, v.small_next, slot, nq);
        out.p[q] = p;
        if (lane == 0) atomicAdd(&v.counters->done[v.depth], 1u);
    }
    __syncwarp();
}

// P2: per cell: the bisection of a kReady cell finished on its list, the tile prefixes, the
// swap count s and the split index i.
//   s = max_x min(f(x), g(x)), f(x) = #{>= cut in [0,x)}, g(x) = #{<= cut in [x,n)}
//   i = min(L_{s+1}, R_s); i == n marks the clamped case (every key below the cut).
// The cell's left tiles go on the swap's work list (one empty item for a cell without pairs:
// the swap kernel finishes every cell). A warp takes a cell of few tiles and listed keys, a
// CTA a larger one, several CTAs one of a level with few cells: each of those bisects the
// whole list, sets the mask bits of its share of the listed keys, and the last one goes on
// (one CTA alone took 270 us for the 65536 listed keys of a root of 2^27 particles, nearly
// all of it the 4 atomics a key).
// One launch where a look-back scan over the level's tiles, its clearing and a kernel per
// cell took three (the scan's 7-9 us and most of the other's 10-15 us a level were latency:
// a binary search over the tiles and a serial walk of 128 positions a lane).
constexpr uint32_t kWarpTiles = 160;  // tiles of a cell a warp takes (5 a lane)
constexpr uint32_t kWarpList = 512;   // listed keys a warp takes (16 a lane)

struct CellsSmem {
    uint32_t bins[kHistBins];
    float edges[kHistBins + 1];
    float list[kWarpList];
    uint32_t red[72];
    uint32_t count;
    float L, R;
    uint32_t it, st;
    uint32_t cross;      // the tile where f crosses g
    uint2 swaps;         // the cell's pieces on the swap's list
    uint32_t last;       // the cell's other CTAs have arrived
    int upper[32];       // each warp's cell that needs patch_upper (-1: none), and its cut
    float cuts[32];
};

// The rest of the reference loop on at most 32 N bracket keys, N a lane (slots past them
// hold R, which no cut in [L, R] exceeds); `below` keys lie below all of them. Every lane.
template <int N>
__device__ __forceinline__ int bisect_list(const float (&kl)[N], uint32_t below, uint32_t n, float ratio,
                                           float &L, float &R, uint32_t &it) {
    for (;;) {
        if (it >= (uint32_t)kMaxIterations) return kCapped;
        const float cut = mid_cut(L, R);
        uint32_t c = 0;
#pragma unroll
        for (int q = 0; q < N; ++q) c += kl[q] < cut;
        ++it;
        const int dir = convergence(below + __reduce_add_sync(0xffffffffu, c), n, ratio);
        if (dir == 0) return kFound;
        if (dir > 0)
            R = cut;
        else
            L = cut;
    }
}

__device__ __forceinline__ void store_bisection(const Level &v, int c, orb_cell_t &cell, float L, float R,
                                                uint32_t it, int st) {
    cell.cutMarginLeft = L;
    cell.cutMarginRight = R;
    cell.foundCut = st == kFound ? 1 : 0;
    v.iters[c] = (uint8_t)it;
    v.state[c] = (uint8_t)st;
    atomicMax(&v.counters->max_iters, it);
    if (st == kCapped) atomicAdd(&v.counters->unfound, 1u);
}

// Mask bits of one listed key (position `pos`) against the final cut.
__device__ __forceinline__ void patch_key(const Level &v, uint32_t t0, uint32_t rel, float k, float cut) {
    const uint32_t t = t0 + rel / (uint32_t)kPTile, in = rel % (uint32_t)kPTile;
    const uint32_t bit = 1u << (in & 31u);
    const size_t w = (size_t)t * kPWords + (in >> 5);
    if (!(k < cut)) {
        atomicOr(&v.ge_bits[w], bit);
        atomicAdd(&v.pt_ge[t], 1u);
    }
    if (!(k > cut)) {
        atomicOr(&v.le_bits[w], bit);
        atomicAdd(&v.pt_le[t], 1u);
    }
}

// The final cut is the classify pass's upper bracket end: keys equal to it are <= cut too.
// (Only a bracket a few floats wide ends there.) Sets their bits: a second read of the cell's
// keys, warp `w` of `nw` taking every nw-th run of kUpperWords mask words, a lane a key.
constexpr int kUpperWords = 16;
__device__ __noinline__ void patch_upper(const Level &v, const float *keys, uint2 rg, uint32_t t0, float cut,
                                         uint32_t w, uint32_t nw) {
    const uint32_t lane = threadIdx.x & 31u, n = rg.y - rg.x, words = (n + 31u) / 32u;
    for (uint32_t w0 = w * kUpperWords; w0 < words; w0 += nw * kUpperWords) {
        float k[kUpperWords];
#pragma unroll
        for (int u = 0; u < kUpperWords; ++u) {
            const uint32_t p = (w0 + (uint32_t)u) * 32u + lane;
            k[u] = p < n ? __ldg(keys + rg.x + p) : __int_as_float(0x7fc00000);
        }
#pragma unroll
        for (int u = 0; u < kUpperWords; ++u) {
            const uint32_t eq = __ballot_sync(0xffffffffu, k[u] == cut), word = w0 + (uint32_t)u;
            if (eq && lane == 0) {  // (a cell's tiles are kPWords words each, one after the other)
                atomicOr(&v.le_bits[(size_t)t0 * kPWords + word], eq);
                atomicAdd(&v.pt_le[t0 + word / (uint32_t)kPWords], (uint32_t)__popc(eq));
            }
        }
    }
}

// One warp: s and i of a cell from its tile prefixes and the crossing tile (see P2) and its
// record. Returns where its pieces start on the swap's list, and their number (fill_swaps).
__device__ uint2 cell_split_point(const Level &v, int c, uint2 rg, uint32_t t0, uint32_t T, uint32_t cross,
                                 uint32_t ge_tot, uint32_t le_tot) {
    const uint32_t lane = threadIdx.x & 31, n = rg.y - rg.x;
    uint32_t s = 0, i = n;
    if (T) {
        const size_t w0 = (size_t)cross * kPWords;
        const uint4 qg = __ldcg(reinterpret_cast<const uint4 *>(v.ge_bits + w0) + lane);
        const uint4 ql = __ldcg(reinterpret_cast<const uint4 *>(v.le_bits + w0) + lane);
        const uint32_t gw[4] = {qg.x, qg.y, qg.z, qg.w}, lw[4] = {ql.x, ql.y, ql.z, ql.w};
        uint32_t tg, tl;
        uint32_t f = v.pt_ge_pre[cross] + warp_excl_scan(__popc(gw[0]) + __popc(gw[1]) + __popc(gw[2]) + __popc(gw[3]), &tg);
        uint32_t g = le_tot - v.pt_le_pre[cross] -
                     warp_excl_scan(__popc(lw[0]) + __popc(lw[1]) + __popc(lw[2]) + __popc(lw[3]), &tl);
        // min(f, g) rises while f < g and falls after: its maximum lies in the first word at
        // whose end f >= g (the tile's last word at the latest)
        uint32_t wa = gw[3], wb = lw[3], wf = 0, wg = 0;
        bool hit = false;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint32_t fe = f + __popc(gw[j]), ge = g - __popc(lw[j]);
            if (!hit && (fe >= ge || j == 3)) {
                wa = gw[j];
                wb = lw[j];
                wf = f;
                wg = g;
                hit = fe >= ge;
            }
            f = fe;
            g = ge;
        }
        const uint32_t hb = __ballot_sync(0xffffffffu, hit);
        const int src = hb ? __ffs(hb) - 1 : 31;
        wa = __shfl_sync(0xffffffffu, wa, src);
        wb = __shfl_sync(0xffffffffu, wb, src);
        wf = __shfl_sync(0xffffffffu, wf, src);
        wg = __shfl_sync(0xffffffffu, wg, src);
        const uint32_t upto = 0xffffffffu >> (31u - lane);
        s = max(min(wf, wg), min(wf + __popc(wa & upto), wg - __popc(wb & upto)));
        s = __reduce_max_sync(0xffffffffu, s);
        i = min(i, warp_select2(v, t0, t0 + T, ge_tot > s, s, s >= 1, le_tot - s));
    }
    const uint32_t left = s ? min(T, (i + (uint32_t)kPTile - 1) / (uint32_t)kPTile) << v.piece_log2 : 1u;
    uint32_t at = 0;
    if (lane == 0) {
        CellPart p;
        p.b = rg.x;
        p.n = n;
        p.s = s;
        p.i = i;
        p.le = le_tot;
        p.t0 = t0;
        p.T = T;
        p.left = left;
        v.part[c] = p;
        v.part_done[c] = v.done_start;
        at = atomicAdd(&v.tot->swaps, left);
    }
    return make_uint2(__shfl_sync(0xffffffffu, at, 0), left);
}
__device__ __forceinline__ void fill_swaps(const Level &v, int c, uint2 w, uint32_t ti, uint32_t nt) {
    for (uint32_t j = ti; j < w.y; j += nt) v.swap_list[w.x + j] = make_uint2((uint32_t)c, j);
}

// A cell of at most kWarpTiles tiles and kWarpList listed keys, by one warp. Every warp of the CTA
// calls it (c < 0: without a cell): cells that need patch_upper get it from all of them (by the
// cell's own warp, 2^20 keys outside a box without extent took 29 ms; 1 ms with the CTA and the
// loop ended by resolve_cell).
__device__ void cells_warp(const Level &v, int c, CellsSmem &sm) {
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const bool any = c >= 0;
    if (!any) c = 0;
    const int slot = level_slot(v, c);
    orb_cell_t &cell = v.heap[slot];
    const uint2 rg = v.ranges[slot];
    const uint32_t n = rg.y - rg.x, t0 = v.ptile_off[c], T = (n + (uint32_t)kPTile - 1) / (uint32_t)kPTile;
    bool upper = false;
    float cut = 0.f;
    if (any && v.state[c] == kReady) {
        const uint32_t m = v.cmp_cnt[c], off = v.cmp_off[c];
        const float ratio = leaf_ratio(cell.nLeafCells);  // src/orbit.cpp:204
        float L = cell.cutMarginLeft, R = cell.cutMarginRight;
        const float hi = R;  // the classify pass's bracket end
        uint32_t it = v.iters[c];
        float kl[kWarpList / 32];
#pragma unroll
        for (int q = 0; q < (int)kWarpList / 32; ++q) {
            const uint32_t j = (uint32_t)q * 32u + lane;
            kl[q] = j < m ? v.cmp_keys[off + j] : R;
        }
        const int st = bisect_list(kl, v.below[c], n, ratio, L, R, it);
        __syncwarp();
        if (lane == 0) store_bisection(v, c, cell, L, R, it, st);
        cut = mid_cut(L, R);
        upper = cut == hi;
#pragma unroll
        for (int q = 0; q < (int)kWarpList / 32; ++q) {
            const uint32_t j = (uint32_t)q * 32u + lane;
            if (j < m) patch_key(v, t0, v.cmp_pos[off + j] - rg.x, kl[q], cut);
        }
        __threadfence();
        __syncwarp();
    }
    if (__syncthreads_or(upper)) {
        if (lane == 0) {
            sm.upper[warp] = upper ? c : -1;
            sm.cuts[warp] = cut;
        }
        __syncthreads();
        for (uint32_t q = 0; q < nw; ++q) {
            const int cq = sm.upper[q];
            if (cq < 0) continue;
            const int sq = level_slot(v, cq);
            patch_upper(v, axis_keys(v, eff_axis(v.heap[sq].cutAxis)), v.ranges[sq], v.ptile_off[cq], sm.cuts[q], warp, nw);
        }
        __threadfence();
        __syncthreads();
    }
    if (!any) return;
    // prefixes within the cell, tiles lane, 32 + lane, ... in a lane
    constexpr int kPer = (int)kWarpTiles / 32;
    uint32_t g[kPer], l[kPer], pg[kPer], pl[kPer];
#pragma unroll
    for (int q = 0; q < kPer; ++q) {
        const uint32_t u = (uint32_t)q * 32u + lane;
        g[q] = u < T ? __ldcg(&v.pt_ge[t0 + u]) : 0u;
        l[q] = u < T ? __ldcg(&v.pt_le[t0 + u]) : 0u;
    }
    uint32_t ge_tot = 0, le_tot = 0;
#pragma unroll
    for (int q = 0; q < kPer; ++q) {
        const uint32_t u = (uint32_t)q * 32u + lane;
        uint32_t tg, tl;
        pg[q] = ge_tot + warp_excl_scan(g[q], &tg);
        pl[q] = le_tot + warp_excl_scan(l[q], &tl);
        ge_tot += tg;
        le_tot += tl;
        if (u < T) {
            v.pt_ge_pre[t0 + u] = pg[q];
            v.pt_le_pre[t0 + u] = pl[q];
        }
    }
    __syncwarp();
    // crossing tile: the first whose end has f >= g (the last always does)
    uint32_t cross = 0;
#pragma unroll
    for (int q = kPer - 1; q >= 0; --q) {
        const uint32_t u = (uint32_t)q * 32u + lane;
        const uint32_t b = __ballot_sync(0xffffffffu, u < T && pg[q] + g[q] >= le_tot - pl[q] - l[q]);
        if (b) cross = (uint32_t)q * 32u + (uint32_t)__ffs(b) - 1u;
    }
    fill_swaps(v, c, cell_split_point(v, c, rg, t0, T, t0 + cross, ge_tot, le_tot), lane, 32);
}

// A larger cell, by the CTA, or by nchunks CTAs of which this is number `chunk`.
template <int NT>
__device__ void cells_cta(const Level &v, int c, uint32_t chunk, uint32_t nchunks, CellsSmem &sm) {
    const uint32_t tid = threadIdx.x, lane = tid & 31;
    const int slot = level_slot(v, c);
    orb_cell_t &cell = v.heap[slot];
    const uint2 rg = v.ranges[slot];
    const uint32_t n = rg.y - rg.x, t0 = v.ptile_off[c], T = (n + (uint32_t)kPTile - 1) / (uint32_t)kPTile;
    if (v.state[c] == kReady) {
        const uint32_t m = v.cmp_cnt[c];
        const float *keys = v.cmp_keys + v.cmp_off[c];
        const uint32_t *pos = v.cmp_pos + v.cmp_off[c];
        const float ratio = leaf_ratio(cell.nLeafCells);  // src/orbit.cpp:204
        float L = cell.cutMarginLeft, R = cell.cutMarginRight;
        const float hi = R;
        uint32_t it = v.iters[c], cand = m, below = v.below[c];  // keys below L
        uint8_t st = kActive;
        // histogram rounds over the bracket's midpoint tree, until the bracket fits a warp
        while (st == kActive && cand > kWarpList) {
            const int K = min(kMaxBinsLog2, 32 - __clz(cand));
            const uint32_t nb = 1u << K;
            for (uint32_t j = tid; j < kHistBins; j += NT) sm.bins[j] = 0u;
            fill_edges(sm.edges, L, R, K, tid, NT);
            __syncthreads();
            const Guess gs = make_guess(L, R, __fdiv_rn((float)nb, __fsub_rn(R, L)), nb);
            // (with the loads a round at a time, and the wide cells' lists below filled by the CTA,
            // the root of 2^27 particles takes 54 us here, 74 before)
            constexpr int kLoads = 8;
            for (uint32_t j0 = tid; j0 < m; j0 += kLoads * NT) {
                float k[kLoads];
#pragma unroll
                for (int q = 0; q < kLoads; ++q) k[q] = j0 + q * NT < m ? keys[j0 + q * NT] : __int_as_float(0x7fc00000);
#pragma unroll
                for (int q = 0; q < kLoads; ++q)
                    if (k[q] >= L && k[q] < R) {
                        uint32_t g;
                        if (!guess_bin(gs, k[q], &g)) g = near_bin(k[q], gs, sm.edges, nb - 1u);
                        atomicAdd(&sm.bins[g], 1u);
                    }
            }
            __syncthreads();
            constexpr uint32_t kPer = kHistBins / NT;  // bins a thread
            uint32_t h[kPer], loc = 0;
#pragma unroll
            for (uint32_t j = 0; j < kPer; ++j) {
                h[j] = sm.bins[tid * kPer + j];
                loc += h[j];
            }
            uint32_t tot, unused;
            uint32_t run = block_excl_scan2(loc, 0u, sm.red, &tot, &unused).x;
#pragma unroll
            for (uint32_t j = 0; j < kPer; ++j) {
                sm.bins[tid * kPer + j] = run;
                run += h[j];
            }
            __syncthreads();
            uint32_t p = 0;
            replay<false>(sm.bins, K, below, n, ratio, 0u, L, R, it, p, st);
            if (st == kActive) {
                cand = (p + 1 < nb ? sm.bins[p + 1] : tot) - sm.bins[p];
                below += sm.bins[p];
            }
            __syncthreads();
        }
        if (st == kActive) {
            // the bracket's keys gathered; warp 0 finishes
            if (tid == 0) sm.count = 0;
            __syncthreads();
#pragma unroll 8
            for (uint32_t j = tid; j < m; j += NT) {
                const float k = keys[j];
                if (k >= L && k < R) {
                    const uint32_t q = atomicAdd(&sm.count, 1u);
                    if (q < kWarpList) sm.list[q] = k;
                }
            }
            __syncthreads();
            if (tid < 32) {
                float kl[kWarpList / 32];
#pragma unroll
                for (int q = 0; q < (int)kWarpList / 32; ++q) {
                    const uint32_t j = (uint32_t)q * 32u + lane;
                    kl[q] = j < cand ? sm.list[j] : R;
                }
                st = (uint8_t)bisect_list(kl, below, n, ratio, L, R, it);
            }
        }
        if (tid == 0) {
            sm.L = L;
            sm.R = R;
            sm.it = it;
            sm.st = st;
        }
        __syncthreads();
        const float cut = mid_cut(sm.L, sm.R);
        for (uint32_t j = chunk * NT + tid; j < m; j += nchunks * NT) patch_key(v, t0, pos[j] - rg.x, keys[j], cut);
        if (cut == hi)
            patch_upper(v, axis_keys(v, eff_axis(cell.cutAxis)), rg, t0, cut, chunk * (NT / 32) + tid / 32, nchunks * (NT / 32));
        __threadfence();
        __syncthreads();
    }
    if (nchunks > 1) {
        if (tid == 0) {
            sm.last = arrive_release(&v.hdone[c], 1u) + 1u == nchunks;
            if (sm.last) acquire();
        }
        __syncthreads();
        if (!sm.last) return;
    }
    // (the cell and its state are the other CTAs' inputs: written once all have arrived)
    if (tid == 0 && v.state[c] == kReady) store_bisection(v, c, cell, sm.L, sm.R, sm.it, (int)sm.st);
    // prefixes within the cell: a run of consecutive tiles a warp, 32 at a time
    const uint32_t warp = tid >> 5;
    constexpr uint32_t kWarps = NT / 32;
    const uint32_t per = (T + kWarps * 32 - 1) / (kWarps * 32) * 32;
    const uint32_t u0 = min(T, warp * per), u1 = min(T, u0 + per);
    uint32_t cg = 0, cl = 0;
#pragma unroll 8
    for (uint32_t u = u0 + lane; u < u1; u += 32) {
        cg += __ldcg(&v.pt_ge[t0 + u]);
        cl += __ldcg(&v.pt_le[t0 + u]);
    }
    // (block_excl_scan2 runs over threads in order: a warp's tiles precede the next warp's)
    uint32_t ge_tot, le_tot;
    const uint2 ex = block_excl_scan2(cg, cl, sm.red, &ge_tot, &le_tot);
    uint32_t f = __shfl_sync(0xffffffffu, ex.x, 0), l = __shfl_sync(0xffffffffu, ex.y, 0);
    if (tid == 0) sm.cross = 0xffffffffu;
    __syncthreads();
    constexpr int kAhead = 4;  // rounds of 32 tiles whose counts are loaded together
    for (uint32_t b0 = u0; b0 < u1; b0 += 32 * kAhead) {
        uint32_t gs[kAhead], ls[kAhead];
#pragma unroll
        for (int q = 0; q < kAhead; ++q) {
            const uint32_t u = b0 + (uint32_t)q * 32u + lane;
            gs[q] = u < u1 ? __ldcg(&v.pt_ge[t0 + u]) : 0u;
            ls[q] = u < u1 ? __ldcg(&v.pt_le[t0 + u]) : 0u;
        }
#pragma unroll
        for (int q = 0; q < kAhead; ++q) {
            const uint32_t b = b0 + (uint32_t)q * 32u, u = b + lane;
            if (b >= u1) break;
            uint32_t tg, tl;
            const uint32_t pf = f + warp_excl_scan(gs[q], &tg), pl = l + warp_excl_scan(ls[q], &tl);
            if (u < u1) {
                v.pt_ge_pre[t0 + u] = pf;
                v.pt_le_pre[t0 + u] = pl;
            }
            // crossing tile: the first whose end has f >= g (the last always does)
            const uint32_t x = __ballot_sync(0xffffffffu, u < u1 && pf + gs[q] >= le_tot - pl - ls[q]);
            if (lane == 0 && x) atomicMin(&sm.cross, t0 + b + (uint32_t)__ffs(x) - 1u);
            f += tg;
            l += tl;
        }
    }
    __syncthreads();
    const bool wide = T > 1024;  // a list worth the CTA's threads
    if (tid < 32) {
        const uint2 w = cell_split_point(v, c, rg, t0, T, sm.cross, ge_tot, le_tot);
        if (!wide) fill_swaps(v, c, w, lane, 32);
        if (tid == 0) sm.swaps = w;
    }
    __syncthreads();  // sm reused by the next cell
    if (wide) {
        fill_swaps(v, c, sm.swaps, tid, NT);
        __syncthreads();
    }
}

// kPerCell: gridDim.x CTAs a cell (levels of few cells); else a warp a cell, the larger ones
// by the CTA.
template <int NT, bool kPerCell>
__global__ void __launch_bounds__(NT) k_part_cells(const __grid_constant__ Level v) {
    pdl_enter();
    __shared__ CellsSmem sm;
    if (level_failed(v)) return;
    auto fits_warp = [&](int c) {
        const uint2 rg = v.ranges[level_slot(v, c)];
        return rg.y - rg.x <= kWarpTiles * (uint32_t)kPTile && !(v.state[c] == kReady && v.cmp_cnt[c] > kWarpList);
    };
    const int warp = (int)threadIdx.x >> 5;
    if (kPerCell) {
        const int c = (int)blockIdx.y;
        const bool fits = fits_warp(c);
        __syncthreads();  // every thread has looked before the state changes
        if (!fits)
            cells_cta<NT>(v, c, blockIdx.x, gridDim.x, sm);
        else if (blockIdx.x == 0)
            cells_warp(v, warp == 0 ? c : -1, sm);
        if (threadIdx.x == 0 && blockIdx.x == 0) add_bytes(v, kKPartCells, 512ull);
        return;
    }
    constexpr int kW = NT / 32;
    const int c0 = (int)blockIdx.x * kW;
    __shared__ uint32_t s_big;  // the CTA's cells a warp cannot take
    if (threadIdx.x == 0) s_big = 0;
    __syncthreads();
    if ((threadIdx.x & 31) == 0 && c0 + warp < v.C && !fits_warp(c0 + warp)) atomicOr(&s_big, 1u << warp);
    __syncthreads();
    uint32_t big = s_big;
    cells_warp(v, c0 + warp < v.C && !((big >> warp) & 1u) ? c0 + warp : -1, sm);
    for (; big; big &= big - 1u) cells_cta<NT>(v, c0 + __ffs(big) - 1, 0u, 1u, sm);
    if (threadIdx.x == 0 && c0 < v.C) add_bytes(v, kKPartCells, 512ull * (unsigned)min(kW, v.C - c0));
}

// Writes the cell-relative positions of the set bits of one tile's mask whose in-cell rank
// lies in [lo, hi) to out[f(rank)], f(rank) = rank - lo (forward) or (top - rank) (reverse).
// Block-cooperative; `sh` holds >= 96 words.
__device__ __forceinline__ void emit_positions(const uint32_t *words, uint32_t rank_base,
                                               uint32_t lo, uint32_t hi, uint32_t rel_base,
                                               bool reverse, uint32_t top, uint32_t *out,
                                               uint32_t *sh) {
    const uint32_t tid = threadIdx.x;
    const uint32_t w = tid < (uint32_t)kPWords ? words[tid] : 0u;
    uint32_t ta, tb;
    const uint2 ex = block_excl_scan2(__popc(w), 0u, sh, &ta, &tb);
    uint32_t r = rank_base + ex.x;
    uint32_t word = w;
    while (word) {
        const uint32_t b = (uint32_t)(__ffs(word) - 1);
        word &= word - 1;
        if (r >= lo && r < hi) out[reverse ? top - r : r - lo] = rel_base + tid * 32u + b;
        ++r;
    }
}

// P4: the Hoare swaps. The CTA of tile t takes the pairs (L_k, R_k) whose left element
// L_k lies in t (k < s); their right partners are the keys <= cut of left-to-right rank
// le_tot-1-k, found in the right tiles' masks. Positions of each side are disjoint
// (L_k < i <= R_k), so the CTAs never touch the same particle.
// Tuning (compile time): pairs per thread per round, and the CTAs per SM the register
// budget is sized for (4 x 256 threads: 64 registers a thread).
#ifndef ORB_SWAP_BATCH
#define ORB_SWAP_BATCH 4
#endif
#ifndef ORB_SWAP_MIN_BLOCKS
#define ORB_SWAP_MIN_BLOCKS 4
#endif
#ifndef ORB_SWAP_THREADS
#define ORB_SWAP_THREADS 256  // threads of a swap CTA (at least kPWords: one mask word each)
#endif
constexpr int kSwapThreads = ORB_SWAP_THREADS;
static_assert(kSwapThreads >= kPWords && kSwapThreads % 32 == 0, "a swap CTA scans a tile's mask words");
// kWt: weighted builds, whose weights move with their particles. kYZ: bit 0 y moves, bit 1 z
// moves (3 normally; the first levels of a build from host memory move x before y and z have
// arrived, see orb_build).
// kFuse: the CTA that brings a cell's last tile also finishes the cell (levels of at most one
// tile a CTA, where a launch less counts); else k_part_finish does. Arrivals between a CTA's
// tiles made the swap of the headline's deep levels 40% slower (570 -> 850 us a level: each
// waits for the SM's stores), so larger levels take the separate launch.
template <bool kWt, int kYZ, bool kFuse>
__global__ void __launch_bounds__(kSwapThreads, ORB_SWAP_MIN_BLOCKS) k_part_swap(const __grid_constant__ Level v, int do_split) {
    pdl_enter();
    if (level_failed(v)) return;
    __shared__ uint32_t posL[kPTile];
    __shared__ uint32_t posR[kPTile];
    __shared__ uint32_t sh[96];
    __shared__ FinishIn s_in;
    const uint32_t total = v.tot->swaps;
    unsigned long long bytes = 0;  // pairs swapped by this CTA
    for (uint32_t w = blockIdx.x; w < total; w += gridDim.x) {
        const uint2 item = v.swap_list[w];
        const int c = (int)item.x;
        const CellPart P = v.part[c];
        const uint32_t tile = item.y >> v.piece_log2, t0 = P.t0, t1 = t0 + P.T, t = t0 + tile;
        const uint32_t s = P.s, le_tot = P.le, b = P.b;
        const uint32_t kt = s ? v.pt_ge_pre[t] : 0u;  // (a cell without pairs has one empty item)
        uint32_t ka = kt, kb = s ? max(kt, min(s, kt + v.pt_ge[t])) : 0u;
        if (v.piece_log2) {  // the item's share of the tile's pairs
            const uint32_t per = ((kb - ka) + (1u << v.piece_log2) - 1u) >> v.piece_log2;
            ka = min(kb, kt + (item.y - (tile << v.piece_log2)) * per);
            kb = min(kb, ka + per);
        }
        const uint32_t cnt = kb - ka;
        if (kFuse && threadIdx.x == 0) s_in = finish_in(v, c);
        if (cnt) {
            // left elements: ranks [ka, kb) of this tile's >= mask, in order
            emit_positions(v.ge_bits + (size_t)t * kPWords, kt, ka, kb, tile * (uint32_t)kPTile, false, 0u,
                           posL, sh);
            // right partners: left-to-right <= ranks [le_tot-kb, le_tot-ka); rank r pairs with
            // k = le_tot-1-r, stored at posR[k - ka] = posR[(le_tot-1-ka) - r]
            const uint32_t ra = le_tot - kb, rb = le_tot - ka;
            const uint32_t u0 = warp_last_at_most(v.pt_le_pre, t0, t1 - 1, ra);
            for (uint32_t u = u0; u < t1 && v.pt_le_pre[u] < rb; ++u)
                emit_positions(v.le_bits + (size_t)u * kPWords, v.pt_le_pre[u], ra, rb,
                               (u - t0) * (uint32_t)kPTile, true, le_tot - 1 - ka, posR, sh);
        }
        __syncthreads();
        // kB pairs per thread per round: every load is issued before any store
        constexpr int kB = ORB_SWAP_BATCH;
        for (uint32_t j0 = 0; j0 < cnt; j0 += kB * blockDim.x) {
            uint32_t pa[kB], pb[kB];
            float xa[kB], xb[kB], ya[kB], yb[kB], za[kB], zb[kB];
            uint32_t ia[kB], ib[kB], wa[kB], wb[kB];
#pragma unroll
            for (int q = 0; q < kB; ++q) {
                const uint32_t j = j0 + q * blockDim.x + threadIdx.x;
                const bool ok = j < cnt;
                pa[q] = ok ? b + posL[j] : 0xffffffffu;
                pb[q] = ok ? b + posR[j] : 0xffffffffu;
                if (ok) {
                    xa[q] = v.x[pa[q]];
                    xb[q] = v.x[pb[q]];
                    if constexpr ((kYZ & 1) != 0) {
                        ya[q] = v.y[pa[q]];
                        yb[q] = v.y[pb[q]];
                    }
                    if constexpr ((kYZ & 2) != 0) {
                        za[q] = v.z[pa[q]];
                        zb[q] = v.z[pb[q]];
                    }
                    if (v.idx) {
                        ia[q] = v.idx[pa[q]];
                        ib[q] = v.idx[pb[q]];
                    }
                    if constexpr (kWt) {
                        wa[q] = v.wt[pa[q]];
                        wb[q] = v.wt[pb[q]];
                    }
                }
            }
#pragma unroll
            for (int q = 0; q < kB; ++q) {
                if (pa[q] == 0xffffffffu) continue;
                v.x[pa[q]] = xb[q];
                v.x[pb[q]] = xa[q];
                if constexpr ((kYZ & 1) != 0) {
                    v.y[pa[q]] = yb[q];
                    v.y[pb[q]] = ya[q];
                }
                if constexpr ((kYZ & 2) != 0) {
                    v.z[pa[q]] = zb[q];
                    v.z[pb[q]] = za[q];
                }
                if (v.idx) {
                    v.idx[pa[q]] = ib[q];
                    v.idx[pb[q]] = ia[q];
                }
                if constexpr (kWt) {
                    v.wt[pa[q]] = wb[q];
                    v.wt[pb[q]] = wa[q];
                }
            }
        }
        bytes += cnt;
        __syncthreads();
        if constexpr (kFuse) {
            __shared__ Kids s_kids;
            __shared__ bool s_last;
            if (threadIdx.x < 32) {
                uint32_t last = 0;
                if (threadIdx.x == 0) {
                    last = arrive_release(&v.part_done[c], 1u) + 1u == P.left ? 1u : 0u;
                    s_last = last != 0;
                    if (last) acquire();
                }
                __syncwarp();  // (the other lanes read the cell's particles too)
                if (__shfl_sync(0xffffffffu, last, 0)) finish_and_plan(v, s_in, P, do_split != 0, s_kids);
            }
            __syncthreads();
            if (s_last) {
                plan_fill(v, s_kids.p[0], threadIdx.x, kSwapThreads);
                plan_fill(v, s_kids.p[1], threadIdx.x, kSwapThreads);
                __syncthreads();
            }
        } else if (threadIdx.x == 0) {
            atomicAdd(&v.part_done[c], 1u);
        }
    }
    // per pair: both elements of x, y, z (and idx, weights) read and written
    if (threadIdx.x == 0 && bytes)
        add_bytes(v, kKPartSwap, (16ull * (1 + (kYZ & 1) + ((kYZ >> 1) & 1)) + (v.idx ? 16ull : 0ull) +
                                  (kWt ? 16ull : 0ull)) * bytes);
}

// P5: the final swap, the split and the children's plan of every cell, a CTA a cell on levels of
// few cells (large maps to fill), else a warp. A cell whose tiles did not all report is left
// alone: its missing count stops the build.
template <bool kPerCell>
__global__ void __launch_bounds__(kThreads) k_part_finish(const __grid_constant__ Level v, int do_split) {
    pdl_enter();
    if (level_failed(v)) return;
    __shared__ Kids s_kids[kThreads / 32];
    __shared__ FinishIn s_in[kThreads / 32];
    const uint32_t warp = threadIdx.x >> 5, nt = kPerCell ? kThreads : 32u;
    const uint32_t ti = kPerCell ? threadIdx.x : threadIdx.x & 31u;
    const int c = kPerCell ? (int)blockIdx.x : (int)(blockIdx.x * (kThreads / 32) + warp);
    Kids &k = s_kids[kPerCell ? 0 : warp];
    if (c < v.C && ti < 32) {
        const CellPart P = v.part[c];
        const uint32_t done = v.part_done[c];
        if (ti == 0) {
            s_in[warp] = finish_in(v, c);
            k.p[0].c = k.p[1].c = -1;
        }
        __syncwarp();
        if (done == P.left) finish_and_plan(v, s_in[warp], P, do_split != 0, k);
    }
    if (kPerCell)
        __syncthreads();
    else
        __syncwarp();
    if (c >= v.C) return;
    plan_fill(v, k.p[0], ti, nt);
    plan_fill(v, k.p[1], ti, nt);
}

// ------------------------------------------------------------------------------------
// Subtrees: once every cell of a level fits one CTA, the rest of each cell's tree (bisection,
// Hoare partition and split of every descendant, breadth first) is built in shared memory
// without moving a particle until the end: a group of warps holds one axis of the cell's keys
// in their original order and the current order as 16-bit positions. A level loads the axis
// its cells cut along (a coalesced copy of 4 B a particle, mostly from L2), reads the keys
// through the positions, and its swaps exchange 2-byte positions. At the end each coordinate
// is loaded once more and written through the positions: in all 4 B a particle and level plus
// 24 B (32 B with the permutation), every access coalesced. The cells of a level are worked on
// side by side, the group's warps divided evenly among them, all in step.
//
// Measured (GB300): the last four levels of 2^27 uniform particles into 2^16 leaves (cells of
// 2^15) take 2.71 ms, against 3.88 ms for a CTA of 256 threads that moved the particles in
// global memory at every level (four such CTAs an SM, its cells re-read from L2).
//
// The kernel is bound by instructions and shared memory, so the bisection avoids exact binning: a histogram by
// the rounded scaled key finds a window [a, b) of floats around the target rank (a few dozen
// keys); the pass that writes the masks counts the keys below a and above b exactly and lists
// those inside; then the reference loop (src/orbit.cpp:146-232) is replayed from the cell's own
// margins: a cut at or below a has a count of at most count(< a), one at or above b at least
// count(< b), so where the exact counts show the first too low and the second too high the
// loop moves that margin (the float test is monotone in the count), and a cut inside the
// window gets its exact count from the list. A cell whose replay meets a cut the window
// cannot settle (many equal keys, a box far wider than its keys) counts every cut over all
// its keys instead, until its bracket is two neighbouring floats. Same cuts, same integer counts, same iterations on every path.
//
// A group is the CTA's 32 warps, or 16, 8 or 2 of them for smaller cells (by size): small
// cells are bound by the latency of their steps, so an SM keeps 2, 4 or 16 in flight. (Cells of
// 2^14, the common size above 2^8 particles a leaf: 2^26 clustered particles into 2^18, six
// levels, 4.00 ms with one on an SM, 2.48 with two. So a group of 16 has half the bins, and the list
// holds positions only.)
// ------------------------------------------------------------------------------------
constexpr int kSubLevels = kSubMaxLevels;
constexpr int kSubCells = 1 << (kSubLevels - 1);  // cells of the deepest level split
constexpr int kSubThreads = 1024;                 // of the CTA, one on an SM
constexpr uint32_t kSubWindowList = 256;          // most listed keys of a cell (8 a lane)

struct SubCell {
    int id, leaves, axis;
    float lower[3], upper[3];
    uint16_t b, m;  // first position within the root cell, particles
};

// Bisection and partition state of one cell of the level.
enum : uint32_t { kSubOpen = 0, kSubDone = 1, kSubWindow = 2, kSubCount = 3 };
struct SubState {
    float L, R;          // the bisection's bracket
    float a, b;          // the window (kSubOpen: being narrowed; kSubWindow: classified)
    float ratio;         // the test's share of the keys, leaf_ratio() of the cell
    uint32_t mode;       // kSubOpen, kSubWindow, kSubCount (counts every cut), kSubDone
    uint16_t it, found;
    uint32_t cand;       // keys in the window by the last histogram (~0: none yet)
    uint32_t cnt;        // kSubCount: keys below the cut
    uint32_t nlist;      // listed keys
    uint32_t tot;        // keys >= cut | keys <= cut << 16
    uint32_t cross, s, i;
};

template <int NW>
struct SubSmem {
    // a level's cells together (16 warps: what two cells of 2^14 on an SM leave room for)
    static constexpr uint32_t kBins = NW == 32 ? 2048 : (NW >= 8 ? 1024 : 256);
    static constexpr uint32_t kLists = NW == 32 ? 1024 : (NW == 16 ? 1280 : (NW == 8 ? 512 : 256));
    // cells up to this size: one warp's registers
    static constexpr uint32_t kDirect = NW == 16 ? 768 : 256;
    SubCell cell[2][kSubCells];
    SubState state[kSubCells];
    uint32_t bins[kBins];
    uint16_t lpos[kLists];  // the listed keys' positions within their cell
    uint32_t part[NW];
    uint32_t axes;    // axes the level's cells cut along
    uint32_t counted; // ... those of cells too large for one warp's registers
    uint32_t more, direct;
    uint32_t max_it, unfound, degenerate;
    int item, root;
    alignas(8) unsigned long long arrived;  // mbarrier of the key copies
};

// Shared memory of a group: SubSmem, keys (up to three words of misalignment), mask words and
// their prefixes (a partial word a cell), order.
__host__ __device__ constexpr uint32_t sub_words(uint32_t nmax) { return nmax / 32 + kSubCells + 2; }
template <int NW>
__host__ __device__ constexpr uint32_t sub_bytes(uint32_t nmax) {
    return ((uint32_t)((sizeof(SubSmem<NW>) + 15) / 16 * 16) + (nmax + 4) * 4 + sub_words(nmax) * 12 + nmax * 2 + 15) / 16 * 16;
}
// particles of a cell a group of 32, 16, 8, 2 warps takes
constexpr uint32_t kSub32 = kSubMaxParticles, kSub16 = 16400, kSub8 = 6656, kSub2 = 1088;
constexpr uint32_t kSubBytes = 232448;  // all of a CTA's shared memory
static_assert(sub_bytes<32>(kSub32) <= kSubBytes && 2 * sub_bytes<16>(kSub16) <= kSubBytes && 4 * sub_bytes<8>(kSub8) <= kSubBytes && 16 * sub_bytes<2>(kSub2) <= kSubBytes,
              "the smaller groups' slices");

// Levels below a cell: the same for every cell of the level in a single build (v.sub_levels);
// in a batch (powers of two, built to their leaves) log2 of its leaf count.
__device__ __forceinline__ int levels_below(const Level &v, int leaves) {
    return v.sub_levels ? v.sub_levels : (leaves > 1 ? 31 - __clz((uint32_t)leaves) : 0);
}

// Flag for k_subtree: every cell of the level fits a CTA and has at most `max_levels`
// (<= kSubLevels) levels below it; for the host, the largest cell. Then the cells with levels below them, by class (all of
// the first class on levels of few cells, v.sub_wide), in order. One CTA.
__global__ void __launch_bounds__(1024) k_subtree_check(const __grid_constant__ Level v, int max_levels) {
    pdl_enter();
    __shared__ uint32_t sh[96];
    const bool failed = level_failed(v);
    uint32_t mx = 0, ml = 0;
    for (int c = threadIdx.x; c < v.C; c += blockDim.x) {
        const int slot = level_slot(v, c);
        const uint2 rg = v.ranges[slot];
        mx = max(mx, rg.y - rg.x);
        ml = max(ml, (uint32_t)levels_below(v, v.heap[slot].nLeafCells));
    }
    mx = block_max(mx, sh);
    ml = block_max(ml, sh);
    const bool take = !failed && mx <= kSub32 && (int)ml <= min(max_levels, kSubLevels);
    // v.sub_list: four stretches of v.C cells, one a class
    uint32_t n0 = 0, n1 = 0, n2 = 0, n3 = 0;
    for (int base = 0; take && base < v.C; base += (int)blockDim.x) {
        const int c = base + (int)threadIdx.x;
        int k = 4;
        if (c < v.C) {
            const int slot = level_slot(v, c);
            const uint2 rg = v.ranges[slot];
            const uint32_t n = rg.y - rg.x;
            if (v.heap[slot].nLeafCells > 1)
                k = v.sub_wide || n > kSub16 ? 0 : (n > kSub8 ? 1 : (n > kSub2 ? 2 : 3));
        }
        uint32_t ta, tb;
        const uint2 ex = block_excl_scan2((k == 0 ? 1u : 0u) | (k == 1 ? 0x10000u : 0u),
                                          (k == 2 ? 1u : 0u) | (k == 3 ? 0x10000u : 0u), sh, &ta, &tb);
        if (k == 0) v.sub_list[n0 + (ex.x & 0xffffu)] = c;
        if (k == 1) v.sub_list[v.C + n1 + (ex.x >> 16)] = c;
        if (k == 2) v.sub_list[2 * v.C + n2 + (ex.y & 0xffffu)] = c;
        if (k == 3) v.sub_list[3 * v.C + n3 + (ex.y >> 16)] = c;
        n0 += ta & 0xffffu;
        n1 += ta >> 16;
        n2 += tb & 0xffffu;
        n3 += tb >> 16;
    }
    if (v.win_cnt)
        for (int w = threadIdx.x; w < kMaxWindows; w += blockDim.x) v.win_cnt[w] = 0u;
    if (threadIdx.x == 0) {
        v.skip[0] = take ? 1u : 0u;
        v.skip[1] = failed || (int)ml > min(max_levels, kSubLevels) ? 0xffffffffu : mx;
        v.counters->sub_cells[0] = n0;
        v.counters->sub_cells[1] = n1;
        v.counters->sub_cells[2] = n2;
        v.counters->sub_cells[3] = n3;
        for (int k = 0; k < 4; ++k) v.counters->sub_next[k] = 0u;
        if (v.hwin) {
            __threadfence_system();
            *(volatile uint32_t *)&v.hwin->decision = take ? 1u : 2u;
        }
    }
}

extern __shared__ __align__(16) unsigned char sub_mem[];

// One group of NW warps: the cells of one class, from its work queue. `slice`: where the
// group's shared memory starts (named here, not passed as a pointer, so that every access is a
// shared-memory one); ti: thread of the group; bar: its named barrier. False: a copy did not come;
// the build is flagged and the group has left its queue and this shared memory.
template <int NW>
__device__ __forceinline__ bool sub_group(const Level &v, uint32_t slice, uint32_t ti, int bar) {
    unsigned char *const mem = sub_mem + slice;
    constexpr int kClass = NW == 32 ? 0 : (NW == 16 ? 1 : (NW == 8 ? 2 : 3));
    constexpr uint32_t NT = NW * 32, nmax = NW == 32 ? kSub32 : (NW == 16 ? kSub16 : (NW == 8 ? kSub8 : kSub2)), nwords = sub_words(nmax);
    constexpr uint32_t kBins = SubSmem<NW>::kBins, kLists = SubSmem<NW>::kLists, kSubDirect = SubSmem<NW>::kDirect;
    constexpr int kU = 8;  // words of a warp in flight
    auto sync = [&]() {
        if (NW == 32)
            __syncthreads();
        else
            asm volatile("bar.sync %0, %1;" ::"r"(bar), "n"((int)NT) : "memory");
    };
    SubSmem<NW> &sm = *reinterpret_cast<SubSmem<NW> *>(mem);
    uint32_t *keys = reinterpret_cast<uint32_t *>(mem + (sizeof(SubSmem<NW>) + 15) / 16 * 16);
    uint2 *mask = reinterpret_cast<uint2 *>(keys + nmax + 4);  // .x: key >= cut, .y: key <= cut
    uint32_t *pre = reinterpret_cast<uint32_t *>(mask + nwords);
    uint16_t *order = reinterpret_cast<uint16_t *>(pre + nwords);
    // the pairs to swap (the keys are done then): a cell's left positions, then its right ones
    uint16_t *pairs = reinterpret_cast<uint16_t *>(keys);
    const uint32_t lane = ti & 31, warp = ti >> 5, lt = (1u << lane) - 1u;
    const uint32_t keys_at = (uint32_t)__cvta_generic_to_shared(keys);
    const uint32_t ncells = v.counters->sub_cells[kClass];
    const int *list = v.sub_list + kClass * v.C;
    unsigned long long bytes = 0;
    // Copies the n words at src into keys[off ...] (off: src's misalignment in words, so that
    // 16-byte pieces stay aligned on both sides): one bulk copy for the whole pieces, plain loads
    // for the rest. begin_load after a barrier that ends the keys' last use; end_load, then a
    // barrier, before they are read, and the group leaves if any of its threads' waits ran out
    // (come_all). A wait polls at most v.copy_polls times (kCopyPolls: about a second, far beyond
    // any copy).
    const uint32_t arrived = (uint32_t)__cvta_generic_to_shared(&sm.arrived);
    uint32_t parity = 0;
    if (ti == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(arrived) : "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    sync();
    // each thread's last plain access to the keys, before the barrier ahead of a bulk copy
    auto done_with_keys = [&]() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); };
    auto begin_load = [&](const void *from, uint32_t n) -> uint32_t {
        const uint32_t *src = reinterpret_cast<const uint32_t *>(from);
        const uint32_t off = (uint32_t)(reinterpret_cast<uintptr_t>(src) >> 2) & 3u;
        const uint32_t head = min(n, (4u - off) & 3u), body = (n - head) & ~3u;
        if (ti == 0 && !v.drop_copies) {
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(arrived), "r"(4u * body) : "memory");
            if (body)
                asm volatile(
                    "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                        keys_at + 4 * (off + head)),
                    "l"(src + head), "r"(4u * body), "r"(arrived)
                    : "memory");
        }
        if (ti < head) keys[off + ti] = __ldcg(src + ti);
        if (ti >= 32 && ti - 32 < n - head - body) keys[off + head + body + ti - 32] = __ldcg(src + head + body + ti - 32);
        return off;
    };
    auto wait_copy = [&](uint32_t phase, uint32_t polls) -> bool {
        uint32_t ok = 0;
        for (uint32_t spins = 0; !ok && spins < polls; ++spins)
            asm volatile(
                "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n selp.b32 %0, 1, 0, p;\n}"
                : "=r"(ok)
                : "r"(arrived), "r"(phase), "r"(kCopyPollNs)
                : "memory");
        return ok != 0;
    };
    auto end_load = [&]() -> bool {
        const bool ok = wait_copy(parity, v.copy_polls);
        parity ^= 1u;
        return ok;
    };
    // The barrier, and whether every thread came with `ok` (a vote in the barrier: a flag in shared
    // memory made a tree of six levels 1% slower).
    auto come_all = [&](bool ok) -> bool {
        if (NW == 32) return __syncthreads_and(ok) != 0;
        uint32_t all;
        asm volatile("{\n .reg .pred p, q;\n setp.ne.u32 p, %1, 0;\n bar.red.and.pred q, %2, %3, p;\n selp.b32 %0, 1, 0, q;\n}"
                     : "=r"(all)
                     : "r"((uint32_t)ok), "r"(bar), "n"((int)NT)
                     : "memory");
        return all != 0;
    };
    // Where not all copies came: the group leaves, its own copy (if one is under way after all)
    // waited for once more.
    auto leave = [&]() {
        if (ti == 0) atomicExch(&v.counters->error, 1u);
        if (!v.drop_copies) wait_copy(parity ^ 1u, kCopyPolls);
        return false;
    };
    auto take = [&]() -> int {
        const uint32_t k = atomicAdd(&v.counters->sub_next[kClass], 1u);
        return k < ncells ? list[k] : -1;
    };
    auto prefetch = [&](const void *p, uint32_t words) {  // whole 16-byte pieces
        const uintptr_t a = (reinterpret_cast<uintptr_t>(p) + 15) & ~(uintptr_t)15;
        const uintptr_t e = (reinterpret_cast<uintptr_t>(p) + 4ull * words) & ~(uintptr_t)15;
        if (e > a)
            asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(a), "r"((uint32_t)(e - a)) : "memory");
    };
    // A group takes its next cell while it works on one, unless there are no more cells than
    // groups: the first groups to start then took two each, and the others, a few microseconds
    // later, none (2^20 particles, 32 cells of 2^15 on 32 CTAs: 142 or 270 us).
    const bool ahead = ncells > gridDim.x * (32 / NW);
    int next = -1;  // thread 0: the cell after this one
    bool started = false;
    for (;;) {
        if (ti == 0) {
            // this cell, and the next one, whose particles start their way into L2 meanwhile
            if (NW == 32 && !ahead)
                next = !started && blockIdx.x < ncells ? list[blockIdx.x] : -1;
            else if (!started || !ahead)
                next = take();
            started = true;
            sm.item = next;
            if (ahead && next >= 0) {
                next = take();
                if (next >= 0) {
                    const uint2 r = v.ranges[level_slot(v, next)];
                    prefetch(v.x + r.x, r.y - r.x);
                    prefetch(v.y + r.x, r.y - r.x);
                    prefetch(v.z + r.x, r.y - r.x);
                    if (v.idx) prefetch(v.idx + r.x, r.y - r.x);
                }
            }
            sm.max_it = sm.unfound = sm.degenerate = 0;
            sm.axes = sm.counted = 0;
            if (sm.item >= 0) {
                const int slot = level_slot(v, sm.item);
                const orb_cell_t &h = v.heap[slot];
                const uint2 rg = v.ranges[slot];
                SubCell &sc = sm.cell[0][0];
                sc.id = h.id;
                sc.leaves = h.nLeafCells;
                sc.axis = h.cutAxis;
                for (int a = 0; a < 3; ++a) {
                    sc.lower[a] = h.lower[a];
                    sc.upper[a] = h.upper[a];
                }
                sc.b = 0;
                sc.m = (uint16_t)(rg.y - rg.x);
                sm.root = slot;
            }
        }
        sync();
        const int c = sm.item;
        if (c < 0) break;
        const int root = sm.root, root_id = sm.cell[0][0].id;
        const uint32_t n = sm.cell[0][0].m, first = v.ranges[root].x;
        const int levels = levels_below(v, sm.cell[0][0].leaves);
        // heap slot of a descendant: slot - id is the instance's heap base
        const int heap0 = root - root_id;
        uint32_t off = begin_load(axis_keys(v, eff_axis(sm.cell[0][0].axis)) + first, n);  // the root's keys
        for (uint32_t p = ti; p < n; p += NT) order[p] = (uint16_t)p;
        bool loading = true;  // a copy of an axis is under way
        for (int l = 0; l < levels; ++l) {
            SubCell *const cells = sm.cell[l & 1];
            const uint32_t nq = 1u << l;
            // cell q's warps: gs of them (at least one), this warp is number gw of cell q0 and,
            // with more cells than warps, takes q0 + qs, ... too (then gs = 1)
            const uint32_t gs = max(1u, (uint32_t)NW >> l), q0 = warp / gs, gw = warp % gs, qs = NW / gs;
            const uint32_t nb = kBins >> l, lslots = kLists >> l, cap = min(kSubWindowList, lslots);
            if (ti < nq) {
                const SubCell &sc = cells[ti];
                SubState &s = sm.state[ti];
                const int a = eff_axis(sc.axis);
                s.L = s.a = sc.lower[a];  // setCutMargin, src/cell.h:123-126
                s.R = s.b = sc.upper[a];
                s.ratio = leaf_ratio(sc.leaves);  // src/orbit.cpp:204
                s.mode = sc.m ? kSubOpen : kSubDone;  // no key: the first cut is found (count 0 of 0)
                s.it = s.found = sc.m ? 0 : 1;
                s.cand = 0xffffffffu;
                s.nlist = s.s = 0;
                s.i = sc.m;
                atomicOr(&sm.axes, 1u << a);
                if (sc.m > kSubDirect) atomicOr(&sm.counted, 1u << a);
            }
            sync();
            const uint32_t axes = sm.axes, counted = sm.counted;
            const float *kf = reinterpret_cast<const float *>(keys);
            // f(word, key) for this warp's words of cell q, a run of consecutive ones (lanes past the
            // cell's end hold NaN); a position's key is the one its order entry names
            auto for_words = [&](uint32_t q, auto f) {
                const uint32_t m = cells[q].m, W = (m + 31) / 32, run = (W + gs - 1) / gs;
                uint32_t w = min(W, gw * run);
                const uint32_t end = min(W, w + run), full = min(m / 32, end);
                const uint16_t *ord = order + cells[q].b + lane + w * 32u;
                for (; w + kU <= full; w += kU, ord += kU * 32) {
                    uint32_t o[kU];
                    float k[kU];
#pragma unroll
                    for (int u = 0; u < kU; ++u) o[u] = ord[u * 32];
#pragma unroll
                    for (int u = 0; u < kU; ++u) k[u] = kf[o[u]];
#pragma unroll
                    for (int u = 0; u < kU; ++u) f(w + (uint32_t)u, k[u], Flag<true>());
                }
                for (; w < full; ++w, ord += 32) f(w, kf[*ord], Flag<true>());
                if (w < end) f(w, lane < (m & 31u) ? kf[*ord] : __int_as_float(0x7fc00000), Flag<false>());
            };
            // masks of cell q against lo and hi (see k_part_classify), the keys between listed;
            // returns this lane's keys that are not below hi
            auto classify = [&](uint32_t q, float lo, float hi) -> uint32_t {
                uint2 *mk = mask + ((uint32_t)cells[q].b >> 5) + q;
                const uint32_t vm = (1u << (cells[q].m & 31u)) - 1u;  // the partial word's positions
                uint32_t above = 0;
                for_words(q, [&](uint32_t w, float k, auto full) {
                    constexpr bool kFull = decltype(full)::value;
                    const uint32_t valid = kFull ? 0xffffffffu : vm;
                    const bool not_below = !(k < hi);
                    const uint32_t gb = __ballot_sync(0xffffffffu, not_below) & valid;
                    const uint32_t lb = __ballot_sync(0xffffffffu, !(k >= lo)) & valid;
                    above += not_below;
                    if (lane == 0) mk[w] = make_uint2(gb, lb);
                });
                // the unresolved keys to the list, a lane a word
                __syncwarp();
                const uint32_t W = (cells[q].m + 31u) / 32u, run = (W + gs - 1) / gs;
                const uint32_t w0 = min(W, gw * run), w1 = min(W, w0 + run);
                for (uint32_t w = w0 + lane; w < w1; w += 32) {
                    const uint2 x = mk[w];
                    uint32_t e = ~(x.x | x.y) & (w * 32u + 32u <= cells[q].m ? 0xffffffffu : vm);
                    if (!e) continue;
                    uint32_t at = atomicAdd(&sm.state[q].nlist, (uint32_t)__popc(e));
                    for (; e && at < lslots; e &= e - 1u, ++at) {
                        const uint32_t p = w * 32u + (uint32_t)__ffs(e) - 1u;
                        sm.lpos[q * lslots + at] = (uint16_t)p;
                    }
                }
                return above;
            };
            for (int ax = 0; ax < 3; ++ax) {
                if (!((axes >> ax) & 1u)) continue;
                if (!loading) off = begin_load(axis_keys(v, ax) + first, n);
                loading = false;
                kf = reinterpret_cast<const float *>(keys) + off;
                bytes += 4ull * n;
                auto mine = [&](uint32_t q) { return eff_axis(cells[q].axis) == ax; };
                // rounds: histogram of the keys over the window (keys outside it in the end
                // bins), then the window narrowed to the bins of the ranks around the target
                auto counts = [&](uint32_t q) {
                    return mine(q) && cells[q].m > kSubDirect && sm.state[q].mode == kSubOpen && sm.state[q].cand > cap;
                };
                if (ti == 0) sm.direct = 0;
                if (!((counted >> ax) & 1u)) {
                    if (!come_all(end_load())) return leave();
                }
                for (int r = 0; (counted >> ax) & 1u; ++r) {
                    for (uint32_t j = ti; j < kBins; j += NT) sm.bins[j] = 0u;
                    if (ti == 0) sm.more = 0;
                    if (!come_all(r > 0 || end_load())) return leave();
                    bool any = false;
                    for (uint32_t q = q0; q < nq; q += qs) {
                        if (!counts(q)) continue;
                        any = true;
                        const float a = sm.state[q].a, scale = __frcp_rn(__fsub_rn(sm.state[q].b, a));
                        const float top = (float)(nb - 1u);
                        // the float 2^23 + g holds bin g in its low bits: 4 times its encoding plus
                        // `at` is the bin's address
                        const uint32_t at = (uint32_t)__cvta_generic_to_shared(sm.bins + q * nb) - 4u * 0x4b000000u;
                        for_words(q, [&](uint32_t, float k, auto full) {
                            const float t = __saturatef(__fmul_rn(__fsub_rn(k, a), scale));  // NaN: bin 0
                            const uint32_t e = __float_as_uint(__fmaf_rn(t, top, 8388608.0f));
                            if (decltype(full)::value || k == k)
                                asm volatile("red.shared.add.u32 [%0], 1;" ::"r"(4u * e + at) : "memory");
                        });
                    }
                    sync();
                    // the bins of the ranks 4 below and above ratio * m: a cut the test accepts has
                    // a count within 3 of that
                    const uint32_t per = nb / (gs * 32u);
                    auto narrow = [&](uint32_t q, uint32_t j0, uint32_t run) {
                        SubState &s = sm.state[q];
                        const uint32_t target = (uint32_t)(s.ratio * (float)cells[q].m), r0 = target - 4u, r1 = target + 4u;
                        const float a = s.a, step = __fdiv_rn(__fsub_rn(s.b, a), (float)(nb - 1u));
                        for (uint32_t j = j0; j < j0 + per; ++j) {
                            const uint32_t h = sm.bins[q * nb + j];
                            // bin j holds the keys rounded to j: [j - 1/2, j + 1/2) steps above a
                            if (run <= r0 && r0 < run + h) {
                                s.L = __fadd_rn(a, __fmul_rn((float)j - 0.53125f, step));
                                s.cnt = run;
                            }
                            if (run <= r1 && r1 < run + h) {
                                s.R = __fadd_rn(a, __fmul_rn((float)j + 0.53125f, step));
                                s.cross = run + h;
                            }
                            run += h;
                        }
                    };
                    // (s.L, s.R, s.cnt and s.cross carry the new window and its ranks here; the
                    // bracket is set again below)
                    if (gs == 1) {
                        for (uint32_t q = q0; q < nq; q += qs) {
                            if (!counts(q)) continue;
                            uint32_t loc = 0, tot;
                            for (uint32_t j = 0; j < per; ++j) loc += sm.bins[q * nb + lane * per + j];
                            const uint32_t ex = warp_excl_scan(loc, &tot);
                            if (lane == 0) {
                                sm.state[q].L = sm.state[q].R = __int_as_float(0x7fc00000);
                                sm.state[q].cnt = sm.state[q].cross = 0;
                            }
                            __syncwarp();
                            narrow(q, lane * per, ex);
                        }
                    } else {
                        uint32_t loc = 0, wtot;
                        if (any)
                            for (uint32_t j = 0; j < per; ++j) loc += sm.bins[q0 * nb + (gw * 32u + lane) * per + j];
                        const uint32_t ex = warp_excl_scan(loc, &wtot);
                        if (lane == 0) {
                            sm.part[warp] = wtot;
                            if (any && gw == 0) {
                                sm.state[q0].L = sm.state[q0].R = __int_as_float(0x7fc00000);
                                sm.state[q0].cnt = sm.state[q0].cross = 0;
                            }
                        }
                        sync();
                        const uint32_t before = __reduce_add_sync(0xffffffffu, lane < gw ? sm.part[warp - gw + lane] : 0u);
                        if (any) narrow(q0, (gw * 32u + lane) * per, before + ex);
                    }
                    sync();
                    for (uint32_t q = q0; q < nq; q += qs) {
                        if (gw || lane || !counts(q)) continue;
                        SubState &s = sm.state[q];
                        const uint32_t cand = s.cross - s.cnt;
                        const float na = s.L, nbnd = s.R;
                        const int a = eff_axis(cells[q].axis);
                        s.L = cells[q].lower[a];
                        s.R = cells[q].upper[a];
                        s.cnt = 0;  // (from here on: the classify pass's count)
                        if (!(na < nbnd) || (cand > cap && (r == 3 || cand >= s.cand))) {
                            s.mode = kSubCount;  // ranks outside the bins (NaN keys), or no narrowing
                        } else {
                            s.a = na;
                            s.b = nbnd;
                            s.cand = cand;
                            if (cand > cap) sm.more = 1;
                        }
                    }
                    sync();
                    const bool again = sm.more != 0;
                    sync();  // (more is cleared by the next round)
                    if (!again) break;
                }
                // small cells: the whole loop by one warp, the keys in its registers; the others:
                // masks and list against the window
                for (uint32_t q = q0; q < nq; q += qs) {
                    if (!mine(q)) continue;
                    SubState &s = sm.state[q];
                    const uint32_t m = cells[q].m;
                    if (m <= kSubDirect) {
                        if (gw || s.mode == kSubDone) continue;
                        float kl[kSubDirect / 32], L = s.L, R = s.R;
                        uint32_t it = 0;
#pragma unroll
                        for (int j = 0; j < (int)kSubDirect / 32; ++j) {
                            const uint32_t p = (uint32_t)j * 32u + lane;
                            kl[j] = p < m ? kf[order[cells[q].b + p]] : __int_as_float(0x7fc00000);  // NaN: never below
                        }
                        const int st = bisect_list(kl, 0u, m, s.ratio, L, R, it);
                        __syncwarp();
                        if (lane == 0) {
                            s.L = L;
                            s.R = R;
                            s.it = (uint16_t)it;
                            s.found = st == kFound;
                            s.mode = kSubDone;
                        }
                    } else if (s.mode == kSubOpen) {
                        uint32_t above = classify(q, s.a, s.b);
                        // (lanes past the cell's end hold NaN, counted by the last word's warp)
                        above = __reduce_add_sync(0xffffffffu, above);
                        if (lane == 0 && above) atomicAdd(&s.cnt, above);
                    }
                }
                sync();
                // the window's exact counts, and the replay of the loop on the list
                for (uint32_t q = q0; q < nq; q += qs) {
                    SubState &s = sm.state[q];
                    const uint32_t m = cells[q].m;
                    if (gw || !mine(q) || m <= kSubDirect || s.mode == kSubDone) continue;
                    uint32_t mode = s.mode;
                    const uint32_t nl = s.nlist;
                    if (mode == kSubOpen && nl <= cap) {
                        const uint32_t wb = ((uint32_t)cells[q].b >> 5) + q;
                        // keys at or above b, and NaN (without the partial word's empty lanes)
                        const uint32_t g = s.cnt - ((m & 31u) ? 32u - (m & 31u) : 0u);
                        const uint32_t below = m - g - nl;
                        // NaN keys are in g and never below a cut: count(< b) = below + nl all the same
                        const float ratio = s.ratio;
                        const bool low = convergence(below, m, ratio) < 0, high = convergence(below + nl, m, ratio) > 0;
                        const float a = s.a, b = s.b;
                        float kl[kSubWindowList / 32], L = s.L, R = s.R;
#pragma unroll
                        for (int j = 0; j < (int)kSubWindowList / 32; ++j) {
                            const uint32_t e = (uint32_t)j * 32u + lane;
                            kl[j] = e < nl ? kf[order[cells[q].b + sm.lpos[q * lslots + e]]] : __int_as_float(0x7fc00000);
                        }
                        uint32_t it = 0;
                        int st = kActive;
                        while (st == kActive) {
                            if (it >= (uint32_t)kMaxIterations) {
                                st = kCapped;
                                break;
                            }
                            const float cut = mid_cut(L, R);
                            int dir;
                            if (cut <= a) {
                                if (!low) break;
                                dir = -1;
                            } else if (cut >= b) {
                                if (!high) break;
                                dir = 1;
                            } else {
                                uint32_t cc = 0;
#pragma unroll
                                for (int j = 0; j < (int)kSubWindowList / 32; ++j) cc += kl[j] < cut;
                                dir = convergence(below + __reduce_add_sync(0xffffffffu, cc), m, ratio);
                            }
                            ++it;
                            if (dir == 0)
                                st = kFound;
                            else if (dir > 0)
                                R = cut;
                            else
                                L = cut;
                        }
                        const float cut = mid_cut(L, R);
                        if (st != kActive && cut > a && cut < b) {
                            // the listed keys' bits against the final cut
#pragma unroll
                            for (int j = 0; j < (int)kSubWindowList / 32; ++j) {
                                const uint32_t e = (uint32_t)j * 32u + lane;
                                if (e < nl) {
                                    const uint32_t p = sm.lpos[q * lslots + e], bit = 1u << (p & 31u);
                                    if (!(kl[j] < cut)) atomicOr(&mask[wb + (p >> 5)].x, bit);
                                    if (!(kl[j] > cut)) atomicOr(&mask[wb + (p >> 5)].y, bit);
                                }
                            }
                            mode = kSubWindow;
                            if (lane == 0) {
                                s.L = L;
                                s.R = R;
                                s.it = (uint16_t)it;
                                s.found = st == kFound;
                                s.mode = kSubWindow;
                            }
                        }
                    }
                    __syncwarp();
                    if (mode != kSubWindow && lane == 0) {
                        s.mode = kSubCount;
                        sm.direct = 1;
                    }
                }
                sync();
                if (sm.direct) {
                    // cells the window did not settle: every cut counted over all the keys
                    for (int it = 0; it < kMaxIterations; ++it) {
                        if (ti < nq) sm.state[ti].cnt = 0;
                        if (ti == 0) sm.more = 0;
                        sync();
                        for (uint32_t q = q0; q < nq; q += qs) {
                            if (!mine(q) || sm.state[q].mode != kSubCount) continue;
                            const float cut = mid_cut(sm.state[q].L, sm.state[q].R);
                            uint32_t cc = 0;
                            for_words(q, [&](uint32_t, float k, auto) { cc += k < cut; });
                            cc = __reduce_add_sync(0xffffffffu, cc);
                            if (lane == 0 && cc) atomicAdd(&sm.state[q].cnt, cc);
                        }
                        sync();
                        if (ti < nq && mine(ti) && sm.state[ti].mode == kSubCount) {
                            SubState &s = sm.state[ti];
                            const float cut = mid_cut(s.L, s.R);
                            const uint32_t was_l = __float_as_uint(s.L), was_r = __float_as_uint(s.R);
                            ++s.it;
                            const int dir = convergence(s.cnt, cells[ti].m, s.ratio);
                            if (dir == 0) {
                                s.found = 1;
                                s.mode = kSubDone;
                            } else if (dir > 0) {
                                s.R = cut;
                            } else {
                                s.L = cut;
                            }
                            // a bracket that stays as it is gives the same cut up to the cap
                            if (dir != 0 && was_l == __float_as_uint(s.L) && was_r == __float_as_uint(s.R)) {
                                s.it = kMaxIterations;
                                s.mode = kSubDone;
                            } else if (dir != 0) {
                                sm.more = 1;
                            }
                        }
                        sync();
                        const bool again = sm.more != 0;
                        sync();
                        if (!again) break;
                    }
                }
                // masks against the final cut, where the window did not give them
                for (uint32_t q = q0; q < nq; q += qs) {
                    if (!mine(q) || sm.state[q].mode == kSubWindow) continue;
                    const float cut = mid_cut(sm.state[q].L, sm.state[q].R);
                    classify(q, next_above(cut), cut);
                }
                done_with_keys();
                sync();
            }
            // prefixes of the masks' counts (>= in the low half of a word, <= in the high half)
            // and the word where #{>= before} crosses #{<= after}
            auto popcounts = [&](uint32_t wb, uint32_t w0, uint32_t w1) {
                uint32_t t = 0;
                for (uint32_t w = w0; w < w1; ++w) {
                    const uint2 x = mask[wb + w];
                    t += (uint32_t)__popc(x.x) + ((uint32_t)__popc(x.y) << 16);
                }
                return t;
            };
            auto prefix = [&](uint32_t q, uint32_t wb, uint32_t w0, uint32_t w1, uint32_t run, uint32_t le_tot) {
                for (uint32_t w = w0; w < w1; ++w) {
                    const bool was = w > 0 && (run & 0xffffu) >= le_tot - (run >> 16);
                    const uint2 x = mask[wb + w];
                    pre[wb + w] = run;
                    run += (uint32_t)__popc(x.x) + ((uint32_t)__popc(x.y) << 16);
                    if (!was && (run & 0xffffu) >= le_tot - (run >> 16)) sm.state[q].cross = w;
                }
            };
            if (gs == 1) {
                for (uint32_t q = q0; q < nq; q += qs) {
                    const uint32_t W = ((uint32_t)cells[q].m + 31) / 32, pw = (W + 31) / 32, wb = ((uint32_t)cells[q].b >> 5) + q;
                    const uint32_t w0 = min(W, lane * pw), w1 = min(W, w0 + pw);
                    uint32_t tot;
                    const uint32_t ex = warp_excl_scan(popcounts(wb, w0, w1), &tot);
                    if (lane == 0) sm.state[q].tot = tot;
                    prefix(q, wb, w0, w1, ex, tot >> 16);
                }
                __syncwarp();
            } else {
                const uint32_t W = ((uint32_t)cells[q0].m + 31) / 32, pw = (W + gs * 32u - 1) / (gs * 32u);
                const uint32_t wb = ((uint32_t)cells[q0].b >> 5) + q0;
                const uint32_t w0 = min(W, (gw * 32u + lane) * pw), w1 = min(W, w0 + pw);
                uint32_t wtot;
                const uint32_t ex = warp_excl_scan(popcounts(wb, w0, w1), &wtot);
                if (lane == 0) sm.part[warp] = wtot;
                sync();
                const uint32_t pv = lane < gs ? sm.part[warp - gw + lane] : 0u;
                const uint32_t before = __reduce_add_sync(0xffffffffu, lane < gw ? pv : 0u);
                const uint32_t tot = __reduce_add_sync(0xffffffffu, pv);
                if (gw == 0 && lane == 0) sm.state[q0].tot = tot;
                prefix(q0, wb, w0, w1, before + ex, tot >> 16);
                sync();
            }
            // The swap count s = max over x of min(#>= in [0,x), #<= in [x,m)): it lies in that word
            // (every warp of the cell finds it). Then the pairs, a lane a word: left elements by
            // rank (pair k: the key >= cut of rank k), right ones (the key <= cut of rank le-1-k),
            // and the split index i = min(L_{s+1}, R_s). A word's 16 or so bits one after the other
            // in a lane cost a sixth of the instructions of a warp a word.
            for (uint32_t q = q0; q < nq; q += qs) {
                SubState &s = sm.state[q];
                const uint32_t b = cells[q].b, W = ((uint32_t)cells[q].m + 31) / 32, wb = (b >> 5) + q;
                if (!W) continue;
                const uint32_t x = s.cross, le_tot = s.tot >> 16;
                const uint2 cw = mask[wb + x];
                const uint32_t f = pre[wb + x] & 0xffffu, g = le_tot - (pre[wb + x] >> 16), upto = 0xffffffffu >> (31u - lane);
                const uint32_t ns = __reduce_max_sync(
                    0xffffffffu, max(min(f, g), min(f + __popc(cw.x & upto), g - __popc(cw.y & upto))));
                if (gw == 0 && lane == 0) s.s = ns;
                const uint32_t first_le = le_tot - ns;  // ranks from here on are partners
                uint16_t *const pl = pairs + 2 * b, *const pr = pl + cells[q].m;
                if (gw == 0) {  // the crossing word, a lane a bit: it can hold both kinds, and i
                    const uint32_t kg = f + __popc(cw.x & lt), kl = le_tot - g + __popc(cw.y & lt);
                    const bool isg = (cw.x >> lane) & 1u, isl = (cw.y >> lane) & 1u;
                    if (isg && kg < ns) pl[kg] = (uint16_t)(b + x * 32u + lane);
                    if (isl && kl >= first_le) pr[le_tot - 1u - kl] = (uint16_t)(b + x * 32u + lane);
                    if ((isg && kg == ns) || (isl && kl == first_le && ns)) atomicMin(&s.i, x * 32u + lane);
                }
                // words before it: every key >= cut is a left element; words behind it: every key <=
                // cut a partner. A lane takes words of its own run, each lane starting elsewhere in
                // it, so the lanes' ranks (16 a word apart) fall on different banks.
                const uint32_t run = (W + 31) / 32;
                for (uint32_t j = gw, r0 = lane % run; j < run; j += gs) {
                    uint32_t o = j + r0;
                    if (o >= run) o -= run;
                    const uint32_t w = lane * run + o;
                    if (w >= W || w == x) continue;
                    const uint2 k = mask[wb + w];
                    const uint32_t at = pre[wb + w], rgt = at & 0xffffu, rl = at >> 16;
                    const bool behind = w > x;
                    uint32_t e = behind ? k.y : k.x;
                    uint16_t *dst = behind ? pr + (le_tot - 1u - rl) : pl + rgt;
                    const int step = behind ? -1 : 1;
                    if (behind) {
                        if (rgt <= ns && ns < rgt + (uint32_t)__popc(k.x))
                            atomicMin(&s.i, w * 32u + select_in_word(k.x, ns - rgt));
                        if (e && rl == first_le && ns) atomicMin(&s.i, w * 32u + (uint32_t)__ffs(e) - 1u);
                    }
                    const uint32_t base = b + w * 32u - 1u;
                    for (; e; e &= e - 1u, dst += step) *dst = (uint16_t)(base + (uint32_t)__ffs(e));
                }
            }
            sync();
            // the swaps (the two sides' positions are disjoint)
            for (uint32_t q = q0; q < nq; q += qs) {
                const uint16_t *const pl = pairs + 2 * (uint32_t)cells[q].b, *const pr = pl + cells[q].m;
                for (uint32_t k = gw * 32u + lane; k < sm.state[q].s; k += gs * 32u) {
                    const uint32_t pa = pl[k], pb = pr[k];
                    const uint16_t oa = order[pa], ob = order[pb];
                    order[pa] = ob;
                    order[pb] = oa;
                }
            }
            done_with_keys();
            sync();
            if (l + 1 == levels && n) off = begin_load(v.x + first, n);  // for the final pass
            // the final swap, the split (Cell::cut, src/cell.h:78-100) and the children, a thread a cell
            if (ti < nq) {
                const SubCell sc = cells[ti];
                const SubState &s = sm.state[ti];
                const uint32_t b = sc.b, m = sc.m, i = s.i;
                if (i < m) {
                    const uint16_t oa = order[b + i];
                    order[b + i] = order[b + m - 1];
                    order[b + m - 1] = oa;
                } else {
                    atomicAdd(&sm.degenerate, 1u);
                }
                orb_cell_t &h = v.heap[heap0 + sc.id];
                h.cutMarginLeft = s.L;
                h.cutMarginRight = s.R;
                h.foundCut = (uint8_t)s.found;
                atomicMax(&sm.max_it, (uint32_t)s.it);
                if (!s.found) atomicAdd(&sm.unfound, 1u);
                orb_cell_t cell;
                cell.id = sc.id;
                cell.nLeafCells = sc.leaves;
                cell.cutAxis = sc.axis;
                cell.cutMarginLeft = s.L;
                cell.cutMarginRight = s.R;
                for (int a = 0; a < 3; ++a) {
                    cell.lower[a] = sc.lower[a];
                    cell.upper[a] = sc.upper[a];
                }
                orb_cell_t kid[2];
                split_child(cell, 0, kid[0], v.counters);
                split_child(cell, 1, kid[1], v.counters);
#pragma unroll
                for (int w = 0; w < 2; ++w) {
                    const int slot = heap0 + kid[w].id;
                    const uint32_t kb = w ? b + i : b, km = w ? m - i : i;
                    v.heap[slot] = kid[w];
                    v.ranges[slot] = make_uint2(first + kb, first + kb + km);
                    if (l + 1 < levels) {
                        SubCell &o = sm.cell[(l + 1) & 1][2 * ti + w];
                        o.id = kid[w].id;
                        o.leaves = kid[w].nLeafCells;
                        o.axis = kid[w].cutAxis;
                        for (int a = 0; a < 3; ++a) {
                            o.lower[a] = kid[w].lower[a];
                            o.upper[a] = kid[w].upper[a];
                        }
                        o.b = (uint16_t)kb;
                        o.m = (uint16_t)km;
                    }
                }
            }
            if (ti == 0) sm.axes = sm.counted = 0;
            sync();
        }
        // the particles, one array after the other
        uint32_t *const arr[4] = {reinterpret_cast<uint32_t *>(v.x), reinterpret_cast<uint32_t *>(v.y),
                                  reinterpret_cast<uint32_t *>(v.z), v.idx};
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            if (!n || !arr[a]) continue;  // (without particles the coordinates may be null)
            uint32_t *dst = arr[a] + first;
            if (a > 0) off = begin_load(dst, n);
            if (!come_all(end_load())) return leave();
            const uint32_t *from = keys + off;
            uint32_t p = ti;
            for (; p + 7 * NT < n; p += 8 * NT) {
                uint32_t x[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) x[u] = from[order[p + u * NT]];
#pragma unroll
                for (int u = 0; u < 8; ++u) dst[p + u * NT] = x[u];
            }
            for (; p < n; p += NT) dst[p] = from[order[p]];
            done_with_keys();
            sync();
            bytes += 8ull * n;
        }
        if (ti == 0) {
            atomicMax(&v.counters->max_iters, sm.max_it);
            if (sm.unfound) atomicAdd(&v.counters->unfound, sm.unfound);
            if (sm.degenerate) atomicAdd(&v.counters->degenerate, sm.degenerate);
        }
        if (v.hwin) {
            // the cell is final: every thread's writes made visible beyond the GPU, then the
            // last cell of its window reports the window's particle range to the host
            __threadfence_system();
            sync();
            if (ti == 0) {
                const uint32_t w = (uint32_t)c / v.win_cells;
                const uint32_t c0 = w * v.win_cells, c1 = min(c0 + v.win_cells, (uint32_t)v.C) - 1u;
                if (atomicAdd(&v.win_cnt[w], 1u) == c1 - c0) {
                    __threadfence_system();
                    const uint2 r = make_uint2(v.ranges[level_slot(v, (int)c0)].x,
                                               v.ranges[level_slot(v, (int)c1)].y);
                    volatile uint32_t *hr = &v.hwin->range[w].x;
                    hr[0] = r.x;
                    hr[1] = r.y;
                    __threadfence_system();
                    *(volatile uint32_t *)&v.hwin->done[w] = 1u;
                }
            }
        }
    }
    if (ti == 0 && bytes) add_bytes(v, kKSubtree, bytes);
    return true;
}

// The level's cells, largest class first: all of the CTA's warps on one cell, then groups of
// 16, 8 and 2 warps on their own slices of its shared memory. A class is not begun by a CTA one of
// whose groups left the one before.
__global__ void __launch_bounds__(kSubThreads) k_subtree(const __grid_constant__ Level v) {
    pdl_enter();
    if (*(volatile const uint32_t *)v.skip != 1u) return;  // the level kernels run instead
    const uint32_t tid = threadIdx.x;
    bool ok = true;
    if (v.counters->sub_cells[0]) ok = sub_group<32>(v, 0u, tid, 0);
    if (!__syncthreads_and(ok)) return;
    if (v.counters->sub_cells[1]) {
        const uint32_t k = tid / 512;
        ok = sub_group<16>(v, k * sub_bytes<16>(kSub16), tid % 512, 1 + (int)k);
    }
    if (!__syncthreads_and(ok)) return;
    if (v.counters->sub_cells[2]) {
        const uint32_t k = tid / 256;
        ok = sub_group<8>(v, k * sub_bytes<8>(kSub8), tid % 256, 1 + (int)k);
    }
    if (!__syncthreads_and(ok)) return;
    if (v.counters->sub_cells[3]) {
        const uint32_t k = tid / 64;
        sub_group<2>(v, k * sub_bytes<2>(kSub2), tid % 64, (int)k);
    }
}

// ------------------------------------------------------------------------------------
// Weighted builds: the reference's bisection loop on integer weight sums instead of counts
// (the thesis's weighted ORB, documentation/notes.tex:259-271; never implemented by the
// reference). A pass bins the weights of an active cell's bracket into its midpoint tree (the
// reference's own cuts, binned exactly as in the count passes) and replays up to its depth of
// iterations on the prefix sums with the weighted test; the first pass also sums the weights
// below the bracket and the cell's total. Integer sums: the same results in any order.
//
// A cell whose tiles one CTA reads (all cells of at most one tile, but on levels of few cells)
// is bisected to the end in one launch: up to kWDirect keys with the keys and weights in the
// CTA's registers, every cut's weight summed (2.5 us a cell of 2^11 keys, against 12 with
// histograms; 4096 cells of 3900: 120 us, against 160),
// more with the bins in shared memory. Larger cells take kWPasses launches, the CTA that brings
// the last piece replaying; levels of few cells deal quarter tiles to the CTAs. A bin is two 32-bit sums, of the weights' low and high
// halves (the high one is touched only by weights above 65535): shared memory has no 64-bit
// add of its own, and an add that loops on compare-and-swap bound the passes (2^24 clustered
// particles into 2^14 leaves: 4.0 ms of count passes with 64-bit bins, 256 a pass, four
// launches a level and the descent for every key).
// ------------------------------------------------------------------------------------
__device__ __forceinline__ unsigned long long block_sum_u64(unsigned long long x,
                                                            unsigned long long *sh) {
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    __syncthreads();
    if (lane == 0) sh[warp] = x;
    __syncthreads();
    unsigned long long t = 0;
    for (int w = 0; w < nw; ++w) t += sh[w];
    return t;
}

// convergence_weighted() prepared for one cell: with W below 2^32 (k <= 2^30) the products fit
// 64 bits, and n |D| < 3 k W is |D| < ceil(3 k W / n) for the integer |D|, one division a cell
// in place of two 128-bit products a step (a third of the deep levels' passes).
struct WeightTest {
    unsigned long long W, half_w, limit;
    uint32_t n;
    int32_t k;
    __device__ __forceinline__ WeightTest(unsigned long long w_cell, uint32_t n_, int32_t leaves)
        : W(w_cell), half_w(0), limit(0), n(n_), k(leaves) {
        if (!(W >> 32)) {
            half_w = (unsigned long long)((k + 1) / 2) * W;
            const unsigned long long b = 3ull * (unsigned long long)k * W;
            limit = n ? (b + (n - 1)) / n : 0ull;
            if (b + (n - 1) < b) limit = b / n + (b % n ? 1ull : 0ull);
        }
    }
    __device__ __forceinline__ int dir(unsigned long long w_left) const {
        if (W >> 32) return convergence_weighted(w_left, W, n, k);
        const long long D = (long long)((unsigned long long)k * w_left) - (long long)half_w;
        const unsigned long long ad = (unsigned long long)(D < 0 ? -D : D);
        if (D == 0 || ad < limit) return 0;
        return D > 0 ? 1 : -1;
    }
};

// Tree depth of a pass over a cell of n keys that one CTA finishes: about two keys a bin, the
// full depth for cells of more than a tile (so kWPasses launches reach the iteration cap; cells
// dealt in pieces take it too).
__device__ __forceinline__ int weighted_depth(uint32_t n) {
    return max(4, min(kMaxBinsLog2, 30 - __clz(max(n, 1u))));
}
static_assert(kWPasses * kMaxBinsLog2 >= kMaxIterations, "the weighted passes reach the cap");
constexpr uint32_t kWDirect = 16 * kThreads;
constexpr uint32_t kWFlush = 4;  // tiles whose low halves fit a 32-bit bin
static_assert((unsigned long long)kWFlush * kTile * 0xffffull < (1ull << 32), "low halves of a run of tiles");

// The cell a CTA is working on, in shared memory.
struct WeightCell {
    const float *keys;
    float L, R;
    int K;
    uint32_t base, end, t0;
    Guess gs;
    unsigned long long below, tot;  // weight below L; the cell's weight
    uint32_t it, state, last;
};

struct WeightSmem {
    union {
        uint32_t half[2][kHistBins];      // low and high halves' sums
        unsigned long long pre[kHistBins];  // the replay's prefix sums
    };
    float edge[kHistBins + 1];
    unsigned long long red[kThreads / 32];
    uint32_t sum[2][2][kThreads / 32];  // direct sums by parity of the step: halves, a warp each
    WeightCell cell;
    uint32_t run[2], next;
};

// Replay of up to K iterations on the finished bins of cell c (in shared memory, or added up
// in global memory by several CTAs), every thread; the cell's bracket and state in sm.cell.
template <bool kWide>
__device__ __noinline__ void weighted_replay(const Level &v, int c, bool global, WeightSmem &sm) {
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    WeightCell &w = sm.cell;
    const uint32_t nb = 1u << w.K, per = max(1u, nb / kThreads);
    unsigned long long h[kHistBins / kThreads], run = 0;
    unsigned long long *g = v.whist + v.hist_off[c];
#pragma unroll
    for (int j = 0; j < (int)(kHistBins / kThreads); ++j) {
        h[j] = 0;
        const uint32_t b = tid * per + (uint32_t)j;
        if ((uint32_t)j < per && b < nb) {
            if (global) {
                h[j] = __ldcg(g + b);  // other CTAs' atomics: from L2
                g[b] = 0ull;
            } else {
                h[j] = (unsigned long long)sm.half[0][b] + ((unsigned long long)sm.half[1][b] << 16);
            }
        }
        run += h[j];
    }
    unsigned long long inc = run;
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= (uint32_t)o) inc += t;
    }
    if (lane == 31) sm.red[warp] = inc;
    __syncthreads();  // (and every bin is read)
    for (uint32_t k = 0; k < warp; ++k) inc += sm.red[k];
    run = inc - run;
#pragma unroll
    for (int j = 0; j < (int)(kHistBins / kThreads); ++j) {
        const uint32_t b = tid * per + (uint32_t)j;
        if ((uint32_t)j < per && b < nb) sm.pre[b] = run;
        run += h[j];
    }
    __syncthreads();
    const uint32_t n = w.end - w.base;
    float L = w.L, R = w.R;
    uint32_t it = w.it, pos = 0;
    uint8_t st = kActive;
    unsigned long long finite = ~0ull;  // (kWide) the weight of the keys below +inf, see replay()
    auto attempt = [&]() -> bool {
        const WeightTest test(w.tot, n, v.heap[level_slot(v, c)].nLeafCells);
        uint32_t width = nb;
        for (int step = 0; step < w.K; ++step) {
            if (it >= (uint32_t)kMaxIterations) break;
            const uint32_t half = width >> 1;
            unsigned long long wl = w.below + sm.pre[pos + half];
            if (kWide && overflowed(mid_cut(L, R))) {
                if (finite == ~0ull) return false;
                wl = mid_cut(L, R) > 0.f ? finite : 0ull;
            }
            ++it;
            const int dir = test.dir(wl);
            if (dir == 0) {
                st = kFound;
                break;
            }
            const float cut = mid_cut(L, R);
            if (dir > 0) {
                R = cut;
            } else {
                L = cut;
                pos += half;
            }
            width = half;
        }
        if (st == kActive && it >= (uint32_t)kMaxIterations) st = kCapped;
        return true;
    };
    if (kWide) {  // a trial run by every thread
        if (!attempt()) {
            finite = 0;
            for (uint32_t p = w.base + tid; p < w.end; p += kThreads)
                if (__ldg(w.keys + p) < __int_as_float(0x7f800000)) finite += __ldg(v.wt + p);
            finite = block_sum_u64(finite, sm.red);
        }
        L = w.L, R = w.R, it = w.it, pos = 0, st = kActive;
        __syncthreads();
    }
    if (tid == 0) {
        attempt();
        // the weight below the new bracket: below the old one plus the bins left of it
        w.below += sm.pre[pos];
        w.L = L;
        w.R = R;
        w.it = it;
        w.state = st;
        w.gs = make_guess(L, R, __fdiv_rn((float)nb, __fsub_rn(R, L)), nb);
    }
    __syncthreads();
}

// The whole loop of a cell of at most kPer keys a thread by the CTA, keys and weights in registers.
template <uint32_t kPer>
__device__ __noinline__ void weighted_direct(const Level &v, int c, WeightSmem &sm) {
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    WeightCell &w = sm.cell;
    const int32_t leaves = v.heap[level_slot(v, c)].nLeafCells;
    const uint32_t n = w.end - w.base;
    float k[kPer], L = w.L, R = w.R;
    uint32_t x[kPer];
#pragma unroll
    for (int j = 0; j < (int)kPer; ++j) {
        const uint32_t p = (uint32_t)j * kThreads + tid;
        k[j] = p < n ? __ldg(w.keys + w.base + p) : __int_as_float(0x7fc00000);  // NaN: never below
        x[j] = p < n ? __ldg(v.wt + w.base + p) : 0u;
    }
    // the CTA's sum of the weights of the keys below cut, in every thread; one barrier a step
    uint32_t step = 0;
    auto below = [&](float cut, bool all) -> unsigned long long {
        uint32_t lo = 0, hi = 0;
#pragma unroll
        for (int j = 0; j < (int)kPer; ++j) {
            const uint32_t y = all || k[j] < cut ? x[j] : 0u;
            lo += y & 0xffffu;
            hi += y >> 16;
        }
        lo = __reduce_add_sync(0xffffffffu, lo);
        hi = __reduce_add_sync(0xffffffffu, hi);
        uint32_t(*s)[kThreads / 32] = sm.sum[step++ & 1u];
        if (lane == 0) {
            s[0][warp] = lo;
            s[1][warp] = hi;
        }
        __syncthreads();
        lo = __reduce_add_sync(0xffffffffu, lane < kThreads / 32 ? s[0][lane] : 0u);
        hi = __reduce_add_sync(0xffffffffu, lane < kThreads / 32 ? s[1][lane] : 0u);
        return (unsigned long long)lo + ((unsigned long long)hi << 16);
    };
    const WeightTest test(below(0.f, true), n, leaves);
    uint32_t it = 0;
    int st = kActive;
    while (st == kActive) {
        if (it >= (uint32_t)kMaxIterations) {
            st = kCapped;
            break;
        }
        const float cut = mid_cut(L, R);
        ++it;
        const int dir = test.dir(below(cut, false));
        if (dir == 0)
            st = kFound;
        else if (dir > 0)
            R = cut;
        else
            L = cut;
    }
    __syncthreads();  // every thread has left the cell and the sums
    if (tid == 0) {
        w.L = L;
        w.R = R;
        w.it = it;
        w.state = (uint32_t)st;
        w.below = 0;
    }
    __syncthreads();
}

// A later pass's round that leaves a warp many keys in the bracket, mostly equal ones (see
// bracket_tile): bits `in` of its lanes' keys at p0, p0 + kThreads, ...; 32 at a time, the first
// one's bin found once and its equals' weights added together. (A tile of equal keys took 85 us,
// two additions to the same words a key; half of 6.4 million particles on one point, 2^14 leaves,
// whose large cell's tiles are a few CTAs' runs among small cells: 7.1 -> 4.6 ms.)
__device__ __noinline__ void tied_weights(const uint32_t *wt, uint32_t p0, uint32_t in, WeightSmem &sm) {
    const uint32_t lane = threadIdx.x & 31u, top = (1u << sm.cell.K) - 1u;
    const float *keys = sm.cell.keys;
    float tie = __int_as_float(0x7fc00000);
    uint32_t bin = 0;
    auto bin_of = [&](float k) -> uint32_t {
        uint32_t b;
        return guess_bin(sm.cell.gs, k, &b) ? b : near_bin(k, sm.cell.gs, sm.edge, top);
    };
#pragma unroll 1
    for (uint32_t any = __reduce_or_sync(0xffffffffu, in); any; any &= any - 1u) {
        const uint32_t u = (uint32_t)__ffs(any) - 1u, p = p0 + u * kThreads;
        const bool mine = (in >> u) & 1u;
        const uint32_t first = (uint32_t)__ffs(__ballot_sync(0xffffffffu, mine)) - 1u;
        const float k = mine ? __ldg(keys + p) : 0.0f;
        const uint32_t y = mine ? __ldg(wt + p) : 0u;
        const float t = __shfl_sync(0xffffffffu, k, (int)first);
        if (t != tie) bin = bin_of(t);
        tie = t;
        const bool same = mine && k == t;
        const uint32_t lo = __reduce_add_sync(0xffffffffu, same ? y & 0xffffu : 0u);
        const uint32_t hi = __reduce_add_sync(0xffffffffu, same ? y >> 16 : 0u);
        if (lane == first) {
            atomicAdd(&sm.half[0][bin], lo);
            if (hi) atomicAdd(&sm.half[1][bin], hi);
        } else if (mine && !same && y) {
            const uint32_t b = bin_of(k);
            atomicAdd(&sm.half[0][b], y & 0xffffu);
            if (y >> 16) atomicAdd(&sm.half[1][b], y >> 16);
        }
    }
}

// A run of consecutive tiles a CTA, so that a cell's bins go to global memory once a run and a cell of
// several tiles ends in its CTA's first pass (apart, 2^26 particles into 2^16 leaves took 2% longer).
// kFew: levels of cells of at most 1024 keys on average. If some have several tiles all the same,
// these, next to each other in the plan and with many times the keys, would be a few CTAs' runs: the
// tiles are dealt apart, and those of cells that are done passed over a CTA's width at a time. (Half
// of 6.4 million particles on one point: 2^19 leaves 52.1 ms in runs, 12.9 apart, 2^14 4.6 and 3.8. An
// instance of its own: the choice at run time was 2 to 3% of 2^24 particles into 2^11 to 2^14 leaves.)
template <bool kWide, bool kFew>
__global__ void __launch_bounds__(kThreads, 4) k_whist(const __grid_constant__ Level v, uint32_t pieces) {
    pdl_enter();
    __shared__ WeightSmem sm;
    if (v.pass == 0 && level_failed(v)) return;
    // every cell of the level finished in an earlier pass
    if (v.pass > 0 && *(volatile uint32_t *)&v.counters->any_active[v.pass - 1] == 0u) return;
    WeightCell &w = sm.cell;
    const uint32_t tid = threadIdx.x;
    const uint32_t piece = (uint32_t)kTile / pieces;  // keys of a piece; `pieces` of them a tile
    unsigned long long bytes = 0;
    const uint64_t total = (v.tot->tiles >> 32) * pieces;
    const bool apart = kFew && total != (uint64_t)v.C * pieces;
    if (tid == 0) {
        sm.run[0] = apart ? blockIdx.x : (uint32_t)(total * blockIdx.x / gridDim.x);
        sm.run[1] = apart ? (uint32_t)total : (uint32_t)(total * (blockIdx.x + 1) / gridDim.x);
    }
    __syncthreads();
    const uint32_t t_end = sm.run[1];
    int cur = -1;
    uint32_t ntiles = 0, held = 0;  // pieces of the cell so far; of them in the shared bins
    bool flushed = false, direct = false;
    unsigned long long below = 0, tot = 0;  // this thread's weights below L, and all (first pass)
    auto clear = [&]() {
        for (uint32_t j = tid; j < (1u << w.K); j += kThreads) sm.half[0][j] = sm.half[1][j] = 0u;
    };
    auto flush = [&]() {  // the shared bins to the cell's global ones
        __syncthreads();
        unsigned long long *g = v.whist + v.hist_off[cur];
        for (uint32_t j = tid; j < (1u << w.K); j += kThreads) {
            const unsigned long long x =
                (unsigned long long)sm.half[0][j] + ((unsigned long long)sm.half[1][j] << 16);
            if (x) atomicAdd(&g[j], x);
        }
        __syncthreads();
        flushed = true;
        held = 0;
    };
    // keys [e0, e1) of the cell; first: every weight is read (the total, the weight below L),
    // later: those of the bracket's keys
    auto tile = [&](uint32_t e0, uint32_t e1, bool first) {
        const float *keys = w.keys;
        const Guess gs = w.gs;
        const float L = w.L, R = w.R;
        const uint32_t top = (1u << w.K) - 1u;
        auto add = [&](float k, uint32_t x) {
            uint32_t b;
            if (!guess_bin(gs, k, &b)) b = near_bin(k, gs, sm.edge, top);
            atomicAdd(&sm.half[0][b], x & 0xffffu);
            if (x >> 16) atomicAdd(&sm.half[1][b], x >> 16);
        };
        if (!first) {
            // 16 keys of a thread in flight, the weights of the bracket's keys only
            constexpr int kLoads = 16;
            for (uint32_t p0 = e0 + tid; p0 < e1; p0 += kThreads * kLoads) {
                float k[kLoads];
#pragma unroll
                for (int u = 0; u < kLoads; ++u) {
                    const uint32_t p = p0 + (uint32_t)u * kThreads;
                    k[u] = p < e1 ? __ldg(keys + p) : __int_as_float(0x7fc00000);  // NaN: not binned
                }
                uint32_t in = 0;
#pragma unroll
                for (int u = 0; u < kLoads; ++u) in |= (uint32_t)(k[u] >= L && k[u] < R) << u;
                if (p0 - tid + kThreads * kLoads <= e1 &&  // (a whole round: every lane is here)
                    __reduce_add_sync(0xffffffffu, (uint32_t)__popc(in)) > kTies) {
                    tied_weights(v.wt, p0, in, sm);
                    continue;
                }
                for (; in; in &= in - 1u) {
                    const uint32_t p = p0 + ((uint32_t)__ffs(in) - 1u) * kThreads, y = __ldg(v.wt + p);
                    if (y) add(__ldg(keys + p), y);
                }
            }
            if (tid == 0) bytes += 4ull * (e1 - e0);
            return;
        }
        constexpr int kLoads = 8;
        for (uint32_t p0 = e0 + tid; p0 < e1; p0 += kThreads * kLoads) {
            float k[kLoads];
            uint32_t x[kLoads], any = 0;
#pragma unroll
            for (int u = 0; u < kLoads; ++u) {
                const uint32_t p = p0 + (uint32_t)u * kThreads;
                k[u] = p < e1 ? __ldg(keys + p) : __int_as_float(0x7fc00000);
                x[u] = p < e1 ? __ldg(v.wt + p) : 0u;
            }
#pragma unroll
            for (int u = 0; u < kLoads; ++u) any |= x[u];
            if (any < (1u << 29)) {  // eight weights below 2^29 add up in 32 bits
                uint32_t all = 0, low = 0;
#pragma unroll
                for (int u = 0; u < kLoads; ++u) {
                    all += x[u];
                    low += k[u] < L ? x[u] : 0u;
                }
                tot += all;
                below += low;
            } else {
#pragma unroll
                for (int u = 0; u < kLoads; ++u) {
                    tot += x[u];
                    if (k[u] < L) below += x[u];
                }
            }
            if (gs.span) {  // each guess corrected by the edges either side of it, as in edges_key
#pragma unroll
                for (int u = 0; u < kLoads; ++u) {
                    const uint32_t t = __float_as_uint(__fmaf_rn(__fsub_rn(k[u], gs.L), gs.scale, 2048.0f)) - 0x45000000u;
                    const uint32_t g = min(t >> 12, top);
                    const float a = sm.edge[g], b = sm.edge[g + 1];
                    const uint32_t bin = g + (k[u] >= b ? 1u : 0u) - (k[u] < a ? 1u : 0u);
                    if (k[u] >= L && k[u] < R) {
                        atomicAdd(&sm.half[0][bin], x[u] & 0xffffu);
                        if (x[u] >> 16) atomicAdd(&sm.half[1][bin], x[u] >> 16);
                    }
                }
                continue;
            }
#pragma unroll
            for (int u = 0; u < kLoads; ++u)
                if (k[u] >= L && k[u] < R && x[u]) add(k[u], x[u]);
        }
        if (tid == 0) bytes += 8ull * (e1 - e0);
    };
    auto end_cell = [&]() {
        const uint32_t tiles = (w.end - w.base + (uint32_t)kTile - 1) / (uint32_t)kTile * pieces;
        const bool whole = ntiles == tiles && !flushed, first = v.pass == 0;
        if (first && !direct) {
            below = block_sum_u64(below, sm.red);
            tot = block_sum_u64(tot, sm.red);
        }
        __syncthreads();
        bool last = true;
        if (direct) {
            if (w.end - w.base <= 8 * kThreads)
                weighted_direct<8>(v, cur, sm);
            else
                weighted_direct<16>(v, cur, sm);
        } else if (whole) {
            if (tid == 0 && first) {
                w.below = below;
                w.tot = tot;
            }
            __syncthreads();
            weighted_replay<kWide>(v, cur, false, sm);
            while (w.state == kActive) {  // the rest of the loop, on this CTA's own cell
                clear();
                fill_edges(sm.edge, w.L, w.R, w.K, tid, kThreads);
                __syncthreads();
                tile(w.base, w.end, false);
                __syncthreads();
                weighted_replay<kWide>(v, cur, false, sm);
            }
        } else {
            if (tid == 0 && first) {
                if (below) atomicAdd(&v.wbelow[cur], below);
                if (tot) atomicAdd(&v.wtot[cur], tot);
            }
            flush();
            if (tid == 0) {
                w.last = arrive_release(&v.hdone[cur], ntiles) + ntiles == tiles;
                if (w.last) {
                    acquire();
                    w.below = __ldcg(&v.wbelow[cur]);
                    w.tot = __ldcg(&v.wtot[cur]);
                }
            }
            __syncthreads();
            last = w.last != 0;
            if (last) weighted_replay<kWide>(v, cur, true, sm);
        }
        if (last && tid == 0) {
            orb_cell_t &cell = v.heap[level_slot(v, cur)];
            cell.cutMarginLeft = w.L;
            cell.cutMarginRight = w.R;
            cell.foundCut = w.state == kFound ? 1 : 0;
            v.iters[cur] = (uint8_t)w.it;
            v.state[cur] = (uint8_t)w.state;
            v.wbelow[cur] = w.below;
            v.hdone[cur] = 0;
            if (w.state != kActive) atomicMax(&v.counters->max_iters, w.it);
            if (w.state == kCapped) atomicAdd(&v.counters->unfound, 1u);
            if (w.state == kActive) {
                v.counters->any_active[v.pass] = 1u;
                if (v.pass == v.last_pass) atomicExch(&v.counters->error, 1u);
            }
        }
        __syncthreads();  // the cell and its bins are free for the next one
        ntiles = 0;
        below = tot = 0;
        flushed = false;
    };
    int skip_c = -1;  // an inactive cell whose tiles are being passed over
    const uint32_t t_step = apart ? gridDim.x : 1u;
    for (uint32_t t = sm.run[0]; t < t_end; t += t_step) {
        const int c = (int)v.htile_cell[t / pieces];
        if (c == skip_c) continue;
        if (c != cur) {
            // a cell with a tile still to come is not resolved in this pass: its state stands
            if (v.state[c] != kActive) {
                if (!kFew) {
                    skip_c = c;
                } else {  // on to this CTA's next tile of an active cell
                    if (tid == 0) sm.next = t + kThreads * t_step;
                    __syncthreads();
                    const uint32_t u = t + (tid + 1u) * t_step;
                    if (u < t_end && v.state[v.htile_cell[u / pieces]] == kActive) atomicMin(&sm.next, u);
                    __syncthreads();
                    t = sm.next - t_step;
                    __syncthreads();
                }
                continue;
            }
            if (cur >= 0) end_cell();
            cur = c;
            held = 0;
            if (tid == 0) {
                const int slot = level_slot(v, c);
                const orb_cell_t &cell = v.heap[slot];
                const uint2 rg = v.ranges[slot];
                w.keys = axis_keys(v, eff_axis(cell.cutAxis));
                w.L = cell.cutMarginLeft;
                w.R = cell.cutMarginRight;
                w.K = pieces > 1 ? kMaxBinsLog2 : weighted_depth(rg.y - rg.x);
                w.base = rg.x;
                w.end = rg.y;
                w.t0 = v.tile_off[c];
                w.it = v.iters[c];
                w.below = v.pass ? v.wbelow[c] : 0ull;
                w.tot = v.pass ? v.wtot[c] : 0ull;
                const uint32_t nb = 1u << w.K;
                w.gs = make_guess(w.L, w.R, __fdiv_rn((float)nb, __fsub_rn(w.R, w.L)), nb);
            }
            __syncthreads();
            direct = pieces == 1 && w.end - w.base <= kWDirect;
            if (!direct) {
                clear();
                fill_edges(sm.edge, w.L, w.R, w.K, tid, kThreads);
                __syncthreads();
            }
        } else if (held == kWFlush * pieces) {
            flush();
            clear();
            __syncthreads();
        }
        const uint32_t e0 = min(w.end, w.base + (t - w.t0 * pieces) * piece);
        if (!direct) tile(e0, min(w.end, e0 + piece), v.pass == 0);
        if (direct && tid == 0) bytes += 8ull * (w.end - w.base);
        ++ntiles;
        ++held;
    }
    if (cur >= 0) end_cell();
    if (tid == 0 && bytes) add_bytes(v, kKWHist, bytes);
}

// Weighted cells of at most 256 keys by a warp each, the whole loop, on levels of such cells on
// average (then k_whist finds the larger ones, if any). A CTA a cell with a barrier a step took 17 us
// a cell of many equal keys: 340783 particles on 1000 points into 2^16 leaves, the last level's 32768
// cells 1046 us; 121 here and 50 for k_whist to pass them over. (As an instance of k_whist with a warp
// a cell 357, and the other instances' registers suffered: 0.6% of 16 million particles.)
constexpr int kWWarpKeys = 256;
__global__ void __launch_bounds__(kThreads, kTileBlocksPerSm) k_wbisect_tile(const __grid_constant__ Level v) {
    pdl_enter();
    if (level_failed(v)) return;
    const uint32_t lane = threadIdx.x & 31;
    const int nwarps = (int)(gridDim.x * (blockDim.x >> 5));
    for (int c = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5); c < v.C; c += nwarps) {
        if (v.state[c] != kActive) continue;
        const int slot = level_slot(v, c);
        const uint2 rg = v.ranges[slot];
        const uint32_t n = rg.y - rg.x;
        if (n > (uint32_t)kWWarpKeys) continue;
        orb_cell_t &cell = v.heap[slot];
        const float *keys = axis_keys(v, eff_axis(cell.cutAxis));
        constexpr int kPer = kWWarpKeys / 32;
        float k[kPer], L = cell.cutMarginLeft, R = cell.cutMarginRight;
        uint32_t x[kPer];
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            const uint32_t p = (uint32_t)j * 32u + lane;
            k[j] = p < n ? __ldg(keys + rg.x + p) : __int_as_float(0x7fc00000);  // NaN: never below
            x[j] = p < n ? __ldg(v.wt + rg.x + p) : 0u;
        }
        auto below = [&](float cut, bool all) -> unsigned long long {
            uint32_t lo = 0, hi = 0;
#pragma unroll
            for (int j = 0; j < kPer; ++j) {
                const uint32_t y = all || k[j] < cut ? x[j] : 0u;
                lo += y & 0xffffu;
                hi += y >> 16;
            }
            return (unsigned long long)__reduce_add_sync(0xffffffffu, lo) +
                   ((unsigned long long)__reduce_add_sync(0xffffffffu, hi) << 16);
        };
        const WeightTest test(below(0.f, true), n, cell.nLeafCells);
        uint32_t it = 0;
        uint8_t st = kActive;
        while (st == kActive) {
            if (it >= (uint32_t)kMaxIterations) {
                st = kCapped;
                break;
            }
            const float cut = mid_cut(L, R);
            ++it;
            const int dir = test.dir(below(cut, false));
            if (dir == 0)
                st = kFound;
            else if (dir > 0)
                R = cut;
            else
                L = cut;
        }
        __syncwarp();
        if (lane == 0) {
            cell.cutMarginLeft = L;
            cell.cutMarginRight = R;
            cell.foundCut = st == kFound ? 1 : 0;
            v.iters[c] = (uint8_t)it;
            v.state[c] = st;
            atomicMax(&v.counters->max_iters, it);
            if (st == kCapped) atomicAdd(&v.counters->unfound, 1u);
            add_bytes(v, kKBisectTile, 8ull * n);
        }
    }
}

// ------------------------------------------------------------------------------------
// Service count-left: one plain pass at getCut() per cell, found cells skipped.
// ------------------------------------------------------------------------------------
__global__ void __launch_bounds__(kThreads) k_count_left(const __grid_constant__ Level v) {
    pdl_enter();
    __shared__ uint32_t s_red[32];
    const uint32_t total = (uint32_t)(v.tot->tiles >> 32);
    for (uint32_t t = blockIdx.x; t < total; t += gridDim.x) {
        const TileRef tr = tile_ref(v, t);
        const orb_cell_t &cell = v.heap[tr.slot];
        if (cell.foundCut) continue;
        const float cut = cell_cut(cell);
        uint32_t cnt = 0;
        for_keys(axis_keys(v, eff_axis(cell.cutAxis)), tr.e0, tr.e1, [&](float k) { cnt += k < cut; });
        cnt = block_sum(cnt, s_red);
        if (threadIdx.x == 0) {
            if (cnt) atomicAdd(&v.out_counts[tr.c], cnt);
            add_bytes(v, kKCountLeft, 4ull * (tr.e1 - tr.e0));
        }
    }
}

// ------------------------------------------------------------------------------------
// Seeded generators (bit-identical with the CPU oracle's generator)
// ------------------------------------------------------------------------------------
__device__ __forceinline__ uint64_t mix64(uint64_t z) {
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}
__device__ __forceinline__ uint64_t draw(uint64_t seed_mix, uint64_t counter) {
    return mix64(seed_mix + counter * 0xD1B54A32D192ED03ull);
}
__device__ __forceinline__ float unit_coord(uint64_t u) {
    return __fsub_rn(__fmul_rn(__uint2float_rn((uint32_t)(u >> 40)), 0x1p-24f), 0.5f);
}
__device__ __forceinline__ double unit_double(uint64_t u) {
    return __dmul_rn(__ull2double_rn(u >> 11), 0x1p-53);
}

__global__ void k_gen_uniform(uint64_t seed, uint64_t n, float *x, float *y, float *z) {
    const uint64_t sm = mix64(seed);
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x) {
        x[i] = unit_coord(draw(sm, 3 * i + 0));
        y[i] = unit_coord(draw(sm, 3 * i + 1));
        z[i] = unit_coord(draw(sm, 3 * i + 2));
    }
}

struct PlummerTable {
    float centre[64 * 3];
    double scale[64];
};

__global__ void k_gen_plummer(uint64_t seed, uint64_t n, PlummerTable tab, float *x, float *y,
                              float *z) {
    const uint64_t sm = mix64(seed);
    const float hi = 0x1.fffffep-2f;  // nextafter(0.5f, -1)
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t c = i * 64;
        const uint64_t sel = draw(sm, c) >> 40;
        float p[3];
        if (sel * 10 < 9ull * (1ull << 24)) {
            const int k = (int)(draw(sm, c + 1) % 64);
            double w = unit_double(draw(sm, c + 2));
            w = fmax(w, unit_double(draw(sm, c + 3)));
            w = fmax(w, unit_double(draw(sm, c + 4)));
            const double r = __ddiv_rn(__dmul_rn(tab.scale[k], w),
                                       __dsqrt_rn(__dsub_rn(1.0, __dmul_rn(w, w))));
            double v0 = 1.0, v1 = 0.0, v2 = 0.0, q = 1.0;
            for (int t = 0; t < 19; ++t) {
                const double u0 = __dsub_rn(__dmul_rn(2.0, unit_double(draw(sm, c + 5 + 3 * t + 0))), 1.0);
                const double u1 = __dsub_rn(__dmul_rn(2.0, unit_double(draw(sm, c + 5 + 3 * t + 1))), 1.0);
                const double u2 = __dsub_rn(__dmul_rn(2.0, unit_double(draw(sm, c + 5 + 3 * t + 2))), 1.0);
                const double qq = __dadd_rn(__dadd_rn(__dmul_rn(u0, u0), __dmul_rn(u1, u1)), __dmul_rn(u2, u2));
                if (qq > 0.0 && qq <= 1.0) {
                    v0 = u0;
                    v1 = u1;
                    v2 = u2;
                    q = qq;
                    break;
                }
            }
            const double s = __ddiv_rn(r, __dsqrt_rn(q));
            const double vv[3] = {v0, v1, v2};
            for (int a = 0; a < 3; ++a) {
                const float f = __double2float_rn(__dadd_rn((double)tab.centre[3 * k + a], __dmul_rn(vv[a], s)));
                p[a] = fminf(fmaxf(f, -0.5f), hi);
            }
        } else {
            for (int a = 0; a < 3; ++a) p[a] = unit_coord(draw(sm, c + 2 + a));
        }
        x[i] = p[0];
        y[i] = p[1];
        z[i] = p[2];
    }
}

// The reference's xorshf96 stream (src/services/init.cu:11-25): thread g continues the
// stream from starts[g] (its state after g * chunk draws, computed on the host by a GF(2)
// jump) for `chunk` draws; draw j is coordinate j % 3 of particle j / 3. Value:
// (float)z / 2^64 - 0.5 (exact scaling, then the subtraction rounded once: the reference's
// double subtraction rounded to float gives the same float).
__global__ void k_gen_xorshf96(const unsigned long long *starts, uint64_t draws, uint32_t chunk,
                               float *x, float *y, float *z) {
    const uint64_t g = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint64_t j0 = g * chunk;
    if (j0 >= draws) return;
    unsigned long long sx = starts[3 * g], sy = starts[3 * g + 1], sz = starts[3 * g + 2];
    const uint64_t j1 = min(draws, j0 + chunk);
    float *dst[3] = {x, y, z};
    for (uint64_t j = j0; j < j1; ++j) {
        sx ^= sx << 16;
        sx ^= sx >> 5;
        sx ^= sx << 1;
        const unsigned long long t = sx;
        sx = sy;
        sy = sz;
        sz = t ^ sx ^ sy;
        const float q = __fmul_rn(__ull2float_rn(sz), 0x1p-64f);
        dst[j % 3][j / 3] = __fsub_rn(q, 0.5f);
    }
}

__global__ void k_copy_instances(const uint32_t *src, uint32_t *dst, const BatchRoot *roots, int k) {
    for (int i = blockIdx.y; i < k; i += gridDim.y) {
        const BatchRoot r = roots[i];
        for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < r.n; p += gridDim.x * blockDim.x)
            dst[r.offset + p] = src[r.offset + p];
    }
}

// Box-Muller pairs from the counter-based stream: coordinate a of particle i uses draws
// (seed, 2*(3i+a)) and (seed, 2*(3i+a)+1).
__global__ void k_displace(float *x, float *y, float *z, uint64_t offset, uint64_t n,
                           uint64_t seed, float sigma, float lo0, float lo1, float lo2,
                           float hi0, float hi1, float hi2) {
    const uint64_t sm = mix64(seed);
    float *c[3] = {x, y, z};
    const float lo[3] = {lo0, lo1, lo2};
    const float hi[3] = {nextafterf(hi0, lo0), nextafterf(hi1, lo1), nextafterf(hi2, lo2)};
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x) {
        for (int a = 0; a < 3; ++a) {
            const uint64_t q = 2 * (3 * i + a);
            const float u1 = ((float)(uint32_t)(draw(sm, q) >> 40) + 1.0f) * 0x1p-24f;  // (0, 1]
            const float u2 = (float)(uint32_t)(draw(sm, q + 1) >> 40) * 0x1p-24f;       // [0, 1)
            const float g = sqrtf(-2.0f * logf(u1)) * cospif(2.0f * u2);
            const float p = c[a][offset + i] + sigma * g;
            c[a][offset + i] = fminf(fmaxf(p, lo[a]), hi[a]);
        }
    }
}

__global__ void k_iota_u32(uint32_t *dst, uint64_t n) {
    for (uint64_t p = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; p < n;
         p += (uint64_t)gridDim.x * blockDim.x)
        dst[p] = (uint32_t)p;
}

__global__ void k_gather_u32(uint32_t *dst, const uint32_t *src, const uint32_t *perm, uint64_t off,
                             uint64_t n) {
    for (uint64_t p = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; p < n;
         p += (uint64_t)gridDim.x * blockDim.x)
        dst[off + p] = src[off + perm[off + p]];
}

#ifndef ORB_GATHER_QUADS
#define ORB_GATHER_QUADS 4  // quads of a thread in flight in the stage gather
#endif
// Staged builds from host memory: a coordinate that arrived after the first levels moved the
// other coordinates takes their order through the permutation, dst[p] = src[idx[p]].
__global__ void __launch_bounds__(256) k_stage_gather(float *__restrict__ dst, const float *__restrict__ src,
                                                      const uint32_t *__restrict__ idx, uint64_t n,
                                                      BuildCounters *ctr) {
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    const uint64_t g = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint64_t n4 = n / 4;  // dst and idx are 16-byte aligned allocations
    const uint4 *idx4 = reinterpret_cast<const uint4 *>(idx);
    float4 *dst4 = reinterpret_cast<float4 *>(dst);
    // kQ quads per thread and step: all index loads, then all 4 kQ gathers, in flight
    constexpr int kQ = ORB_GATHER_QUADS;
    uint64_t q = g;
    for (; q + (kQ - 1) * stride < n4; q += kQ * stride) {
        uint4 i[kQ];
#pragma unroll
        for (int u = 0; u < kQ; ++u) i[u] = idx4[q + u * stride];
        float4 a[kQ];
#pragma unroll
        for (int u = 0; u < kQ; ++u) a[u] = make_float4(src[i[u].x], src[i[u].y], src[i[u].z], src[i[u].w]);
#pragma unroll
        for (int u = 0; u < kQ; ++u) dst4[q + u * stride] = a[u];
    }
    for (; q < n4; q += stride) {
        const uint4 i = idx4[q];
        dst4[q] = make_float4(src[i.x], src[i.y], src[i.z], src[i.w]);
    }
    for (uint64_t p = n4 * 4 + g; p < n; p += stride) dst[p] = src[idx[p]];
    // per particle: its index and the gathered value read, the value written
    if (g == 0) atomicAdd(&ctr->bytes[kKStageGather], 12ull * n);
}

inline int grid_for(uint64_t n, int threads, int cap) {
    uint64_t g = (n + threads - 1) / threads;
    if (g < 1) g = 1;
    if (g > (uint64_t)cap) g = cap;
    return (int)g;
}

}  // namespace

// ------------------------------------------------------------------------------------
// Launchers
// ------------------------------------------------------------------------------------
void launch_init_batch(const Level &v, const BatchRoot *roots, int k, uint64_t n_total,
                       cudaStream_t st) {
    (void)n_total;
    if (k > 0) k_init_batch<<<dim3(64, (unsigned)(k < 65535 ? k : 65535)), 256, 0, st>>>(v, roots, k);
}

void launch_init(const Level &v, uint64_t n, const float lower[3], const float upper[3],
                 uint32_t d, int heap_cells, cudaStream_t st) {
    uint64_t work = n > (uint64_t)heap_cells * 13 ? n : (uint64_t)heap_cells * 13;
    k_init<<<grid_for(work, 256, 152 * 16), 256, 0, st>>>(v, (uint32_t)n, lower[0], lower[1],
                                                        lower[2], upper[0], upper[1], upper[2], d,
                                                        heap_cells);
}

// A level kernel on the stream, with the programmatic-dependent-launch attribute when the
// context uses it (the kernels wait for their predecessor in pdl_enter()).
template <class... P, class... A>
void launch_kernel(bool pdl, void (*kern)(P...), dim3 grid, dim3 block, size_t smem,
                   cudaStream_t st, A... args) {
    if (!pdl) {
        kern<<<grid, block, smem, st>>>(args...);
        return;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kern, args...);
}

template <bool kFuse>
void launch_swap(bool p, const Level &v, int grid, int arg, cudaStream_t st) {
    const dim3 T(kSwapThreads);
    if (v.wt)
        launch_kernel(p, k_part_swap<true, 3, kFuse>, dim3(grid), T, 0, st, v, arg);
    else if (!v.y)
        launch_kernel(p, k_part_swap<false, 0, kFuse>, dim3(grid), T, 0, st, v, arg);
    else if (!v.z)
        launch_kernel(p, k_part_swap<false, 1, kFuse>, dim3(grid), T, 0, st, v, arg);
    else
        launch_kernel(p, k_part_swap<false, 3, kFuse>, dim3(grid), T, 0, st, v, arg);
}

void launch_level_kernel(Kernel k, const Level &v, int grid, int arg, cudaStream_t st) {
    const bool p = v.pdl != 0;
    const dim3 T(kThreads);
    const unsigned per_cell_warps = (unsigned)grid_for((uint64_t)v.C * 32, kThreads, 1 << 30);
    switch (k) {
        case kKPlan: launch_kernel(p, k_plan, dim3(per_cell_warps), T, 0, st, v); break;
        case kKHist:  // arg: 1 first pass, all cells dense; 2 first pass of a sampled level
            if (v.wide)
                launch_kernel(p, arg == 2 ? k_hist<kHFirstSampled, kThreads, true> : k_hist<kHRest, kThreads, true>, dim3(grid), T, 0, st, v);
            else if (arg == 2)
                launch_kernel(p, k_hist<kHFirstSampled, kThreads>, dim3(grid), T, 0, st, v);
            else if (v.hist_threads == 1024)
                launch_kernel(p, arg ? k_hist<kHFirstDense, 1024> : k_hist<kHRest, 1024>, dim3(grid), dim3(1024), 0, st, v);
            else if (v.hist_threads == 512)
                launch_kernel(p, arg ? k_hist<kHFirstDense, 512> : k_hist<kHRest, 512>, dim3(grid), dim3(512), 0, st, v);
            else
                launch_kernel(p, arg ? k_hist<kHFirstDense, kThreads> : k_hist<kHRest, kThreads>, dim3(grid), T, 0, st, v);
            break;
        case kKBisectTile: launch_kernel(p, v.wt ? k_wbisect_tile : k_bisect_tile, dim3(grid), T, 0, st, v); break;
        case kKSubtreeCheck: launch_kernel(p, k_subtree_check, dim3(1), dim3(1024), 0, st, v, arg); break;
        case kKSubtree: launch_kernel(p, k_subtree, dim3(grid), dim3(kSubThreads), kSubBytes, st, v); break;
        case kKBisectCta:
            launch_kernel(p, k_bisect_cta, dim3(grid), dim3(kCtaThreads), kCtaSmemBytes, st, v);
            break;
        case kKPartClassify: launch_kernel(p, arg == 4 ? k_part_classify<4> : k_part_classify<1>, dim3(grid), T, 0, st, v); break;
        case kKPartCells:
            // grid = the SM count: levels of few cells take large CTAs, several a cell
            if (v.C <= grid)
                launch_kernel(p, k_part_cells<1024, true>, dim3((unsigned)std::max(1, std::min(64, grid / v.C)), v.C),
                              dim3(1024), 0, st, v);
            else
                launch_kernel(p, k_part_cells<kThreads, false>, dim3(per_cell_warps), T, 0, st, v);
            break;
        case kKPartSwap:
            if (v.fuse)
                launch_swap<true>(p, v, grid, arg, st);
            else
                launch_swap<false>(p, v, grid, arg, st);
            break;
        case kKPartFinish:  // grid = the SM count
            if (v.C <= grid)
                launch_kernel(p, k_part_finish<true>, dim3(v.C), T, 0, st, v, arg);
            else
                launch_kernel(p, k_part_finish<false>, dim3(per_cell_warps), T, 0, st, v, arg);
            break;
        case kKWHist: {
            auto *k = v.few_tiles ? (v.wide ? k_whist<true, true> : k_whist<false, true>)
                                   : (v.wide ? k_whist<true, false> : k_whist<false, false>);
            launch_kernel(p, k, dim3(grid), T, 0, st, v, (uint32_t)arg);
            break;
        }
        case kKCountLeft: launch_kernel(p, k_count_left, dim3(grid), T, 0, st, v); break;
        case kKSample:
            launch_kernel(p, k_sample_bin, dim3(kSampleMax / kSamplePerCta, (unsigned)min(v.C, 65535)),
                          dim3(kSampleThreads), 0, st, v);
            break;
        case kKSamplePick:
            launch_kernel(p, k_sample_pick, dim3((unsigned)min(v.C, 65535)), dim3(kPickThreads), 0, st, v);
            break;
        default: break;
    }
}

cudaError_t configure_kernels() {
    const cudaError_t e = cudaFuncSetAttribute(k_bisect_cta, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)kCtaSmemBytes);
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(k_subtree, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSubBytes);
}

int swap_blocks_per_sm() {
    // the swap's CTAs walk the tiles grid-stride: one resident wave, none waiting behind it
    static const int blocks = [] {
        int b = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_part_swap<false, 3, false>, kSwapThreads, 0) != cudaSuccess ||
            b < 1) {
            cudaGetLastError();
            b = ORB_SWAP_MIN_BLOCKS;
        }
        return b;
    }();
    return blocks;
}

void launch_copy_instances(const uint32_t *src, uint32_t *dst, const BatchRoot *roots, int k,
                           cudaStream_t st) {
    if (k > 0)
        k_copy_instances<<<dim3(64, (unsigned)(k < 65535 ? k : 65535)), 256, 0, st>>>(src, dst, roots, k);
}

void launch_displace(float *x, float *y, float *z, uint64_t offset, uint64_t n, uint64_t seed,
                     float sigma, const float lower[3], const float upper[3], cudaStream_t st) {
    if (n == 0) return;
    k_displace<<<grid_for(n, 256, 152 * 16), 256, 0, st>>>(x, y, z, offset, n, seed, sigma, lower[0],
                                                          lower[1], lower[2], upper[0], upper[1],
                                                          upper[2]);
}

void launch_iota_u32(uint32_t *dst, uint64_t n, cudaStream_t st) {
    if (n) k_iota_u32<<<grid_for(n, 256, 152 * 16), 256, 0, st>>>(dst, n);
}

void launch_stage_gather(float *dst, const float *src, const uint32_t *idx, uint64_t n,
                         BuildCounters *ctr, int num_sms, cudaStream_t st) {
    if (n) k_stage_gather<<<grid_for((n + 3) / 4, 256, num_sms * 8), 256, 0, st>>>(dst, src, idx, n, ctr);
}

void launch_gather_u32(uint32_t *dst, const uint32_t *src, const uint32_t *perm, uint64_t off,
                       uint64_t n, cudaStream_t st) {
    if (n) k_gather_u32<<<grid_for(n, 256, 152 * 16), 256, 0, st>>>(dst, src, perm, off, n);
}

void launch_gen_xorshf96(const unsigned long long *starts, uint64_t draws, uint32_t chunk,
                         float *x, float *y, float *z, cudaStream_t st) {
    const uint64_t threads = (draws + chunk - 1) / chunk;
    k_gen_xorshf96<<<(unsigned)((threads + 127) / 128), 128, 0, st>>>(starts, draws, chunk, x, y, z);
}

void launch_gen_uniform(uint64_t seed, uint64_t n, float *x, float *y, float *z,
                        cudaStream_t st) {
    k_gen_uniform<<<grid_for(n, 256, 152 * 32), 256, 0, st>>>(seed, n, x, y, z);
}

void launch_gen_plummer(uint64_t seed, uint64_t n, const float *centres, const double *scales,
                        float *x, float *y, float *z, cudaStream_t st) {
    PlummerTable tab;
    for (int i = 0; i < 64 * 3; ++i) tab.centre[i] = centres[i];
    for (int i = 0; i < 64; ++i) tab.scale[i] = scales[i];
    k_gen_plummer<<<grid_for(n, 256, 152 * 32), 256, 0, st>>>(seed, n, tab, x, y, z);
}

}  // namespace orb
