// Internal declarations of the ORB engine: device helpers shared by the kernels and the
// launch interface the host driver uses. Nothing here is part of the C ABI.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "orb/orb.h"
#include "orb_leaf_ratio.h"

namespace orb {

static_assert(sizeof(orb_cell_t) == 52, "orb_cell_t must keep the reference's 52-byte Cell layout");

constexpr int kMaxIterations = 32;   // bisection cap, src/orbit.cpp:149
constexpr int kTile = 16384;         // keys per tile of the count-left passes
constexpr int kPTile = 4096;         // positions per tile of the partition passes
constexpr int kPWords = kPTile / 32; // bitmask words per partition tile
constexpr int kMaxBinsLog2 = 11;     // deepest midpoint tree one histogram pass resolves
// Histogram passes per level: their midpoint trees have depth 11, so 3 passes (33 iterations)
// reach the 32-iteration cap of every cell. A first pass that is discarded (a warm or sampled bracket that missed the
// cut) costs one more, hence 4 for levels that may have one.
constexpr int kHistPasses = 4;
constexpr int kColdHistPasses = 3;
static_assert(kHistPasses <= 4, "BuildCounters::any_active holds the passes");
constexpr int kThreads = 256;
// resident CTAs of the count-left pass (its launch bound: 65536 / (256 x 6) = 40 registers)
#ifndef ORB_HIST_BLOCKS_PER_SM
#define ORB_HIST_BLOCKS_PER_SM 6
#endif
constexpr int kHistBlocksPerSm = ORB_HIST_BLOCKS_PER_SM;
constexpr int kHistBlocks512 = 3;  // ... and of its CTAs of 512 threads
constexpr int kTileBlocksPerSm = 4;  // resident CTAs of the one-warp cell bisection
constexpr uint32_t kSubMaxParticles = 33024;  // largest cell one subtree CTA takes (2^15 + 256)
// Warm builds: hints apply to the levels above the first one of at least two cells per SM whose
// cells are expected to have at most this many particles and that is at most tune.subtree_levels
// above the leaves; where the device finds a larger cell there, to all levels. (Which levels start
// from hints decides the trees, so the line stays where it was whatever the subtree kernel takes.)
constexpr uint32_t kHintSubMax = 34816;
constexpr uint32_t kSubDefaultLevels = 4;     // default of tune.subtree_levels
constexpr int kSubMaxLevels = 6;              // deepest tree one subtree CTA finishes

// Weighted builds: launches of the weighted pass a level (11 iterations each for cells of more
// than one tile; smaller cells are finished by the first).
constexpr int kWPasses = 3;

// kSmall: at most kWarpKeys keys, one warp bisects it
// kReady: its bracket holds few enough keys for a list: the classify pass lists them and
// k_part_cells finishes the bisection on the list
enum CellState : uint8_t { kActive = 0, kFound = 1, kCapped = 2, kSmall = 3, kReady = 4 };
constexpr int kWarpKeys = 1024;      // cells up to this size bisect in one warp's registers
constexpr int kMaxLevels = 30;       // d is at most 2^30
// The subtree kernel's wait for a copy of keys: its polls at most, and the nanoseconds after which
// the hardware is asked to end one (2^20 of them were measured to take 3.8 s, 2^18 a second).
constexpr uint32_t kCopyPolls = 1u << 18, kCopyPollNs = 1000;

// Kernel kinds, for launch counting, event timing and algorithmic-byte accounting.
enum Kernel : int {
    kKInit = 0,
    kKPlan,
    kKHist,
    kKPartClassify,
    kKPartCells,
    kKPartSwap,
    kKPartFinish,
    kKCountLeft,
    kKGenerate,
    kKBisectCta,
    kKBisectTile,
    kKSubtreeCheck,
    kKSubtree,
    kKSample,
    kKSamplePick,
    kKWHist,
    kKStageGather,
    kNumKernels
};
static_assert(kNumKernels <= 32, "BuildCounters::bytes holds 32 kernel kinds");
extern const char *const kKernelNames[kNumKernels];

// Totals of one level's plan. A level's cells take their tiles, histogram bins and list slots
// from these counters (one allocation per cell, in the order the cells become known).
struct PlanTotals {
    unsigned long long tiles;  // count tiles << 32 | partition tiles
    unsigned long long pools;  // histogram cells << 32 | list slots
    uint32_t swaps;            // partition tiles with pairs to swap (the swap's work list)
    uint32_t pad_;
};

// What the partition found for one cell (32 bytes, read at once by the swap).
struct CellPart {
    uint32_t b, n;   // first particle, particles
    uint32_t s, i;   // Hoare swaps, split index (cell-relative; n when clamped)
    uint32_t le;     // keys <= cut
    uint32_t t0, T;  // first partition tile, tiles
    uint32_t left;   // tiles that can hold left elements of pairs
};

// Device-side counters of one build (read back at the end).
struct BuildCounters {
    uint32_t degenerate;
    uint32_t zero_volume;
    uint32_t unfound;
    uint32_t max_iters;
    uint32_t any_active[4];  // histogram pass p left a cell active
    uint32_t error;       // set when a step could not be finished (see level_late, k_subtree's waits)
    uint32_t done[kMaxLevels + 1];  // cells whose children (or leaves) are final, per level
    PlanTotals plan[2];   // levels 1, 3, ... and 2, 4, ...
    uint32_t warm_cells;  // warm builds: cells that started from a hinted bracket
    uint32_t warm_resets; // ... whose hinted bracket missed the target (restarted cold)
    uint32_t pred_cells;  // cells whose first count pass used a sampled bracket
    uint32_t pred_misses; // ... whose sampled bracket did not hold the cut (binned again)
    uint32_t sub_cells[4];  // the subtree kernel's cells by class, and its work queues
    uint32_t sub_next[4];
    unsigned long long bytes[32];  // algorithmic bytes per Kernel kind
};

// Builds from host memory: the subtree kernel reports, per window of consecutive root cells,
// when every cell of the window is final, into pinned host memory that the host polls while
// the kernel runs; the host then copies the window's particles back while later windows are
// still being built.
constexpr int kMaxWindows = 64;
struct HostWindows {
    uint32_t decision;           // 0 not yet, 1 the subtree kernel finishes the tree, 2 refused
    uint32_t done[kMaxWindows];  // 1: window w final, its particles in range[w]
    uint2 range[kMaxWindows];
};

// Everything a level's kernels need. Cells of the level are heap slots [base, base + C)
// unless `slots` is non-null (batched builds, service calls over an arbitrary cell list).
// The partition of a level plans the next one: whoever finishes a cell allocates its
// children's tiles and writes their tile maps and state.
struct Level {
    float *x, *y, *z;
    uint32_t *idx;          // original particle index (perm), may be null
    orb_cell_t *heap;
    uint2 *ranges;          // {begin, end} per heap slot, absolute positions
    const int *slots;       // optional explicit slot list [C]
    int base;
    int C;
    int pass;               // histogram pass index within the level
    int last_pass;          // index of the level's last histogram pass
    uint32_t depth;         // index of the level within the build (0: the root's)
    // the next level: its cells (0: none is planned), where a cell's children stand among
    // them (child_map[c] = 4 x index of the first child | bit per child in the level; null:
    // 2c and 2c+1) and the cells the one-warp bisection takes there (up to small_next
    // particles; larger ones get count tiles)
    int next_C;
    const int *child_map;
    uint32_t small_next;
    uint32_t small;         // ... on this level (k_plan, k_init)
    int wide;               // 1: the box reaches 2^127, where midpoints overflow
    int few_tiles;          // weighted, 1: cells of at most 1024 keys on average
    uint32_t hist_threads;  // threads of a count pass's CTA (kThreads, 512 or 1024)
    uint32_t plan_bins;     // cells with count tiles get a list and, with several tiles, bins (1);
                            // bins for all (2); neither (0)
    // plan
    PlanTotals *tot, *tot_next;
    uint32_t *tile_off;     // [C] first count tile of each cell
    uint32_t *htile_cell;   // [tiles] cell of each count-left tile
    uint32_t *ptile_off;    // [C] first partition tile of each cell
    uint32_t *ptile_cell;   // [ptiles] cell of each partition tile
    uint32_t *hist_off;     // [C] first bin of each cell in the histogram pool
    uint8_t *state;         // [C] CellState
    uint8_t *iters;         // [C] bisection iterations done
    uint32_t *hist;         // histogram pool (kept all-zero between passes)
    uint32_t *hdone;        // [C] count tiles finished in the current pass
    uint32_t *below;        // [C] keys below the left margin
    uint32_t *inb;          // [C] keys inside the current bracket (n before the first pass)
    // bracket keys the classify pass lists for a kReady cell (their keys and positions)
    uint32_t *cmp_off;      // [C] first list slot of each cell
    uint32_t *cmp_cnt;      // [C] keys written to the list
    float *cmp_keys;        // the lists
    uint32_t *cmp_pos;
    // sampled first pass: leaves [lo, hi) of the first pass's midpoint tree predicted to hold
    // the cut (k_sample_bin, k_sample_pick); that pass counts the keys below leaf lo and bins
    // only the keys of [lo, hi). Packed (lo | hi << 12 | flag); 0: no prediction (dense)
    uint32_t *pred;         // [C]
    float pred_sigmas;      // half-width of the sampled bracket in standard errors (0: off)
    // partition
    uint32_t *ge_bits;      // [ptiles * kPWords] bit p: key >= cut
    uint32_t *le_bits;      // [ptiles * kPWords] bit p: key <= cut
    uint32_t *pt_ge;        // [ptiles] set bits per tile
    uint32_t *pt_le;
    uint32_t *pt_ge_pre;    // [ptiles] exclusive prefix within the cell
    uint32_t *pt_le_pre;
    CellPart *part;         // [C]
    uint2 *swap_list;       // [ptiles + cells] (cell, piece within the cell) of the swap's work: the
                            // tiles with left elements, each in 2^piece_log2 pieces
    uint32_t piece_log2;
    uint32_t *part_done;    // [C] tiles swapped
    int fuse;               // 1: the swap kernel finishes the cells (else k_part_finish)
    uint32_t done_start;    // what part_done starts from (0; the test hook's offset otherwise)
    uint32_t *out_counts;   // service calls: per-cell result
    const orb_cell_t *cells_in;  // service calls: the cells, which k_plan puts at their slots
    uint32_t sparse_per_tile;  // a bracket of at most this many keys a count tile is listed
    int pdl;                // level kernels launched with programmatic dependent launch
    // warm builds (null otherwise): per heap slot the previous tree's cut and w x its extent
    // (x NaN: no hint) and that tree's cut axis
    const float2 *hint;     // (cut, w x extent) from the previous tree
    const int *hint_axis;
    uint8_t *warm;          // [C] 1 while a hinted bracket is not yet checked
    int plan_hint;          // 1: the cells being planned start from their hints
    // subtrees: [0] 1 when one CTA per cell finishes the tree from this level down, [1] the level's
    // largest cell (~0: no subtree would help); null when not attempted
    uint32_t *skip;
    int *sub_list;          // [4 C] the subtree kernel's cells by class
    int sub_levels;         // levels below every cell (0: by its leaf count)
    int sub_wide;           // 1: all of a CTA's warps on every cell (levels of few cells)
    uint32_t copy_polls;    // most polls of a wait for a copy of keys
    int drop_copies;        // test hook: no copy of keys is made
    // window reports (null otherwise): the host-mapped reports, a finished-cell counter per
    // window, root cells per window
    HostWindows *hwin;
    uint32_t *win_cnt;
    uint32_t win_cells;
    // weighted builds (null otherwise): an integer weight per particle, moved with it, and
    // per cell of the level with several tiles its weight bins (at hist_off, kept all-zero
    // between passes), the weight below its bracket and its total weight
    uint32_t *wt;
    unsigned long long *whist;
    unsigned long long *wbelow;
    unsigned long long *wtot;
    uint32_t prev_C;        // cells of the level above (checked against counters->done)
    BuildCounters *counters;
};

__device__ __forceinline__ int level_slot(const Level &v, int c) {
    return v.slots ? v.slots[c] : v.base + c;
}

__device__ __forceinline__ int eff_axis(int a) { return a < 0 ? 0 : a; }

// getCut(), src/cell.h:74-76: float sum, halved (exact, no FMA, no FTZ).
__device__ __forceinline__ float mid_cut(float lo, float hi) {
    return __fmul_rn(__fadd_rn(hi, lo), 0.5f);
}

// src/orbit.cpp:204-208: difference = int(float(cl) - float(c) * ratio), found when
// |difference| < 3, else the right margin moves for a positive difference and the left one
// otherwise. ratio = leaf_ratio(nLeafCells) (0.5f when the leaf count is even). The
// uint->float roundings above 2^24 are kept. Returns 0 found, +1 right margin, -1 left.
__device__ __forceinline__ int convergence(uint32_t count_left, uint32_t count, float ratio) {
    float prod = __fmul_rn(__uint2float_rn(count), ratio);
    float diff = __fsub_rn(__uint2float_rn(count_left), prod);
    int difference = __float2int_rz(diff);
    if (difference > -3 && difference < 3) return 0;
    return difference > 0 ? 1 : -1;
}

// The weighted test (no counterpart in the reference, whose thesis specifies weighted ORB,
// documentation/notes.tex:259-271, and whose code never implements it): the reference's
// |W_left - ratio W| < 3 (src/orbit.cpp:204-208) with the tolerance scaled by the cell's
// mean weight W/n, exact in 128-bit integers: D = k W_left - ceil(k/2) W for k leaves;
// found when D == 0 or n |D| < 3 k W; else +1 (D > 0, the right margin moves) or -1. With
// unit weights: |cl - ratio c| < 3 exactly, the reference's float32 test wherever that test
// is exact (fewer than 2^24 particles, an even k).
__device__ __forceinline__ int convergence_weighted(unsigned long long w_left,
                                                    unsigned long long w_cell, uint32_t n,
                                                    int32_t n_leaf) {
    const __int128 k = n_leaf, half = (n_leaf + 1) / 2;
    const __int128 D = k * (__int128)w_left - half * (__int128)w_cell;
    const unsigned __int128 ad = (unsigned __int128)(D < 0 ? -D : D);
    if (D == 0 || (unsigned __int128)n * ad < (unsigned __int128)3 * (unsigned __int128)k * w_cell)
        return 0;
    return D > 0 ? 1 : -1;
}

__device__ __forceinline__ const float *axis_keys(const Level &v, int axis) {
    return axis == 0 ? v.x : (axis == 1 ? v.y : v.z);
}

// Level slices of the reference's driver for a root of d leaves (src/orbit.cpp:104-107,
// src/cell.h:65-72): level l (from 1) takes the heap cells [2^(l-1)-1, b_l] with
// b_l = min(getNCellsOnLastLevel(), 2^l) - 2, getNCellsOnLastLevel() = 2d - 2^ceil(log2 d).
// For a power of two that is every cell of the level. For other d the reference's loop
// stops at getNLevels() - 1 = ceil(log2 d) - 1, and a slice may come out partial or empty
// (b_l < 2^(l-1)-1; the reference then calls its services with a non-positive cell count,
// which is undefined; here such a level has no cells).
struct Slices {
    uint32_t depth;  // getNLevels()
    uint32_t last;   // getNCellsOnLastLevel()
    bool pow2;
    explicit Slices(uint32_t d) {
        depth = 0;
        while ((1ull << depth) < d) ++depth;
        last = (uint32_t)(2ull * d - (1ull << depth));
        pow2 = (d & (d - 1)) == 0;
    }
    // most split levels: log2(d) for a power of two, else the reference's bound
    uint32_t max_levels() const { return pow2 ? depth : (depth ? depth - 1 : 0); }
    int first(uint32_t l) const { return (1 << (l - 1)) - 1; }
    int count(uint32_t l) const {
        const int b = (int)std::min<uint64_t>(last, 1ull << l) - 2;
        return std::max(0, b - first(l) + 1);
    }
    // heap cells a build of `levels` levels fills: ids [0, 2 b + 3) for the last level with
    // cells (children 2b+1, 2b+2 of its last cell b), the root alone without levels
    uint64_t filled(uint32_t levels) const {
        uint64_t f = 1;
        for (uint32_t l = 1; l <= levels; ++l)
            if (count(l) > 0) f = 2ull * (uint64_t)(first(l) + count(l) - 1) + 3;
        return f;
    }
};

// Root of one instance of a batched build.
struct BatchRoot {
    uint32_t offset;     // first particle
    uint32_t n;          // particles
    uint32_t d;          // leaf cells
    uint32_t heap_base;  // heap slot of the root
    int32_t cell;        // its index among level 1's cells (-1: no split level)
    float lower[3], upper[3];
};

// Host-side launchers (orb_kernels.cu). `grid` is the CTA count of the tile loops.
void launch_init(const Level &v, uint64_t n, const float lower[3], const float upper[3],
                 uint32_t d, int heap_cells, cudaStream_t st);
void launch_level_kernel(Kernel k, const Level &v, int grid, int arg, cudaStream_t st);
void launch_init_batch(const Level &v, const BatchRoot *roots, int k, uint64_t n_total,
                       cudaStream_t st);
// dst[p] = src[p] for the positions of every instance (2-D grid: instance x particles)
void launch_copy_instances(const uint32_t *src, uint32_t *dst, const BatchRoot *roots, int k,
                           cudaStream_t st);
// Gaussian displacement of the particles [offset, offset+n): x += sigma * N(0,1) per
// coordinate, clamped to [lower, nextafter(upper, lower)] (seeded, counter-based)
void launch_displace(float *x, float *y, float *z, uint64_t offset, uint64_t n, uint64_t seed,
                     float sigma, const float lower[3], const float upper[3], cudaStream_t st);
cudaError_t configure_kernels();  // once per device (dynamic shared memory limits)
int swap_blocks_per_sm();         // resident CTAs of the swap kernel per SM (its grid)
void launch_gen_uniform(uint64_t seed, uint64_t n, float *x, float *y, float *z,
                        cudaStream_t st);
// `draws` draws of the reference's xorshf96 stream, thread g from starts[3g..3g+2] for `chunk`
void launch_gen_xorshf96(const unsigned long long *starts, uint64_t draws, uint32_t chunk,
                         float *x, float *y, float *z, cudaStream_t st);
void launch_gen_plummer(uint64_t seed, uint64_t n, const float *centres, const double *scales,
                        float *x, float *y, float *z, cudaStream_t st);

// Makes the pages of a host buffer resident (its bytes keep their values), see orb_api.cu.
void touch_pages(void *ptr, size_t bytes, bool meanwhile);

// Context internals used by the request server (orb_server.cu).
cudaStream_t ctx_stream(orb_ctx *ctx);
void ctx_disable_graphs(orb_ctx *ctx);
void launch_iota_u32(uint32_t *dst, uint64_t n, cudaStream_t st);  // dst[p] = p
// gather: dst[off+p] = src[off + perm[off+p]] for p < n (instance-relative permutation)
void launch_stage_gather(float *dst, const float *src, const uint32_t *idx, uint64_t n,
                         BuildCounters *ctr, int num_sms, cudaStream_t st);
void launch_gather_u32(uint32_t *dst, const uint32_t *src, const uint32_t *perm, uint64_t off,
                       uint64_t n, cudaStream_t st);

}  // namespace orb
