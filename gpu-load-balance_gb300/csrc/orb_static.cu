// orb_count_left_static: count-left for callers that may not allocate device memory.
//
// Simulation codes that call the ORB services from inside their time-step loop often own
// the whole device through their own memory pool, reserved at start-up: a cudaMalloc there
// either fails or fragments the pool, and cudaMalloc/cudaFree synchronise the device, which
// stalls the caller's other streams. orb_count_left needs a context whose buffers are
// allocated on first use; this entry point needs no context and allocates nothing. Its
// scratch (per-cell tile offsets and their chunks' totals) is the file-scope device array
// below, for ORB_STATIC_MAX_CELLS cells; every GPU that loads the library holds it
// (65536 + 64 words, 256 KiB) until the process exits.
#include <cuda_runtime.h>

#include <mutex>

#include "orb_internal.cuh"

namespace {

constexpr uint32_t kMaxCells = ORB_STATIC_MAX_CELLS;
constexpr uint32_t kTileKeys = 2048;   // keys a warp counts at a time
constexpr uint32_t kChunk = 1024;      // cells a plan CTA takes
constexpr uint32_t kChunks = kMaxCells / kChunk;
static_assert(kChunks <= 64, "two chunks a lane in k_static_count");
constexpr int kMaxDevices = 64;

// [0, kMaxCells): first tile of each cell within its chunk; [kMaxCells, kMaxCells + kChunks):
// the chunks' tiles.
static __device__ __align__(256) uint32_t g_count_scratch[kMaxCells + kChunks];

struct DeviceSetup {
    bool done;
    uint32_t *scratch;  // device address of g_count_scratch on that device
    int sms;
};
std::mutex g_setup_mu;
DeviceSetup g_setup[kMaxDevices];

// Once per device, with that device current: resolve the array's device address. Host
// code must not pass `g_count_scratch` itself to a kernel: on the host that name is a
// host-side stand-in, not a device address. The address is kept for the life of the
// process, so the entry point must not be called on a device after cudaDeviceReset there
// (the module, and with it the array, is loaded again at another address).
cudaError_t setup_device(int dev, DeviceSetup *out) {
    std::lock_guard<std::mutex> g(g_setup_mu);
    if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
    DeviceSetup &s = g_setup[dev];
    if (!s.done) {
        void *p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_count_scratch);
        if (e != cudaSuccess) return e;
        int sms = 0;
        e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (e != cudaSuccess) return e;
        s.scratch = static_cast<uint32_t *>(p);
        s.sms = sms;
        s.done = true;
    }
    *out = s;
    return cudaSuccess;
}

// Range of a cell, or an empty range when its id or range is outside the caller's map.
__device__ __forceinline__ uint2 cell_range(const orb_cell_t &c, const uint32_t *ranges,
                                            uint32_t n_ranges, uint64_t n) {
    if (c.id < 0 || (uint32_t)c.id >= n_ranges) return make_uint2(0u, 0u);
    const uint32_t b = ranges[2 * c.id], e = ranges[2 * c.id + 1];
    if (b > e || (uint64_t)e > n) return make_uint2(0u, 0u);
    return make_uint2(b, e);
}

// A CTA a chunk of cells, a thread a cell: its tiles (none for a found cell), their exclusive
// prefix within the chunk, and a zero in the output of every cell that is counted.
__global__ void __launch_bounds__(kChunk) k_static_plan(const orb_cell_t *cells, uint32_t C,
                                                        const uint32_t *ranges, uint32_t n_ranges,
                                                        uint64_t n, uint32_t *out, uint32_t *scratch) {
    __shared__ uint32_t warp_tot[32];
    const uint32_t tid = threadIdx.x, c = blockIdx.x * kChunk + tid;
    uint32_t mine = 0;
    if (c < C && !cells[c].foundCut) {
        const uint2 r = cell_range(cells[c], ranges, n_ranges, n);
        mine = (r.y - r.x + kTileKeys - 1) / kTileKeys;
        out[c] = 0u;
    }
    const int lane = tid & 31, warp = tid >> 5;
    uint32_t inc = mine;
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += t;
    }
    if (lane == 31) warp_tot[warp] = inc;
    __syncthreads();
    const uint32_t w = warp_tot[lane];
    const uint32_t before = __reduce_add_sync(0xffffffffu, lane < warp ? w : 0u);
    if (c < C) scratch[c] = before + inc - mine;
    if (tid == kChunk - 1) scratch[kMaxCells + blockIdx.x] = before + inc;
}

// A warp a tile, the CTA's eight warps on consecutive ones: two searches find its cell (the
// chunk among the lanes' prefixes, then 32 cells a probe), 16-byte loads, and one add per cell
// and CTA. Bound by HBM for many keys, by the chain of small loads ahead of them for few. The
// former form (a scan by one CTA, a CTA a tile of 8192 keys with 4-byte loads and a binary
// search, counters in scratch copied out by a third kernel) took 47 us for 2^24 clustered
// particles in 1024 cells, a quarter of them found; this takes 18.
__global__ void __launch_bounds__(256) k_static_count(const float *x, const float *y, const float *z,
                                                      const orb_cell_t *cells, uint32_t C,
                                                      const uint32_t *ranges, uint32_t n_ranges,
                                                      uint64_t n, uint32_t *out, const uint32_t *scratch) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    __shared__ uint32_t s_cell[8], s_cnt[8];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t chunks = (C + kChunk - 1) / kChunk;
    // first tile of chunks 2 lane and 2 lane + 1 (past the last chunk: all the tiles)
    const uint32_t ta = 2 * lane < chunks ? scratch[kMaxCells + 2 * lane] : 0u;
    const uint32_t tb = 2 * lane + 1 < chunks ? scratch[kMaxCells + 2 * lane + 1] : 0u;
    unsigned long long inc = (unsigned long long)ta + tb;
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= (uint32_t)o) inc += t;
    }
    const unsigned long long total = __shfl_sync(0xffffffffu, inc, 31);
    const unsigned long long b0 = inc - ta - tb, b1 = b0 + ta;
    for (unsigned long long g = 8ull * blockIdx.x; g < total; g += 8ull * gridDim.x) {
        const unsigned long long t = g + warp;
        uint32_t c = 0xffffffffu, cnt = 0;
        if (t < total) {  // warp-uniform
            const uint32_t below = (uint32_t)__popc(__ballot_sync(0xffffffffu, 2 * lane < chunks && b0 <= t)) +
                                   (uint32_t)__popc(__ballot_sync(0xffffffffu, 2 * lane + 1 < chunks && b1 <= t));
            const uint32_t chunk = below - 1u;  // the last chunk that starts at or before t
            const unsigned long long base =
                __shfl_sync(0xffffffffu, (chunk & 1u) ? b1 : b0, (int)(chunk >> 1));
            const uint32_t local = (uint32_t)(t - base);
            const uint32_t *off = scratch + chunk * kChunk;
            const uint32_t len = min(kChunk, C - chunk * kChunk);
            // the last cell that starts at or before `local`, 32 probes a round
            uint32_t lo = 0;
            for (uint32_t step = kChunk / 32; step; step = step > 1 ? 1 : 0) {
                const uint32_t p = lo + lane * step;
                const bool ok = p < len && off[p] <= local;
                lo += ((uint32_t)__popc(__ballot_sync(0xffffffffu, ok)) - 1u) * step;
            }
            c = chunk * kChunk + lo;
            const orb_cell_t &cell = cells[c];
            const uint2 r = cell_range(cell, ranges, n_ranges, n);
            const int axis = cell.cutAxis < 0 ? 0 : cell.cutAxis;
            const float *keys = axis == 0 ? x : (axis == 1 ? y : z);
            const float cut = orb::mid_cut(cell.cutMarginLeft, cell.cutMarginRight);  // getCut()
            const uint32_t e0 = r.x + (local - off[lo]) * kTileKeys, e1 = min(r.y, e0 + kTileKeys);
            const uintptr_t addr = reinterpret_cast<uintptr_t>(keys + e0);
            const uint32_t a0 = min(e1, e0 + (uint32_t)(((16u - (addr & 15u)) & 15u) >> 2));
            const uint32_t n4 = (e1 - a0) >> 2;
            if (lane < a0 - e0) cnt += __ldg(keys + e0 + lane) < cut;
            const float4 *k4 = reinterpret_cast<const float4 *>(keys + a0);
#pragma unroll 8
            for (uint32_t i = lane; i < n4; i += 32) {
                const float4 q = __ldg(k4 + i);
                cnt += (q.x < cut) + (q.y < cut) + (q.z < cut) + (q.w < cut);
            }
            const uint32_t tail = a0 + (n4 << 2);
            if (lane < e1 - tail) cnt += __ldg(keys + tail + lane) < cut;
            cnt = __reduce_add_sync(0xffffffffu, cnt);
        }
        if (lane == 0) {
            s_cell[warp] = c;
            s_cnt[warp] = cnt;
        }
        __syncthreads();
        if (warp == 0) {
            // the warps' counts added up per cell, by each cell's first warp
            const uint32_t mc = lane < 8 ? s_cell[lane] : 0xffffffffu;
            const uint32_t peers = __match_any_sync(0xffffffffu, mc);
            if (mc != 0xffffffffu && lane == (uint32_t)__ffs(peers) - 1u) {
                uint32_t sum = 0;
                for (uint32_t p = peers; p; p &= p - 1u) sum += s_cnt[__ffs(p) - 1];
                if (sum) atomicAdd(&out[mc], sum);
            }
        }
        __syncthreads();
    }
}

}  // namespace

extern "C" orb_status orb_count_left_static(const float *x, const float *y, const float *z,
                                            uint64_t n, const orb_cell_t *cells,
                                            uint32_t n_cells, const uint32_t *ranges,
                                            uint32_t n_ranges, uint32_t *out, void *stream) {
    if (n_cells == 0) return ORB_OK;
    if (n_cells > kMaxCells) return ORB_ERR_CAPACITY;  // more cells than the static scratch holds
    if (!cells || !ranges || !out || (n > 0 && (!x || !y || !z))) return ORB_ERR_INVALID_ARGUMENT;
    if (n >= (1ull << 31)) return ORB_ERR_CAPACITY;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return ORB_ERR_CUDA;
    DeviceSetup s;
    if (setup_device(dev, &s) != cudaSuccess) return ORB_ERR_CUDA;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    k_static_plan<<<(n_cells + kChunk - 1) / kChunk, kChunk, 0, st>>>(cells, n_cells, ranges, n_ranges, n, out,
                                                                     s.scratch);
    // the count kernel's launch overlaps the plan's (it waits for it in griddepcontrol.wait)
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)s.sms * 8);
    cfg.blockDim = dim3(256);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (cudaLaunchKernelEx(&cfg, k_static_count, x, y, z, cells, n_cells, ranges, n_ranges, n, out,
                           (const uint32_t *)s.scratch) != cudaSuccess) {
        cudaGetLastError();
        return ORB_ERR_CUDA;
    }
    return cudaGetLastError() == cudaSuccess ? ORB_OK : ORB_ERR_CUDA;
}
