// flk_grid_noalloc: the grid build of one flock step (cell keys, bucket
// offsets, stable sorted order) for callers that cannot allocate device memory.
//
// Who needs it: code that runs where cudaMalloc is off limits -- a host
// application that owns every byte of device memory through its own pool and
// forbids libraries from allocating behind its back, a real-time loop where
// cudaMalloc's implicit device synchronisation would stall the frame, or a
// plugin loaded into a process whose memory budget is fixed up front. Such a
// caller hands in device buffers for the inputs and outputs; everything else
// the passes need (histogram, the unsorted slots and counters) lives in one
// file-scope device array, g_flk_noalloc_scratch, sized for at most
// FLK_NOALLOC_MAX_BIRDS birds. Every GPU that loads this library holds that
// array (about 1.5 MiB) until the process exits.
//
// The array's name in host code is only a host-side handle, not a device
// address, so every call looks the address up with cudaGetSymbolAddress on the
// current device and passes the pointer to the kernels. Nothing is cached
// across calls, so a device reset between calls (which reloads the module and
// moves the array) cannot leave a stale address behind. The call is blocking:
// it synchronises its stream before it returns.
//
// All calls share the one array and it keeps the previous call's contents:
// each call clears the parts that must start at zero. Calls that overlap on the
// GPU (different streams or threads, same device) race on the array and give
// wrong results; serialise them. Later calls are right again: a call's barrier
// counters are its own (one of BARRIERS sets in turn, cleared half a turn before).
//
// A call is latency: at 131,072 birds three clears, four kernels and the error
// word's copy took 49 us, of which the host's launches were nearly all. The
// passes (clear, hash and count, exclusive scan, scatter by arrival rank,
// per-bucket sort by bird) are phases of one cooperative kernel with two buckets
// and at most one bird per thread, a bounded grid barrier between them, and the
// error word goes straight to a page-locked host word. (One 16-CTA cluster with
// its hardware barrier took 76 us: too few SMs for the atomics and the sort.)
// The outputs equal flk_step_debug's keys/offsets/sorted bit for bit.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdint>
#include <cstring>
#include <string>

#include "../../include/flock_gb300.h"
#include "flock_params.h"

namespace flk {
void set_last_error(const std::string& msg);  // flock_abi.cpp
}

namespace {

constexpr uint32_t MAX_BIRDS = FLK_NOALLOC_MAX_BIRDS;
constexpr uint32_t MAX_BUCKETS = 2u * FLK_NOALLOC_MAX_BIRDS;  // buckets_for(MAX_BIRDS)
constexpr uint32_t FULL = 0xFFFFFFFFu;

// Byte layout of the scratch array (each region 256-byte aligned).
constexpr size_t OFF_COUNTS = 0;                                  // MAX_BUCKETS u32
constexpr size_t OFF_TMP = OFF_COUNTS + MAX_BUCKETS * 4ull;       // MAX_BIRDS u32
constexpr size_t OFF_CTL = OFF_TMP + MAX_BIRDS * 4ull;            // CTL_WORDS u32
constexpr uint32_t BARRIERS = 32;  // calls until a set of barrier counters is used again
// an error; birds per tile; the barriers' counters (arrived, turns: 16 words a set)
enum { CTL_ERROR = 0, CTL_SUM = 64, CTL_BARRIER = 128, CTL_WORDS = CTL_BARRIER + 16 * BARRIERS };
enum { ARRIVED = 0, TURN = 8 };
constexpr size_t SCRATCH_BYTES = OFF_CTL + CTL_WORDS * 4ull;
constexpr int THREADS = 1024;        // per CTA
constexpr uint32_t TILE = 4096;      // buckets per CTA in the scan
constexpr uint32_t SPIN_LIMIT = 1u << 20;  // polls of a barrier before it gives up

static_assert(OFF_CTL % 256 == 0, "scratch regions stay 256-byte aligned");

}  // namespace

static __device__ __align__(256) unsigned char g_flk_noalloc_scratch[SCRATCH_BYTES];

namespace {

struct Scratch {
    uint32_t* counts;
    uint32_t* tmp;
    uint32_t* ctl;
};

Scratch carve(unsigned char* base) {
    return Scratch{reinterpret_cast<uint32_t*>(base + OFF_COUNTS), reinterpret_cast<uint32_t*>(base + OFF_TMP),
                   reinterpret_cast<uint32_t*>(base + OFF_CTL)};
}

__device__ __forceinline__ int cell1(float x) { return (int)floorf(__fmul_rn(x, flk::INV_CELL)); }

// Loads of what another CTA wrote in an earlier phase.
__device__ __forceinline__ uint32_t ld(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ uint4 ld(const uint4* p) {
    uint4 v;
    asm volatile("ld.global.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(p)
                 : "memory");
    return v;
}
// Orders every earlier access of the grid's threads before every later one (a
// cooperative launch: all CTAs are resident). The wait is bounded: false, in
// every thread of a CTA, where it gave up.
__device__ __forceinline__ bool grid_barrier(uint32_t* bar, uint32_t* status) {
    __shared__ uint32_t s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        volatile uint32_t* turn = bar + TURN;
        const uint32_t now = *turn;
        uint32_t polls = 0;
        __threadfence();
        if (atomicAdd(&bar[ARRIVED], 1u) == gridDim.x - 1u) {
            bar[ARRIVED] = 0;
            __threadfence();
            *turn = now + 1u;
        } else {
            while (*turn == now && polls < SPIN_LIMIT) ++polls;
        }
        __threadfence();
        s_ok = polls < SPIN_LIMIT;
        if (polls == SPIN_LIMIT) *(volatile uint32_t*)status = 1u;
    }
    __syncthreads();
    return s_ok != 0;
}
__device__ __forceinline__ uint32_t warp_inclusive(uint32_t x, uint32_t lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(FULL, x, o);
        if ((int)lane >= o) x += y;
    }
    return x;
}

// The birds (tmp[s0 .. s0 + L)) of one bucket in bird order, by one warp.
__device__ __forceinline__ void sort_bucket(const uint32_t* tmp, uint32_t s0, uint32_t L, uint32_t* __restrict__ sorted,
                                            uint32_t lane) {
    if (L <= 32) {
        uint32_t x = lane < L ? ld(&tmp[s0 + lane]) : 0xFFFFFFFFu;
#pragma unroll
        for (int k = 2; k <= 32; k <<= 1) {
#pragma unroll
            for (int j = k >> 1; j > 0; j >>= 1) {
                const uint32_t y = __shfl_xor_sync(FULL, x, j);
                const bool up = (lane & k) == 0, lower = (lane & j) == 0;
                x = (lower == up) ? min(x, y) : max(x, y);
            }
        }
        if (lane < L) sorted[s0 + lane] = x;
        return;
    }
    for (uint32_t c0 = 0; c0 < L; c0 += 32) {
        const bool has = c0 + lane < L;
        const uint32_t x = has ? ld(&tmp[s0 + c0 + lane]) : 0xFFFFFFFFu;
        uint32_t rank = 0;
        for (uint32_t j0 = 0; j0 < L; j0 += 32) {
            const uint32_t y = (j0 + lane < L) ? ld(&tmp[s0 + j0 + lane]) : 0xFFFFFFFFu;
#pragma unroll 8
            for (int q = 0; q < 32; ++q) rank += __shfl_sync(FULL, y, q) < x;
        }
        if (has) sorted[s0 + rank] = x;
    }
}

constexpr int PHASES = 5;  // clear, count, scan, scatter, order

// buckets: a power of two of at least 2^16, and at least 2n; buckets / 2 threads.
// *status: zero at the start, an error word where there was one.
// FUSED: every phase, with barrier set `arg` (a cooperative launch); otherwise
// phase `arg` alone, the arrival ranks waiting in `sorted` for the scatter.
template <bool FUSED>
__global__ void __launch_bounds__(THREADS, 1) k_na_grid(const float4* __restrict__ pos, uint32_t n, uint32_t buckets,
                                                        uint32_t* keys, uint32_t* offsets, uint32_t* sorted, Scratch s,
                                                        uint32_t* status, uint32_t arg) {
    __shared__ uint32_t s_warp[THREADS / 32], s_tile[MAX_BUCKETS / TILE];
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, v = blockIdx.x * THREADS + tid;
    const bool mine = v < n;  // this thread's bird
    uint32_t* bar = s.ctl + CTL_BARRIER + 16 * arg;
    const auto runs = [&](uint32_t phase) { return FUSED || arg == phase; };
    float4 p = make_float4(0.f, 0.f, 0.f, 0.f);
    uint32_t b = 0, arrival = 0;
    if (mine && (FUSED || arg == 1)) p = pos[v];
    if (tid < MAX_BUCKETS / TILE) s_tile[tid] = 0;
    if (runs(0)) {
        reinterpret_cast<uint2*>(s.counts)[v] = make_uint2(0u, 0u);
        if (v < MAX_BUCKETS / TILE) s.ctl[CTL_SUM + v] = 0;
        if (FUSED && v < 16) s.ctl[CTL_BARRIER + 16 * ((arg + BARRIERS / 2) % BARRIERS) + v] = 0;
    }
    if (FUSED && !grid_barrier(bar, status)) return;
    // hash and count, each tile of buckets as a whole as well
    if (runs(1)) {
        if (!FUSED) __syncthreads();  // s_tile is clear
        if (mine) {
            b = (((uint32_t)cell1(p.x) * 73856093u) ^ ((uint32_t)cell1(p.y) * 19349663u) ^
                 ((uint32_t)cell1(p.z) * 83492791u)) & (buckets - 1u);
            arrival = atomicAdd(&s.counts[b], 1u);
            keys[v] = b;
            atomicAdd(&s_tile[b / TILE], 1u);
            if (!FUSED) sorted[v] = arrival;
        }
        __syncthreads();
        if (tid < MAX_BUCKETS / TILE && s_tile[tid]) atomicAdd(&s.ctl[CTL_SUM + tid], s_tile[tid]);
    }
    if (FUSED && !grid_barrier(bar, status)) return;
    // exclusive scan, a tile per CTA (half of the CTAs)
    const uint32_t tiles = buckets / TILE;  // 16 to 64
    if (runs(2) && blockIdx.x < tiles) {
        const uint4 c = ld(reinterpret_cast<const uint4*>(s.counts + blockIdx.x * TILE) + tid);
        uint32_t before = 0;  // birds of the tiles before
        for (uint32_t t = lane; t < blockIdx.x; t += 32) before += ld(&s.ctl[CTL_SUM + t]);
        const uint32_t sum = c.x + c.y + c.z + c.w, inc = warp_inclusive(sum, lane);
        if (lane == 31) s_warp[warp] = inc;
        __syncthreads();
        const uint32_t tot = s_warp[lane], pre = warp_inclusive(tot, lane);
        uint32_t run = __reduce_add_sync(FULL, before) + __shfl_sync(FULL, pre - tot, warp) + inc - sum;
        uint4 o;
        o.x = run; run += c.x;
        o.y = run; run += c.y;
        o.z = run; run += c.z;
        o.w = run; run += c.w;
        reinterpret_cast<uint4*>(offsets + blockIdx.x * TILE)[tid] = o;
        if (blockIdx.x == tiles - 1 && tid == THREADS - 1) offsets[buckets] = run;
    }
    if (FUSED && !grid_barrier(bar, status)) return;
    // scatter by arrival rank
    if (runs(3) && mine) {
        if (!FUSED) {
            b = keys[v];
            arrival = sorted[v];
        }
        const uint32_t to = ld(&offsets[b]) + arrival;
        if (to < n) s.tmp[to] = v;
        else *(volatile uint32_t*)status = 2u;
    }
    if (FUSED && !grid_barrier(bar, status)) return;
    // each occupied bucket in bird order, a warp each; a warp looks through 32
    // buckets at a time, the CTAs' warps in turn
    if (!runs(4)) return;
    for (uint32_t b0 = (warp * gridDim.x + blockIdx.x) * 32u; b0 < buckets; b0 += gridDim.x * THREADS) {
        const uint32_t s0 = ld(&offsets[b0 + lane]), L = ld(&s.counts[b0 + lane]);
        uint32_t some = __ballot_sync(FULL, L != 0);
        while (some) {
            const int k = __ffs(some) - 1;
            some &= some - 1;
            const uint32_t from = __shfl_sync(FULL, s0, k), len = __shfl_sync(FULL, L, k);
            if (from + len < from || from + len > n) {
                if (lane == 0) *(volatile uint32_t*)status = 2u;
                continue;
            }
            sort_bucket(s.tmp, from, len, sorted, lane);
        }
    }
}

// A page-locked word per device that the kernel reports to. Its device address
// is looked up on every call, and the words locked again where a device reset
// has undone that; null: the error word is copied back instead.
constexpr int STATUS_DEVICES = 64;
alignas(4096) uint32_t g_status[STATUS_DEVICES * 16];
uint32_t* status_word(int dev) {
    void* d = nullptr;
    if (cudaHostGetDevicePointer(&d, g_status, 0) != cudaSuccess) {
        (void)cudaHostRegister(g_status, sizeof g_status, cudaHostRegisterPortable | cudaHostRegisterMapped);
        d = nullptr;
        if (cudaHostGetDevicePointer(&d, g_status, 0) != cudaSuccess) d = nullptr;
        (void)cudaGetLastError();
    }
    return d ? static_cast<uint32_t*>(d) + (dev % STATUS_DEVICES) * 16 : nullptr;
}

int na_fail(int code, const std::string& m) {
    flk::set_last_error(m);  // reported by flk_last_error()
    return code;
}

// The last call's number on each device: which barrier counters the next one uses.
std::atomic<uint32_t> g_calls[STATUS_DEVICES];

// separate: five launches whatever the device holds; spoil: leaves the call's
// barrier counters as calls that overlapped might.
int grid_noalloc(const float* pos4, uint32_t n, uint32_t* keys, uint32_t* offsets, uint32_t* sorted, void* stream,
                 bool separate, bool spoil) {
    if (n > MAX_BIRDS)
        return na_fail(FLK_ERR_CAPACITY, "flk_grid_noalloc: " + std::to_string(n) + " birds exceeds the maximum of " +
                                             std::to_string(MAX_BIRDS) + " this entry point's fixed scratch holds");
    if (!offsets || (n && (!pos4 || !keys || !sorted)))
        return na_fail(FLK_ERR_ARG, "flk_grid_noalloc: null device pointer");
    // float4 loads of pos4 and 16-byte stores into offsets need 16-byte alignment
    if ((reinterpret_cast<uintptr_t>(pos4) | reinterpret_cast<uintptr_t>(offsets)) & 15u)
        return na_fail(FLK_ERR_ARG, "flk_grid_noalloc: pos4 and offsets must be 16-byte aligned");
    // the scratch array's device address on the current device, looked up on
    // every call (cheap next to the stream synchronisation below)
    void* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_flk_noalloc_scratch);
    if (e != cudaSuccess) return na_fail(FLK_ERR_CUDA, std::string("cudaGetSymbolAddress: ") + cudaGetErrorString(e));
    unsigned char* base = static_cast<unsigned char*>(p);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    uint64_t want = 1;
    while (want < (uint64_t)n * 2) want <<= 1;
    const uint32_t B = (uint32_t)(want < (1u << 16) ? (1u << 16) : want);  // n <= MAX_BIRDS keeps B <= 2^22
    const Scratch s = carve(base);
    int dev = 0;
    e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return na_fail(FLK_ERR_CUDA, std::string("cudaGetDevice: ") + cudaGetErrorString(e));
    uint32_t* word = status_word(dev);
    if (word) *(volatile uint32_t*)&g_status[(dev % STATUS_DEVICES) * 16] = 0;
    else if ((e = cudaMemsetAsync(s.ctl + CTL_ERROR, 0, 4, st)) != cudaSuccess)
        return na_fail(FLK_ERR_CUDA, std::string("cudaMemsetAsync: ") + cudaGetErrorString(e));
    uint32_t* status = word ? word : s.ctl + CTL_ERROR;
    const float4* pos = reinterpret_cast<const float4*>(pos4);
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeCooperative;
    at.val.cooperative = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(B / 2 / THREADS);  // 32 to 128 CTAs
    cfg.blockDim = dim3(THREADS);
    cfg.stream = st;
    const uint32_t set = g_calls[dev % STATUS_DEVICES].fetch_add(1) % BARRIERS;
    const auto phases = [&] {
        cfg.numAttrs = 0;
        cudaError_t r = cudaMemsetAsync(s.ctl + CTL_BARRIER + 16 * ((set + BARRIERS / 2) % BARRIERS), 0, 64, st);
        for (uint32_t k = 0; k < PHASES && r == cudaSuccess; ++k)
            r = cudaLaunchKernelEx(&cfg, k_na_grid<false>, pos, n, B, keys, offsets, sorted, s, status, k);
        return r;
    };
    uint32_t err = 0;
    // the error word once the stream is done
    const auto finish = [&] {
        err = 0;
        cudaError_t r = word ? cudaSuccess : cudaMemcpyAsync(&err, status, 4, cudaMemcpyDeviceToHost, st);
        if (r == cudaSuccess) r = cudaStreamSynchronize(st);
        if (r == cudaSuccess && word) err = *(volatile uint32_t*)&g_status[(dev % STATUS_DEVICES) * 16];
        return r;
    };
    if (!separate) {
        cfg.attrs = &at;
        cfg.numAttrs = 1;
        e = cudaLaunchKernelEx(&cfg, k_na_grid<true>, pos, n, B, keys, offsets, sorted, s, status, set);
        if (e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorNotSupported) {
            (void)cudaGetLastError();
            separate = true;
        }
    }
    if (separate) e = phases();
    if (e != cudaSuccess) return na_fail(FLK_ERR_CUDA, std::string("launch: ") + cudaGetErrorString(e));
    e = finish();
    if (e == cudaSuccess && err == 1) {  // a barrier gave up: clear its counters, do without
        if (word) *(volatile uint32_t*)&g_status[(dev % STATUS_DEVICES) * 16] = 0;
        e = cudaMemsetAsync(s.ctl, 0, CTL_WORDS * 4, st);
        if (e == cudaSuccess) e = phases();
        if (e == cudaSuccess) e = finish();
    }
    if (e == cudaSuccess && spoil) {
        e = cudaMemsetAsync(s.ctl + CTL_BARRIER + 16 * set, 1, 16 * 4, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    }
    if (e != cudaSuccess) return na_fail(FLK_ERR_CUDA, std::string("flk_grid_noalloc: ") + cudaGetErrorString(e));
    if (err) return na_fail(FLK_ERR_DEVICE, "flk_grid_noalloc: device error word " + std::to_string(err));
    return FLK_OK;
}

}  // namespace

extern "C" int flk_grid_noalloc(const float* pos4, uint32_t n, uint32_t* keys, uint32_t* offsets, uint32_t* sorted,
                                void* stream) {
    return grid_noalloc(pos4, n, keys, offsets, sorted, stream, false, false);
}

extern "C" int flk_debug_grid_noalloc(const float* pos4, uint32_t n, uint32_t* keys, uint32_t* offsets,
                                      uint32_t* sorted, void* stream, int32_t separate, int32_t spoil) {
    return grid_noalloc(pos4, n, keys, offsets, sorted, stream, separate != 0, spoil != 0);
}
