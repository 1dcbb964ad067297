// GB300 (sm_103a) kernels and host engine for the starling-flock step.
//
// One step (reference order, crates/flock-ref/src/model.rs:182-200 and
// cuda/flock.cu:453-470): time += DT; rebuild the cell grid from the current
// positions; every bird with time >= next_decision decides from a snapshot;
// every bird integrates. The passes here:
//
//   k_hash_count  cell key per bird + bucket histogram with warp-aggregated
//                 atomics (one per run of adjacent lanes with one bucket);
//                 records each bird's arrival rank. Production steps bucket
//                 birds by a row lattice, grid-reporting steps by the
//                 reference's hash.
//   k_place       production steps: run starts from the histogram, tile by tile
//                 (whole rows), each tile's place from its flock's cursor;
//                 clears the histogram.
//   k_scan        grid-reporting steps: single-pass decoupled look-back
//                 exclusive scan of the histogram into the canonical offsets;
//                 clears the histogram. Bounded waits.
//   k_scatter     bird -> slot in its bucket's run (arrival order).
//   k_order       one thread per place: orders each bucket by bird index (the
//                 canonical stable order), writes the positions in that order
//                 (the view) and the deciding-bird records; in one step of
//                 MOVE_EVERY also moves the birds' state into the other of the
//                 flock's two state buffers in that order.
//   k_decide      eight lanes per deciding bird, one CTA of 24, 28 or 32 warps per
//                 SM: the rows of the bird's 2R neighbourhood are listed as ranges
//                 and swept, hits are compacted over the group and finished
//                 together, and a reduce-scatter of shuffles sums them
//                 (k_decide_sets: grid-reporting steps).
//   k_integrate   banked flight, streaming float4 over the state's slots; its
//                 last block advances the flock clocks, makes a moved state's
//                 buffer current and resets the step counters.
//                 In runs of steps it counts the next step's grid as well.
//
// Exactness: the file is compiled with -fmad=false, and the expressions that
// decide set membership use explicit round-to-nearest intrinsics, so cell
// keys, the sorted order and all four neighbour sets equal the CPU oracle's
// bit for bit. Sums run in lane order instead of bird order, so forces agree
// to rounding (about 1e-7 relative), not bit for bit.
#include <cuda.h>
#include <cuda_runtime.h>
#include <sys/mman.h>
#include <unistd.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>

#include "flock_engine.h"
#include "flock_params.h"
#include "k_decide.cuh"
#include "k_decide_sets.cuh"
#include "k_decide_staged.cuh"
#include "k_fp64.cuh"
#include "k_grid.cuh"
#include "k_integrate.cuh"
#include "k_small.cuh"

namespace flk {

#define FLK_CUDA(call)                                                                                    \
    do {                                                                                                  \
        cudaError_t e_ = (call);                                                                          \
        if (e_ != cudaSuccess) {                                                                          \
            throw Error{-3, std::string(#call) + ": " + cudaGetErrorString(e_)};                          \
        }                                                                                                 \
    } while (0)

const char* device_error_text(uint32_t word) {
    switch (word) {
        case DEV_OK: return "no device error";
        case DEV_SCAN_TIMEOUT: return "a scan look-back wait gave up (error word 1)";
        case DEV_BAD_RANGE: return "a bucket range or slot fell outside its array and was skipped (error word 2)";
        case DEV_STAGE_TIMEOUT: return "a staged decide's bulk copies did not land in time (error word 3)";
        default: return "unknown device error word";
    }
}

uint32_t buckets_for(uint32_t n) {
    uint64_t want = 1;
    while (want < (uint64_t)n * 2) want <<= 1;
    return (uint32_t)std::min<uint64_t>(std::max<uint64_t>(want, 1u << 16), 1u << 22);
}

// ---------------------------------------------------------------------------
// host engine
// ---------------------------------------------------------------------------
// Device memory cache shared by every engine of the process, per device.
// cudaMalloc of the large arrays and cudaFree (which synchronises the whole
// device) cost more than a short run of steps, so an engine's blocks go back
// to the cache when it releases them (after its streams have finished with
// them) and the next engine that asks for a block of the same rounded size
// on that device takes it. At most CACHE_CAP bytes stay cached per device;
// beyond that, blocks are freed.
namespace {
constexpr int CACHE_DEVICES = 64;
constexpr size_t CACHE_CAP = 16ull << 30;
struct DevCache {
    std::mutex mu;
    std::multimap<size_t, void*> free_blocks;  // rounded size -> block
    std::map<void*, size_t> sizes;             // every block handed out: its rounded size
    size_t cached = 0;
};
DevCache g_cache[CACHE_DEVICES];

size_t round_bytes(size_t b) {
    const size_t g = b <= (1u << 20) ? 4096 : (2u << 20);
    return (b + g - 1) / g * g;
}

void* cache_alloc(int dev, size_t bytes) {
    const size_t rb = round_bytes(std::max<size_t>(bytes, 1));
    DevCache& c = g_cache[dev % CACHE_DEVICES];
    {
        std::lock_guard<std::mutex> lk(c.mu);
        auto it = c.free_blocks.find(rb);
        if (it != c.free_blocks.end()) {
            void* p = it->second;
            c.free_blocks.erase(it);
            c.cached -= rb;
            return p;
        }
    }
    void* p = nullptr;
    cudaError_t e = cudaMalloc(&p, rb);
    if (e == cudaErrorMemoryAllocation) {
        (void)cudaGetLastError();
        // give the cached blocks back and try once more
        std::lock_guard<std::mutex> lk(c.mu);
        for (auto& kv : c.free_blocks) {
            cudaFree(kv.second);
            c.sizes.erase(kv.second);
        }
        c.free_blocks.clear();
        c.cached = 0;
        e = cudaMalloc(&p, rb);
    }
    if (e != cudaSuccess) throw Error{-3, std::string("cudaMalloc: ") + cudaGetErrorString(e)};
    std::lock_guard<std::mutex> lk(c.mu);
    c.sizes[p] = rb;
    return p;
}

// The caller guarantees that no work in flight uses p.
void cache_free(int dev, void* p) {
    if (!p) return;
    DevCache& c = g_cache[dev % CACHE_DEVICES];
    std::lock_guard<std::mutex> lk(c.mu);
    auto it = c.sizes.find(p);
    if (it == c.sizes.end()) return;  // never for a block from cache_alloc
    const size_t rb = it->second;
    if (c.cached + rb > CACHE_CAP) {
        cudaFree(p);
        c.sizes.erase(it);
        return;
    }
    c.free_blocks.emplace(rb, p);
    c.cached += rb;
}

// Streams of released engines, a few per device (creating and destroying a pair
// costs as much as a short run). A stream is returned idle.
constexpr size_t STREAM_CAP = 32;
struct StreamCache {
    std::mutex mu;
    std::vector<cudaStream_t> free_streams;
};
StreamCache g_streams[CACHE_DEVICES];

cudaStream_t stream_get(int dev) {
    StreamCache& c = g_streams[dev % CACHE_DEVICES];
    {
        std::lock_guard<std::mutex> lk(c.mu);
        if (!c.free_streams.empty()) {
            cudaStream_t s = c.free_streams.back();
            c.free_streams.pop_back();
            return s;
        }
    }
    cudaStream_t s = nullptr;
    FLK_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
    return s;
}
void stream_put(int dev, cudaStream_t s) {
    if (!s) return;
    StreamCache& c = g_streams[dev % CACHE_DEVICES];
    std::lock_guard<std::mutex> lk(c.mu);
    if (c.free_streams.size() < STREAM_CAP) c.free_streams.push_back(s);
    else cudaStreamDestroy(s);
}

// Page-locked host blocks (host_alloc): engines' control blocks and result
// arrays. They are private anonymous memory, page-locked afterwards: memory from
// cudaHostAlloc is one mapping that a forked child shares with its parent, so a
// child would see its array change as the parent's next result takes the block
// (both kinds copy at the link's rate: 1M birds read in 336 us, opened in 315).
// Mapping and locking cost about a millisecond per 25 MB, so released blocks
// wait here for the next of their size, at most HOST_CAP bytes of them. Result
// arrays that callers hold are page-locked up to RESULT_CAP bytes in all: a program
// that keeps every frame must not lock the host's memory away.
constexpr size_t HOST_CAP = 2ull << 30, RESULT_CAP = 2ull << 30;
struct HostCache {
    struct Block {
        size_t bytes;
        bool result;  // counted in `results`
    };
    std::mutex mu;
    std::multimap<size_t, void*> free_blocks;
    std::map<void*, Block> blocks;  // every block there is
    size_t cached = 0, results = 0;
};
HostCache g_host;

// Per device, set up once for the process: the radius factor table
// (params.rs:61-65 evaluated with the host libm, 65,536 powf calls) and the
// streaming kernels' resident CTAs per SM.
struct DevStatic {
    std::once_flag once;
    float* radius_table = nullptr;
    int fit[10] = {};
    int small_clusters[SMALL_SIZES] = {};  // k_small clusters of SMALL_CTAS >> k CTAs resident at once
};
DevStatic g_static[CACHE_DEVICES];

// Launch of k_small for `flocks` flocks of at most nmax birds, `ctas` CTAs each
// (*at: the cluster).
cudaLaunchConfig_t small_config(uint32_t flocks, uint32_t ctas, uint32_t nmax, cudaLaunchAttribute* at) {
    at->id = cudaLaunchAttributeClusterDimension;
    at->val.clusterDim.x = ctas;
    at->val.clusterDim.y = at->val.clusterDim.z = 1;
    cudaLaunchConfig_t c{};
    c.gridDim = dim3(flocks * ctas);
    c.blockDim = dim3(SMALL_THREADS);
    c.dynamicSmemBytes = small_smem_bytes(nmax);
    c.attrs = at;
    c.numAttrs = 1;
    return c;
}
}  // namespace

static thread_local uint32_t t_fail_locks = 0;  // test hook: host_alloc calls of this thread that still fail
void fail_locks(uint32_t count) { t_fail_locks = count; }

// A page-locked block of at least `bytes`, or null where the host gives none or
// (result) callers hold RESULT_CAP bytes of results. Sizes are rounded up to a
// quarter of their power of two (a page at least).
void* host_alloc(size_t bytes, bool result) {
    if (t_fail_locks) return --t_fail_locks, nullptr;
    size_t unit = (size_t)sysconf(_SC_PAGESIZE);
    while (unit * 8 < bytes) unit *= 2;
    const size_t rb = std::max<size_t>(unit, (bytes + unit - 1) / unit * unit);
    {
        std::lock_guard<std::mutex> lk(g_host.mu);
        if (result && g_host.results + rb > RESULT_CAP) return nullptr;
        if (result) g_host.results += rb;
        auto it = g_host.free_blocks.find(rb);
        if (it != g_host.free_blocks.end()) {
            void* p = it->second;
            g_host.free_blocks.erase(it);
            g_host.cached -= rb;
            g_host.blocks[p].result = result;
            return p;
        }
    }
    void* p = mmap(nullptr, rb, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS | MAP_POPULATE, -1, 0);
    if (p != MAP_FAILED && cudaHostRegister(p, rb, cudaHostRegisterPortable | cudaHostRegisterMapped) != cudaSuccess) {
        (void)cudaGetLastError();
        munmap(p, rb);
        p = MAP_FAILED;
    }
    std::lock_guard<std::mutex> lk(g_host.mu);
    if (p == MAP_FAILED) {
        if (result) g_host.results -= rb;
        return nullptr;
    }
    g_host.blocks[p] = {rb, result};
    return p;
}

// Gives a block of host_alloc back (no copy in flight may use it). False where p is
// none.
bool host_free(void* p) {
    if (!p) return false;
    std::lock_guard<std::mutex> lk(g_host.mu);
    auto it = g_host.blocks.find(p);
    if (it == g_host.blocks.end()) return false;
    const size_t rb = it->second.bytes;
    if (it->second.result) g_host.results -= rb;
    it->second.result = false;
    if (g_host.cached + rb > HOST_CAP) {
        if (cudaHostUnregister(p) != cudaSuccess) (void)cudaGetLastError();
        munmap(p, rb);
        g_host.blocks.erase(it);
        return true;
    }
    g_host.free_blocks.emplace(rb, p);
    g_host.cached += rb;
    return true;
}

// An engine's control blocks, out and in: page-locked, or ordinary memory where the host locks
// no more (its copies then return when they are done).
static uint8_t* control_alloc(size_t bytes) {
    void* p = host_alloc(bytes);
    if (!p && !(p = std::malloc(bytes))) throw Error{-3, "host allocation failed"};
    return static_cast<uint8_t*>(p);
}
static void control_free(uint8_t*& p) {
    if (!host_free(p)) std::free(p);
    p = nullptr;
}

template <class T>
T* Engine::dalloc(size_t n, size_t* acct) {
    if (n == 0) n = 1;
    void* p = cache_alloc(device_, n * sizeof(T));
    *acct += n * sizeof(T);
    return static_cast<T*>(p);
}
template <class T>
void Engine::dfree(T*& p) {
    if (!p) return;
    // the engine's queued work may still use the block: let it finish first
    if (!idle_) {
        cudaStreamSynchronize(stream_);
        cudaStreamSynchronize(copy_);
    }
    cache_free(device_, p);
    p = nullptr;
}

// What CUDA knows of the memory at p: nothing of ordinary host memory (type 0).
namespace {
struct Known {
    unsigned int type = 0, managed = 0;
    unsigned long long at = 0, start = 0;  // device address; start and size of its range
    size_t size = 0;
};
Known known(const void* p) {
    using Query = CUresult (*)(unsigned int, CUpointer_attribute*, void**, CUdeviceptr);
    static const Query query = [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult found;
        if (cudaGetDriverEntryPointByVersion("cuPointerGetAttributes", &f, 12000, cudaEnableDefault, &found) !=
                cudaSuccess || found != cudaDriverEntryPointSuccess) {
            (void)cudaGetLastError();
            f = nullptr;
        }
        return reinterpret_cast<Query>(f);
    }();
    Known k;
    CUpointer_attribute what[] = {CU_POINTER_ATTRIBUTE_MEMORY_TYPE, CU_POINTER_ATTRIBUTE_IS_MANAGED,
                                  CU_POINTER_ATTRIBUTE_DEVICE_POINTER, CU_POINTER_ATTRIBUTE_RANGE_START_ADDR,
                                  CU_POINTER_ATTRIBUTE_RANGE_SIZE};
    void* to[] = {&k.type, &k.managed, &k.at, &k.start, &k.size};
    if (!query || query(5, what, to, (CUdeviceptr)(uintptr_t)p) != CUDA_SUCCESS) {
        k = Known{};
        k.type = ~0u;  // not known to be ordinary either
    }
    return k;
}
}  // namespace

// The device address of host memory [p, p + bytes) that lies in one page-locked
// range, or null: where it is not page-locked, only part of it is (two
// registrations may lie within it and pages between them that a kernel must not
// touch; device addresses equal host addresses, so the ends alone do not tell),
// or the kernels' 4-byte words would not be aligned (a float32 view at an odd byte
// offset: the copy engine takes any address, a load or store does not).
static void* mapped(const Known& k, const void* p, size_t bytes) {
    if (reinterpret_cast<uintptr_t>(p) % sizeof(float)) return nullptr;
    if (k.type != CU_MEMORYTYPE_HOST || k.managed || !k.at || k.at < k.start) return nullptr;
    const size_t before = (size_t)(k.at - k.start);
    return before < k.size && bytes <= k.size - before ? reinterpret_cast<void*>((uintptr_t)k.at) : nullptr;
}
void* mapped(const void* p, size_t bytes) { return mapped(known(p), p, bytes); }

Engine::Engine(int device) {
    if (device < 0) FLK_CUDA(cudaGetDevice(&device));
    device_ = device;
    FLK_CUDA(cudaSetDevice(device_));
    FLK_CUDA(cudaDeviceGetAttribute(&num_sms_, cudaDevAttrMultiProcessorCount, device_));
    stream_ = stream_get(device_);
    copy_ = stream_get(device_);
    ensure_block(16);
    DevStatic& ds = g_static[device_ % CACHE_DEVICES];
    std::call_once(ds.once, [&] {
        std::vector<float> tab(RADIUS_TABLE);
        for (int n = 0; n < RADIUS_TABLE; ++n) {
            const float nn = (float)(n > 1 ? n : 1);
            tab[n] = powf(N_C / nn, RADIUS_EXP);
        }
        FLK_CUDA(cudaMalloc(&ds.radius_table, RADIUS_TABLE * sizeof(float)));  // held for the process
        FLK_CUDA(cudaMemcpy(ds.radius_table, tab.data(), tab.size() * 4, cudaMemcpyHostToDevice));
        auto fit = [](auto kernel) {
            int n = 0;
            FLK_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, 256, 0));
            return std::max(1, n);
        };
        const int f[10] = {fit(k_hash_count<false>), fit(k_hash_count<true>),  fit(k_scatter), fit(k_order<false>),
                          fit(k_order<true>),       fit(k_integrate<false>), fit(k_integrate<true>),
                          fit(k_decide_f64),        fit(k_integrate_f64),    fit(k_compare_f64)};
        std::copy(f, f + 10, ds.fit);
        FLK_CUDA(cudaFuncSetAttribute(k_small, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)small_smem_bytes(SMALL_CLUSTER)));
        FLK_CUDA(cudaFuncSetAttribute(k_small, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
        for (int k = 0; k < SMALL_SIZES; ++k) {
            const uint32_t ctas = SMALL_CTAS >> k;
            cudaLaunchAttribute at{};
            cudaLaunchConfig_t c = small_config(1, ctas, std::min(SMALL_CLUSTER, ctas * SMALL_THREADS), &at);
            if (cudaOccupancyMaxActiveClusters(&ds.small_clusters[k], k_small, &c) != cudaSuccess) {
                (void)cudaGetLastError();
                ds.small_clusters[k] = 0;  // no such cluster here: another size or the separate kernels run
            }
        }
    });
    if (!ds.radius_table) throw Error{-3, "radius table set-up failed on this device"};
    radius_table_ = ds.radius_table;
    set_shape(shape_);  // decide's shared memory may exceed the default 48 KB per CTA
}

Engine::~Engine() {
    cudaSetDevice(device_);
    if (stream_) cudaStreamSynchronize(stream_);
    if (copy_) cudaStreamSynchronize(copy_);
    idle_ = true;  // nothing is in flight: the blocks below go back without another wait
    destroy_graphs();
    dfree(ar_.A); dfree(ar_.B); dfree(ar_.C); dfree(ar_.D); dfree(ar_.id); dfree(ar_.next);
    dfree(key_); dfree(arrival_); dfree(tmp_); dfree(due_);
    dfree(view_); dfree(counts_); dfree(offsets_); dfree(tile_end_); dfree(even_);
    dfree(status_); dfree(sets_);
    dfree(block_); dfree(staging_); dfree(inv_);
    control_free(h_up_);
    host_free(h_bounce_);
    dfree(dec64_); dfree(out64_); dfree(active_); dfree(err64_);
    stream_put(device_, copy_);
    stream_put(device_, stream_);
}

// Marks the captured graphs as out of date (sizes, pointers or launch shapes
// changed); the next ensure_graph recaptures and updates them in place.
void Engine::free_graphs() {
    chunk_graph_.stale = step_graph_.stale = true;
    same_runs_ = 0;
}

void Engine::destroy_graphs() {
    for (StepGraph* g : {&chunk_graph_, &step_graph_}) {
        if (g->exec) cudaGraphExecDestroy(g->exec);
        *g = StepGraph{};
    }
}

size_t Engine::bytes_for(uint32_t n) {
    // state 2 x 72 B (two buffers) + scratch (key, arrival 4 B each; tmp 8 B;
    // due record 48 B; view 16 B) + buckets (histogram, offsets 4 B each; one and
    // a half to three buckets per bird; the tiles' few bytes per 4,096 of them are
    // within the allocations' rounding)
    const size_t b = production_buckets(n);
    return (size_t)n * (144 + 80) + b * 8 + (b / SCAN_TILE) * 4 + 256;
}

// Steps from one that moves the state into cell order to the next. Measured per
// step at 1M / 16.7M birds: every step 130 / 1,851 us, one in 4 130 / 1,774, in 8
// 124 / 1,755, in 16 123 / 1,738, in 64 the same.
static constexpr uint32_t MOVE_EVERY = 16;

// Flocks of at most this many birds are packed by slot: 2,000 birds read in 14.9
// against 17.4 us through the inverse order, 16,000 in 24.6 against 22.7.
static constexpr uint32_t PACK_DIRECT = 8192;
// Into a staging buffer, whose lines the L2 cache assembles, by slot up to this
// size: 100,000 birds 50.7 against 61 us.
static constexpr uint32_t PACK_STAGED = 131072;

// Results of at most this many bytes for ordinary memory go by way of a page-locked
// block and the CPU. The driver's own copy of them to such memory costs a read 18 or
// 28 us, by process (1 bird 28 -> 16.5, 500 28 -> 18, 2,000 28 -> 22.6); a larger one
// 20 (4,000 birds; 28 by way of the block).
static constexpr size_t BOUNCE = 128 << 10;

// staged positions a k_decide_staged CTA holds
static constexpr uint32_t STAGE_CAP = 4096;

static constexpr size_t decide_bytes(int threads) { return (size_t)(threads / 32) * sizeof(WarpSmem); }

// A caller's reservation (decide_extra_smem) is accepted against these sizes of a
// warp's and a staged CTA's memory, those of the first kernels that took one, so
// that what a caller may reserve does not change with decide's own use. A launch
// that would exceed the CTA's limit together with its reservation asks for the limit:
// no kernel touches the reserved part, and such a CTA has its SM to itself anyway.
static constexpr size_t RESERVE_WARP = 1568, RESERVE_STAGED_WARP = 1344, RESERVE_STAGED = 73920;

size_t Engine::decide_smem(bool sets) const {
    if (sets) return 0;
    const int w = shape_.decide_threads / 32;
    const size_t own = shape_.decide_kind == 1 ? staged_smem_bytes(w, STAGE_CAP) : (size_t)w * sizeof(WarpSmem);
    return std::max(own, std::min(own + shape_.decide_extra_smem, smem_optin_));
}

// k_decide with `threads` picked by the engine (pick_decide) or the caller's (0).
static auto decide_kernel(int threads) {
    return threads == DECIDE_FEW ? k_decide<DECIDE_FEW> : threads == DECIDE_SOME ? k_decide<DECIDE_SOME>
                                                                                 : k_decide<DECIDE_MANY>;
}

void Engine::decide_occupancy(int* blocks_per_sm, int* threads, size_t* smem_bytes) const {
    std::vector<uint32_t> sizes;
    for (int id : flock_ids()) sizes.push_back(flock_size(id));
    const int picked = pick_decide(sizes);
    const size_t smem = picked ? decide_bytes(picked) : decide_smem(false);
    const int t = picked ? picked : shape_.decide_threads;
    int n = 0;
    if (shape_.decide_kind == 1)
        FLK_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_decide_staged, t, smem));
    else
        FLK_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, decide_kernel(picked), t, smem));
    *blocks_per_sm = n;
    *threads = t;
    *smem_bytes = smem;
}

void Engine::set_shape(const LaunchShape& s) {
    int optin = 0;
    FLK_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device_));
    const size_t w = (size_t)(s.decide_threads / 32);
    if (s.decide_kind != 0 && s.decide_kind != 1) throw Error{-1, "decide kind must be 0 (direct) or 1 (staged)"};
    const size_t need = std::max(w * RESERVE_WARP,
                                 s.decide_kind == 1 ? w * RESERVE_STAGED_WARP + RESERVE_STAGED : (size_t)0) +
                        s.decide_extra_smem;
    if (need > (size_t)optin)
        throw Error{-1, "decide would need " + std::to_string(need) + " B of shared memory per CTA, above the " +
                            std::to_string(optin) + " B a CTA may have"};
    if (!(s.cell >= 2.0f && s.cell <= 16.0f)) throw Error{-1, "production cell edge must lie in [2, 16] m"};
    shape_ = s;
    smem_optin_ = (size_t)optin;
    decide_threads_ = pick_decide();
    // decide's dynamic shared memory grows with its CTA size; allow past 48 KB
    auto allow = [](auto kernel, size_t bytes) {
        FLK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
    };
    allow(k_decide<DECIDE_MANY>, decide_smem(false));
    allow(k_decide<DECIDE_SOME>, decide_bytes(DECIDE_SOME));
    allow(k_decide<DECIDE_FEW>, decide_bytes(DECIDE_FEW));
    if (s.decide_kind == 1)
        FLK_CUDA(cudaFuncSetAttribute(k_decide_staged, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)decide_smem(false)));
    // the streaming kernels' resident CTAs per SM, queried once per device
    const int* f = g_static[device_ % CACHE_DEVICES].fit;
    fit_.hash[0] = f[0];
    fit_.hash[1] = f[1];
    fit_.scatter = f[2];
    fit_.order[0] = f[3];
    fit_.order[1] = f[4];
    fit_.integrate[0] = f[5];
    fit_.integrate[1] = f[6];
    fit_.decide_f64 = f[7];
    fit_.integrate_f64 = f[8];
    fit_.compare_f64 = f[9];
    free_graphs();
}

void Engine::ensure_arena(uint32_t need) {
    if (need <= cap_) return;
    // both buffers of a field share one allocation indexed by 32-bit slots
    if (need >= (1u << 31)) throw Error{-5, "arena above 2^31 birds"};
    uint32_t ncap = std::max<uint32_t>(need, cap_ ? cap_ + cap_ / 2 : need);
    ncap = std::min<uint32_t>(ncap, (1u << 31) - 1);
    size_t acct = 0;
    Arena na{};
    na.cap = ncap;
    na.A = dalloc<float4>((size_t)ncap * 2, &acct);
    na.B = dalloc<float4>((size_t)ncap * 2, &acct);
    na.C = dalloc<float4>((size_t)ncap * 2, &acct);
    na.D = dalloc<float4>((size_t)ncap * 2, &acct);
    na.id = dalloc<uint32_t>((size_t)ncap * 2, &acct);
    na.next = dalloc<float>((size_t)ncap * 2, &acct);
    if (used_) {
        for (size_t p = 0; p < 2; ++p) {
            const size_t o = p * cap_, n = p * ncap;
            FLK_CUDA(cudaMemcpyAsync(na.A + n, ar_.A + o, (size_t)used_ * 16, cudaMemcpyDeviceToDevice, stream_));
            FLK_CUDA(cudaMemcpyAsync(na.B + n, ar_.B + o, (size_t)used_ * 16, cudaMemcpyDeviceToDevice, stream_));
            FLK_CUDA(cudaMemcpyAsync(na.C + n, ar_.C + o, (size_t)used_ * 16, cudaMemcpyDeviceToDevice, stream_));
            FLK_CUDA(cudaMemcpyAsync(na.D + n, ar_.D + o, (size_t)used_ * 16, cudaMemcpyDeviceToDevice, stream_));
            FLK_CUDA(cudaMemcpyAsync(na.id + n, ar_.id + o, (size_t)used_ * 4, cudaMemcpyDeviceToDevice, stream_));
            FLK_CUDA(cudaMemcpyAsync(na.next + n, ar_.next + o, (size_t)used_ * 4, cudaMemcpyDeviceToDevice, stream_));
        }
        FLK_CUDA(cudaStreamSynchronize(stream_));
    }
    dev_bytes_ -= (size_t)cap_ * 144;
    dfree(ar_.A); dfree(ar_.B); dfree(ar_.C); dfree(ar_.D); dfree(ar_.id); dfree(ar_.next);
    ar_ = na;
    dev_bytes_ += acct;
    cap_ = ncap;
    free_graphs();
}

int Engine::add_flock(uint32_t n, float time, const float* words) {
    FLK_CUDA(cudaSetDevice(device_));
    // first-fit into a hole, else append
    uint32_t sbase = used_;
    bool from_hole = false;
    for (auto& h : free_ranges_) {
        if (h.second >= n) {
            sbase = h.first;
            h.first += n;
            h.second -= n;
            from_hole = true;
            break;
        }
    }
    if (!from_hole) {
        ensure_arena(used_ + n);
        used_ += n;
    }
    free_ranges_.erase(std::remove_if(free_ranges_.begin(), free_ranges_.end(),
                                      [](const std::pair<uint32_t, uint32_t>& h) { return h.second == 0; }),
                       free_ranges_.end());
    if (n) {
        const size_t bytes = (size_t)n * WORDS * 4;
        const Known at = known(words);
        const float* src = static_cast<const float*>(mapped(at, words, bytes));
        if (!src) {  // by way of a staging copy
            ensure_staging(bytes);
            FLK_CUDA(cudaMemcpyAsync(staging_, words, bytes, cudaMemcpyHostToDevice, stream_));
            src = staging_;
        }
        k_unpack<<<pack_blocks(n), PACK_WARPS * 32, 0, stream_>>>(src, n, sbase, ar_);  // buffer 0
        FLK_CUDA(cudaGetLastError());
        // Page-locked words are read after the launches return: the caller may
        // change them, or give their memory back, as soon as this call does.
        // Ordinary memory has been staged by then (200 flocks of 300 birds added in
        // 4.4 ms with a wait each, 2.5 without).
        if (at.type || known(reinterpret_cast<const char*>(words) + bytes - 1).type)
            FLK_CUDA(cudaStreamSynchronize(stream_));
    }
    Slot s;
    s.n = n;
    s.sbase = sbase;
    s.buckets = buckets_for(n);
    s.remaining = 0;
    s.time = time;
    s.live = true;
    int id = -1;
    for (size_t k = 0; k < slots_.size(); ++k)
        if (!slots_[k].live) { id = (int)k; break; }
    if (id < 0) {
        id = (int)slots_.size();
        slots_.push_back(s);
    } else {
        slots_[id] = s;
    }
    return id;
}

bool Engine::has_flock(int id) const { return id >= 0 && id < (int)slots_.size() && slots_[id].live; }
uint32_t Engine::flock_size(int id) const { return has_flock(id) ? slots_[id].n : 0; }
std::vector<int> Engine::flock_ids() const {
    std::vector<int> ids;
    for (size_t k = 0; k < slots_.size(); ++k)
        if (slots_[k].live) ids.push_back((int)k);
    return ids;
}

// The control block and the flock table share one device block and one
// page-locked host block each way, so that a call waits for the GPU once: the
// steps, then one copy of the error word, clocks and countdowns.
void Engine::ensure_block(uint32_t flocks) {
    if (h_up_ && flocks <= table_cap_) return;
    const uint32_t cap = std::max(flocks, table_cap_ * 2);
    const size_t bytes = BLOCK_TABLE + (size_t)cap * sizeof(FlockDesc);
    size_t acct = 0;
    uint8_t* nb = dalloc<uint8_t>(bytes, &acct);
    if (block_) FLK_CUDA(cudaMemcpyAsync(nb, block_, BLOCK_TABLE, cudaMemcpyDeviceToDevice, stream_));
    else FLK_CUDA(cudaMemsetAsync(nb, 0, BLOCK_TABLE, stream_));
    dev_bytes_ += acct - (block_ ? BLOCK_TABLE + (size_t)table_cap_ * sizeof(FlockDesc) : 0);
    dfree(block_);
    block_ = nb;
    ctl_ = reinterpret_cast<StepCtl*>(block_);
    table_d_ = reinterpret_cast<FlockDesc*>(block_ + BLOCK_TABLE);
    table_cap_ = cap;
    FLK_CUDA(cudaStreamSynchronize(stream_));  // the last upload has left its host block
    control_free(h_up_);
    h_up_ = control_alloc(2 * bytes);
    h_down_ = h_up_ + bytes;
    ctl_seen_ = false;
    free_graphs();
}

// Waits for the stream and reads the control block and the table back.
void Engine::fetch() {
    const size_t bytes = BLOCK_TABLE + table_h_.size() * sizeof(FlockDesc);
    FLK_CUDA(cudaMemcpyAsync(h_down_, block_, bytes, cudaMemcpyDeviceToHost, stream_));
    FLK_CUDA(cudaStreamSynchronize(stream_));
    ctl_seen_ = true;
    uploading_ = false;
    if (!device_ahead_) return;
    device_ahead_ = false;
    const FlockDesc* t = reinterpret_cast<const FlockDesc*>(h_down_ + BLOCK_TABLE);
    for (size_t k = 0; k < table_h_.size(); ++k) {
        table_h_[k] = t[k];
        if (table_ids_[k] < 0) continue;  // removed since the table was built
        Slot& s = slots_[table_ids_[k]];
        s.time = t[k].time;
        s.remaining = t[k].remaining;
        s.parity = t[k].parity;
    }
}

void Engine::sync_times() {
    // The device table holds the live clocks and countdowns once steps have
    // run; until then the host copy is authoritative (it may hold step counts
    // set since the last run that the device has not seen yet).
    if (device_ahead_ && !table_h_.empty()) fetch();
}

void Engine::remove_flock(int id) {
    if (!has_flock(id)) throw Error{-4, "unknown flock id"};
    sync_times();
    // the slot id may be reused before the table is rebuilt: detach it
    for (int& t : table_ids_)
        if (t == id) t = -1;
    Slot& s = slots_[id];
    s.live = false;
    if (s.n) {
        free_ranges_.push_back({s.sbase, s.n});
        std::sort(free_ranges_.begin(), free_ranges_.end());
        std::vector<std::pair<uint32_t, uint32_t>> merged;
        for (auto& h : free_ranges_) {
            if (!merged.empty() && merged.back().first + merged.back().second == h.first) merged.back().second += h.second;
            else merged.push_back(h);
        }
        // a hole at the end of the arena returns to the tail
        if (!merged.empty() && merged.back().first + merged.back().second == used_) {
            used_ = merged.back().first;
            merged.pop_back();
        }
        free_ranges_ = merged;
    }
    table_dirty_ = true;
}

float Engine::flock_time(int id) {
    if (!has_flock(id)) throw Error{-4, "unknown flock id"};
    sync_times();
    return slots_[id].time;
}

int Engine::add_flock_async(uint32_t n, float time, const float* words) {
    FLK_CUDA(cudaSetDevice(device_));
    // the state crosses the link on the copy stream while the compute stream
    // keeps running; a stream-ordered staging buffer is unpacked once it lands
    float* stage = nullptr;
    cudaEvent_t landed = nullptr;
    if (n) {
        const size_t bytes = (size_t)n * WORDS * 4;
        FLK_CUDA(cudaMallocAsync((void**)&stage, bytes, copy_));
        FLK_CUDA(cudaMemcpyAsync(stage, words, bytes, cudaMemcpyHostToDevice, copy_));
        FLK_CUDA(cudaEventCreateWithFlags(&landed, cudaEventDisableTiming));
        FLK_CUDA(cudaEventRecord(landed, copy_));
    }
    const int id = add_flock(0, time, nullptr);  // reserves the slot; its state follows
    if (n) {
        Slot& s = slots_[id];
        // move the empty reservation to a real range of n birds
        uint32_t sbase = used_;
        bool from_hole = false;
        for (auto& h : free_ranges_) {
            if (h.second >= n) {
                sbase = h.first;
                h.first += n;
                h.second -= n;
                from_hole = true;
                break;
            }
        }
        if (!from_hole) {
            ensure_arena(used_ + n);
            used_ += n;
        }
        free_ranges_.erase(std::remove_if(free_ranges_.begin(), free_ranges_.end(),
                                          [](const std::pair<uint32_t, uint32_t>& h) { return h.second == 0; }),
                           free_ranges_.end());
        s.n = n;
        s.sbase = sbase;
        s.buckets = buckets_for(n);
        FLK_CUDA(cudaStreamWaitEvent(stream_, landed, 0));
        k_unpack<<<pack_blocks(n), PACK_WARPS * 32, 0, stream_>>>(stage, n, sbase, ar_);  // buffer 0
        FLK_CUDA(cudaGetLastError());
        FLK_CUDA(cudaFreeAsync(stage, stream_));
        FLK_CUDA(cudaEventDestroy(landed));
    }
    return id;
}

void Engine::read_flock_async(int id, float* time, float* words, cudaEvent_t done) {
    if (!has_flock(id)) throw Error{-4, "unknown flock id"};
    FLK_CUDA(cudaSetDevice(device_));
    sync_times();
    const Slot& s = slots_[id];
    if (time) *time = s.time;
    if (s.n) {
        // pack on the compute stream (ordered after the steps that wrote the
        // state), copy out on the copy stream while the next chunk runs
        const size_t bytes = (size_t)s.n * WORDS * 4;
        const bool inverse = s.n > PACK_STAGED;
        float* stage = nullptr;
        FLK_CUDA(cudaMallocAsync((void**)&stage, bytes + (inverse ? (size_t)s.n * 4 : 0), stream_));
        enqueue_pack(stage, s, inverse ? reinterpret_cast<uint32_t*>(stage + (size_t)s.n * WORDS) : nullptr);
        cudaEvent_t packed;
        FLK_CUDA(cudaEventCreateWithFlags(&packed, cudaEventDisableTiming));
        FLK_CUDA(cudaEventRecord(packed, stream_));
        FLK_CUDA(cudaStreamWaitEvent(copy_, packed, 0));
        FLK_CUDA(cudaMemcpyAsync(words, stage, bytes, cudaMemcpyDeviceToHost, copy_));
        FLK_CUDA(cudaFreeAsync(stage, copy_));
        FLK_CUDA(cudaEventDestroy(packed));
    }
    FLK_CUDA(cudaEventRecord(done, copy_));
}

void Engine::read_flock(int id, float* time, float* words) {
    if (!has_flock(id)) throw Error{-4, "unknown flock id"};
    FLK_CUDA(cudaSetDevice(device_));
    sync_times();
    const Slot& s = slots_[id];
    if (time) *time = s.time;
    if (!s.n) return;
    const size_t bytes = (size_t)s.n * WORDS * 4;
    float* dst = static_cast<float*>(mapped(words, bytes));
    const bool bounce = !dst && bytes <= BOUNCE && bounce_block();
    if (bounce) dst = bounce_at_;
    if (!dst) ensure_staging(bytes);
    const bool inverse = s.n > (dst ? PACK_DIRECT : PACK_STAGED);
    if (inverse && s.n > inv_cap_) {
        dev_bytes_ -= (size_t)inv_cap_ * 4;
        dfree(inv_);
        inv_ = dalloc<uint32_t>(s.n, &dev_bytes_);
        inv_cap_ = s.n;
    }
    enqueue_pack(dst ? dst : staging_, s, inverse ? inv_ : nullptr);
    if (!dst) FLK_CUDA(cudaMemcpyAsync(words, staging_, bytes, cudaMemcpyDeviceToHost, stream_));
    FLK_CUDA(cudaStreamSynchronize(stream_));
    if (bounce) std::memcpy(words, h_bounce_, bytes);
}

// The engine's page-locked block for small results; false where the host locks no more.
bool Engine::bounce_block() {
    if (!h_bounce_) {
        h_bounce_ = static_cast<uint8_t*>(host_alloc(BOUNCE));
        bounce_at_ = h_bounce_ ? static_cast<float*>(mapped(h_bounce_, BOUNCE)) : nullptr;
    }
    return bounce_at_ != nullptr;
}

void Engine::ensure_staging(size_t bytes) {
    if (bytes <= staging_cap_) return;
    dev_bytes_ -= staging_cap_;
    dfree(staging_);
    staging_ = dalloc<float>(bytes / 4, &dev_bytes_);
    staging_cap_ = bytes;
}

int Engine::pack_blocks(uint32_t n) const {
    return (int)std::min<uint32_t>((n + PACK_WARPS * 32 - 1) / (PACK_WARPS * 32), (uint32_t)num_sms_ * 8);
}

// The flock's words in bird order to dst (device or mapped host memory); inv:
// room for its inverse order, or null to pack by slot.
void Engine::enqueue_pack(float* dst, const Slot& s, uint32_t* inv) {
    const uint32_t base = (s.parity & 1u) * cap_ + s.sbase;
    if (inv) k_inverse<<<pack_blocks(s.n), 256, 0, stream_>>>(inv, s.n, base, ar_);
    k_pack<<<pack_blocks(s.n), PACK_WARPS * 32, 0, stream_>>>(dst, s.n, base, ar_, inv);
    FLK_CUDA(cudaGetLastError());
}

void Engine::set_remaining(const std::vector<int>& ids, const std::vector<uint32_t>& steps) {
    sync_times();
    for (auto& s : slots_) s.remaining = 0;
    for (size_t k = 0; k < ids.size(); ++k) {
        if (!has_flock(ids[k])) throw Error{-4, "unknown flock id"};
        slots_[ids[k]].remaining = steps[k];
    }
    table_dirty_ = true;
}

void Engine::set_flock_remaining(int id, uint32_t steps) {
    if (!has_flock(id)) throw Error{-4, "unknown flock id"};
    // a flock that is not in the device table has no device-side countdown to
    // read back, so the host need not wait for work in flight
    if (std::find(table_ids_.begin(), table_ids_.end(), id) != table_ids_.end()) sync_times();
    slots_[id].remaining = steps;
    table_dirty_ = true;
}

uint32_t Engine::flock_remaining(int id) {
    if (!has_flock(id)) throw Error{-4, "unknown flock id"};
    sync_times();
    return slots_[id].remaining;
}

std::vector<uint32_t> Engine::remaining_of(const std::vector<int>& ids) {
    sync_times();
    std::vector<uint32_t> out;
    for (int id : ids) {
        if (!has_flock(id)) throw Error{-4, "unknown flock id"};
        out.push_back(slots_[id].remaining);
    }
    return out;
}

double Engine::time_run(uint32_t steps) {
    FLK_CUDA(cudaSetDevice(device_));
    prepare(false);
    cudaEvent_t e0, e1;
    FLK_CUDA(cudaEventCreate(&e0));
    FLK_CUDA(cudaEventCreate(&e1));
    // capture (if needed) before the timed region so the events bracket launches only
    const uint32_t chunk = (uint32_t)std::max(1, shape_.graph_chunk);
    if (!table_h_.empty() && steps >= chunk && !small_ctas()) ensure_graph(chunk_graph_, chunk);
    FLK_CUDA(cudaEventRecord(e0, stream_));
    run(steps);
    FLK_CUDA(cudaEventRecord(e1, stream_));
    FLK_CUDA(cudaEventSynchronize(e1));
    float ms = 0;
    FLK_CUDA(cudaEventElapsedTime(&ms, e0, e1));
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    return ms;
}

__global__ void k_flush(uint4* __restrict__ buf, size_t n16, uint32_t salt) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n16; i += (size_t)gridDim.x * blockDim.x)
        buf[i] = make_uint4(salt, (uint32_t)i, salt, (uint32_t)i);
}

void Engine::time_steps_cold(uint32_t steps, size_t flush_bytes, float* ms_per_step) {
    FLK_CUDA(cudaSetDevice(device_));
    prepare(false);
    if (table_h_.empty() || steps == 0) return;
    uint4* flush = nullptr;
    const size_t n16 = flush_bytes / 16;
    size_t flush_acct = 0;
    if (n16) flush = dalloc<uint4>(n16, &flush_acct);
    // Each timed step is one launch of a single-step graph that runs the step as
    // a multi-step run does: its integrate also counts the next step's grid, so
    // the step has no hash pass of its own. The first step's grid is counted
    // before the timed region and one untimed step after it consumes the grid
    // the last timed step counted: every timed step counts every bird once, and
    // the histogram ends clear.
    cudaGraphExec_t one[2] = {nullptr, nullptr};  // without and with moving the state
    for (int move = 0; move < 2; ++move) {
        cudaGraph_t g;
        FLK_CUDA(cudaStreamBeginCapture(stream_, cudaStreamCaptureModeThreadLocal));
        enqueue_step(false, nullptr, false, false, true, move != 0);
        FLK_CUDA(cudaStreamEndCapture(stream_, &g));
        cudaError_t e = cudaGraphInstantiate(&one[move], g, 0);
        cudaGraphDestroy(g);
        FLK_CUDA(e);
    }
    std::vector<cudaEvent_t> ev(2 * (size_t)steps);
    for (auto& x : ev) FLK_CUDA(cudaEventCreate(&x));
    enqueue_hash();
    for (uint32_t s = 0; s < steps; ++s) {
        if (n16) k_flush<<<num_sms_ * 4, 256, 0, stream_>>>(flush, n16, s);
        FLK_CUDA(cudaEventRecord(ev[2 * s], stream_));
        FLK_CUDA(cudaGraphLaunch(one[s % MOVE_EVERY == 0], stream_));
        FLK_CUDA(cudaEventRecord(ev[2 * s + 1], stream_));
    }
    enqueue_step(false, nullptr, false, false, false);
    FLK_CUDA(cudaGetLastError());
    FLK_CUDA(cudaStreamSynchronize(stream_));
    for (uint32_t s = 0; s < steps; ++s) FLK_CUDA(cudaEventElapsedTime(&ms_per_step[s], ev[2 * s], ev[2 * s + 1]));
    for (auto& x : ev) cudaEventDestroy(x);
    for (auto& x : one) cudaGraphExecDestroy(x);
    dfree(flush);
    const uint32_t ran = steps + 1;
    for (size_t k = 0; k < table_h_.size(); ++k) {
        const uint32_t left = table_h_[k].remaining > ran ? table_h_[k].remaining - ran : 0;
        table_h_[k].remaining = left;
        if (table_ids_[k] >= 0) slots_[table_ids_[k]].remaining = left;
    }
    table_dirty_ = true;
}

// Bucket count of a production step (one that reports no keys; any count
// gives the same sets): the power of two at or above 3n/2, at least 2^13 (a
// lattice of 21 x 43 x 43 m at the 4 m cell) and at most 2^27. At the flock's
// density (0.5 birds per m^3, two and a half per occupied bucket) the lattice holds
// four to eight times the flock's volume; a flock that spreads wraps it, at a cost
// of two thirds of a candidate per bucket visited at most.
uint32_t production_buckets(uint32_t n) {
    uint64_t want = 1;
    while (want < (uint64_t)n + n / 2) want <<= 1;
    return (uint32_t)std::min<uint64_t>(std::max<uint64_t>(want, 1u << 13), 1u << 27);
}

void Engine::prepare(bool grid_output) {
    if (table_dirty_ || table_grid_output_ != grid_output) {
        sync_times();
        rebuild_table(grid_output);
    }
}

void Engine::rebuild_table(bool grid_output) {
    table_grid_output_ = grid_output;
    std::vector<FlockDesc> t;
    std::vector<int> ids;
    uint32_t V = 0;
    uint64_t Bt = 0;
    for (size_t k = 0; k < slots_.size(); ++k) {
        const Slot& s = slots_[k];
        if (!s.live || s.remaining == 0) continue;
        FlockDesc d{};
        d.vbase = V;
        d.n = s.n;
        d.sbase = s.sbase;
        d.bbase = (uint32_t)Bt;
        d.buckets = grid_output ? s.buckets : production_buckets(s.n);
        d.remaining = s.remaining;
        d.time = s.time;
        d.parity = s.parity;
        t.push_back(d);
        ids.push_back((int)k);
        V += s.n;
        Bt += d.buckets;
    }
    if (Bt >= (1ull << 32) - SCAN_TILE) throw Error{-5, "too many buckets in one batch"};
    ensure_block((uint32_t)t.size());
    if (uploading_) FLK_CUDA(cudaStreamSynchronize(stream_));  // the host block is still being read
    if (!t.empty()) {
        std::memcpy(h_up_, t.data(), t.size() * sizeof(FlockDesc));
        FLK_CUDA(cudaMemcpyAsync(table_d_, h_up_, t.size() * sizeof(FlockDesc), cudaMemcpyHostToDevice, stream_));
    }
    uploading_ = !t.empty();
    // a captured graph bakes in sizes and pointers, not the table contents
    const bool same_shape = t.size() == table_h_.size() && V == V_ && (uint32_t)Bt == Btot_;
    table_h_ = t;
    table_ids_ = ids;
    V_ = V;
    Btot_ = (uint32_t)Bt;
    decide_threads_ = pick_decide();
    if (!same_shape) free_graphs();
    ensure_scratch();
    table_dirty_ = false;
    device_ahead_ = false;  // the device table now equals the host copy
}

// Threads of decide's CTAs: by how many turns of the chip's warps a step's
// deciding birds (a tenth of the table's, four to a warp, or one in small flocks)
// take. Measured on both sides of the lines (birds: us a step): 200,000: 24 warps
// per SM 35, 32 40; 500,000: 24 62-64, 32 63; 300,000: 28 40.4, 32 44.2; 1M: 28
// 105, 32 110; 8M: 28 727, 32 727; 16.7M: 28 1,525, 32 1,512. A caller's own launch
// shape is used as it is (0).
int Engine::pick_decide() const {
    std::vector<uint32_t> sizes;
    for (const FlockDesc& d : table_h_) sizes.push_back(d.n);
    return pick_decide(sizes);
}
int Engine::pick_decide(const std::vector<uint32_t>& sizes) const {
    const LaunchShape own;
    if (shape_.decide_kind != own.decide_kind || shape_.decide_threads != own.decide_threads ||
        shape_.decide_blocks_per_sm != own.decide_blocks_per_sm || shape_.decide_extra_smem != own.decide_extra_smem)
        return 0;
    uint64_t birds = 0;  // four per warp
    for (uint32_t n : sizes) birds += n < SMALL_FLOCK ? (uint64_t)n * DECIDE_GROUPS : n;
    const auto turn = [&](int threads) { return (uint64_t)num_sms_ * (threads / 32) * DECIDE_GROUPS * 10; };
    return birds <= 2 * turn(DECIDE_FEW) ? DECIDE_FEW : birds <= 50 * turn(DECIDE_SOME) ? DECIDE_SOME : DECIDE_MANY;
}

void Engine::ensure_scratch() {
    if (V_ > scratch_V_ || !key_) {
        const uint32_t nv = std::max<uint32_t>(V_, scratch_V_ + scratch_V_ / 2);
        dev_bytes_ -= (size_t)scratch_V_ * 80;
        if (sets_) dev_bytes_ -= (size_t)scratch_V_ * 32;
        dfree(key_); dfree(arrival_); dfree(tmp_); dfree(due_); dfree(view_); dfree(sets_);
        key_ = dalloc<uint32_t>(nv, &dev_bytes_);
        arrival_ = dalloc<uint32_t>(nv, &dev_bytes_);
        tmp_ = dalloc<uint2>(nv, &dev_bytes_);
        due_ = dalloc<DueRec>(nv, &dev_bytes_);
        size_t past_end = 0;  // (read by decide's lanes without a candidate; not counted)
        view_ = dalloc<float4>((size_t)nv + DECIDE_LANES, &past_end);
        dev_bytes_ += (size_t)nv * sizeof(float4);
        scratch_V_ = nv;
        free_graphs();
    }
    if (Btot_ > scratch_B_) {
        const uint32_t nb = Btot_;
        dev_bytes_ -= (size_t)scratch_B_ * 8 + (scratch_B_ / SCAN_TILE) * 13;
        dfree(counts_); dfree(offsets_); dfree(tile_end_); dfree(even_); dfree(status_);
        counts_ = dalloc<uint32_t>(nb, &dev_bytes_);
        offsets_ = dalloc<uint32_t>(nb, &dev_bytes_);
        tile_end_ = dalloc<uint32_t>(nb / SCAN_TILE, &dev_bytes_);
        even_ = dalloc<uint8_t>(nb / SCAN_TILE, &dev_bytes_);
        status_ = dalloc<unsigned long long>(nb / SCAN_TILE, &dev_bytes_);
        FLK_CUDA(cudaMemsetAsync(counts_, 0, (size_t)nb * 4, stream_));
        FLK_CUDA(cudaMemsetAsync(even_, 0, nb / SCAN_TILE, stream_));
        FLK_CUDA(cudaMemsetAsync(status_, 0, (size_t)(nb / SCAN_TILE) * 8, stream_));
        scratch_B_ = nb;
        free_graphs();
    }
}

// Grid of a persistent pass: `per_sm` CTAs per SM, but no more CTAs than
// there are work items (`items` split into `per_cta` per CTA).
static int pgrid(int sms, int per_sm, uint64_t items, uint64_t per_cta) {
    const uint64_t need = (items + per_cta - 1) / per_cta;
    return (int)std::max<uint64_t>(1, std::min<uint64_t>((uint64_t)sms * per_sm, need));
}

void Engine::enqueue_step(bool sets, cudaEvent_t* ev, bool f64, bool hash, bool fuse_next, bool move) {
    device_ahead_ = true;
    const int nfl = (int)table_h_.size();
    // grid of a bird-parallel pass whose kernel fits `f` CTAs per SM
    auto sgrid = [&](int f) { return pgrid(num_sms_, std::min(shape_.stream_blocks_per_sm, f), V_, 256); };
    const uint32_t ntiles = Btot_ / SCAN_TILE;
    const float cell = shape_.cell, inv_cell = 1.0f / shape_.cell;  // production cells
    if (ev) FLK_CUDA(cudaEventRecord(ev[0], stream_));
    if (sets) clear_counted();
    if (sets)  // a grid-reporting step: the reference's cell hash
        k_hash_count<false><<<sgrid(fit_.hash[0]), 256, 0, stream_>>>(table_d_, nfl, V_, ar_, key_, arrival_, counts_,
                                                                      INV_CELL);
    else if (hash)
        enqueue_hash();
    if (ev) FLK_CUDA(cudaEventRecord(ev[1], stream_));
    if (sets)
        k_scan<<<ntiles, SCAN_THREADS, 0, stream_>>>(table_d_, nfl, counts_, offsets_, tile_end_, even_, ntiles,
                                                     status_, ctl_);
    else
        k_place<<<ntiles, SCAN_THREADS, 0, stream_>>>(table_d_, nfl, counts_, offsets_, tile_end_, even_);
    if (ev) FLK_CUDA(cudaEventRecord(ev[2], stream_));
    k_scatter<<<sgrid(fit_.scatter), 256, 0, stream_>>>(table_d_, nfl, V_, ar_, key_, arrival_, offsets_, tmp_, ctl_);
    if (move)
        k_order<true><<<sgrid(fit_.order[1]), 256, 0, stream_>>>(table_d_, nfl, V_, ctl_, tmp_, ar_, view_, due_,
                                                                           wide_radius(cell));
    else
        k_order<false><<<sgrid(fit_.order[0]), 256, 0, stream_>>>(table_d_, nfl, V_, ctl_, tmp_, ar_, view_, due_,
                                                                           wide_radius(cell));
    if (f64) {  // FP64 evaluation from the input state, before the f32 passes change it
        k_decide_f64<<<pgrid(num_sms_, fit_.decide_f64, V_, 8), 256, 0, stream_>>>(table_d_, V_, ctl_, due_, offsets_, tile_end_, ar_,
                                                                                   dec64_, err64_, cell, inv_cell);
        k_integrate_f64<<<sgrid(fit_.integrate_f64), 256, 0, stream_>>>(table_d_, nfl, V_, ar_, dec64_, out64_);
    }
    if (ev) FLK_CUDA(cudaEventRecord(ev[3], stream_));
    const int dthreads = decide_threads_ ? decide_threads_ : shape_.decide_threads;
    const int dblocks = pgrid(num_sms_, shape_.decide_blocks_per_sm, V_, (uint64_t)DECIDE_GROUPS * (dthreads / 32));
    if (sets) {
        k_decide_sets<<<pgrid(num_sms_, 4, V_, 8), 256, 0, stream_>>>(table_d_, V_, ctl_, due_, offsets_, tile_end_, ar_,
                                                                      radius_table_, sets_);
    } else if (shape_.decide_kind == 1) {
        k_decide_staged<<<dblocks, dthreads, decide_smem(false), stream_>>>(
            table_d_, V_, ctl_, due_, offsets_, tile_end_, ar_, view_, radius_table_, cell, inv_cell, STAGE_CAP);
    } else {
        decide_kernel(decide_threads_)<<<dblocks, dthreads, decide_threads_ ? decide_bytes(dthreads) : decide_smem(false), stream_>>>(
            table_d_, V_, ctl_, due_, offsets_, tile_end_, ar_, view_, radius_table_, cell, inv_cell);
    }
    if (ev) FLK_CUDA(cudaEventRecord(ev[4], stream_));
    if (fuse_next && !sets)
        k_integrate<true><<<sgrid(fit_.integrate[1]), 256, 0, stream_>>>(table_d_, nfl, V_, ar_, counts_, key_,
                                                                         arrival_, ctl_, inv_cell, move);
    else
        k_integrate<false><<<sgrid(fit_.integrate[0]), 256, 0, stream_>>>(table_d_, nfl, V_, ar_, counts_, key_,
                                                                          arrival_, ctl_, inv_cell, move);
    counted_ = fuse_next && !sets;
    if (f64) k_compare_f64<<<sgrid(fit_.compare_f64), 256, 0, stream_>>>(table_d_, nfl, V_, ar_, active_, out64_, err64_);
    if (ev) FLK_CUDA(cudaEventRecord(ev[5], stream_));
}

// A run that failed between two steps has left the next step's grid counted.
void Engine::clear_counted() {
    if (!counted_) return;
    FLK_CUDA(cudaMemsetAsync(counts_, 0, (size_t)scratch_B_ * 4, stream_));
    counted_ = false;
}

void Engine::enqueue_hash() {
    device_ahead_ = true;
    clear_counted();
    const int grid = pgrid(num_sms_, std::min(shape_.stream_blocks_per_sm, fit_.hash[1]), V_, 256);
    k_hash_count<true><<<grid, 256, 0, stream_>>>(table_d_, (int)table_h_.size(), V_, ar_, key_, arrival_, counts_,
                                                  1.0f / shape_.cell);
    counted_ = true;
}

void Engine::enqueue_steps(uint32_t n) {
    for (uint32_t i = 0; i < n; ++i) enqueue_step(false, nullptr, false, i == 0, i + 1 < n, i % MOVE_EVERY == 0);
}

// CTAs per flock where the table's flocks all run as one cluster each (k_small), or
// 0: the largest cluster of which all the flocks' are on the chip together, if its
// threads are as many as the largest flock's birds. How many clusters fit depends on
// the GPU's own layout (one GB300 holds nine of 16 CTAs, 18 of 8, 36 of 4, 74 of 2;
// another 7, 15, 36, 76), so it is asked for. Measured against the separate kernels
// on the former where each size takes over (us a step): 9 flocks of 1,000 birds (16 CTAs)
// 9.7 / 21.1, of 4,000 20.7 / 26.2; 18 flocks (8) of 1,000 11.6 / 22.6, of 4,000
// 32 / 32; 20 flocks (4) of 2,000 18.8 / 28.3; 37 flocks (2) of 1,000 17.2 / 27.5;
// 150 flocks (1) of 500 15.9 / 33.9. Clusters in a second turn take as long again.
uint32_t Engine::small_ctas(size_t flocks, uint32_t nmax) const {
    if (shape_.decide_kind != 0 || !flocks) return 0;
    for (int k = 0; k < SMALL_SIZES; ++k) {
        const uint32_t ctas = SMALL_CTAS >> k;
        if (nmax <= std::min(SMALL_CLUSTER, ctas * SMALL_THREADS) &&
            (int)flocks <= g_static[device_ % CACHE_DEVICES].small_clusters[k])
            return ctas;
    }
    return 0;
}

uint32_t Engine::small_ctas() const {
    uint32_t nmax = 0;
    for (const FlockDesc& d : table_h_) nmax = std::max(nmax, d.n);
    return small_ctas(table_h_.size(), nmax);
}

uint32_t Engine::small_ctas_of_all() const {
    uint32_t nmax = 0;
    const std::vector<int> ids = flock_ids();
    for (int id : ids) nmax = std::max(nmax, flock_size(id));
    return small_ctas(ids.size(), nmax);
}

// A launch runs at most SMALL_STEPS steps, 0.1 s or so.
void Engine::enqueue_small(uint32_t steps, uint32_t ctas) {
    device_ahead_ = true;
    uint32_t nmax = 1;
    for (const FlockDesc& d : table_h_) nmax = std::max(nmax, d.n);
    cudaLaunchAttribute at{};
    cudaLaunchConfig_t c = small_config((uint32_t)table_h_.size(), ctas, nmax, &at);
    c.stream = stream_;
    for (uint32_t done = 0; done < steps;) {
        const uint32_t part = std::min(steps - done, SMALL_STEPS);
        FLK_CUDA(cudaLaunchKernelEx(&c, k_small, table_d_, part, nmax, ctl_, ar_, (const float*)radius_table_,
                                    shape_.cell, 1.0f / shape_.cell));
        done += part;
    }
}

// Captures `steps` production steps (1: the step alone, its grid counted before
// and counting the next one's) as graph g, unless it is there and current. When
// only sizes, pointers or launch shapes changed since the last capture (a flock
// joined or left, a buffer grew), the new capture has the same nodes, and
// cudaGraphExecUpdate rewrites the executable graph's parameters instead of
// instantiating a new one (launches already in flight keep their old
// parameters). A different length, or an update the runtime refuses,
// instantiates afresh.
// False where the runtime gives no graph: the steps then go launch by launch (a
// capture that fails changes nothing, a counted grid included).
bool Engine::ensure_graph(StepGraph& sg, uint32_t steps) {
    if (sg.exec && sg.steps == steps && !sg.stale) return true;
    const auto failed = [] {
        (void)cudaGetLastError();  // leaves no sticky error
        return false;
    };
    if (fail_captures_) return --fail_captures_, false;
    cudaGraph_t g = nullptr;
    if (cudaStreamBeginCapture(stream_, cudaStreamCaptureModeThreadLocal) != cudaSuccess) return failed();
    const bool counted = counted_;
    counted_ = false;
    if (&sg == &step_graph_) enqueue_step(false, nullptr, false, false, true, false);
    else enqueue_steps(steps);
    counted_ = counted;
    if (cudaStreamEndCapture(stream_, &g) != cudaSuccess) return failed();
    if (sg.exec && sg.steps == steps) {
        cudaGraphExecUpdateResultInfo info;
        if (cudaGraphExecUpdate(sg.exec, g, &info) == cudaSuccess) {
            cudaGraphDestroy(g);
            sg.stale = false;
            ++graph_updates_;
            return true;
        }
        (void)cudaGetLastError();  // the refused update leaves no sticky error
    }
    if (sg.exec) cudaGraphExecDestroy(sg.exec);
    sg = StepGraph{};
    const cudaError_t e = cudaGraphInstantiate(&sg.exec, g, 0);
    cudaGraphDestroy(g);
    if (e != cudaSuccess) {
        sg = StepGraph{};
        return failed();
    }
    sg.steps = steps;
    ++graph_instantiations_;
    return true;
}

void Engine::launch_graph(const StepGraph& sg) {
    if (fail_launch_ && --fail_launch_ == 0) throw Error{-3, "graph launch failed (test hook)"};
    FLK_CUDA(cudaGraphLaunch(sg.exec, stream_));
}

// A kernel launch takes the host about 7 us, a graph launch no more, and a
// mid-size step's five kernels 28 us on the GPU: launched one by one they keep it
// waiting (37,501 birds: 38 us a step against 29 in graphs). A step graph is
// cheap to capture (five nodes), so any run of a few steps goes through it. A
// graph of a whole chunk has no gap between its steps (us a step, step graphs
// against chunk graphs: 8,193 birds 26.0 / 23.7, 37,501 29.6 / 26.3, 100,000
// 31.7 / 27.7, 300,000 45.6 / 42.7, 1M 109 / 105), but each of its launches moves
// the state, not one step in MOVE_EVERY (chunks of one step: 1M 134 / 136, 3M 324 /
// 346; of two: 3M 308 / 310, 16.7M 1,526 / 1,596; of ten: 3M 291 / 289, 16.7M 1,490 /
// 1,491). It is built for runs of ten chunks and, up to a million birds per step of
// a chunk, for the third run of a table that stays the same, a served pool's chunks
// among them (its median latency under a Poisson load 14.8 -> 13.5 ms), while the
// GPU is busy with a chunk. The launches are the captured ones, so the results are
// the same.
void Engine::enqueue_run(uint32_t steps) {
    if (const uint32_t ctas = small_ctas()) {
        enqueue_small(steps, ctas);
        return;
    }
    device_ahead_ = true;
    const uint32_t chunk = (uint32_t)std::max(1, shape_.graph_chunk);
    uint32_t done = 0;
    if (steps >= chunk) {
        const bool ready = chunk_graph_.exec && chunk_graph_.steps == chunk && !chunk_graph_.stale;
        if (ready || steps >= 10 * chunk || (same_runs_ >= 2 && V_ / 1000000u <= chunk)) {
            if (!ready) {
                enqueue_singly(chunk);
                done = chunk;
            }
            if (ensure_graph(chunk_graph_, chunk)) {
                for (; done + chunk <= steps; done += chunk) launch_graph(chunk_graph_);
                since_move_ = (chunk - 1) % MOVE_EVERY + 1;  // a chunk's first step moves the state
                for (int id : table_ids_)
                    if (id >= 0) slots_[id].fresh = false;
            }
        }
        ++same_runs_;
    }
    if (done < steps) enqueue_singly(steps - done);
}

// `n` steps, one launch of the step graph each. The steps that move the state
// (the first one on flocks still in the order they were added in, then one in
// MOVE_EVERY) and the last one, which counts no next grid, go pass by pass.
void Engine::enqueue_singly(uint32_t n) {
    for (int id : table_ids_)
        if (id >= 0 && slots_[id].fresh) since_move_ = MOVE_EVERY;
    bool graphed = n >= 4 || (n >= 2 && step_graph_.exec && !step_graph_.stale);
    for (uint32_t i = 0; i < n; ++i) {
        const bool last = i + 1 == n, move = since_move_ >= MOVE_EVERY;
        if (move) {
            since_move_ = 0;
            for (int id : table_ids_)
                if (id >= 0) slots_[id].fresh = false;
        }
        ++since_move_;
        // (captured while the steps before are running: first pass of a frame of
        // 100,000 birds 265 us, 300 with the capture ahead of them)
        if (graphed && !last && !move) graphed = ensure_graph(step_graph_, 1);
        if (!graphed || last || move) {
            enqueue_step(false, nullptr, false, i == 0, !last, move);
            continue;
        }
        if (i == 0) enqueue_hash();
        launch_graph(step_graph_);
    }
}

void Engine::run(uint32_t steps) {
    FLK_CUDA(cudaSetDevice(device_));
    prepare(false);
    if (table_h_.empty() || steps == 0) return;
    enqueue_run(steps);
    FLK_CUDA(cudaGetLastError());
    // host mirror of the countdown (clocks are read back on demand)
    bool finished = false;
    for (size_t k = 0; k < table_h_.size(); ++k) {
        const uint32_t left = table_h_[k].remaining > steps ? table_h_[k].remaining - steps : 0;
        table_h_[k].remaining = left;
        if (table_ids_[k] >= 0) slots_[table_ids_[k]].remaining = left;
        finished |= left == 0;
    }
    // flocks that reached zero leave the table at the next run (their clocks
    // are read back from the device table before it is rebuilt)
    if (finished) table_dirty_ = true;
}

void Engine::run_timed(uint32_t steps, uint32_t warmup, PassTimes* out) {
    FLK_CUDA(cudaSetDevice(device_));
    prepare(false);
    PassTimes pt{};
    if (table_h_.empty() || steps == 0) {
        if (out) *out = pt;
        return;
    }
    std::vector<cudaEvent_t> ev((size_t)steps * 6);
    for (auto& e : ev) FLK_CUDA(cudaEventCreate(&e));
    for (uint32_t s = 0; s < steps; ++s)
        enqueue_step(false, &ev[(size_t)s * 6], false, true, false, s % MOVE_EVERY == 0);
    FLK_CUDA(cudaGetLastError());
    FLK_CUDA(cudaStreamSynchronize(stream_));
    warmup = std::min(warmup, steps);
    for (uint32_t s = warmup; s < steps; ++s) {
        cudaEvent_t* e = &ev[(size_t)s * 6];
        for (int p = 0; p < 5; ++p) {
            float ms = 0;
            FLK_CUDA(cudaEventElapsedTime(&ms, e[p], e[p + 1]));
            pt.ms[p] += ms;
        }
    }
    pt.timed_steps = (int)(steps - warmup);
    if (pt.timed_steps > 0) {
        for (int p = 0; p < 5; ++p) {
            pt.ms[p] /= pt.timed_steps;
            pt.total_ms += pt.ms[p];
        }
    }
    for (auto& e : ev) cudaEventDestroy(e);
    sync_times();  // clocks and countdowns from the device table
    table_dirty_ = true;
    if (out) *out = pt;
}

void Engine::step_debug(std::vector<GridDebug>* out) {
    FLK_CUDA(cudaSetDevice(device_));
    prepare(true);  // the canonical bucket counts the reported grid is defined with
    if (table_h_.empty()) return;
    if (!sets_) sets_ = dalloc<uint32_t>((size_t)scratch_V_ * 8, &dev_bytes_);
    FLK_CUDA(cudaMemsetAsync(sets_, 0, (size_t)V_ * 8 * 4, stream_));
    const std::vector<FlockDesc> before = table_h_;
    enqueue_step(true);
    FLK_CUDA(cudaGetLastError());
    FLK_CUDA(cudaStreamSynchronize(stream_));
    // a grid the device gave up on is not interpreted
    if (const uint32_t err = check_device_error()) {
        table_dirty_ = true;
        device_ahead_ = true;
        throw Error{-6, std::string("device: ") + device_error_text(err)};
    }
    std::vector<uint32_t> key(V_), offs((size_t)Btot_), sets((size_t)V_ * 8);
    FLK_CUDA(cudaMemcpy(key.data(), key_, (size_t)V_ * 4, cudaMemcpyDeviceToHost));
    FLK_CUDA(cudaMemcpy(offs.data(), offsets_, (size_t)Btot_ * 4, cudaMemcpyDeviceToHost));
    FLK_CUDA(cudaMemcpy(sets.data(), sets_, (size_t)V_ * 8 * 4, cudaMemcpyDeviceToHost));
    // bird index per slot in both buffers: the step read buf[parity] (keys are
    // per old slot) and wrote buf[parity ^ 1] (sorted order, sets per new slot)
    std::vector<uint32_t> ids[2];
    for (int k = 0; k < 2; ++k) {
        ids[k].resize(used_);
        if (used_)
            FLK_CUDA(cudaMemcpy(ids[k].data(), ar_.id + (size_t)k * cap_, (size_t)used_ * 4, cudaMemcpyDeviceToHost));
    }
    out->clear();
    for (const FlockDesc& d : before) {
        const std::vector<uint32_t>& oid = ids[d.parity & 1u];
        const std::vector<uint32_t>& nid = ids[(d.parity & 1u) ^ 1u];
        GridDebug g;
        g.keys.assign(d.n, 0);
        g.sets.assign((size_t)d.n * 8, 0);
        g.sorted.resize(d.n);
        for (uint32_t i = 0; i < d.n; ++i) {
            const uint32_t bo = oid[d.sbase + i], bn = nid[d.sbase + i];
            if (bo >= d.n || bn >= d.n) throw Error{-6, "bird index out of range in step_debug"};
            g.keys[bo] = key[d.vbase + i] - d.bbase;
            g.sorted[i] = bn;  // view index vbase + i holds bird bn
            std::copy(sets.begin() + (size_t)(d.vbase + i) * 8, sets.begin() + (size_t)(d.vbase + i + 1) * 8,
                      g.sets.begin() + (size_t)bn * 8);
        }
        g.offsets.resize((size_t)d.buckets + 1);
        const uint32_t o0 = offs[d.bbase];
        for (uint32_t b = 0; b < d.buckets; ++b) g.offsets[b] = offs[(size_t)d.bbase + b] - o0;
        g.offsets[d.buckets] = d.n;
        if (o0 != d.vbase) throw Error{-6, "grid offsets of a flock do not start at its view base"};
        out->push_back(std::move(g));
    }
    sync_times();  // clocks and countdowns from the device table
    table_dirty_ = true;
}

void Engine::step_f64(std::vector<std::vector<double>>* out, std::vector<std::array<double, 4>>* report) {
    FLK_CUDA(cudaSetDevice(device_));
    prepare(false);  // production buckets: the FP64 passes use the lattice index
    out->clear();
    report->clear();
    if (table_h_.empty()) return;
    if (V_ > f64_V_ || !dec64_) {
        dfree(dec64_);
        dfree(out64_);
        dec64_ = dalloc<double>((size_t)V_ * 8, &dev_bytes_);
        out64_ = dalloc<double>((size_t)V_ * 15, &dev_bytes_);
        f64_V_ = V_;
    }
    const size_t nfl = table_h_.size();
    if (nfl > active_cap_ || !active_) {
        dfree(active_);
        dfree(err64_);
        active_cap_ = (uint32_t)nfl;
        active_ = dalloc<uint8_t>(active_cap_, &dev_bytes_);
        err64_ = dalloc<uint32_t>((size_t)active_cap_ * 4, &dev_bytes_);
    }
    const std::vector<FlockDesc> before = table_h_;
    std::vector<uint8_t> act(nfl);
    for (size_t k = 0; k < nfl; ++k) act[k] = before[k].remaining > 0;
    FLK_CUDA(cudaMemcpyAsync(active_, act.data(), nfl, cudaMemcpyHostToDevice, stream_));
    FLK_CUDA(cudaMemsetAsync(err64_, 0, nfl * 16, stream_));
    enqueue_step(false, nullptr, true);
    FLK_CUDA(cudaGetLastError());
    std::vector<uint32_t> err(nfl * 4);
    FLK_CUDA(cudaMemcpyAsync(err.data(), err64_, nfl * 16, cudaMemcpyDeviceToHost, stream_));
    std::vector<double> o64((size_t)V_ * 15);
    FLK_CUDA(cudaMemcpyAsync(o64.data(), out64_, o64.size() * 8, cudaMemcpyDeviceToHost, stream_));
    std::vector<uint32_t> ids[2];
    for (int k = 0; k < 2; ++k) {
        ids[k].resize(used_);
        if (used_)
            FLK_CUDA(cudaMemcpyAsync(ids[k].data(), ar_.id + (size_t)k * cap_, (size_t)used_ * 4,
                                     cudaMemcpyDeviceToHost, stream_));
    }
    FLK_CUDA(cudaStreamSynchronize(stream_));
    for (size_t f = 0; f < nfl; ++f) {
        const FlockDesc& d = before[f];
        std::vector<double> w;
        std::array<double, 4> r{0.0, 0.0, 0.0, 0.0};
        if (d.remaining) {
            float ep, ev;
            std::memcpy(&ep, &err[4 * f], 4);
            std::memcpy(&ev, &err[4 * f + 1], 4);
            r = {ep, ev, (double)err[4 * f + 2], (double)err[4 * f + 3]};
            // view index vbase + i sits in slot sbase + i of the copy the step wrote
            const std::vector<uint32_t>& nid = ids[(d.parity & 1u) ^ 1u];
            w.resize((size_t)d.n * 15);
            for (uint32_t i = 0; i < d.n; ++i) {
                const uint32_t bird = nid[d.sbase + i];
                if (bird >= d.n) throw Error{-6, "bird index out of range in step_f64"};
                std::memcpy(&w[(size_t)bird * 15], &o64[(size_t)(d.vbase + i) * 15], 15 * 8);
            }
        }
        out->push_back(std::move(w));
        report->push_back(r);
    }
}

void Engine::sync() {
    FLK_CUDA(cudaSetDevice(device_));
    if (device_ahead_) fetch();
    else FLK_CUDA(cudaStreamSynchronize(stream_));
}

uint32_t Engine::check_device_error() {
    FLK_CUDA(cudaSetDevice(device_));
    if (device_ahead_ || !ctl_seen_) fetch();
    StepCtl* c = reinterpret_cast<StepCtl*>(h_down_);
    const uint32_t error = c->error;
    if (error) {
        c->error = 0;
        FLK_CUDA(cudaMemsetAsync(&ctl_->error, 0, 4, stream_));
        FLK_CUDA(cudaStreamSynchronize(stream_));
    }
    return error;
}

void Engine::arm_scan_timeout(uint32_t skip_tile, uint32_t spin_limit) {
    FLK_CUDA(cudaSetDevice(device_));
    const uint32_t v[2] = {skip_tile + 1u, spin_limit};
    FLK_CUDA(cudaMemcpyAsync(&ctl_->scan_skip1, v, sizeof v, cudaMemcpyHostToDevice, stream_));
    FLK_CUDA(cudaStreamSynchronize(stream_));
}

void Engine::counters(unsigned long long* due, unsigned long long* cand, unsigned long long* pairs) {
    FLK_CUDA(cudaSetDevice(device_));
    StepCtl c;
    FLK_CUDA(cudaMemcpyAsync(&c, ctl_, sizeof c, cudaMemcpyDeviceToHost, stream_));
    FLK_CUDA(cudaStreamSynchronize(stream_));
    if (due) *due = c.due_total;
    if (cand) *cand = c.cand_total;
    if (pairs) *pairs = c.pair_total;
}

}  // namespace flk

