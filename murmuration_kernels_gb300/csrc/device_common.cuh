// Device helpers shared by the step's passes: f32 vector arithmetic with
// explicit round-to-nearest operations (no FMA contraction), the reference's
// forward/side/body_up (crates/flock-ref/src/model.rs:15-38), the cell hash
// (cuda/flock.cu:77-83), warp utilities and relaxed loads/stores.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "flock_engine.h"
#include "flock_params.h"

namespace flk {

constexpr uint32_t FULL = 0xFFFFFFFFu;
constexpr int SCAN_THREADS = 256;
constexpr int SCAN_ITEMS = 16;
constexpr uint32_t SCAN_TILE = SCAN_THREADS * SCAN_ITEMS;  // 4096 buckets per tile
constexpr uint32_t SCAN_SPIN_LIMIT = 1u << 22;             // look-back polls before giving up
constexpr uint32_t FLAG_A = 1u, FLAG_P = 2u;
// Flocks below this many birds are decided by a whole warp per bird instead of
// eight lanes: 2,000 birds 23.1 -> 19.9 us a step, 7,000 24.1 -> 21.0; a batch
// of 24 flocks of 1e3 to 2e5 birds pays 3 % for the line at 8,192 and 15 % at
// 32,768, where a flock alone still gained.
constexpr uint32_t SMALL_FLOCK = 8192u;

// ---------------------------------------------------------------------------
// device helpers
// ---------------------------------------------------------------------------
struct f3 {
    float x, y, z;
};
__device__ __forceinline__ f3 mk(float x, float y, float z) { return f3{x, y, z}; }
__device__ __forceinline__ f3 add(f3 a, f3 b) { return mk(__fadd_rn(a.x, b.x), __fadd_rn(a.y, b.y), __fadd_rn(a.z, b.z)); }
__device__ __forceinline__ f3 sub(f3 a, f3 b) { return mk(__fsub_rn(a.x, b.x), __fsub_rn(a.y, b.y), __fsub_rn(a.z, b.z)); }
__device__ __forceinline__ f3 mul(f3 a, float s) { return mk(__fmul_rn(a.x, s), __fmul_rn(a.y, s), __fmul_rn(a.z, s)); }
__device__ __forceinline__ f3 dvs(f3 a, float s) { return mk(__fdiv_rn(a.x, s), __fdiv_rn(a.y, s), __fdiv_rn(a.z, s)); }
__device__ __forceinline__ float dot(f3 a, f3 b) {
    return __fadd_rn(__fadd_rn(__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y)), __fmul_rn(a.z, b.z));
}
// glam Vec3::cross
__device__ __forceinline__ f3 cross(f3 a, f3 b) {
    return mk(__fsub_rn(__fmul_rn(a.y, b.z), __fmul_rn(b.y, a.z)), __fsub_rn(__fmul_rn(a.z, b.x), __fmul_rn(b.z, a.x)),
              __fsub_rn(__fmul_rn(a.x, b.y), __fmul_rn(b.x, a.y)));
}
__device__ __forceinline__ float len(f3 a) { return __fsqrt_rn(dot(a, a)); }
__device__ __forceinline__ f3 normalize(f3 a) { return mul(a, __fdiv_rn(1.0f, len(a))); }
__device__ __forceinline__ f3 normalize_or_zero(f3 a) {
    const float rcp = __fdiv_rn(1.0f, len(a));
    return (isfinite(rcp) && rcp > 0.0f) ? mul(a, rcp) : mk(0.f, 0.f, 0.f);
}
// f32::clamp (NaN passes through)
__device__ __forceinline__ float clampf(float v, float lo, float hi) {
    if (v < lo) v = lo;
    if (v > hi) v = hi;
    return v;
}
// model.rs:15-38
__device__ __forceinline__ f3 forward(f3 v) { return dot(v, v) > 1e-12f ? normalize(v) : mk(1.f, 0.f, 0.f); }
__device__ __forceinline__ f3 side_of(f3 f) {
    const f3 s = cross(f, mk(0.f, 0.f, 1.f));
    return dot(s, s) > 1e-8f ? normalize(s) : mk(1.f, 0.f, 0.f);
}
__device__ __forceinline__ f3 body_up(f3 f, float beta) {
    const f3 side = side_of(f);
    const f3 up0 = cross(side, f);
    return add(mul(up0, cosf(beta)), mul(side, sinf(beta)));
}
__device__ __forceinline__ f3 xyz(float4 v) { return mk(v.x, v.y, v.z); }

// cuda/flock.cu:77-83: cell = floor(p / 4), bucket = spatial hash & mask.
__device__ __forceinline__ int cell1(float x) { return (int)floorf(__fmul_rn(x, INV_CELL)); }
// Cell of coordinate x in a grid of edge 1 / inv_cell: floor(x * inv_cell),
// monotonic in x for any edge; production steps use the same expression in
// every pass (the edge is a runtime choice, the autotuner's `cell` axis).
__device__ __forceinline__ int pcell(float x, float inv_cell) { return (int)floorf(__fmul_rn(x, inv_cell)); }
__device__ __forceinline__ uint32_t cell_hash(int cx, int cy, int cz) {
    return ((uint32_t)cx * 73856093u) ^ ((uint32_t)cy * 19349663u) ^ ((uint32_t)cz * 83492791u);
}

// Buckets of a production step (one that reports no grid). A bucket is a sixth of
// a cell along x by 2/3 of one along y and z (0.7 x 2.7 x 2.7 m for the 4 m cell),
// and the buckets along x are consecutive: a row. Their birds are contiguous in
// the cell-ordered state, so the part of a row that a search sphere reaches is one
// range of slots, read from two offsets. Finer rows mean fewer candidates and more
// ranges to look up, list and step between. A step at 1M / 16.7M birds and of a
// batch of 64 flocks, us: quarter by half cells (1 x 2 x 2 m, 153 candidates in 14
// rows for 57 birds in the sphere) 119 / 1,680 / 372, 0.67 x 2.67 111 / 1,558 / 336,
// 0.8 x 2.5 the same, 0.75 x 3 116 / 1,638 / 351.
// The coordinates are taken modulo a 2^bx x 2^by x 2^bz lattice (bx + by + bz =
// log2 buckets; bx one more than by). Wider flocks wrap, and a bucket then also
// holds its lattice translate's birds; results do not depend on which places share
// buckets. (With bx two more than by, or x buckets of half a metre, a settled
// flock, twice as wide as high, wraps more often: 64 flocks 338 -> 358 us.) Packed
// as bx | by << 5 | bz << 10.
constexpr float ROWS_PER_CELL = 1.5f, X_PER_CELL = 6.0f;
__device__ __forceinline__ uint32_t row_bits(uint32_t buckets) {
    const uint32_t k = 31u - (uint32_t)__clz(buckets);  // buckets = 2^k, k >= 12
    const uint32_t bz = (k - 1u) / 3u, by = (k - 1u - bz) >> 1, bx = k - by - bz;
    return bx | (by << 5) | (bz << 10);
}
// First bucket of row (cy, cz).
__device__ __forceinline__ uint32_t row_base(int cy, int cz, uint32_t bits) {
    const uint32_t bx = bits & 31u, by = (bits >> 5) & 31u, bz = bits >> 10;
    const uint32_t y = (uint32_t)cy & ((1u << by) - 1u), z = (uint32_t)cz & ((1u << bz) - 1u);
    return (y | (z << by)) << bx;
}
__device__ __forceinline__ uint32_t row_bucket(int cx, int cy, int cz, uint32_t bits) {
    return row_base(cy, cz, bits) | ((uint32_t)cx & ((1u << (bits & 31u)) - 1u));
}
// Loads of what an earlier phase of the same kernel wrote, on any SM of the
// cluster (never through the read-only cache).
__device__ __forceinline__ float4 ld_phase(const float4* p) {
    float4 v;
    asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                 : "l"(p)
                 : "memory");
    return v;
}

// End of bucket b's run: the next bucket's start, or its tile's end where the
// next bucket belongs to another tile (tiles are placed independently).
__device__ __forceinline__ uint32_t bucket_end(const uint32_t* offsets, const uint32_t* tile_end, uint32_t b) {
    return __ldg((b + 1u) % SCAN_TILE ? &offsets[b + 1u] : &tile_end[b / SCAN_TILE]);
}

// Search reach of a deciding bird at p with radius r: 2r inflated so that
// every bird the exact test d2 <= (2r)^2 accepts lies within it, the rounding
// of p -/+ reach covered as well.
__device__ __forceinline__ float search_reach(f3 p, float r) {
    const float rr = __fmul_rn(2.0f, r);
    const float pm = fmaxf(fabsf(p.x), fmaxf(fabsf(p.y), fabsf(p.z)));
    return rr * 1.00001f + 1e-3f + pm * 1e-6f;
}
// Radius above which a bird's box spans more than eight rows along y and z: 4 R (the
// reach is at least 2 R to either side) is more than eight rows' width.
inline float wide_radius(float cell) { return 8.01f * cell / ROWS_PER_CELL / 4.0f; }
// The reference cells that reach touches.
struct SearchBox {
    float reach, reach2;
    int lx, ly, lz;
    long long nx, ny, nz, ncell;
};
__device__ __forceinline__ SearchBox search_box(f3 p, float r) {
    SearchBox b;
    b.reach = search_reach(p, r);
    b.reach2 = b.reach * b.reach;
    b.lx = cell1(p.x - b.reach);
    b.ly = cell1(p.y - b.reach);
    b.lz = cell1(p.z - b.reach);
    b.nx = (long long)cell1(p.x + b.reach) - b.lx + 1;
    b.ny = (long long)cell1(p.y + b.reach) - b.ly + 1;
    b.nz = (long long)cell1(p.z + b.reach) - b.lz + 1;
    // an absurd reach (huge or non-finite radius)
    const bool wide = b.nx > (1 << 20) || b.ny > (1 << 20) || b.nz > (1 << 20);
    b.ncell = wide ? (1ll << 60) : b.nx * b.ny * b.nz;
    return b;
}

__device__ __forceinline__ uint32_t lanemask_lt() {
    uint32_t m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

__device__ __forceinline__ int find_flock_v(const FlockDesc* __restrict__ fl, int nfl, uint32_t v) {
    int lo = 0, hi = nfl - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (__ldg(&fl[mid].vbase) <= v) lo = mid; else hi = mid - 1;
    }
    return lo;
}
__device__ __forceinline__ int find_flock_b(const FlockDesc* __restrict__ fl, int nfl, uint32_t b) {
    int lo = 0, hi = nfl - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (__ldg(&fl[mid].bbase) <= b) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// The flock of every lane's view index, where the lanes' indices v ascend (the
// whole warp calls; an index beyond the table gets the last flock). The lanes
// search the table together, a 32nd of it per round of loads, and step on from
// the first lane's flock: two dependent loads where a binary search's five to
// eight took 1.5 to 2 us of every pass over 30 flocks (a step of 30 flocks below
// 8,000 birds 35.0 -> 31.2 us). BASE: bbase, to search by bucket.
template <uint32_t FlockDesc::*BASE = &FlockDesc::vbase>
__device__ __forceinline__ int warp_flock(const FlockDesc* __restrict__ fl, int nfl, uint32_t v) {
    if (nfl == 1) return 0;
    const int lane = (int)(threadIdx.x & 31u);
    const uint32_t v0 = __shfl_sync(FULL, v, 0);
    int f = 0;
    for (int n = nfl; n > 1;) {
        const int part = (n + 31) >> 5, i = lane * part;
        const int k = 31 - __clz(__ballot_sync(FULL, i < n && __ldg(&(fl[f + i].*BASE)) <= v0));
        f += k * part;
        n = min(part, n - k * part);
    }
    while (f + 1 < nfl && __ldg(&(fl[f + 1].*BASE)) <= v) ++f;
    return f;
}

// Slot - view index of a flock's birds in buffer p (wraps modulo 2^32).
__device__ __forceinline__ uint32_t view_shift(uint32_t sbase, uint32_t vbase, uint32_t p, uint32_t cap) {
    return p * cap + sbase - vbase;
}

__device__ __forceinline__ unsigned long long ld_relaxed(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_relaxed(unsigned long long* p, unsigned long long v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}


}  // namespace flk
