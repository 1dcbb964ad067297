// Passes 1-4 of the step: .flk words <-> arena, cell key + histogram, the
// single-pass decoupled look-back scan, scatter by arrival rank, and the birds'
// positions (or their whole state) in cell order with the deciding-bird list
// (reference cuda/flock.cu:118-179, made stable).
//
// A flock's state lives in one of two buffers (FlockDesc::parity), in the cell
// order of a recent step. Every step orders the birds' positions anew (the view);
// one step in MOVE_EVERY also moves the state into buffer parity ^ 1 in that
// order, and its integrate's last block flips the parity. Because consecutive
// slots hold birds of one neighbourhood, the histogram's atomics aggregate within
// a warp, the scatter writes runs and the gathers read mostly contiguous runs.
#pragma once

#include "device_common.cuh"

namespace flk {


// ---------------------------------------------------------------------------
// .flk words <-> arena (A = pos,roll  B = vel,spin  C = steer,radius  D = next,nb,cen)
// ---------------------------------------------------------------------------
// These move 60-byte records between bird order and the arena's arrays, in
// device memory or straight to and from page-locked host memory. What bounds
// them is the link (193 GB/s out, 211 GB/s in, for a kernel as for the copy
// engine), which wants whole lines: a warp takes 32 records at a time through
// shared memory (rows of 15 words: no bank conflicts), so its 1,920 bytes cross
// as 15 full lines. One thread per record, 15 strided words each, and a staged
// copy after it read 1M birds back in 463 us against 313 on the link.
constexpr int PACK_WARPS = 8;  // per CTA

// Loads bird i of a flock into slot base + i (bird order).
__global__ void __launch_bounds__(PACK_WARPS * 32) k_unpack(const float* __restrict__ w, uint32_t n, uint32_t base,
                                                            Arena s) {
    __shared__ float s_rec[PACK_WARPS][32 * WORDS];
    const uint32_t lane = threadIdx.x & 31;
    float* rec = s_rec[threadIdx.x >> 5];
    for (uint32_t i0 = (blockIdx.x * PACK_WARPS + (threadIdx.x >> 5)) * 32u; i0 < n; i0 += gridDim.x * PACK_WARPS * 32u) {
        const uint32_t words = min(32u, n - i0) * WORDS;
        const float* src = w + (size_t)i0 * WORDS;
        float v[WORDS];
#pragma unroll
        for (int k = 0; k < WORDS; ++k) v[k] = lane + 32u * k < words ? src[lane + 32u * k] : 0.f;
#pragma unroll
        for (int k = 0; k < WORDS; ++k) rec[lane + 32u * k] = v[k];
        __syncwarp();
        if (i0 + lane < n) {
            const float* r = rec + lane * WORDS;
            const uint32_t k = base + i0 + lane;
            s.A[k] = make_float4(r[0], r[1], r[2], r[6]);
            s.B[k] = make_float4(r[3], r[4], r[5], r[7]);
            s.C[k] = make_float4(r[9], r[10], r[11], r[8]);
            s.D[k] = make_float4(r[12], r[13], r[14], 0.f);
            s.id[k] = i0 + lane;
            s.next[k] = r[12];
        }
        __syncwarp();
    }
}

__device__ __forceinline__ void record_words(float* __restrict__ r, const Arena& s, uint32_t k) {
    const float4 a = s.A[k], b = s.B[k], c = s.C[k], d = s.D[k];
    r[0] = a.x; r[1] = a.y; r[2] = a.z;
    r[3] = b.x; r[4] = b.y; r[5] = b.z;
    r[6] = a.w; r[7] = b.w; r[8] = c.w;
    r[9] = c.x; r[10] = c.y; r[11] = c.z;
    r[12] = d.x; r[13] = d.y; r[14] = d.z;
}

// Where each bird of the flock in slots [base, base + n) is: inv[bird] = slot - base.
__global__ void __launch_bounds__(256) k_inverse(uint32_t* __restrict__ inv, uint32_t n, uint32_t base, Arena s) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t bird = s.id[base + i];
        if (bird < n) inv[bird] = i;  // always, for a valid arena
    }
}

// Writes the flock held in slots [base, base + n) (any order) back as .flk
// words in bird order. inv (k_inverse): a CTA gathers 256 consecutive birds and
// writes them as whole 128-byte lines, whatever the alignment of w (partial
// lines halve the link's rate). Without it (small flocks, where a second launch
// costs more than whole lines gain) a warp takes 32 slots and writes each
// record where its bird belongs.
__global__ void __launch_bounds__(PACK_WARPS * 32) k_pack(float* __restrict__ w, uint32_t n, uint32_t base, Arena s,
                                                          const uint32_t* __restrict__ inv) {
    constexpr uint32_t CTA = PACK_WARPS * 32;
    __shared__ float s_rec[CTA * WORDS];
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t head = (uint32_t)(reinterpret_cast<uintptr_t>(w) / 4) & 31u;  // words past a line's start
    for (uint32_t i0 = blockIdx.x * CTA; i0 < n; i0 += gridDim.x * CTA) {
        const uint32_t i = i0 + threadIdx.x;
        uint32_t bird = 0xFFFFFFFFu;
        if (i < n) {
            const uint32_t at = inv ? inv[i] : i;
            if (at < n) {  // always, for a valid arena
                record_words(s_rec + threadIdx.x * WORDS, s, base + at);
                if (!inv) bird = s.id[base + at];
            }
        }
        if (inv) {
            __syncthreads();
            const uint32_t words = min(CTA, n - i0) * WORDS;
            float* dst = w + (size_t)i0 * WORDS;  // as far past a line's start as w: a CTA's part is 120 lines
            for (int k = (int)threadIdx.x - (int)head; k < (int)words; k += CTA)
                if (k >= 0) dst[k] = s_rec[k];
            __syncthreads();
        } else {
            __syncwarp();
            const float* rec = s_rec + (threadIdx.x & ~31u) * WORDS;
            const uint32_t half = lane >> 4, word = lane & 15u;
#pragma unroll 4
            for (uint32_t r = 0; r < 32; r += 2) {
                const uint32_t to = __shfl_sync(FULL, bird, r + half);
                if (to < n && word < WORDS) w[(size_t)to * WORDS + word] = rec[(r + half) * WORDS + word];
            }
            __syncwarp();
        }
    }
}

// ---------------------------------------------------------------------------
// pass 1: cell key + histogram (warp-aggregated atomics)
// ---------------------------------------------------------------------------
// Counts a warp's birds into the histogram: a lane's bird v (act) falls in
// bucket b. Called by all 32 lanes.
__device__ __forceinline__ void count_warp(bool act, uint32_t v, uint32_t b, uint32_t* __restrict__ arrival,
                                           uint32_t* __restrict__ counts) {
    const uint32_t lane = threadIdx.x & 31;
    // Birds come in cell order, so equal buckets sit in runs of adjacent lanes:
    // each maximal run of active lanes with one bucket takes one atomic (its
    // first lane's) for the run's length, and lane k of the run gets rank
    // old + k. A bucket that recurs after a gap takes another atomic; ranks stay
    // distinct, and k_order orders every bucket by bird, so results do not
    // depend on them.
    const uint32_t m = __ballot_sync(FULL, act);
    const uint32_t bp = __shfl_up_sync(FULL, b, 1), bn = __shfl_down_sync(FULL, b, 1);
    const bool head = act && (lane == 0 || !((m >> (lane - 1)) & 1u) || bp != b);
    const bool tail = act && (lane == 31 || !((m >> (lane + 1)) & 1u) || bn != b);
    const uint32_t H = __ballot_sync(FULL, head), E = __ballot_sync(FULL, tail);
    uint32_t le;
    asm("mov.u32 %0, %%lanemask_le;" : "=r"(le));
    const uint32_t h = 31u - (uint32_t)__clz(H & le);  // this lane's run head (active lanes)
    uint32_t old = 0;
    if (head) old = atomicAdd(&counts[b], (uint32_t)__ffs(E >> lane));  // the run ends at lane + len - 1
    old = __shfl_sync(FULL, old, act ? h : lane);
    if (act) arrival[v] = old + (lane - h);
}

// Bucket of position p: ROWS (production steps) the row lattice of cell edge
// 1 / inv_cell; otherwise the reference's 4 m cell and hash, whose keys a
// grid-reporting step returns.
template <bool ROWS>
__device__ __forceinline__ uint32_t bucket_at(const float4 p, uint32_t bbase, uint32_t nb, float inv_cell) {
    if (!ROWS) return bbase + (cell_hash(cell1(p.x), cell1(p.y), cell1(p.z)) & (nb - 1u));
    const float inv_row = __fmul_rn(ROWS_PER_CELL, inv_cell);
    return bbase + row_bucket(pcell(p.x, __fmul_rn(X_PER_CELL, inv_cell)), pcell(p.y, inv_row), pcell(p.z, inv_row),
                              row_bits(nb));
}

template <bool ROWS>
__global__ void __launch_bounds__(256) k_hash_count(const FlockDesc* __restrict__ fl, int nfl, uint32_t V,
                                                    Arena ar, uint32_t* __restrict__ key,
                                                    uint32_t* __restrict__ arrival, uint32_t* __restrict__ counts,
                                                    float inv_cell) {
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t blk = blockIdx.x * blockDim.x; blk < V; blk += stride) {
        const uint32_t v = blk + threadIdx.x;
        bool act = false;
        uint32_t b = 0;
        const FlockDesc* d = &fl[warp_flock(fl, nfl, v)];
        if (v < V) {
            if (__ldg(&d->remaining)) {
                const float4 p = ar.A[v + view_shift(__ldg(&d->sbase), __ldg(&d->vbase), __ldg(&d->parity), ar.cap)];
                b = bucket_at<ROWS>(p, __ldg(&d->bbase), __ldg(&d->buckets), inv_cell);
                key[v] = b;
                act = true;
            }
        }
        count_warp(act, v, b, arrival, counts);
    }
}

// ---------------------------------------------------------------------------
// pass 2 (grid-reporting steps): single-pass decoupled look-back exclusive scan
// ---------------------------------------------------------------------------
__device__ __forceinline__ unsigned long long scan_word(uint32_t epoch, uint32_t flag, uint32_t value) {
    return ((unsigned long long)(epoch & 0x3FFFFFFFu) << 34) | ((unsigned long long)flag << 32) | value;
}

// A bucket's offset is its flock's view base plus the birds in the flock's
// lower buckets, whatever the other flocks do: a flock's buckets are a whole
// number of tiles, so the look-back ends at the flock's first tile. The
// histogram goes back to zero as it is read, ready for the next count.
__global__ void __launch_bounds__(SCAN_THREADS) k_scan(const FlockDesc* __restrict__ fl, int nfl,
                                                       uint32_t* __restrict__ counts, uint32_t* __restrict__ offsets,
                                                       uint32_t* __restrict__ tile_end, uint8_t* __restrict__ even,
                                                       uint32_t ntiles, unsigned long long* __restrict__ status,
                                                       StepCtl* __restrict__ ctl) {
    __shared__ uint32_t s_tile, s_prefix;
    __shared__ uint32_t s_warp[SCAN_THREADS / 32];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) s_tile = atomicAdd(&ctl->scan_ticket, 1u);
    __syncthreads();
    const uint32_t tile = s_tile;
    if (tile >= ntiles) {  // only after an aborted step left the ticket counter off
        if (threadIdx.x == 0) atomicCAS(&ctl->error, 0u, (uint32_t)DEV_BAD_RANGE);
        return;
    }
    const uint32_t epoch = (*(volatile uint32_t*)&ctl->epoch + 1u) & 0x3FFFFFFFu;  // never the cleared flags' 0
    const size_t base = (size_t)tile * SCAN_TILE + (size_t)threadIdx.x * SCAN_ITEMS;
    // test hook (normally 0 / 0): a tile that publishes nothing, a shorter poll limit
    const bool publish = tile + 1u != *(volatile uint32_t*)&ctl->scan_skip1;
    const uint32_t spin = *(volatile uint32_t*)&ctl->scan_spin;
    const uint32_t spin_limit = spin ? spin : SCAN_SPIN_LIMIT;

    uint4 c[SCAN_ITEMS / 4];
    uint4* src = reinterpret_cast<uint4*>(counts + base);
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS / 4; ++k) c[k] = src[k];
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS / 4; ++k) src[k] = make_uint4(0u, 0u, 0u, 0u);
    const int f = find_flock_b(fl, nfl, tile * SCAN_TILE);
    const uint32_t vbase = __ldg(&fl[f].vbase);
    const int first = (int)(__ldg(&fl[f].bbase) / SCAN_TILE);  // the flock's first tile
    uint32_t sum = 0;
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS / 4; ++k) sum += c[k].x + c[k].y + c[k].z + c[k].w;

    // block exclusive scan of the per-thread sums
    uint32_t inc = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(FULL, inc, o);
        if ((int)lane >= o) inc += y;
    }
    if (lane == 31) s_warp[warp] = inc;
    __syncthreads();
    uint32_t wpre = 0, agg = 0;
#pragma unroll
    for (int w = 0; w < SCAN_THREADS / 32; ++w) {
        const uint32_t t = s_warp[w];
        if (w < (int)warp) wpre += t;
        agg += t;
    }
    const uint32_t texcl = wpre + inc - sum;

    if (warp == 0) {
        uint32_t excl = 0;
        if ((int)tile == first) {
            if (lane == 0 && publish) st_relaxed(&status[tile], scan_word(epoch, FLAG_P, agg));
        } else {
            if (lane == 0 && publish) st_relaxed(&status[tile], scan_word(epoch, FLAG_A, agg));
            int pred = (int)tile - 1;
            uint32_t polls = 0;
            while (true) {
                const int idx = pred - (int)lane;
                uint32_t flag = FLAG_P, val = 0;
                while (true) {
                    if (idx >= first) {
                        const unsigned long long w = ld_relaxed(&status[idx]);
                        const bool ok = (uint32_t)(w >> 34) == epoch;
                        flag = ok ? (uint32_t)((w >> 32) & 3u) : 0u;
                        val = (uint32_t)w;
                    }
                    if (__all_sync(FULL, flag != 0)) break;
                    if (++polls > spin_limit) {  // give up: record and let every waiter finish
                        if (lane == 0) atomicCAS(&ctl->error, 0u, (uint32_t)DEV_SCAN_TIMEOUT);
                        flag = FLAG_P;
                        val = 0;
                        break;
                    }
                    __nanosleep(64);
                }
                const uint32_t pm = __ballot_sync(FULL, flag == FLAG_P);
                const int firstp = pm ? __ffs(pm) - 1 : 32;
                uint32_t x = ((int)lane <= firstp) ? val : 0u;
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(FULL, x, o);
                excl += x;
                if (pm) break;
                pred -= 32;
            }
            if (lane == 0 && publish) st_relaxed(&status[tile], scan_word(epoch, FLAG_P, excl + agg));
        }
        if (lane == 0) {
            s_prefix = vbase + excl;
            tile_end[tile] = vbase + excl + agg;
            even[tile] = 0;
        }
    }
    __syncthreads();
    uint32_t run = s_prefix + texcl;
    uint4* dst = reinterpret_cast<uint4*>(offsets + base);
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS / 4; ++k) {
        uint4 o;
        o.x = run; run += c[k].x;
        o.y = run; run += c[k].y;
        o.z = run; run += c[k].z;
        o.w = run; run += c[k].w;
        dst[k] = o;
    }
}

// ---------------------------------------------------------------------------
// pass 2' (production steps): run starts without a look-back
// ---------------------------------------------------------------------------
// Production steps need the buckets of a row contiguous, not the canonical
// order of all rows. A tile of 4,096 buckets is a whole number of rows of one
// flock; its birds get a place in the flock's view region from the flock's
// cursor (one atomic per tile), so no tile waits for another (the look-back
// scan took 18 us at 1M birds, 204 us at 16.7M). Where a tile lands changes no
// result: decide visits rows in the order of its box. The histogram goes back
// to zero as it is read. A flock fills a third to a sixth of its lattice, so
// most tiles are empty: they write nothing when their offsets already are all
// the same (even[tile]).
__global__ void __launch_bounds__(SCAN_THREADS) k_place(FlockDesc* __restrict__ fl, int nfl,
                                                        uint32_t* __restrict__ counts, uint32_t* __restrict__ offsets,
                                                        uint32_t* __restrict__ tile_end, uint8_t* __restrict__ even) {
    __shared__ uint32_t s_warp[SCAN_THREADS / 32], s_base;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, tile = blockIdx.x;
    const size_t base = (size_t)tile * SCAN_TILE + (size_t)threadIdx.x * SCAN_ITEMS;
    const bool was_even = even[tile];  // read before the barrier, written after it
    uint4 c[SCAN_ITEMS / 4];
    uint4* src = reinterpret_cast<uint4*>(counts + base);
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS / 4; ++k) c[k] = src[k];
    // the tile's flock, while the counts are on their way
    const int f = warp == 0 ? warp_flock<&FlockDesc::bbase>(fl, nfl, tile * SCAN_TILE) : 0;
    const uint32_t vbase = warp == 0 ? __ldg(&fl[f].vbase) : 0u;
    uint32_t sum = 0;
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS / 4; ++k) sum += c[k].x + c[k].y + c[k].z + c[k].w;
    if (sum) {
#pragma unroll
        for (int k = 0; k < SCAN_ITEMS / 4; ++k) src[k] = make_uint4(0u, 0u, 0u, 0u);
    }
    uint32_t inc = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(FULL, inc, o);
        if ((int)lane >= o) inc += y;
    }
    if (lane == 31) s_warp[warp] = inc;
    __syncthreads();
    uint32_t wpre = 0, agg = 0;
#pragma unroll
    for (int w = 0; w < SCAN_THREADS / 32; ++w) {
        const uint32_t t = s_warp[w];
        if (w < (int)warp) wpre += t;
        agg += t;
    }
    if (agg == 0 && was_even) return;
    if (threadIdx.x == 0) {
        const uint32_t b = vbase + (agg ? atomicAdd(&fl[f].cursor, agg) : 0u);
        s_base = b;
        tile_end[tile] = b + agg;
        even[tile] = agg == 0;
    }
    __syncthreads();
    uint32_t run = s_base + wpre + inc - sum;
    uint4* dst = reinterpret_cast<uint4*>(offsets + base);
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS / 4; ++k) {
        uint4 o;
        o.x = run; run += c[k].x;
        o.y = run; run += c[k].y;
        o.z = run; run += c[k].z;
        o.w = run; run += c[k].w;
        dst[k] = o;
    }
}

// Flags in the top bits of a scattered bird's two words (bird and view indices
// stay below 2^31): it is the first of its bucket's run; it decides in this step.
constexpr uint32_t HEAD_BIT = 0x80000000u, DUE_BIT = 0x80000000u;

// ---------------------------------------------------------------------------
// pass 3: scatter by arrival rank
// ---------------------------------------------------------------------------
// Each bird goes to a slot of its bucket's run, in arrival order: its bird
// index, its view index in the flock (v - vbase) and two flags. The run's first
// bird is marked, so that the next pass finds a bird's run without its bucket;
// whether it decides is read here, where the decision times are one coalesced
// stream.
__global__ void __launch_bounds__(256) k_scatter(const FlockDesc* __restrict__ fl, int nfl, uint32_t V, Arena ar,
                                                 const uint32_t* __restrict__ key, const uint32_t* __restrict__ arrival,
                                                 const uint32_t* __restrict__ offsets, uint2* __restrict__ tmp,
                                                 StepCtl* __restrict__ ctl) {
    // two birds per thread and iteration (v and v + stride), so each thread has
    // two independent load chains in flight
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t blk = blockIdx.x * blockDim.x; blk < V; blk += 2 * stride) {
        uint32_t bird[2], arr[2], kk[2], at[2];
        bool act[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const uint32_t v = blk + threadIdx.x + u * stride;
            const FlockDesc* d = &fl[warp_flock(fl, nfl, v)];
            act[u] = false;
            if (v < V) {
                if (__ldg(&d->remaining)) {
                    act[u] = true;
                    const uint32_t vbase = __ldg(&d->vbase);
                    const uint32_t st = v + view_shift(__ldg(&d->sbase), vbase, __ldg(&d->parity), ar.cap);
                    bird[u] = ar.id[st];
                    at[u] = (v - vbase) | (__fadd_rn(__ldg(&d->time), DT) >= ar.next[st] ? DUE_BIT : 0u);
                    arr[u] = arrival[v];
                    kk[u] = key[v];
                }
            }
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            if (!act[u]) continue;
            const uint32_t pos = __ldg(&offsets[kk[u]]) + arr[u];
            if (pos < V) tmp[pos] = make_uint2(arr[u] ? bird[u] : bird[u] | HEAD_BIT, at[u]);
            else atomicCAS(&ctl->error, 0u, (uint32_t)DEV_BAD_RANGE);
        }
    }
}

// ---------------------------------------------------------------------------
// pass 4: the birds in cell order
// ---------------------------------------------------------------------------
// One thread per place of the new order. A bucket's birds are ordered by bird
// index: each thread walks its bird's run both ways to the marked first birds and
// counts the lower indices (two birds per occupied production bucket, about 32
// per reference cell), which gives the stable order whatever the arrival order
// was. view receives the bird's position with its slot in .w: all that decide
// reads of most birds. A deciding bird's record goes to decide's list; the records
// of 256 places go out together, their places in the list asked for before the
// ranks are counted, so that neighbours in the list are neighbours in space and
// the list follows the order within the chip's window (longer contiguous parts
// per CTA spread the list over the flock: decide 1.08 -> 1.28 ms at 16.7M birds).
// Decide takes the records of one list by groups of eight lanes and those of the
// other by whole warps, spread over the chip: the birds of small flocks, and birds
// whose radius alone makes their box too wide for a group (wide_radius; NaN too),
// which a group would only mark and its warp come back to, one after the other
// (9,000 birds a hundred times thinner than the benchmark's, radius 7 m, 132 -> 67
// us a step, 1M of them 768 -> 733; dense flocks the same, 1M 128).
// MOVE: the state moves into the flock's other buffer in the new order as well.
// Birds change their neighbourhood slowly (5 cm a step), so the slots of a
// recent order still give mostly contiguous gathers, and most steps leave the
// state where it is: 60 bytes a bird through DRAM instead of 170. Scatter and
// order together at 1M / 16.7M birds: 40 / 521 us when every step moved the
// state and looked its buckets' ends up, 29 / 347 now, 29 / 365 without the bound
// on registers that keeps eight CTAs on an SM. (Two or four places per thread,
// ranks by shuffles within the warp, and the records' headings by whole warps
// gave nothing more or cost more in registers.)
template <bool MOVE>
__global__ void __launch_bounds__(256, MOVE ? 5 : 8) k_order(const FlockDesc* __restrict__ fl, int nfl, uint32_t V,
                                               StepCtl* __restrict__ ctl, const uint2* __restrict__ tmp, Arena ar,
                                               float4* __restrict__ view, DueRec* __restrict__ due,
                                               float wide_radius) {
    __shared__ uint32_t s_cnt[2][8];
    __shared__ uint2 s_base[2];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t it = 0;
    for (uint32_t blk = blockIdx.x * blockDim.x; blk < V; blk += gridDim.x * blockDim.x, it ^= 1u) {
        const uint32_t pos = blk + threadIdx.x;
        int f = -1;
        uint2 x;
        uint32_t st = 0, vbase = 0, n = 0;
        bool is_due = false, small = false;
        float4 a, b, c, e;  // (b, c, next: MOVE or a deciding bird; e: MOVE)
        float next;
        const int own = warp_flock(fl, nfl, pos);
        if (pos < V) {
            f = own;
            if (__ldg(&fl[f].remaining)) {
                x = __ldg(&tmp[pos]);
                vbase = __ldg(&fl[f].vbase);
                n = __ldg(&fl[f].n);
                const uint32_t lv = x.y & ~DUE_BIT;
                if (lv < n) {
                    st = vbase + lv + view_shift(__ldg(&fl[f].sbase), vbase, __ldg(&fl[f].parity), ar.cap);
                    is_due = (x.y & DUE_BIT) != 0;
                    small = n < SMALL_FLOCK;
                    a = ar.A[st];
                    if (MOVE || is_due) {
                        b = ar.B[st];
                        c = ar.C[st];
                        next = ar.next[st];
                    }
                    if (is_due) small = small || !(c.w <= wide_radius);
                    if (MOVE) e = ar.D[st];
                } else {  // never with a consistent grid
                    f = -1;
                    atomicCAS(&ctl->error, 0u, (uint32_t)DEV_BAD_RANGE);
                }
            } else {
                f = -1;
            }
        }
        // two lists: groups' records from the start, warps' from the end; the
        // counts of both ride in one word (256 records at most)
        const uint32_t dm = __ballot_sync(FULL, is_due && !small), ds = __ballot_sync(FULL, is_due && small);
        if (lane == 0) s_cnt[it][warp] = __popc(dm) | (uint32_t)__popc(ds) << 16;
        __syncthreads();
        uint32_t before = 0, all = 0;
#pragma unroll
        for (uint32_t w = 0; w < 8; ++w) {
            if (w == warp) before = all;
            all += s_cnt[it][w];
        }
        uint2 base;  // (thread 0; on its way while the ranks are counted)
        if (threadIdx.x == 0) {
            base.x = all & 0xFFFFu ? atomicAdd(&ctl->due_count, all & 0xFFFFu) : 0u;
            base.y = all >> 16 ? atomicAdd(&ctl->due_small, all >> 16) : 0u;
        }
        uint32_t nv = 0;
        if (f >= 0) {
            const uint32_t id = x.x & ~HEAD_BIT;
            uint32_t s = pos, rank = 0;
            for (uint32_t w = x.x; !(w & HEAD_BIT) && s > vbase;) {
                w = __ldg(&tmp[--s].x);
                rank += (w & ~HEAD_BIT) < id;
            }
            for (uint32_t j = pos + 1; j < vbase + n; ++j) {
                const uint32_t w = __ldg(&tmp[j].x);
                if (w & HEAD_BIT) break;
                rank += w < id;
            }
            nv = s + rank;
            if (MOVE) {
                st = nv + view_shift(__ldg(&fl[f].sbase), vbase, __ldg(&fl[f].parity) ^ 1u, ar.cap);
                ar.A[st] = a;
                ar.B[st] = b;
                ar.C[st] = c;
                ar.D[st] = e;
                ar.id[st] = id;
                ar.next[st] = next;
            }
            view[nv] = make_float4(a.x, a.y, a.z, __uint_as_float(st));
        }
        if (threadIdx.x == 0) s_base[it] = base;
        __syncthreads();
        if (is_due) {
            const uint32_t at = small ? V - 1u - (s_base[it].y + (before >> 16) + __popc(ds & lanemask_lt()))
                                      : s_base[it].x + (before & 0xFFFFu) + __popc(dm & lanemask_lt());
            const f3 fw = forward(xyz(b));
            DueRec r;
            r.pr = make_float4(a.x, a.y, a.z, c.w);
            r.fk = make_float4(fw.x, fw.y, fw.z, __uint_as_float((uint32_t)f));
            r.fl = make_uint4(nv, st, __float_as_uint(len(xyz(b))), __float_as_uint(next));
            due[at] = r;
        }
    }
}

}  // namespace flk
