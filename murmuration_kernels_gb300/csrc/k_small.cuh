// Whole steps of small flocks in one kernel: a thread-block cluster per flock.
//
// A small flock's step is latency. At 2,000 birds the separate kernels move a few
// hundred KB and take 20 us: about 2 us of each of the five is launch, ramp and
// drain, and the rest is chains of loads that miss to L2. (The same passes as
// phases of one kernel, a cluster barrier between them, took 15 us: every phase
// still read from L2 what another SM had written.) Here every CTA of the cluster
// builds the whole grid in its own shared memory from the positions of all the
// birds, decides and flies its own share of them with every candidate a
// shared-memory load away, and publishes their new positions and headings: one
// exchange through L2 and one cluster barrier per step. The kernel runs all the
// steps of the call, and the flocks of a batch do not wait for one another.
//
// Buckets, order within a bucket (bird index), candidate order, the warp-per-bird
// sums, the decision and the flight are those of the separate kernels, so the
// words equal theirs bit for bit, and which of the two runs is free to choose by
// the size of the work alone. The state stays where it is (no reordering); the
// flock's other buffer holds the exchanged positions and headings by bird, two
// of each in turn.
#pragma once

#include "k_decide.cuh"
#include "k_grid.cuh"
#include "k_integrate.cuh"

namespace flk {

// Threads per CTA. Every phase but the decisions is a few instructions and a wait
// per bird, and the decisions are a warp per bird (13 in a CTA at 2,000 birds), so
// registers count for more than warps: 16 warps with 128 registers, us a step, 32
// warps with 64 (and 268 bytes of spills) in brackets: 500 birds 5.9 (7.7), 1,000
// 7.0 (8.6), 2,000 10.2 (11.1), 3,000 12.5 (13.9), 4,096 16.0 (18.7); 20 and 24
// warps lie between, 8 have two rounds of decisions from 1,000 birds on.
constexpr uint32_t SMALL_THREADS = 512;
// CTAs per cluster, at most; halved, down to one, where more flocks share the chip.
constexpr int SMALL_CTAS = 16;
constexpr int SMALL_SIZES = 5;  // cluster sizes: SMALL_CTAS >> 0 .. 4
// The largest flock: its grid and positions fit a CTA's shared memory with room
// to spare, a cluster of 8 has a thread for each, and sorting it costs each CTA less than the launches it saves (us a
// step, this kernel against the separate ones: 500 birds 5.9 / 17.7, 2,000
// 10.2 / 20.2, 3,000 12.5 / 22, 4,096 16 / 22).
constexpr uint32_t SMALL_CLUSTER = 4096;
// Steps of one launch, at most, which keeps a warp's 32-bit counters from running
// over (each of its birds deciding every step with every bird a candidate) and
// bounds a kernel's time.
constexpr uint32_t SMALL_STEPS = 8192;
static_assert((uint64_t)SMALL_STEPS * 32u * SMALL_CLUSTER < 1ull << 32, "32 birds a warp at most");
constexpr uint32_t SMALL_BUCKETS = 8192;                          // every such flock's bucket count
constexpr uint32_t SMALL_PER = SMALL_CLUSTER / SMALL_THREADS;  // birds a thread sorts, at most
static_assert(SMALL_CLUSTER <= SMALL_FLOCK, "the decisions are a warp per bird");
constexpr uint32_t SMALL_VEC = SMALL_BUCKETS / 8 / SMALL_THREADS;  // 16-byte vectors of counters a thread scans
static_assert(SMALL_BUCKETS == SMALL_THREADS * 8 * SMALL_VEC, "whole vectors");

// Per-warp shared memory of the decisions.
struct SmallWarp {
    uint2 row[32];
    uint32_t hit[HIT_CAP * 32];
    float red[16];
    float4 fk;
};
constexpr uint32_t SMALL_REC = 64;  // deciding birds of a CTA whose words wait in shared memory

// Dynamic shared memory for flocks of at most n birds.
inline size_t small_smem_bytes(uint32_t n) {
    return (size_t)((n + 7u) & ~7u) * (sizeof(float4) + 2) + SMALL_BUCKETS * 2 + 16 + SMALL_THREADS * 4 +
           SMALL_THREADS / 32 * sizeof(SmallWarp) + SMALL_REC * 4 * sizeof(float4);
}

// Runs in shared memory: start of each bucket, and the end after the last.
struct SharedRuns {
    const uint16_t* off;
    __device__ __forceinline__ uint32_t start(uint32_t b) const { return off[b]; }
    __device__ __forceinline__ uint32_t end(uint32_t b) const { return off[b + 1u]; }
    __device__ __forceinline__ uint2 tile(uint32_t, uint32_t t) const {
        return make_uint2(off[t * SCAN_TILE], off[(t + 1u) * SCAN_TILE]);
    }
};

// Orders every earlier access of the cluster's threads before every later one.
__device__ __forceinline__ void cluster_barrier() {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// `steps` steps of flock blockIdx.x / (CTAs of a cluster), or as many as it has
// left; nmax: the largest flock of the table.
__global__ void __launch_bounds__(SMALL_THREADS, 1) k_small(FlockDesc* fl, uint32_t steps, uint32_t nmax,
                                                            StepCtl* ctl, Arena ar, const float* __restrict__ rtab,
                                                            float cell, float inv_cell) {
    extern __shared__ __align__(16) unsigned char s_raw[];
    const uint32_t nround = (nmax + 7u) & ~7u;
    float4* s_pos = reinterpret_cast<float4*>(s_raw);                 // by sorted place; .w: bird (bits)
    uint32_t* s_off = reinterpret_cast<uint32_t*>(s_pos + nround);   // 16-bit run starts, two per word
    uint16_t* s_id = reinterpret_cast<uint16_t*>(s_off + SMALL_BUCKETS / 2 + 4);  // birds by bucket, in arrival order
    uint32_t* s_due = reinterpret_cast<uint32_t*>(s_id + nround);  // this CTA's deciding birds: own index, bird << 16
    float4* s_rec = reinterpret_cast<float4*>(s_due + SMALL_THREADS);  // A, B, C, D of the first SMALL_REC of them
    SmallWarp& m = reinterpret_cast<SmallWarp*>(s_rec + SMALL_REC * 4)[threadIdx.x >> 5];
    __shared__ uint32_t s_sum[SMALL_THREADS / 32], s_ndue;
    uint32_t ncta, rank;
    asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(ncta));
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    const FlockDesc d = fl[blockIdx.x / ncta];
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, n = d.n;
    const uint32_t run = min(steps, d.remaining);
    // this CTA's birds: slots [base, base + mine) of the state
    const uint32_t own = (n + ncta - 1) / ncta, from = min(n, rank * own), mine = min(n, from + own) - from;
    const uint32_t base = (d.parity & 1u) * ar.cap + d.sbase + from, other = ((d.parity & 1u) ^ 1u) * ar.cap + d.sbase;
    const uint32_t bits = row_bits(SMALL_BUCKETS), words = SMALL_BUCKETS / 2;
    const float inv_row = __fmul_rn(ROWS_PER_CELL, inv_cell), inv_x = __fmul_rn(X_PER_CELL, inv_cell);
    const SharedRuns runs{reinterpret_cast<const uint16_t*>(s_off)};
    float time = d.time;
    uint32_t cand = 0, pairs = 0, decided = 0, bird = 0;

    if (run && tid < mine) {
        bird = ar.id[base + tid];
        const float4 a = ar.A[base + tid];
        const f3 fw = forward(xyz(ar.B[base + tid]));
        if (bird < n) {  // always, for a valid arena
            ar.A[other + bird] = a;
            ar.C[other + bird] = make_float4(fw.x, fw.y, fw.z, 0.f);
        }
    }
    cluster_barrier();
    for (uint32_t step = 0; step < run; ++step) {
        const float4* pos = ((step & 1u) ? ar.B : ar.A) + other;   // by bird
        const float4* head = ((step & 1u) ? ar.D : ar.C) + other;
        const float t_now = __fadd_rn(time, DT);
        // count: two 16-bit counters per word; a bird keeps its bucket and arrival rank
#pragma unroll
        for (uint32_t k = 0; k < SMALL_VEC; ++k) reinterpret_cast<uint4*>(s_off)[tid * SMALL_VEC + k] = make_uint4(0u, 0u, 0u, 0u);
        if (tid == 0) s_ndue = 0;
        f3 p[SMALL_PER];
        uint32_t at[SMALL_PER];  // bucket | arrival rank << 16
        float4 dec = make_float4(0.f, 0.f, 0.f, 0.f);
        if (tid < mine) dec = ld_phase(&ar.D[base + tid]);
#pragma unroll
        for (uint32_t k = 0; k < SMALL_PER; ++k) {
            if (k * SMALL_THREADS >= n) break;
            if (tid + k * SMALL_THREADS < n) p[k] = xyz(ld_phase(&pos[tid + k * SMALL_THREADS]));
        }
        __syncthreads();
        // which of this CTA's birds decide
        const bool due = tid < mine && t_now >= dec.x;
        const uint32_t dm = __ballot_sync(FULL, due);
        uint32_t dat = 0;
        if (lane == 0 && dm) dat = atomicAdd(&s_ndue, (uint32_t)__popc(dm));
        dat = __shfl_sync(FULL, dat, 0) + __popc(dm & lanemask_lt());
        float4 rec_a, rec_b, rec_c;
        const bool keeps = due && dat < SMALL_REC;
        if (due) s_due[dat] = tid | bird << 16;
        if (keeps) {  // stored below, when the loads have had time to land
            rec_a = ld_phase(&ar.A[base + tid]);
            rec_b = ld_phase(&ar.B[base + tid]);
            rec_c = ld_phase(&ar.C[base + tid]);
        }
#pragma unroll
        for (uint32_t k = 0; k < SMALL_PER; ++k) {
            if (k * SMALL_THREADS >= n) break;
            if (tid + k * SMALL_THREADS < n) {
                const uint32_t b = row_bucket(pcell(p[k].x, inv_x), pcell(p[k].y, inv_row), pcell(p[k].z, inv_row), bits);
                const uint32_t sh = (b & 1u) * 16u;
                at[k] = b | (((atomicAdd(&s_off[b >> 1], 1u << sh) >> sh) & 0xFFFFu) << 16);
            }
        }
        __syncthreads();
        // exclusive scan of the counters, in place
        uint4* vec = reinterpret_cast<uint4*>(s_off) + tid * SMALL_VEC;
        uint4 c[SMALL_VEC];
#pragma unroll
        for (uint32_t k = 0; k < SMALL_VEC; ++k) c[k] = vec[k];
        // a word's two counters (of a sum of words: the total stays below 2^16)
        auto both = [](uint32_t w) { return (w & 0xFFFFu) + (w >> 16); };
        uint32_t sum = 0;
#pragma unroll
        for (uint32_t k = 0; k < SMALL_VEC; ++k) sum += both(c[k].x + c[k].y + c[k].z + c[k].w);
        uint32_t inc = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(FULL, inc, o);
            if ((int)lane >= o) inc += y;
        }
        if (lane == 31) s_sum[warp] = inc;
        __syncthreads();
        {
            const uint32_t v = lane < SMALL_THREADS / 32 ? s_sum[lane] : 0u;
            uint32_t pre = v;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(FULL, pre, o);
                if ((int)lane >= o) pre += y;
            }
            uint32_t at0 = __shfl_sync(FULL, pre - v, warp) + inc - sum;
            auto put = [&at0, &both](uint32_t w) {
                const uint32_t o = at0 | ((at0 + (w & 0xFFFFu)) << 16);
                at0 += both(w);
                return o;
            };
#pragma unroll
            for (uint32_t k = 0; k < SMALL_VEC; ++k) {
                uint4 o;
                o.x = put(c[k].x);
                o.y = put(c[k].y);
                o.z = put(c[k].z);
                o.w = put(c[k].w);
                vec[k] = o;
            }
            if (tid == 0) s_off[words] = n;
        }
        __syncthreads();
        // birds by bucket, then each to its place among its bucket's birds
        if (keeps) {
            s_rec[dat * 4] = rec_a;
            s_rec[dat * 4 + 1] = rec_b;
            s_rec[dat * 4 + 2] = rec_c;
            s_rec[dat * 4 + 3] = dec;
        }
#pragma unroll
        for (uint32_t k = 0; k < SMALL_PER; ++k) {
            if (k * SMALL_THREADS >= n) break;
            if (tid + k * SMALL_THREADS < n)
                s_id[runs.start(at[k] & 0xFFFFu) + (at[k] >> 16)] = (uint16_t)(tid + k * SMALL_THREADS);
        }
        __syncthreads();
#pragma unroll
        for (uint32_t k = 0; k < SMALL_PER; ++k) {
            if (k * SMALL_THREADS >= n) break;
            const uint32_t i = tid + k * SMALL_THREADS;
            if (i < n) {
                const uint32_t s = runs.start(at[k] & 0xFFFFu), e = runs.end(at[k] & 0xFFFFu);
                uint32_t place = s;
                for (uint32_t j = s; j < e; ++j) place += s_id[j] < i;
                s_pos[place] = make_float4(p[k].x, p[k].y, p[k].z, __uint_as_float(i));
            }
        }
        __syncthreads();
        // decide, a warp per bird
        const uint32_t ndue = s_ndue;
        decided += ndue;
        float4 fa = make_float4(0.f, 0.f, 0.f, 0.f), fv = fa;  // for the flight, loaded ahead
        if (tid < mine) {
            fa = ld_phase(&ar.A[base + tid]);
            fv = ld_phase(&ar.B[base + tid]);
        }
        for (uint32_t w = warp; w < ndue; w += SMALL_THREADS / 32) {
            const uint32_t st = base + (s_due[w] & 0xFFFFu), me = s_due[w] >> 16;
            const bool kept = w < SMALL_REC;
            const float4 a = kept ? s_rec[w * 4] : ld_phase(&ar.A[st]), v = kept ? s_rec[w * 4 + 1] : ld_phase(&ar.B[st]),
                         c = kept ? s_rec[w * 4 + 2] : ld_phase(&ar.C[st]), e = kept ? s_rec[w * 4 + 3] : ld_phase(&ar.D[st]);
            const f3 fi = forward(xyz(v));
            DueRec rec;
            rec.pr = make_float4(a.x, a.y, a.z, c.w);
            Bird b;
            load_bird(b, rec);
            // the bird's own place: the one in its bucket that holds it
            const uint32_t bk = row_bucket(pcell(a.x, inv_x), pcell(a.y, inv_row), pcell(a.z, inv_row), bits);
            b.self = 0;
            for (uint32_t j = runs.start(bk); j < runs.end(bk); j += 32) {
                const uint32_t t = min(j + lane, n - 1u);
                const uint32_t eq = __ballot_sync(FULL, __float_as_uint(s_pos[t].w) == me);
                if (eq) {
                    b.self = min(j + (uint32_t)__ffs(eq) - 1u, n - 1u);
                    break;
                }
            }
            const RowBox q = row_box(b, c.w, SMALL_BUCKETS, 0u, 0u, n, inv_cell);
            if (lane == 0) m.fk = make_float4(fi.x, fi.y, fi.z, 0.f);
            __syncwarp();
            Acc acc;
            cand += warp_sums<SHARED>(acc, b, q, SMALL_BUCKETS, m.row, m.hit, &m.fk, runs, s_pos, head, ctl, cell, inv_cell, lane);
            pairs += acc.n_g;
            reduce_bird<32>(acc, m.red, 1u, lane);
            __syncwarp();
            if (lane == 0) {
                const float* r = m.red;
                finish_decision(ar, st, fi, make_float4(a.z, c.w, len(xyz(v)), e.x), mk(r[0], r[1], r[2]),
                                mk(r[3], r[4], r[5]), mk(r[6], r[7], r[8]), mk(r[9], r[10], r[11]),
                                __float2uint_rn(r[12]), __float2uint_rn(r[13]), __float2uint_rn(r[14]),
                                __float2uint_rn(r[15]), rtab);
            }
            __syncwarp();
        }
        __syncthreads();
        // flight; the new positions and headings for the next step
        if (tid < mine) {
            float4 na, nb;
            fly(fa, fv, ld_phase(&ar.C[base + tid]), na, nb);
            ar.A[base + tid] = na;
            ar.B[base + tid] = nb;
            const f3 fw = forward(xyz(nb));
            if (bird < n) {
                (((step & 1u) ? ar.A : ar.B) + other)[bird] = na;
                (((step & 1u) ? ar.C : ar.D) + other)[bird] = make_float4(fw.x, fw.y, fw.z, 0.f);
            }
        }
        time = t_now;
        cluster_barrier();
    }
    if (run && rank == 0 && tid == 0) {
        FlockDesc* out = &fl[blockIdx.x / ncta];
        out->time = time;
        out->remaining = d.remaining - run;
    }
    const uint32_t cand_w = __reduce_add_sync(FULL, cand), pairs_w = __reduce_add_sync(FULL, pairs);
    if (lane == 0) {
        if (cand_w) atomicAdd(&ctl->cand_total, (unsigned long long)cand_w);
        if (pairs_w) atomicAdd(&ctl->pair_total, (unsigned long long)pairs_w);
        if (decided && warp == 0) atomicAdd(&ctl->due_total, (unsigned long long)decided);
    }
}

}  // namespace flk
