// Pass 5: decide (reference crates/flock-ref/src/model.rs:53-145; cuda/flock.cu:190-290)
// of production steps: eight lanes per deciding bird, four birds per warp.
//
// Issue-bound: the candidates' distance tests are the work, and everything
// else a bird needs (its record, the list of its rows, its hits, the sums'
// reduction) was two thirds of the instructions when a whole warp took one
// bird. Eight lanes are the narrowest group whose loads still fill a 128-byte
// line, so a warp does that work for four birds at once.
//
// A bird's candidates are the buckets its inflated 2R sphere touches
// (row_bucket): for every (y, z) row of its box, the sphere's x extent at the
// row's nearest point gives one range of consecutive buckets, i.e. one range of
// the cell-ordered positions (two where the row wraps in the lattice).
// The group lists the non-empty ranges in shared memory, one row per lane, and
// its lanes walk them as one sequence, lane k taking every eighth candidate.
// A member of the 2R set adds its unit offset to the centrality sum at once
// (a float sum, compared to rounding: d * rsqrt(d2), a few ulp); one inside R
// goes to the lane's list of hits, about seven per bird. The hits are compacted
// over the group and finished together (square root, IEEE divisions, Gaussian,
// blind-angle test), so the expensive code runs on full groups. Which lane sums
// which candidate, and in which order, depends on the bird's own neighbourhood
// alone, so a bird's decision does not depend on the birds it shares a warp
// with.
//
// A small flock leaves most of the chip idle, and its step is one bird's chain
// of dependent loads and operations: a whole warp per bird is the shortest one,
// so flocks below SMALL_FLOCK birds are decided that way wherever they are
// (alone or in a batch, so that a flock's result does not depend on it).
// Birds above wide_radius, in any flock, go the same way. Other birds with more than
// FAST_ROWS rows in their box, ROW_CAP non-empty ranges or HIT_CAP hits in one lane
// are done by the whole warp, one at a time, after its others; a box wider than the
// lattice or the flock sweeps the flock's whole range.
#pragma once

#include "device_common.cuh"

namespace flk {

constexpr int DECIDE_LANES = 8;                  // lanes per deciding bird
constexpr int DECIDE_GROUPS = 32 / DECIDE_LANES;  // birds per warp
constexpr uint32_t ROW_CAP = 40;                 // row ranges a group lists
constexpr uint32_t HIT_CAP = 7;                  // hits waiting per lane
constexpr uint32_t FAST_ROWS = 64;               // rows of a box that a group looks through
constexpr uint32_t DECIDE_BATCH = 8;             // birds whose epilogues run together

// Per-warp shared memory. It shares each SM's storage with the L1 cache that
// holds the candidates, so it stays small.
static_assert(ROW_CAP >= 32, "a warp that takes one bird lists 32 ranges at a time");
static_assert(FAST_ROWS < 81, "wide_radius: more than eight rows along y and z are too many for a group");
struct WarpSmem {
    uint2 row[DECIDE_GROUPS][ROW_CAP + 1];                // view ranges (padded against bank conflicts)
    uint32_t hit[DECIDE_GROUPS * HIT_CAP * DECIDE_LANES];  // places of hits, each group's part contiguous
    float4 fk[DECIDE_BATCH];      // the batch's unit headings
    float4 own[DECIDE_BATCH];     // height, radius, speed, next decision
    float red[16][DECIDE_BATCH];  // sums: sep, coh, align, csum xyz; n_all, n_star, n_align, n_g
    uint32_t st[DECIDE_BATCH];    // slot of the bird; ~0: no bird
};
// Keeps what a bird's hits and epilogue need as entry k of the batch.
__device__ __forceinline__ void keep(WarpSmem& m, uint32_t k, const DueRec& rec) {
    m.fk[k] = make_float4(rec.fk.x, rec.fk.y, rec.fk.z, 0.f);
    m.own[k] = make_float4(rec.pr.z, rec.pr.w, __uint_as_float(rec.fl.z), __uint_as_float(rec.fl.w));
}

struct Acc {
    f3 sep, coh, align, csum;
    uint32_t n_all, n_star, n_align, n_g;
};
__device__ __forceinline__ void clear(Acc& a) {
    a.sep = a.coh = a.align = a.csum = mk(0.f, 0.f, 0.f);
    a.n_all = a.n_star = a.n_align = a.n_g = 0;
}

// One deciding bird, as the sweep needs it.
struct Bird {
    f3 p;
    float r2, c2;
    uint32_t self;  // its place in the view
};
__device__ __forceinline__ void load_bird(Bird& b, const DueRec& rec) {
    const float r = rec.pr.w;
    b.p = mk(rec.pr.x, rec.pr.y, rec.pr.z);
    b.r2 = __fmul_rn(r, r);
    const float rr = __fmul_rn(2.0f, r);
    b.c2 = __fmul_rn(rr, rr);
    b.self = rec.fl.x;
}

// A bird's rows: its conservative box in the row lattice.
struct RowBox {
    float reach, reach2;
    int ly, lz;          // first row
    uint32_t ny;         // rows along y
    float inv_ny;
    uint32_t nrows;      // rows of the box
    uint32_t nv;         // rows to list: nrows, or twice that where the x range wraps in the lattice
    uint32_t bits;       // row_bits of the flock's buckets
    uint32_t bbase;      // its first bucket
    uint32_t vbase, vend;  // its view region
    bool lattice;        // the box fits the lattice: no place is listed twice (otherwise the rest is not used)
};

__device__ __forceinline__ RowBox row_box(const Bird& b, float r, uint32_t buckets, uint32_t bbase, uint32_t vbase,
                                          uint32_t n, float inv_cell) {
    RowBox q;
    const float inv_row = __fmul_rn(ROWS_PER_CELL, inv_cell), inv_x = __fmul_rn(X_PER_CELL, inv_cell);
    q.reach = search_reach(b.p, r);
    q.reach2 = q.reach * q.reach;
    q.ly = pcell(b.p.y - q.reach, inv_row);
    q.lz = pcell(b.p.z - q.reach, inv_row);
    const int lx = pcell(b.p.x - q.reach, inv_x), hx = pcell(b.p.x + q.reach, inv_x);
    const int nx = hx - lx + 1, ny = pcell(b.p.y + q.reach, inv_row) - q.ly + 1,
              nz = pcell(b.p.z + q.reach, inv_row) - q.lz + 1;
    q.bits = row_bits(buckets);
    const uint32_t bx = q.bits & 31u, by = (q.bits >> 5) & 31u, bz = q.bits >> 10;
    // the first test keeps the cell numbers far from overflow (an infinite or NaN
    // radius fails it; a NaN coordinate alone does not, and needs not: every
    // distance to such a bird is NaN and fails its own test)
    const float far = fmaxf(fabsf(b.p.x), fmaxf(fabsf(b.p.y), fabsf(b.p.z))) + q.reach;
    q.lattice = far * inv_x < 1e9f && nx <= (1 << bx) && ny <= (1 << by) && nz <= (1 << bz);
    q.ny = (uint32_t)ny;
    q.inv_ny = __fdividef(1.0f, (float)ny);
    q.nrows = (uint32_t)(ny * nz);
    const uint32_t mx = (1u << bx) - 1u;
    q.nv = ((uint32_t)lx & mx) > ((uint32_t)hx & mx) ? 2u * q.nrows : q.nrows;
    q.bbase = bbase;
    q.vbase = vbase;
    q.vend = vbase + n;
    return q;
}
__device__ __forceinline__ RowBox row_box(const Bird& b, float r, const FlockDesc* __restrict__ fd, float inv_cell) {
    return row_box(b, r, __ldg(&fd->buckets), __ldg(&fd->bbase), __ldg(&fd->vbase), __ldg(&fd->n), inv_cell);
}

// Where the buckets' runs are read from.
struct GlobalRuns {
    const uint32_t *offsets, *tile_end;
    __device__ __forceinline__ uint32_t start(uint32_t b) const { return __ldg(&offsets[b]); }
    __device__ __forceinline__ uint32_t end(uint32_t b) const { return bucket_end(offsets, tile_end, b); }
    // Birds of the flock's tile t (buckets from bbase), as a view range.
    __device__ __forceinline__ uint2 tile(uint32_t bbase, uint32_t t) const {
        return make_uint2(start(bbase + t * SCAN_TILE), __ldg(&tile_end[bbase / SCAN_TILE + t]));
    }
};

// The slot range [s, e) of entry i < q.nv of the bird's row list (in view
// indices; empty: s = e). Entries from nrows on are the wrapped parts.
// At the row's nearest point the sphere spans |dx| <= sqrt(reach^2 - dyz^2)
// (dyz^2 a lower bound for any bird of the row). The 1e-4 reach^2 under the
// root, and the reach's own absolute margin, cover the rounding (and the few
// ulp of the reciprocal square root, whose argument is at least 1e-4 reach^2).
// An inconsistent range (only possible if the grid build gave up) is recorded
// and treated as empty.
// Returns whether the entry has buckets at all: its first and last one.
__device__ __forceinline__ bool row_buckets(const RowBox& q, const f3 p, uint32_t i, float cell, float inv_cell,
                                            uint32_t& first, uint32_t& last) {
    const bool second = i >= q.nrows;
    const uint32_t j = second ? i - q.nrows : i;
    const uint32_t iz = (uint32_t)(((float)j + 0.5f) * q.inv_ny), iy = j - iz * q.ny;
    const int cy = q.ly + (int)iy, cz = q.lz + (int)iz;
    const float row = cell * (1.0f / ROWS_PER_CELL);
    const float oy = (float)cy * row, oz = (float)cz * row;
    const float dy = fminf(fmaxf(p.y, oy), oy + row) - p.y;
    const float dz = fminf(fmaxf(p.z, oz), oz + row) - p.z;
    const float dyz2 = dy * dy + dz * dz;
    const float hx2 = (q.reach2 - dyz2) + 1e-4f * q.reach2;
    const float hx = fminf(hx2 * rsqrtf(hx2), q.reach);
    const float inv_x = __fmul_rn(X_PER_CELL, inv_cell);
    const uint32_t mx = (1u << (q.bits & 31u)) - 1u;
    const uint32_t xs = (uint32_t)pcell(p.x - hx, inv_x) & mx, xe = (uint32_t)pcell(p.x + hx, inv_x) & mx;
    const bool wraps = xs > xe;
    const uint32_t rb = q.bbase + row_base(cy, cz, q.bits);
    first = rb + (second ? 0u : xs);
    last = rb + (!second && wraps ? mx : xe);
    return dyz2 <= q.reach2 && (!second || wraps);
}

__device__ __forceinline__ void check_range(const RowBox& q, StepCtl* ctl, uint32_t& s, uint32_t& e) {
    if (e != s && (e < s || s < q.vbase || e > q.vend)) {  // (an empty tile's offsets may be another flock's)
        atomicCAS(&ctl->error, 0u, (uint32_t)DEV_BAD_RANGE);
        s = e = 0;
    }
}

// Lists the non-empty ranges of entries [c0, c0 + most) of the bird's nv in
// shared memory; returns how many there are (those beyond ROW_CAP are not
// listed). Called by the whole warp. With a staging table (k_decide_staged: per
// row of the union box at lo, uy rows along y, its staged offset and first
// place) the ranges are staged indices instead of places in the view.
// U entries per lane and turn, so that U pairs of loads are on their way at once.
template <int W, int U, class Runs>
__device__ __forceinline__ uint32_t list_rows(uint2* __restrict__ rows, const RowBox& q, const f3 p, uint32_t c0,
                                              uint32_t most, uint32_t nv, float cell, float inv_cell,
                                              const Runs& runs, StepCtl* ctl, uint32_t sub, uint32_t gmask,
                                              uint32_t& cand, const uint2* table = nullptr, const int* lo = nullptr,
                                              int uy = 0) {
    uint32_t R = 0;
    __syncwarp();  // the last list is no longer read
#pragma unroll 1
    for (uint32_t k = 0; k < most && __any_sync(FULL, c0 + k < nv); k += U * W) {
        uint32_t s[U], e[U], shift[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            s[u] = e[u] = shift[u] = 0;
            const uint32_t i = c0 + k + u * W + sub;
            if (u && !__any_sync(FULL, i < nv)) continue;
            uint32_t first, last;
            if (i < nv && row_buckets(q, p, i, cell, inv_cell, first, last)) {
                s[u] = runs.start(first);
                e[u] = runs.end(last);
                if (table) {
                    const uint32_t j = i >= q.nrows ? i - q.nrows : i;
                    const uint2 tb = table[(q.ly + (int)(j % q.ny) - lo[1]) + uy * (q.lz + (int)(j / q.ny) - lo[2])];
                    shift[u] = tb.x - tb.y;
                }
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            check_range(q, ctl, s[u], e[u]);
            const uint32_t bm = __ballot_sync(FULL, e[u] > s[u]) & gmask;
            if (e[u] > s[u]) {
                const uint32_t at = R + __popc(bm & lanemask_lt());
                const uint32_t b0 = s[u] + shift[u], b1 = e[u] + shift[u];
                if (at < ROW_CAP) rows[at] = W == 32 ? make_uint2(b0, b1) : make_uint2(b0 - b1, b1);
            }
            R += __popc(bm);
            cand += e[u] - s[u];
        }
    }
    __syncwarp();
    return R;
}

// Where the candidates are read from: VIEW, the positions in cell order that
// k_order wrote, through the read-only cache; STAGED, the same in shared memory
// (k_decide_staged); SHARED, positions in shared memory and headings that an
// earlier phase of this kernel wrote (k_small). A position's .w is the slot (the
// heading's place) of its bird.
enum Source { VIEW = 0, STAGED = 1, SHARED = 2 };
template <int SRC>
__device__ __forceinline__ float4 ldpos(const float4* pos, uint32_t t) {
    return SRC == VIEW ? __ldg(&pos[t]) : pos[t];
}

// One member of the R set (candidate t): the exact unit offset decides the
// blind-cone set.
template <int SRC>
__device__ __forceinline__ float4 ldvel(const float4* vel, const float4 q) {
    const float4* at = &vel[__float_as_uint(q.w)];
    return SRC == SHARED ? ld_phase(at) : __ldg(at);
}
template <int SRC>
__device__ __forceinline__ void take(Acc& a, const f3 p, const float4 fk, const float4 q, const float4 v) {
    const f3 d = mk(__fsub_rn(q.x, p.x), __fsub_rn(q.y, p.y), __fsub_rn(q.z, p.z));
    const float dist = __fsqrt_rn(dot(d, d));
    const f3 dh = dvs(d, fmaxf(dist, 1e-6f));
    a.n_all += 1;
    // the separation Gaussian only weights a sum (compared to rounding), so it
    // takes the fast exponential and a multiplication by 1 / (2 sigma^2)
    float g = 1.0f;
    if (dist > R_H) {
        const float tt = __fsub_rn(dist, R_H);
        g = __expf(__fmul_rn(-__fmul_rn(tt, tt), 1.0f / TWO_SIGMA2));
        a.coh = add(a.coh, dh);
        a.n_star += 1;
    }
    a.sep = sub(a.sep, mul(dh, g));
    if (dot(xyz(fk), dh) >= BLIND_COS) {
        a.align = add(a.align, SRC == SHARED ? xyz(v) : forward(xyz(v)));
        a.n_align += 1;
    }
}

// Finishes the group's waiting hits: compacts the lanes' lists (n entries each,
// lane order) and takes them W at a time. Called by the whole warp.
template <int W, int SRC = VIEW>
__device__ __forceinline__ void take_hits(Acc& a, const f3 p, const float4* __restrict__ fk_at,
                                          uint32_t* __restrict__ hits, uint32_t n, const float4* __restrict__ pos,
                                          const float4* __restrict__ vel, uint32_t sub) {
    uint32_t inc = n;
#pragma unroll
    for (int o = 1; o < W; o <<= 1) {
        const uint32_t y = __shfl_up_sync(FULL, inc, o, W);
        if ((int)sub >= o) inc += y;
    }
    const uint32_t total = __shfl_sync(FULL, inc, W - 1, W);
    uint32_t h[HIT_CAP];
    __syncwarp();
#pragma unroll
    for (uint32_t k = 0; k < HIT_CAP; ++k) h[k] = k < n ? hits[k * W + sub] : 0u;
    __syncwarp();
#pragma unroll
    for (uint32_t k = 0; k < HIT_CAP; ++k)
        if (k < n) hits[inc - n + k] = h[k];
    __syncwarp();
    const float4 fk = *fk_at;
    for (uint32_t k = sub; k < total; k += W) {
        const float4 q = ldpos<SRC>(pos, hits[k]);
        take<SRC>(a, p, fk, q, ldvel<SRC>(vel, q));
    }
    __syncwarp();
}

// Offset d from the deciding bird to candidate position q, and |d|^2. Set
// membership must round exactly as the oracle's chain of separately rounded
// f32 operations, so the test stays in scalar round-to-nearest intrinsics:
// paired f32x2 multiplies and adds were measured to round d2 differently,
// admitting a bird one ulp outside 2R (test_two_birds_one_ulp_outside_2r).
__device__ __forceinline__ float offset2(const Bird& b, const float4 q, f3& d) {
    d = mk(__fsub_rn(q.x, b.p.x), __fsub_rn(q.y, b.p.y), __fsub_rn(q.z, b.p.z));
    return __fadd_rn(__fadd_rn(__fmul_rn(d.x, d.x), __fmul_rn(d.y, d.y)), __fmul_rn(d.z, d.z));
}

// A lane's walk over the listed ranges (length negated, end) as one sequence,
// every DECIDE_LANES-th candidate: e + r is the next candidate of the range that
// ends at e while r < 0; row and last are the shared addresses of the ranges still
// to come. Running off a range, the walk carries its overshoot r into the next one;
// a range shorter than the overshoot costs the lane a turn.
struct Walk {
    int r;
    uint32_t e, row, last;
    __device__ __forceinline__ bool active() const { return r < 0 || row != last; }
    // The next candidate; `none` where the lane has none this turn.
    __device__ __forceinline__ uint32_t next(uint32_t none) {
        if (r >= 0 && row != last) {
            int n;
            asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(n), "=r"(e) : "r"(row));
            r += n;
            row += 8;
        }
        const uint32_t c = r < 0 ? e + r : none;
        if (r < 0) r += DECIDE_LANES;
        return c;
    }
};

// Candidate t at position q (none: the bird itself): its share of the 2R sum,
// and a place in the lane's hit list (shared address hit, STRIDE bytes between
// a lane's entries) when it lies inside R. The same operations as offset2; the
// unit offset of the centrality sum, which is compared to rounding, is
// d * rsqrt(d2), a few ulp off (the floor 1e-12 on d2 matches the 1e-6 floor on
// the distance). A full list (hit at `end`) keeps counting and stores no more.
template <int STRIDE>
__device__ __forceinline__ void test(f3& csum, uint32_t& n_g, const Bird& b, const float4 q, uint32_t t, uint32_t& hit,
                                     uint32_t end) {
    asm volatile(
        "{\n"
        " .reg .pred h, i;\n"
        " .reg .f32 x, y, z, s, u, w;\n"
        " sub.rn.f32 x, %5, %8;\n"
        " sub.rn.f32 y, %6, %9;\n"
        " sub.rn.f32 z, %7, %10;\n"
        " mul.rn.f32 s, x, x;\n"
        " mul.rn.f32 u, y, y;\n"
        " add.rn.f32 s, s, u;\n"
        " mul.rn.f32 u, z, z;\n"
        " add.rn.f32 s, s, u;\n"
        " setp.ne.u32 h, %13, %14;\n"
        " setp.le.and.f32 h, s, %11, h;\n"
        " setp.le.and.f32 i, s, %12, h;\n"
        " max.f32 u, s, 0f2B8CBCCC;\n"  // 1e-12
        " rsqrt.approx.ftz.f32 w, u;\n"
        " @h fma.rn.f32 %0, x, w, %0;\n"
        " @h fma.rn.f32 %1, y, w, %1;\n"
        " @h fma.rn.f32 %2, z, w, %2;\n"
        " @h add.u32 %3, %3, 1;\n"
        " setp.lt.and.u32 h, %4, %16, i;\n"
        " @h st.shared.u32 [%4], %13;\n"
        " @i add.u32 %4, %4, %15;\n"
        "}"
        : "+f"(csum.x), "+f"(csum.y), "+f"(csum.z), "+r"(n_g), "+r"(hit)
        : "f"(q.x), "f"(q.y), "f"(q.z), "f"(b.p.x), "f"(b.p.y), "f"(b.p.z), "f"(b.c2), "f"(b.r2), "r"(t),
          "r"(b.self), "n"(STRIDE), "r"(end));
}

// The same for candidates in global memory, U per lane and turn: walk, loads and
// tests in one block, so that a lane without a candidate needs no stand-in, only
// its predicate: it reads the place that its walk's end and overshoot name (at most
// DECIDE_LANES - 1 beyond the view, which is that much longer than its birds).
// 29 instructions per candidate; as two blocks joined by a chosen candidate 33, and
// compiled as branches 57.
#define FLK_WALK(k)                              \
    " setp.ne.u32 p, %7, %9;\n"                  \
    " setp.ge.and.s32 p, %5, 0, p;\n"            \
    " @p ld.shared.v2.u32 {n, %6}, [%7];\n"      \
    " @p add.s32 %5, %5, n;\n"                   \
    " @p add.u32 %7, %7, 8;\n"                   \
    " setp.lt.s32 v" #k ", %5, 0;\n"             \
    " add.u32 c" #k ", %6, %5;\n"                \
    " @v" #k " add.s32 %5, %5, %18;\n"
#define FLK_LOAD(k)                              \
    " mad.wide.u32 at, c" #k ", 16, %8;\n"       \
    " ld.global.nc.v4.f32 {x" #k ", y" #k ", z" #k ", u}, [at];\n"
#define FLK_TEST(k)                                        \
    " sub.rn.f32 x" #k ", x" #k ", %11;\n"                 \
    " sub.rn.f32 y" #k ", y" #k ", %12;\n"                 \
    " sub.rn.f32 z" #k ", z" #k ", %13;\n"                 \
    " mul.rn.f32 s, x" #k ", x" #k ";\n"                   \
    " mul.rn.f32 u, y" #k ", y" #k ";\n"                   \
    " add.rn.f32 s, s, u;\n"                               \
    " mul.rn.f32 u, z" #k ", z" #k ";\n"                   \
    " add.rn.f32 s, s, u;\n"                               \
    " setp.ne.and.u32 h, c" #k ", %10, v" #k ";\n"         \
    " setp.le.and.f32 h, s, %14, h;\n"                     \
    " setp.le.and.f32 i, s, %15, h;\n"                     \
    " max.f32 u, s, 0f2B8CBCCC;\n" /* 1e-12 */             \
    " rsqrt.approx.ftz.f32 u, u;\n"                        \
    " @h fma.rn.f32 %0, x" #k ", u, %0;\n"                 \
    " @h fma.rn.f32 %1, y" #k ", u, %1;\n"                 \
    " @h fma.rn.f32 %2, z" #k ", u, %2;\n"                 \
    " @h add.u32 %3, %3, 1;\n"                             \
    " setp.lt.and.u32 h, %4, %16, i;\n"                    \
    " @h st.shared.u32 [%4], c" #k ";\n"                   \
    " @i add.u32 %4, %4, %17;\n"
template <int STRIDE, int U>
__device__ __forceinline__ void walk_and_test(f3& csum, uint32_t& n_g, const Bird& b, Walk& w, const float4* pos,
                                              uint32_t& hit, uint32_t end) {
    static_assert(U == 3 || U == 4, "candidates per turn");
    if (U == 3)
        asm volatile("{\n .reg .pred p, h, i, v0, v1, v2;\n .reg .u32 n, c0, c1, c2;\n .reg .u64 at;\n"
                     " .reg .f32 s, u, x0, y0, z0, x1, y1, z1, x2, y2, z2;\n"  //
                     FLK_WALK(0) FLK_WALK(1) FLK_WALK(2) FLK_LOAD(0) FLK_LOAD(1) FLK_LOAD(2)  //
                     FLK_TEST(0) FLK_TEST(1) FLK_TEST(2) "}"
                     : "+f"(csum.x), "+f"(csum.y), "+f"(csum.z), "+r"(n_g), "+r"(hit), "+r"(w.r), "+r"(w.e), "+r"(w.row)
                     : "l"(pos), "r"(w.last), "r"(b.self), "f"(b.p.x), "f"(b.p.y), "f"(b.p.z), "f"(b.c2), "f"(b.r2),
                       "r"(end), "n"(STRIDE), "n"(DECIDE_LANES));
    else
        asm volatile("{\n .reg .pred p, h, i, v0, v1, v2, v3;\n .reg .u32 n, c0, c1, c2, c3;\n .reg .u64 at;\n"
                     " .reg .f32 s, u, x0, y0, z0, x1, y1, z1, x2, y2, z2, x3, y3, z3;\n"  //
                     FLK_WALK(0) FLK_WALK(1) FLK_WALK(2) FLK_WALK(3)  //
                     FLK_LOAD(0) FLK_LOAD(1) FLK_LOAD(2) FLK_LOAD(3)  //
                     FLK_TEST(0) FLK_TEST(1) FLK_TEST(2) FLK_TEST(3) "}"
                     : "+f"(csum.x), "+f"(csum.y), "+f"(csum.z), "+r"(n_g), "+r"(hit), "+r"(w.r), "+r"(w.e), "+r"(w.row)
                     : "l"(pos), "r"(w.last), "r"(b.self), "f"(b.p.x), "f"(b.p.y), "f"(b.p.z), "f"(b.c2), "f"(b.r2),
                       "r"(end), "n"(STRIDE), "n"(DECIDE_LANES));
}
#undef FLK_WALK
#undef FLK_LOAD
#undef FLK_TEST

// Sweeps the R listed ranges of each group's bird, U candidates per lane and
// iteration; returns the hits the lane found (those beyond HIT_CAP are not
// listed). Called by the whole warp.
template <int U, int SRC = VIEW>
__device__ __forceinline__ uint32_t sweep_group(Acc& a, const Bird& b, const uint2* __restrict__ rows, uint32_t R,
                                                uint32_t* __restrict__ hits, const float4* __restrict__ pos,
                                                uint32_t sub) {
    const uint32_t row = (uint32_t)__cvta_generic_to_shared(rows);
    Walk w{(int)sub, 0u, row, row + R * 8u};
    constexpr uint32_t STRIDE = DECIDE_LANES * 4;
    const uint32_t hit0 = (uint32_t)__cvta_generic_to_shared(hits + sub), end = hit0 + HIT_CAP * STRIDE;
    uint32_t hit = hit0;
    while (__any_sync(FULL, w.active())) {
        if (SRC == VIEW) {
            walk_and_test<STRIDE, U>(a.csum, a.n_g, b, w, pos, hit, end);
            continue;
        }
        // lanes without a candidate read the bird's own place (always in range) and discard it
        uint32_t t[U];
        float4 q[U];
#pragma unroll
        for (int u = 0; u < U; ++u) t[u] = w.next(b.self);
#pragma unroll
        for (int u = 0; u < U; ++u) q[u] = ldpos<SRC>(pos, t[u]);
#pragma unroll
        for (int u = 0; u < U; ++u) test<STRIDE>(a.csum, a.n_g, b, q[u], t[u], hit, end);
    }
    return (hit - hit0) / STRIDE;
}

// Sweeps the R <= 32 listed ranges of one bird with the whole warp, packed: the
// ranges are concatenated and swept 32 candidates at a time across their
// boundaries, two chunks per iteration. A lane finds its candidate's range from
// the bitmask of ranges that start in its chunk. Hits are taken whenever a
// lane's list (n entries on entry) fills; returns the entries left.
template <int SRC>
__device__ __forceinline__ uint32_t sweep_warp(Acc& a, const Bird& b, const uint2* __restrict__ rows, uint32_t R,
                                               uint32_t* __restrict__ hits, uint32_t n, const float4* __restrict__ pos,
                                               uint32_t lane, const float4* __restrict__ fk,
                                               const float4* __restrict__ vel) {
    const uint2 r = lane < R ? rows[lane] : make_uint2(0u, 0u);
    uint32_t inc = r.y - r.x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(FULL, inc, o);
        if ((int)lane >= o) inc += y;
    }
    const uint32_t T = __shfl_sync(FULL, inc, 31);  // candidates in all
    const uint32_t P = inc - (r.y - r.x);            // where this lane's range starts
    const uint32_t D = r.x - P;                      // candidate i of this range is place i + D
    // the chunk this lane's range starts in, and its bit there (lanes >= R: none)
    const uint32_t pch = lane < R ? P >> 5 : 0xFFFFFFFFu, pbit = 1u << (P & 31u);
    const uint32_t lemask = 0xFFFFFFFFu >> (31u - lane);
    uint32_t r0 = 0;  // ranges started before the current chunk
    constexpr uint32_t STRIDE = 128;
    const uint32_t hit0 = (uint32_t)__cvta_generic_to_shared(hits + lane), end = hit0 + HIT_CAP * STRIDE;
    uint32_t hit = hit0 + n * STRIDE;
    for (uint32_t c0 = 0, ch = 0; c0 < T; c0 += 64, ch += 2) {
        const uint32_t bA = __reduce_or_sync(FULL, pch == ch ? pbit : 0u);
        const uint32_t bB = __reduce_or_sync(FULL, pch == ch + 1 ? pbit : 0u);
        const uint32_t iA = c0 + lane, iB = iA + 32;
        const uint32_t rA = r0 + __popc(bA & lemask) - 1, rB = r0 + __popc(bA) + __popc(bB & lemask) - 1;
        uint32_t tA = iA + __shfl_sync(FULL, D, rA & 31), tB = iB + __shfl_sync(FULL, D, rB & 31);
        r0 += __popc(bA) + __popc(bB);
        if (iA >= T) tA = b.self;
        if (iB >= T) tB = b.self;
        const float4 qA = ldpos<SRC>(pos, tA), qB = ldpos<SRC>(pos, tB);
        test<STRIDE>(a.csum, a.n_g, b, qA, tA, hit, end);
        test<STRIDE>(a.csum, a.n_g, b, qB, tB, hit, end);
        if (__any_sync(FULL, hit + 2 * STRIDE > end)) {
            take_hits<32, SRC>(a, b.p, fk, hits, (hit - hit0) / STRIDE, pos, vel, lane);
            hit = hit0;
        }
    }
    return (hit - hit0) / STRIDE;
}

// Reduces the group's sums over its W lanes (a reduce-scatter of the 16
// values: with each halving a lane keeps half of them) into red, `stride` apart. The counts are small integers, so their f32 sums are exact.
template <int W>
__device__ __forceinline__ void reduce_bird(const Acc& a, float* red, uint32_t stride, uint32_t sub) {
    float v[16] = {a.sep.x,   a.sep.y,   a.sep.z,   a.coh.x,  a.coh.y,  a.coh.z,
                   a.align.x, a.align.y, a.align.z, a.csum.x, a.csum.y, a.csum.z,
                   (float)a.n_all, (float)a.n_star, (float)a.n_align, (float)a.n_g};
    int len = 16;
#pragma unroll
    for (int o = W / 2; o >= 1; o >>= 1) {
        const bool upper = (sub & (uint32_t)o) != 0;
        if (len > 1) {
            len >>= 1;
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                if (k < len) {
                    const float send = upper ? v[k] : v[k + len], keep = upper ? v[k + len] : v[k];
                    v[k] = __fadd_rn(keep, __shfl_xor_sync(FULL, send, o));
                }
            }
        } else {
            v[0] = __fadd_rn(v[0], __shfl_xor_sync(FULL, v[0], o));
        }
    }
    constexpr int PER = W >= 16 ? 1 : 16 / W;  // values a lane holds
    const uint32_t first = W > 16 ? sub / (W / 16) : sub * PER;
    if (W <= 16 || sub % (W / 16) == 0) {
#pragma unroll
        for (int k = 0; k < PER; ++k) red[(first + k) * stride] = v[k];
    }
}

// params.rs:61-65 with the tabulated factor
__device__ __forceinline__ float radius_step(float r, uint32_t n, const float* __restrict__ rtab) {
    const float factor = n < (uint32_t)RADIUS_TABLE ? __ldg(&rtab[n]) : powf(__fdiv_rn(N_C, (float)n), RADIUS_EXP);
    return clampf(__fmul_rn(r, factor), R_H, R_MAX);
}

// Finishes a bird from its sums (model.rs:95-144), one lane per bird, in the
// oracle's order of operations.
__device__ __forceinline__ void finish_decision(const Arena& ar, uint32_t st, f3 fi, const float4 own, f3 sep, f3 coh,
                                                f3 align, f3 csum, uint32_t n_all, uint32_t n_star,
                                                uint32_t n_align, uint32_t n_g, const float* __restrict__ rtab) {
    f3 force = mk(0.f, 0.f, 0.f);
    if (n_all > 0) force = add(force, mul(sep, __fdiv_rn(W_SEP, (float)n_all)));
    const float cen = n_g > 0 ? __fdiv_rn(len(csum), (float)n_g) : 0.0f;
    if (n_star > 0) force = add(force, mul(normalize_or_zero(coh), __fmul_rn(W_COH, cen)));
    const f3 al = n_align > 0 ? sub(dvs(align, (float)n_align), fi) : mk(0.f, 0.f, 0.f);
    force = add(force, mul(al, W_ALIGN));
    const float roost = __fmul_rn(W_ROOST_V, clampf(__fdiv_rn(__fsub_rn(Z0, own.x), H_ROOST_V), -1.0f, 1.0f));
    force = add(force, mul(mk(0.f, 0.f, 1.f), roost));
    force = add(force, mul(fi, __fmul_rn(MASS / TAU, __fsub_rn(V0, own.z))));
    ar.C[st] = make_float4(force.x, force.y, force.z, radius_step(own.y, n_all, rtab));
    const float next = __fadd_rn(own.w, DU);
    ar.D[st] = make_float4(next, __uint_as_float(n_all), cen, 0.f);
    ar.next[st] = next;
}

// The batch's decisions, one lane per bird.
__device__ __forceinline__ void epilogue(const WarpSmem& m, uint32_t k, const Arena& ar,
                                         const float* __restrict__ rtab) {
    const uint32_t st = m.st[k];
    if (st == 0xFFFFFFFFu) return;
    finish_decision(ar, st, xyz(m.fk[k]), m.own[k], mk(m.red[0][k], m.red[1][k], m.red[2][k]),
                    mk(m.red[3][k], m.red[4][k], m.red[5][k]), mk(m.red[6][k], m.red[7][k], m.red[8][k]),
                    mk(m.red[9][k], m.red[10][k], m.red[11][k]), __float2uint_rn(m.red[12][k]),
                    __float2uint_rn(m.red[13][k]), __float2uint_rn(m.red[14][k]), __float2uint_rn(m.red[15][k]), rtab);
}

// One bird's sums by the whole warp: the rows where its box fits the lattice and
// they are few against the flock, otherwise the flock's whole range (of
// `buckets` buckets). rows, hits:
// shared memory for 32 ranges and HIT_CAP hits per lane; fk: the bird's heading
// in shared memory. Returns the candidates.
template <int SRC, class Runs>
__device__ __forceinline__ uint32_t warp_sums(Acc& a, const Bird& b, const RowBox& q, uint32_t buckets,
                                              uint2* __restrict__ rows, uint32_t* __restrict__ hits, const float4* fk,
                                              const Runs& runs, const float4* pos, const float4* vel, StepCtl* ctl,
                                              float cell, float inv_cell, uint32_t lane) {
    clear(a);
    uint32_t n = 0, cand = 0;
    if (q.lattice && (q.nv <= 32u || (unsigned long long)q.nv * 8u < q.vend - q.vbase)) {
        for (uint32_t c0 = 0; c0 < q.nv; c0 += 32) {
            const uint32_t R = list_rows<32, 1>(rows, q, b.p, c0, 32, q.nv, cell, inv_cell, runs, ctl, lane, FULL,
                                             cand);
            n = sweep_warp<SRC>(a, b, rows, R, hits, n, pos, lane, fk, vel);
        }
    } else {
        // the tiles in order: where the placement put them changes no sum
        const uint32_t tiles = buckets / SCAN_TILE;
        for (uint32_t t0 = 0; t0 < tiles; t0 += 32) {
            uint2 r = make_uint2(0u, 0u);
            if (t0 + lane < tiles) r = runs.tile(q.bbase, t0 + lane);
            if (r.y < r.x || r.x < q.vbase || r.y > q.vend) r = make_uint2(0u, 0u);  // (an empty tile's may be another flock's)
            const uint32_t some = __ballot_sync(FULL, r.y > r.x);
            __syncwarp();
            if (r.y > r.x) rows[__popc(some & lanemask_lt())] = r;
            __syncwarp();
            cand += r.y - r.x;
            n = sweep_warp<SRC>(a, b, rows, __popc(some), hits, n, pos, lane, fk, vel);
        }
    }
    take_hits<32, SRC>(a, b.p, fk, hits, n, pos, vel, lane);
    return cand;
}

// A record whose bird an eight-lane group does not finish is marked in its
// flock index; the warp comes back to it after its other birds.
constexpr uint32_t WIDE_MARK = 0x80000000u;

// One record's bird by the whole warp. Returns the lane's candidates and pairs.
__device__ __noinline__ uint2 warp_bird(WarpSmem& m, const DueRec* __restrict__ rec_at,
                                        const FlockDesc* __restrict__ fl, StepCtl* __restrict__ ctl,
                                        const uint32_t* __restrict__ offsets, const uint32_t* __restrict__ tile_end,
                                        Arena ar, const float4* __restrict__ view, const float* __restrict__ rtab,
                                        float cell, float inv_cell, uint32_t lane) {
    const DueRec rec = *rec_at;
    Bird b;
    load_bird(b, rec);
    const RowBox q = row_box(b, rec.pr.w, &fl[__float_as_uint(rec.fk.w) & ~WIDE_MARK], inv_cell);
    __syncwarp();
    if (lane == 0) {
        keep(m, 0, rec);
        m.st[0] = rec.fl.y;
    }
    __syncwarp();
    Acc a;
    const uint32_t cand = warp_sums<VIEW>(a, b, q, __ldg(&fl[__float_as_uint(rec.fk.w) & ~WIDE_MARK].buckets),
                                          &m.row[0][0], m.hit, &m.fk[0], GlobalRuns{offsets, tile_end}, view, ar.B, ctl,
                                          cell, inv_cell, lane);
    reduce_bird<32>(a, &m.red[0][0], DECIDE_BATCH, lane);
    __syncwarp();
    if (lane == 0) epilogue(m, 0, ar, rtab);
    __syncwarp();
    return make_uint2(cand, a.n_g);
}

// The birds of small flocks and those with a radius above wide_radius (their records
// fill the list from its end), one per warp, spread over the CTAs.
__device__ __forceinline__ void small_birds(WarpSmem& m, uint32_t V, uint32_t nsmall, const DueRec* __restrict__ due,
                                            const FlockDesc* __restrict__ fl, StepCtl* __restrict__ ctl,
                                            const uint32_t* __restrict__ offsets,
                                            const uint32_t* __restrict__ tile_end, const Arena& ar,
                                            const float4* __restrict__ view, const float* __restrict__ rtab,
                                            float cell, float inv_cell, uint32_t lane, uint32_t& cand,
                                            uint32_t& pairs) {
    for (uint32_t i = (threadIdx.x >> 5) * gridDim.x + blockIdx.x; i < nsmall; i += gridDim.x * (blockDim.x >> 5)) {
        const uint2 c = warp_bird(m, &due[V - 1u - i], fl, ctl, offsets, tile_end, ar, view, rtab, cell, inv_cell, lane);
        cand += c.x;
        pairs += c.y;
    }
}

// The marked records among the DECIDE_GROUPS from e on.
__device__ __forceinline__ void wide_quad(WarpSmem& m, uint32_t e, uint32_t ndue, const DueRec* due,
                                          const FlockDesc* __restrict__ fl, StepCtl* __restrict__ ctl,
                                          const uint32_t* __restrict__ offsets, const uint32_t* __restrict__ tile_end,
                                          const Arena& ar, const float4* __restrict__ view,
                                          const float* __restrict__ rtab, float cell, float inv_cell, uint32_t lane,
                                          uint32_t& cand, uint32_t& pairs) {
    for (uint32_t k = e; k < min(e + DECIDE_GROUPS, ndue); ++k) {
        if (!(*(const volatile uint32_t*)&due[k].fk.w & WIDE_MARK)) continue;  // the same in every lane
        const uint2 c = warp_bird(m, &due[k], fl, ctl, offsets, tile_end, ar, view, rtab, cell, inv_cell, lane);
        cand += c.x;
        pairs += c.y;
    }
}

// The per-warp counter totals.
__device__ __forceinline__ void count_work(uint32_t lane, bool first, uint32_t ndue, uint32_t cand, uint32_t pairs,
                                           StepCtl* __restrict__ ctl) {
    const uint32_t cand_w = __reduce_add_sync(FULL, cand), pairs_w = __reduce_add_sync(FULL, pairs);
    if (lane == 0) {
        if (cand_w) atomicAdd(&ctl->cand_total, (unsigned long long)cand_w);
        if (pairs_w) atomicAdd(&ctl->pair_total, (unsigned long long)pairs_w);
        if (first) atomicAdd(&ctl->due_total, (unsigned long long)ndue);
    }
}

// Dynamic shared memory: one WarpSmem per warp. 64 registers per thread, so
// one 1024-thread CTA fills an SM, and all its warps take consecutive records,
// i.e. neighbouring birds, and share their candidates in L1.
// THREADS: of a CTA. A warp's registers decide how many of its loads are on their
// way at once, the number of warps how much of their latency others hide: with up
// to two rounds of deciding birds per warp 24 warps are best (37,501 birds 28.2 ->
// 24.8 us a step against 32 warps, 100,000 29.4 -> 26.6), up to about 50 rounds 28
// (1M birds 110 -> 105, 3M the same), beyond that 32 (16.7M birds 1,525 -> 1,512).
// The sums' order, and so every bit, is the same.
constexpr int DECIDE_FEW = 768, DECIDE_SOME = 896, DECIDE_MANY = 1024;
template <int THREADS>
__global__ void __launch_bounds__(THREADS, 1) k_decide(const FlockDesc* __restrict__ fl, uint32_t V,
                                                    StepCtl* __restrict__ ctl,
                                                    DueRec* __restrict__ due,
                                                    const uint32_t* __restrict__ offsets,
                                                    const uint32_t* __restrict__ tile_end, Arena ar,
                                                    const float4* __restrict__ view, const float* __restrict__ rtab,
                                                    float cell, float inv_cell) {
    extern __shared__ __align__(16) unsigned char s_raw[];
    WarpSmem& m = reinterpret_cast<WarpSmem*>(s_raw)[threadIdx.x >> 5];
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t g = lane / DECIDE_LANES, sub = lane % DECIDE_LANES;
    const uint32_t gmask = ((1u << DECIDE_LANES) - 1u) << (g * DECIDE_LANES);
    const uint32_t ndue = *(volatile uint32_t*)&ctl->due_count, nsmall = *(volatile uint32_t*)&ctl->due_small;
    uint32_t cand = 0, pairs = 0, slot = 0;
    uint32_t* hits = m.hit + g * (HIT_CAP * DECIDE_LANES);

    // Warp w of CTA c takes the records of a round at (c, w), so that a CTA works
    // on neighbouring birds, which share candidates in L1; the records of the
    // last, partial round go to the CTAs in turn, so that no SM has a whole round
    // more than another.
    const uint32_t quads = (ndue + DECIDE_GROUPS - 1) / DECIDE_GROUPS, warp = threadIdx.x >> 5;
    const uint32_t all = gridDim.x * (blockDim.x >> 5);
    auto quad = [&](uint32_t r0) {  // of the round that starts at r0
        return r0 + (r0 + all <= quads ? blockIdx.x * (blockDim.x >> 5) + warp : warp * gridDim.x + blockIdx.x);
    };
    bool any_wide = false;
    for (uint32_t r0 = 0; r0 < quads; r0 += all) {
        const uint32_t qd = quad(r0);
        if (qd >= quads) break;
        const uint32_t e = qd * DECIDE_GROUPS;
        const bool has = e + g < ndue;
        Bird b;
        bool fast;
        uint32_t R, st;
        {
            const DueRec rec = due[has ? e + g : e];  // everything the setup needs, one place
            load_bird(b, rec);
            st = rec.fl.y;
            if (sub == 0) keep(m, slot + g, rec);
            const RowBox q = row_box(b, rec.pr.w, &fl[__float_as_uint(rec.fk.w)], inv_cell);
            fast = q.lattice && q.nrows <= FAST_ROWS;
            R = list_rows<DECIDE_LANES, 2>(m.row[g], q, b.p, 0, 2 * FAST_ROWS, has && fast ? q.nv : 0u, cell,
                                        inv_cell, GlobalRuns{offsets, tile_end}, ctl, sub, gmask, cand);
        }
        fast = fast && R <= ROW_CAP;
        Acc a;
        clear(a);
        uint32_t n = sweep_group<THREADS == DECIDE_MANY ? 3 : 4>(a, b, m.row[g], fast ? R : 0u, hits, view, sub);
        const uint32_t over = __ballot_sync(FULL, n > HIT_CAP);
        fast = fast && !(over & gmask);
        take_hits<DECIDE_LANES>(a, b.p, &m.fk[slot + g], hits, fast ? n : 0u, view, ar.B, sub);
        reduce_bird<DECIDE_LANES>(a, &m.red[0][slot + g], DECIDE_BATCH, sub);
        if (fast) pairs += a.n_g;
        if (sub == 0) {
            m.st[slot + g] = has && fast ? st : 0xFFFFFFFFu;
            if (has && !fast) due[e + g].fk.w = __uint_as_float(__float_as_uint(due[e + g].fk.w) | WIDE_MARK);
        }
        any_wide |= __any_sync(FULL, has && !fast);
        slot += DECIDE_GROUPS;
        if (slot == DECIDE_BATCH) {
            __syncwarp();
            if (lane < DECIDE_BATCH) epilogue(m, lane, ar, rtab);
            __syncwarp();
            slot = 0;
        }
    }
    if (slot) {
        __syncwarp();
        if (lane < slot) epilogue(m, lane, ar, rtab);
        __syncwarp();
    }
    small_birds(m, V, nsmall, due, fl, ctl, offsets, tile_end, ar, view, rtab, cell, inv_cell, lane, cand, pairs);
    if (any_wide) {
        __syncwarp();  // the marks are written
        for (uint32_t r0 = 0; r0 < quads; r0 += all) {
            const uint32_t qd = quad(r0);
            if (qd >= quads) break;
            wide_quad(m, qd * DECIDE_GROUPS, ndue, due, fl, ctl, offsets, tile_end, ar, view, rtab, cell, inv_cell,
                      lane, cand, pairs);
        }
    }
    count_work(lane, blockIdx.x == 0 && threadIdx.x < 32, ndue + nsmall, cand, pairs, ctl);
}

}  // namespace flk
