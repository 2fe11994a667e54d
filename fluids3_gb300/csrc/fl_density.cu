// The density pass (computePressure, fluids4.0/fluid_kernels.cu:112-149).
//
// The search block of a cell is gridSrch^2 rows of cells; a row's cells are
// consecutive in x, so their points are one run of slots, and the reference
// loop (cells in y, z, x order, members in slot order) visits the rows in
// order and each row in ascending slots.
//
// k_density_rows: a thread per point walks its rows, the warp's pair lists
// written through shared memory (ring_walk). For gridSrch > 2, whose small
// cells leave few candidates that are not pairs.
//
// k_density: a warp per 32 consecutive slots, for gridSrch 2, whose block
// holds about twenty candidates per pair. It walks the union of its points'
// rows once:
//   1. Staging. 32 slots a time, coalesced; a candidate outside the box of
//      the warp's points widened by the support radius is dropped, the others
//      are appended to a buffer in shared memory, in visiting order.
//   2. Filter, on the tensor cores. With coordinates rounded to whole
//      thousandths of the box, d^2 - r^2 of 16 points against 8 candidates is
//      one m16n8k16 product of half-precision integers, exact in FP32; r is h
//      widened by the most that rounding can move a distance. Its sign bits
//      become one bit per (point, candidate).
//   3. Sum. Each lane visits the set bits of its own point in order and
//      evaluates the pair exactly as the reference does (same test, same
//      rounding, same order), so neither the filter nor the candidates that
//      another point of the warp brought in change a bit of the result.
//
// Two classes of tiles go other ways (crowded_tile, packed_tile below): crowded
// ones that are few are shared by whole blocks of k_density, packed ones that
// are many are walked apart, without the filter, by k_density_packed.
//
// What bounds it: instruction issue (104 warp instructions a point of the wave
// tank of 1,000,000 after 5 steps, half of them the sum's: about 24 visits a
// warp, the lanes' mean being 16). A thread per point over flag-pruned
// candidates took 157, and its chain of dependent loads left small scenes
// waiting: 2,048 points 35.0 us then, 18.4 now; 65,536: 46.1, 24.7; 1,000,000
// (wave tank, with the events around it): 189, 136. With gridSrch 3 (250,000
// points, 165 candidates and 70 pairs a point) the rows take 69 us, the old
// loop took 118 and the filter 140: there every third candidate is a pair, and
// a warp's points come from more runs than one. Staging a row's run in shared
// memory for the warp took 112 (most warps then walk two runs).
//
// The tensor instruction is mma.sync: a tile of 16 x 8 with a depth of 16 has
// too little work for tcgen05's descriptors, and the accumulator's signs
// are wanted in registers at once.
#include <algorithm>
#include <type_traits>

#include <cuda_fp16.h>

#include "fl_internal.h"

namespace {

#include "fl_device.cuh"
#include "fl_step.cuh"
#include "fl_crowd.cuh"

constexpr int kCap = 192;                       // candidates staged per round
constexpr int kFill = kCap - 32;                // a round stops staging past this
constexpr int kWords = kCap / 32;               // mask words per point
constexpr int kMaskRow = kWords + 1;            // (odd: the rows of a tile fall on distinct banks)
// per warp, in words: candidates (position, slot), the product columns of 32
// of them, and the points' product rows, whose place the masks then take
constexpr int kWarpWords = kCap * 4 + 32 * 8 + 32 * 8;
static_assert(32 * kMaskRow <= 32 * 8, "the masks fit where the product rows were");
// Runs of points that a warp takes one by one, and cells that its points may lie
// in; beyond, the lanes walk alone: in spray, a run's union of blocks holds few
// candidates of any one point. Density launch of 1,000,000 points spread evenly,
// cells of 2h with 1, 2, 3, 5 and 8 points: 44, 50, 59, 75, 81 us with 6 cells,
// 134, 94, 88, 83, 81 with as many as there are (8 runs then), 44, 50, 57, 72, 88
// with 4. The wave tank (1,000,000) after 4 steps 136, 153, 136, the dam break
// (65,536) 28.1, 30.8, 29.4; with 2 runs that took 33.1.
constexpr int kMaxSegments = 4, kMaxCells = 6;
constexpr float kUnits = 1000.0f;               // half the widest side of the box, in units (2 x stays exact in half)
constexpr float kBase = 2048.0f;                // squares are split into kBase * high + low, both exact in half
constexpr float kFar = 6.0e4f;                  // times kBase: beyond any square
constexpr int kDensityThreads = 128;
constexpr int kRowsThreads = 256, kMaxThreads = 1024;   // k_density_rows: up to the first, and beyond

__device__ __forceinline__ uint32_t half2_bits(float lo, float hi) {
    const __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t *>(&h);
}
// v / scale rounded to a whole number, for |v / scale + offset| < 2^22.
__device__ __forceinline__ float whole(float v, float scale, float offset) {
    constexpr float kRound = 12582912.0f;   // 1.5 * 2^23: adding it leaves no fraction bits
    return __fmaf_rn(v, scale, kRound + offset) - kRound;
}

// d = A (16 points x 16) . B (16 x 8 candidates): lane (g, t) holds rows g and
// g + 8, columns 2t, 2t + 1, 2t + 8, 2t + 9 of A and the same rows of column
// g of B, and gets columns 2t, 2t + 1 of rows g (d0, d1) and g + 8 (d2, d3).
// a row's words: its lanes' (2t, 2t + 1), (2t + 8, 2t + 9) for t = 0..3.
__device__ __forceinline__ void mma_16x8x16(float (&d)[4], uint2 r0, uint2 r1, uint2 b) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(r0.x), "r"(r1.x), "r"(r0.y), "r"(r1.y), "r"(b.x), "r"(b.y), "f"(0.0f));
}

// What a pair needs of the parameters: from the launch's constants, or (BATCH)
// held here, not read through the scene table for every pair.
template <bool BATCH>
struct PairParams {
    const DevParams &P;
    __device__ explicit PairParams(const DevParams &p) : P(p) {}
    __device__ float rd2() const { return P.rd2; }
    __device__ float d2() const { return P.d2; }
    __device__ uint32_t cap() const { return (uint32_t)P.hcap; }
};
template <>
struct PairParams<true> {
    float r, d;
    uint32_t c;
    __device__ explicit PairParams(const DevParams &p) : r(p.rd2), d(p.d2), c((uint32_t)p.hcap) {}
    __device__ float rd2() const { return r; }
    __device__ float d2() const { return d; }
    __device__ uint32_t cap() const { return c; }
};

// One point's running sum and pair list.
struct Sum {
    float4 p;
    float sum;
    uint32_t nh;
    uint32_t *next;      // where its next pair goes (entries 32 words apart)
};

// Adds the pair with the candidate at q (slot j) if it passes the
// reference's test. Branch-free: a miss adds +0.0, which leaves the sum's
// bits unchanged (it starts at +0.0 and its terms are positive). The list
// store is predicated by hand: compiled as a branch it cost 25 instructions
// per candidate, a quarter of the pass.
template <bool BATCH>
__device__ __forceinline__ void visit(Sum &s, const PairParams<BATCH> &c, float4 q, uint32_t j, bool on) {
    float dx2, dy2;
    const uint64_t dxy = sub2(pk2(s.p.x, s.p.y), pk2(q.x, q.y));
    const float dz = s.p.z - q.z;
    up2(mul2(dxy, dxy), dx2, dy2);
    const float dsq = dx2 + dy2 + dz * dz;
    const bool hit = on && dsq < c.rd2() && dsq > 0.0f;
    float t = (c.rd2() - dsq) * c.d2();
    t = t * t * t;
    s.sum += hit ? t : 0.0f;
    const uint32_t cap = hit ? c.cap() : 0u;
    asm volatile("{\n.reg .pred p;\nsetp.lt.u32 p, %2, %3;\n@p st.global.u32 [%0], %1;\n}" ::"l"(s.next), "r"(j),
                 "r"(s.nh), "r"(cap));
    s.next += hit ? 32 : 0;
    s.nh += hit ? 1u : 0u;
}

// One point by itself: every slot of its search block, kAhead positions
// requested before the first of them is used.
constexpr uint32_t kAhead = 4;
template <bool BATCH>
__device__ __forceinline__ void walk(const DevParams &P, Sum &s, uint32_t gc, const float4 *__restrict__ pos,
                                     const uint32_t *__restrict__ off) {
    const PairParams<BATCH> pp(P);
    const int srch = P.gridSrch, rows = srch * srch;
    const uint32_t *at = off + ((int)gc - P.nadj);
    uint32_t j = at[0], j1 = at[srch];
    for (int r = 1;; r++) {
        uint32_t nj = 0, nj1 = 0;
        if (r < rows) {   // the next row's bounds while this one is walked
            const int a = P.adj[r * srch];
            nj = at[a];
            nj1 = at[a + srch];
        }
        for (; j < j1; j += kAhead) {
            float4 q[kAhead];
#pragma unroll
            for (uint32_t k = 0; k < kAhead; k++) q[k] = pos[min(j + k, j1 - 1u)];
#pragma unroll
            for (uint32_t k = 0; k < kAhead; k++) visit(s, pp, q[k], j + k, j + k < j1);
        }
        if (r >= rows) break;
        j = nj;
        j1 = nj1;
    }
}

// The sums of the warp's points in `seg` (consecutive points of one row of
// cells, a few cells apart at most). All lanes call it.
template <bool BATCH>
__device__ __forceinline__ void segment(const DevParams &P, Sum &s, unsigned seg, uint32_t gc,
                                        const float4 *__restrict__ pos, const uint32_t *__restrict__ off,
                                        uint32_t *s_warp) {
    float4 *const s_cand = reinterpret_cast<float4 *>(s_warp);
    uint32_t *const s_col = s_warp + kCap * 4, *const s_mask = s_col + 32 * 8;
    const unsigned lane = lane_id();
    const int g = (int)(lane >> 2), t = (int)(lane & 3u);
    const bool mine = (seg >> lane) & 1u;
    const int first = __ffs(seg) - 1, last = 31 - __clz(seg);
    const uint32_t ca = __shfl_sync(0xffffffffu, gc, first), cb = __shfl_sync(0xffffffffu, gc, last);
    constexpr int srch = 2, rows = 4;
    // the rows of the search block: lane r holds row r's slots [lo, hi)
    uint32_t lo = 0, hi = 0;
    if ((int)lane < rows) {
        const int at = ((int)(lane >> 1) * P.gridRes.z + (int)(lane & 1u)) * P.gridRes.x - P.nadj;
        lo = off[(int)ca + at];
        hi = off[(int)cb + at + srch];
    }
    const Box box = box_of(s.p, seg);
    const float ox = box.ox, oy = box.oy, oz = box.oz;
    const float bx = box.ex + P.band, by = box.ey + P.band, bz = box.ez + P.band;   // a candidate's largest offset
    // units: a distance between rounded points is off by at most sqrt(3) < 1.8
    const float k = kUnits / fmaxf(fmaxf(bx, by), bz);
    const float qx = -ox * k, qy = -oy * k, qz = -oz * k;
    const float reach = sqrtf(P.rd2) * k + 1.8f, reach2 = ceilf(reach * reach) + 4.0f;
    const int cx = __float2int_rz((s.p.x - P.gridMin.x) * P.gridDelta.x), cxa = __shfl_sync(0xffffffffu, cx, first);
    const PairParams<BATCH> pp(P);
    const int rel = cx - cxa;   // the point's block starts this many cells into the rows
    const int span = __shfl_sync(0xffffffffu, rel, last);
    // With points of at most three cells the product also leaves each point
    // the candidates of its own block: it holds which cell the point is in,
    // and per cell whether the candidate lies past its block (those before it
    // are more than a cell, and so more than h, away). Else the masks are cut
    // below.
    const bool cut = !(span <= 2 && P.cellw.x > P.band);
    __syncwarp();
    {   // row: -2 (x, y, z), kBase, 1, |x|^2 as (high, low), the cell
        float x = 0.0f, y = 0.0f, z = 0.0f, high = kFar, low = 0.0f;
        if (mine) {
            x = whole(s.p.x, k, qx), y = whole(s.p.y, k, qy), z = whole(s.p.z, k, qz);
            const float n2 = x * x + y * y + z * z;
            high = whole(n2, 1.0f / kBase, 0.0f), low = n2 - high * kBase;
        }
        uint4 *row = reinterpret_cast<uint4 *>(s_mask + lane * 8);
        row[0] = make_uint4(half2_bits(-2.0f * x, -2.0f * y), half2_bits(-2.0f * z, kBase), half2_bits(1.0f, high),
                            half2_bits(low, !cut && rel == 0 ? kBase : 0.0f));
        row[1] = make_uint4(half2_bits(!cut && rel == 1 ? kBase : 0.0f, !cut && rel == 2 ? kBase : 0.0f), 0u, 0u, 0u);
    }
    __syncwarp();
    uint2 a[4];
#pragma unroll
    for (int q = 0; q < 4; q++) a[q] = *reinterpret_cast<const uint2 *>(s_mask + (g + 8 * q) * 8 + 2 * t);
    // cells along the row from the end of cell ca's block
    const int past0 = cxa + 1;
    const bool half0 = (seg & 0xffffu) != 0, half1 = (seg >> 16) != 0;

    int r = -1;
    uint32_t jb = 0, j1 = 0;
    bool have = true;
    float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
    auto next = [&]() {   // the next 32 slots: jb (the current row to j1), their positions in q
        jb += 32;
        while (jb >= j1) {
            if (++r >= rows) { have = false; return; }
            jb = __shfl_sync(0xffffffffu, lo, r);
            j1 = __shfl_sync(0xffffffffu, hi, r);
        }
        q = pos[min(jb + lane, j1 - 1u)];
    };
    next();
    while (have) {
        int cnt = 0;
        while (have && cnt <= kFill) {
            const uint32_t j = jb + lane;
            const float4 p = q;
            const bool keep = j < j1 && fabsf(p.x - ox) <= bx && fabsf(p.y - oy) <= by && fabsf(p.z - oz) <= bz;
            next();
            const unsigned kept = __ballot_sync(0xffffffffu, keep);
            if (keep) s_cand[cnt + __popc(kept & ((1u << lane) - 1u))] = make_float4(p.x, p.y, p.z, __uint_as_float(j));
            cnt += __popc(kept);
        }
        if (cnt == 0) break;
        const int words = (cnt + 31) >> 5;
        uint32_t *const row = s_mask + lane * kMaskRow;
        uint8_t *mb = reinterpret_cast<uint8_t *>(s_mask + g * kMaskRow) + t;
        __syncwarp();
        for (int w = 0; w < words; w++, mb += 4) {
            // this word's columns, a lane each: (x, y, z), |y|^2 - r^2 as
            // (high, low), kBase, 1, and per cell whether the candidate is
            // past its block; past the last candidate, near no point
            const int e = w * 32 + (int)lane;
            float x = 0.0f, y = 0.0f, z = 0.0f, high = kFar, low = 0.0f;
            int past = 0;
            if (e < cnt) {
                const float4 p = s_cand[e];
                x = whole(p.x, k, qx), y = whole(p.y, k, qy), z = whole(p.z, k, qz);
                const float n2 = x * x + y * y + z * z - reach2;
                high = whole(n2, 1.0f / kBase, 0.0f), low = n2 - high * kBase;
                past = __float2int_rz((p.x - P.gridMin.x) * P.gridDelta.x) - past0;
            }
            constexpr uint32_t kOneHalf = 0x3c00u, kFarHalf = 0x7b53u;
            uint4 *const col = reinterpret_cast<uint4 *>(s_col + lane * 8);
            col[0] = make_uint4(half2_bits(x, y), half2_bits(z, high), half2_bits(low, kBase),
                                past >= 0 ? kOneHalf | kFarHalf << 16 : kOneHalf);
            col[1] = make_uint4(past >= 2 ? kFarHalf | kFarHalf << 16 : past >= 1 ? kFarHalf : 0u, 0u, 0u, 0u);
            __syncwarp();
            // column 2t + b of tile k is candidate 8t + 2k + b, so a lane's
            // eight signs of a row are byte t of the row's mask word
            uint2 b[4];
#pragma unroll
            for (int k = 0; k < 4; k++)
                b[k] = *reinterpret_cast<const uint2 *>(s_col + ((g >> 1) * 8 + 2 * k + (g & 1)) * 8 + 2 * t);
#pragma unroll
            for (int h = 0; h < 2; h++) {
                if (!(h ? half1 : half0)) continue;
                uint32_t m0 = 0, m1 = 0;
#pragma unroll
                for (int k = 3; k >= 0; k--) {
                    float d[4];
                    mma_16x8x16(d, a[2 * h], a[2 * h + 1], b[k]);
                    m0 = __funnelshift_l(__float_as_uint(d[1]), m0, 1);
                    m0 = __funnelshift_l(__float_as_uint(d[0]), m0, 1);
                    m1 = __funnelshift_l(__float_as_uint(d[3]), m1, 1);
                    m1 = __funnelshift_l(__float_as_uint(d[2]), m1, 1);
                }
                mb[(16 * h) * kMaskRow * 4] = (uint8_t)m0;
                mb[(16 * h + 8) * kMaskRow * 4] = (uint8_t)m1;
            }
            __syncwarp();
            if (cut) {   // leave each point the candidates of its own search block
                uint32_t v = 0;
                for (int k = 0; k <= span; k++) {
                    const unsigned in = __ballot_sync(0xffffffffu, (uint32_t)(past + srch - k) < (uint32_t)srch);
                    if (rel == k) v = in;
                }
                row[w] &= v;
            }
        }
        __syncwarp();
        if (mine) {
            // the set bits in order, the lanes in step; a word without one is
            // idled through (its record, one past the word, is in the buffer)
            const int end = words - 1;
            const float4 *from = s_cand;
            uint32_t m = row[0];
            int w = 0;
            do {
                const float4 p = from[__clz(__brev(m))];
                visit(s, pp, p, __float_as_uint(p.w), m != 0u);
                m &= m - 1u;
                if (m == 0u && w < end) {
                    from += 32;
                    m = row[++w];
                }
            } while (m != 0u || w < end);
        }
        __syncwarp();
    }
}

// The points of a warp, each by itself, for rows that leave few candidates
// that are not pairs. All lanes call it. The lanes' pair counts drift apart, so
// a list entry stored when its pair was found went to a line of its own a lane;
// now entry t waits in `ring` (shared memory: kRing entries a lane) until all
// lanes have reached it. One at `lim` or past it, ahead of the slowest lane by
// more than the ring holds, is stored at once. 250,000 points with gridSrch 3:
// 96 us with every entry stored when found, 81 with 16 entries a lane, 69 with
// 32; 40 resident warps of 48 registers, 48 of 40 took 81.
constexpr uint32_t kRing = 32;
constexpr uint32_t kRingAhead = 4;
template <bool BATCH>
__device__ __forceinline__ void ring_visit(Sum &s, const PairParams<BATCH> &c, float4 q, uint32_t j, uint32_t k,
                                           uint32_t left, uint32_t lim, uint32_t past, uint32_t ring) {
    float dx2, dy2;
    const uint64_t dxy = sub2(pk2(s.p.x, s.p.y), pk2(q.x, q.y));
    const float dz = s.p.z - q.z;
    up2(mul2(dxy, dxy), dx2, dy2);
    const float dsq = dx2 + dy2 + dz * dz;
    float t = (c.rd2() - dsq) * c.d2();
    t = t * t * t;
    asm volatile(
        "{\n"
        ".reg .pred hit, in, out;\n"
        ".reg .u32 at, d;\n"
        ".reg .u64 to;\n"
        "setp.lt.u32 hit, %2, %3;\n"
        "setp.lt.and.f32 hit, %4, %5, hit;\n"
        "setp.gt.and.f32 hit, %4, 0f00000000, hit;\n"
        "setp.lt.and.u32 in, %1, %10, hit;\n"
        "sub.u32 d, %1, %10;\n"
        "setp.lt.and.u32 out, d, %11, hit;\n"
        "and.b32 at, %1, %9;\n"
        "mad.lo.u32 at, at, 128, %8;\n"
        "@in st.shared.u32 [at], %6;\n"
        "mad.wide.u32 to, %1, 128, %12;\n"
        "@out st.global.u32 [to], %6;\n"
        "@hit add.rn.f32 %0, %0, %7;\n"
        "@hit add.u32 %1, %1, 1;\n"
        "}"
        : "+f"(s.sum), "+r"(s.nh)
        : "r"(k), "r"(left), "f"(dsq), "f"(c.rd2()), "r"(j), "f"(t), "r"(ring), "n"(kRing - 1u), "r"(lim), "r"(past),
          "l"(s.next)
        : "memory");
}
// (s.next stays at the list's start.)
template <bool BATCH>
__device__ __forceinline__ void ring_walk(const DevParams &P, Sum &s, bool active, uint32_t gc,
                                          const float4 *__restrict__ pos, const uint32_t *__restrict__ off,
                                          uint32_t *ring) {
    const PairParams<BATCH> pp(P);
    const int srch = P.gridSrch, own = srch * srch,
              rows = BATCH ? (int)__reduce_max_sync(0xffffffffu, (unsigned)own) : own;
    const uint32_t *at = off + (active ? (int)gc - P.nadj : 0);
    uint32_t j = 0, j1 = 0;
    if (active) { j = at[0]; j1 = at[srch]; }
    const uint32_t cap = pp.cap(), sring = (uint32_t)__cvta_generic_to_shared(ring + lane_id());
    uint32_t done = 0, lim = min(kRing, cap);   // entries that all lanes have written; the ring's end
    uint32_t d0 = 0, d1 = 0;                    // entries [d0, d1) were stored at once
    for (int r = 1;; r++) {
        uint32_t nj = 0, nj1 = 0;
        if (r < own && active) {   // the next row's bounds while this one is walked
            const int a = P.adj[r * srch];
            nj = at[a];
            nj1 = at[a + srch];
        }
        const uint32_t past = cap - lim;
        const float4 *from = pos + j;   // (read a few slots past the row's end, and past the last point)
        for (; j < j1; j += kRingAhead, from += kRingAhead) {
            float4 q[kRingAhead];
#pragma unroll
            for (uint32_t k = 0; k < kRingAhead; k++) q[k] = from[k];
            const uint32_t left = j1 - j;
#pragma unroll
            for (uint32_t k = 0; k < kRingAhead; k++) ring_visit(s, pp, q[k], j + k, k, left, lim, past, sring);
        }
        const bool end = r >= rows;
        uint32_t low = end ? __reduce_max_sync(0xffffffffu, s.nh)
                           : __reduce_min_sync(0xffffffffu, active ? s.nh : 0xffffffffu);
        low = low == 0xffffffffu ? 0u : min(low, cap);
        const uint32_t held = min(lim, s.nh);
        for (uint32_t t = done; t < low; t++)
            if (t < held && t - d0 >= d1 - d0) s.next[32u * t] = ring[(t & (kRing - 1u)) * 32u + lane_id()];
        if (end) break;
        done = max(done, low);
        if (s.nh > lim && done >= d1) d0 = lim, d1 = s.nh;
        if (s.nh <= lim || d1 == s.nh) lim = min(done + kRing, cap);
        j = nj;
        j1 = nj1;
    }
}

// A point's results: its density, pair count and pair record.
__device__ __forceinline__ void finish(const DevParams &P, const Sum &s, int i, bool active,
                                       const float4 *__restrict__ veval, float *__restrict__ press,
                                       uint32_t *__restrict__ hitcnt, float4 *__restrict__ pairdata) {
    if (!active) {
        press[i] = 0.0f;
        hitcnt[i] = 0;
        return;
    }
    float d = s.sum * P.pmass * P.poly6kern;
    if (d == 0.0f) d = 1.0f;
    press[i] = d;
    hitcnt[i] = s.nh;
    const float4 e = veval[i];
    pairdata[2 * (size_t)i] = make_float4(s.p.x, s.p.y, s.p.z, d);
    pairdata[2 * (size_t)i + 1] = make_float4(e.x, e.y, e.z, 0.0f);
}

// Blocks of up to 256 threads are compiled for 40 resident warps (above); the
// larger ones a caller may pin or the tuner times (fl_set_launch_shapes) have
// an instantiation of their own: one block of 1,024 threads and its rings,
// 128 KB, fit a multiprocessor, two do not.
template <bool BATCH, int MOST>
__global__ void __launch_bounds__(MOST, MOST == kRowsThreads ? 1280 / kRowsThreads : 1)
k_density_rows(const __grid_constant__ DevParams P0, const SceneTab T, int n, const float4 *pos,
               const uint32_t *gcell, const uint32_t *off, const float4 *veval,
               float *press, uint32_t *hitlist, uint32_t *hitcnt,
               float4 *pairdata) {
    follow_previous();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const DevParams &P = (BATCH && i < n) ? T.params[T.point_scene[i]] : P0;
    const uint32_t gc = (i < n) ? gcell[i] : kUndef;
    const bool active = gc != kUndef;
    Sum s;
    s.p = active ? pos[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    s.sum = 0.0f;
    s.nh = 0;
    s.next = hitlist + list_at(P, i, 0);
    extern __shared__ __align__(16) uint32_t s_dyn[];
    ring_walk<BATCH>(P, s, active, gc, pos, off, s_dyn + (threadIdx.x >> 5) * (32 * kRing));
    if (i < n) finish(P, s, i, active, veval, press, hitcnt, pairdata);
}

// A crowded tile, by a whole block (fl_crowd.cuh). Alone, its warp would walk
// thousands of candidates in one chain: the density launch of 65,536 points
// after 160 steps of a collapse (up to 4,967 pairs a point) took 1,063 us, now
// 385; of 32,768 after 100 steps 174, now 119. Six blocks a multiprocessor
// hide one another's waits (two: 580 us).
constexpr int kCrowdSlots = 16;       // candidates a warp and round
constexpr int kCrowdBlocksPerSm = 6;
struct CrowdShared {              // per warp
    float4 cand[2][kCrowdSlots];            // position, slot
    float term[2][kCrowdSlots][32];         // per candidate and point
    uint32_t hits[2][32];                   // per point: its pairs among the candidates
    int kept[2];
};
static_assert(sizeof(CrowdShared) <= kWarpWords * sizeof(uint32_t), "a warp's shared memory holds its share");

// A call, not inlined: the other tiles' code keeps its registers.
template <bool BATCH>
__device__ __noinline__ void crowded_tile(const DevParams &P0, const SceneTab &T, uint32_t tile, int n,
                                             const float4 *__restrict__ pos, const uint32_t *__restrict__ gcell,
                                             const uint32_t *__restrict__ off, const float4 *__restrict__ veval,
                                             float *__restrict__ press, uint32_t *__restrict__ hitlist,
                                             uint32_t *__restrict__ hitcnt, float4 *__restrict__ pairdata,
                                             uint32_t *s_dyn) {
    const unsigned lane = lane_id();
    const int warp = (int)(threadIdx.x >> 5), from = blockDim.x > 32 ? 1 : 0;   // the first evaluating warp
    auto shared_of = [&](int w) -> CrowdShared & { return *reinterpret_cast<CrowdShared *>(s_dyn + w * kWarpWords); };
    CrowdShared &own_sh = shared_of(warp);
    const int i = (int)(tile * 32u + lane);
    const uint32_t gc = (i < n) ? gcell[i] : kUndef;
    const bool active = gc != kUndef;
    const DevParams &P = (BATCH && i < n) ? T.params[T.point_scene[i]] : P0;
    Sum s;
    s.p = active ? pos[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    s.sum = 0.0f;
    s.nh = 0;
    s.next = hitlist + list_at(P, i, 0);
    const unsigned act = __ballot_sync(0xffffffffu, active);
    unsigned heads = segment_heads(gc, active);
    while (heads) {
        const unsigned seg = next_segment(heads, act);
        const DevParams &PS = BATCH ? T.params[T.point_scene[i - (int)lane + __ffs(seg) - 1]] : P0;
        const Box box = box_of(s.p, seg);
        const float bx = box.ex + PS.band, by = box.ey + PS.band, bz = box.ez + PS.band;
        const float rd2 = PS.rd2, d2 = PS.d2;
        crowd_segment<kCrowdSlots>(
            PS, seg, gc, off, [&](bool ok, uint32_t j) { return ok ? pos[j] : make_float4(0.f, 0.f, 0.f, 0.f); },
            [&](float4 q) { return fabsf(q.x - box.ox) <= bx && fabsf(q.y - box.oy) <= by && fabsf(q.z - box.oz) <= bz; },
            [&](int buf, int e, uint32_t j, float4 q) { own_sh.cand[buf][e] = make_float4(q.x, q.y, q.z, __uint_as_float(j)); },
            [&](int buf, int kept, RowRange own) {
                uint32_t hits = 0;
#pragma unroll 4
                for (int e = 0; e < kept; e++) {
                    const float4 q = own_sh.cand[buf][e];
                    const float dx = s.p.x - q.x, dy = s.p.y - q.y, dz = s.p.z - q.z;
                    const float dsq = dx * dx + dy * dy + dz * dz;
                    const bool hit = dsq < rd2 && dsq > 0.0f && __float_as_uint(q.w) - own.lo < own.len;
                    float t = (rd2 - dsq) * d2;
                    t = t * t * t;
                    own_sh.term[buf][e][lane] = hit ? t : 0.0f;
                    hits |= (hit ? 1u : 0u) << e;
                }
                for (int e = kept; e & 3; e++) own_sh.term[buf][e][lane] = 0.0f;   // whole groups of four
                own_sh.hits[buf][lane] = hits;
                if (lane == 0) own_sh.kept[buf] = kept;
            },
            [&](int buf, int w) {
                const CrowdShared &sh = shared_of(w + from);
                const int kept = sh.kept[buf];
                for (int e = 0; e < kept; e += 4) {   // a miss adds +0.0; four loads a round trip
                    float t[4];
#pragma unroll
                    for (int u = 0; u < 4; u++) t[u] = sh.term[buf][e + u][lane];
#pragma unroll
                    for (int u = 0; u < 4; u++) s.sum += t[u];
                }
                uint32_t hits = sh.hits[buf][lane], k = s.nh;
                s.nh += __popc(hits);
                for (; hits && k < (uint32_t)PS.hcap; k++, s.next += 32, hits &= hits - 1u)
                    *s.next = __float_as_uint(sh.cand[buf][__ffs(hits) - 1].w);
            });
    }
    if (warp == 0 && i < n) finish(P, s, i, active, veval, press, hitcnt, pairdata);
}

// Whether the tiles of a class are set apart for whole blocks: while they are
// fewer than would keep every warp of those blocks busy by itself. Density
// launch with and without sharing, dam break after 90 steps: 65,536 points 172
// and 290 us, 1,048,576 points 823 and 470 us.
__host__ __device__ __forceinline__ bool shared_tiles(uint32_t count, int workers) { return count < 3u * (uint32_t)workers; }

// A packed tile by one warp, for when there are such tiles for every warp.
// Points that close together are nearly all pairs of one another, so nothing is
// filtered but by the tile's box: all lanes test every candidate, in order, four
// of them a round trip to shared memory and two an instruction (packed FP32).
// Bound by the FP32 pipe. Wave tank of 4,000,000 points after 250, 300 and 340
// steps (largest cell 14,051, 17,717, 97,686), density launches: 20.5, 49.3 and
// 139 ms by the filter, 12.5, 27.1 and 69.3 so; 1,000,000 points after 400 steps
// 27.6 and 13.4.
constexpr int kPackedCap = 256;                    // candidates staged per round
constexpr int kPackedRow = kPackedCap + 4;         // x, y, z, slot: a row each; a round's last four are made whole
constexpr int kPackedThreads = 128, kPackedBlocksPerSm = 8;

template <bool BATCH>
__device__ __forceinline__ void packed_tile(const DevParams &P0, const SceneTab &T, uint32_t tile, int n,
                                         const float4 *__restrict__ pos, const uint32_t *__restrict__ gcell,
                                         const uint32_t *__restrict__ off, const float4 *__restrict__ veval,
                                         float *__restrict__ press, uint32_t *__restrict__ hitlist,
                                         uint32_t *__restrict__ hitcnt, float4 *__restrict__ pairdata,
                                         uint32_t *s_warp) {
    const unsigned lane = lane_id(), below = (1u << lane) - 1u;
    float *const s_x = reinterpret_cast<float *>(s_warp), *const s_y = s_x + kPackedRow, *const s_z = s_y + kPackedRow;
    uint32_t *const s_slot = s_warp + 3 * kPackedRow;
    const int i = (int)(tile * 32u + lane);
    const uint32_t gc = (i < n) ? gcell[i] : kUndef;
    const bool active = gc != kUndef;
    const DevParams &P = (BATCH && i < n) ? T.params[T.point_scene[i]] : P0;
    Sum s;
    s.p = active ? pos[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    s.sum = 0.0f;
    s.nh = 0;
    s.next = hitlist + list_at(P, i, 0);
    const unsigned act = __ballot_sync(0xffffffffu, active);
    unsigned heads = segment_heads(gc, active);
    while (heads) {
        const unsigned seg = next_segment(heads, act);
        const bool mine = (seg >> lane) & 1u;
        const int first = __ffs(seg) - 1, last = 31 - __clz(seg);
        const DevParams &PS = BATCH ? T.params[T.point_scene[i - (int)lane + first]] : P0;
        const int ca = (int)__shfl_sync(0xffffffffu, gc, first), cb = (int)__shfl_sync(0xffffffffu, gc, last);
        const Box box = box_of(s.p, seg);
        const float bx = box.ex + PS.band, by = box.ey + PS.band, bz = box.ez + PS.band;
        const float rd2 = PS.rd2, d2 = PS.d2, none = __int_as_float(0x7fffffff);   // (NaN passes no test)
        const uint32_t cap = (uint32_t)PS.hcap;
        const float px = mine ? s.p.x : none;
        const uint64_t x2 = pk2(px, px), y2 = pk2(s.p.y, s.p.y), z2 = pk2(s.p.z, s.p.z), r2 = pk2(rd2, rd2),
                       k2 = pk2(d2, d2);
        RowRange own = {0u, 0xffffffffu};
        // candidate e (its distance and term) is a pair: the next of the list
        // while it has room (ROOM), and the next term of the sum
        auto pair = [&](auto room, auto ranges, int e, float dsq, float t) {
            bool hit = dsq < rd2 && dsq > 0.0f;
            if (decltype(ranges)::value) hit = hit && s_slot[e] - own.lo < own.len;
            s.sum += hit ? t : 0.0f;
            if (decltype(room)::value) {
                if (hit && s.nh < cap) s.next[32u * s.nh] = s_slot[e];
            }
            s.nh += hit ? 1u : 0u;
        };
        auto round = [&](auto room, auto ranges, int count) {
            for (int e = 0; e < count; e += 4) {
                const float4 x = *reinterpret_cast<const float4 *>(s_x + e), y = *reinterpret_cast<const float4 *>(s_y + e),
                             z = *reinterpret_cast<const float4 *>(s_z + e);
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const uint64_t dx = sub2(x2, h ? pk2(x.z, x.w) : pk2(x.x, x.y)),
                                   dy = sub2(y2, h ? pk2(y.z, y.w) : pk2(y.x, y.y)),
                                   dz = sub2(z2, h ? pk2(z.z, z.w) : pk2(z.x, z.y));
                    float xa, xb, ya, yb, za, zb, ta, tb;
                    up2(mul2(dx, dx), xa, xb);
                    up2(mul2(dy, dy), ya, yb);
                    up2(mul2(dz, dz), za, zb);
                    const float da = xa + ya + za, db = xb + yb + zb;   // (in scalar: see pk2)
                    const uint64_t t = mul2(sub2(r2, pk2(da, db)), k2);
                    up2(mul2(mul2(t, t), t), ta, tb);
                    pair(room, ranges, e + 2 * h, da, ta);
                    pair(room, ranges, e + 2 * h + 1, db, tb);
                }
            }
        };
        int cnt = 0;
        auto drain = [&]() {
            if (lane < 4) s_x[cnt + (int)lane] = none;
            __syncwarp();
            const std::true_type yes;
            const std::false_type no;
            if (__any_sync(0xffffffffu, mine && s.nh < cap)) round(yes, yes, cnt);
            else if (ca != cb) round(no, yes, cnt);
            else round(no, no, cnt);
            cnt = 0;
            __syncwarp();
        };
        for (int r = 0; r < 4; r++) {
            const int at = ((r >> 1) * PS.gridRes.z + (r & 1)) * PS.gridRes.x - PS.nadj;
            const uint32_t lo = off[ca + at], hi = off[cb + at + 2];
            if (ca != cb && mine) {   // points of several cells: each takes its own block's candidates
                own.lo = off[(int)gc + at];
                own.len = off[(int)gc + at + 2] - own.lo;
            }
            if (lo == hi) continue;
            float4 next = pos[min(lo + lane, hi - 1u)];
            for (uint32_t jb = lo; jb < hi; jb += 32u) {
                const float4 q = next;
                const uint32_t j = jb + lane;
                next = pos[min(j + 32u, hi - 1u)];
                const bool keep = j < hi && fabsf(q.x - box.ox) <= bx && fabsf(q.y - box.oy) <= by && fabsf(q.z - box.oz) <= bz;
                const unsigned kept = __ballot_sync(0xffffffffu, keep);
                if (keep) {
                    const int e = cnt + __popc(kept & below);
                    s_x[e] = q.x, s_y[e] = q.y, s_z[e] = q.z;
                    s_slot[e] = j;
                }
                cnt += __popc(kept);
                if (cnt > kPackedCap - 32) drain();
            }
            if (ca != cb && cnt) drain();   // the next row has other ranges
        }
        if (cnt) drain();
    }
    if (i < n) finish(P, s, i, active, veval, press, hitcnt, pairdata);
}

// Whether packed tiles are walked apart: too many to be shared, and not few
// beside the crowded ones (they are done before the others begin, so a launch
// of few of them ends in waits). Density of the wave tank by the filter | so:
// 4,000,000 points after 160, 170 and 180 steps (12,630, 15,690 and 18,935
// packed tiles, 0.28, 0.36 and 0.47 of the crowded) 2.21 | 2.26, 2.41 | 2.41,
// 2.66 | 2.58 ms; 1,000,000 after 210 (3,877, 0.72) 1.23 | 1.08.
__device__ __forceinline__ bool walked_apart(uint32_t crowded, uint32_t packed, int workers) {
    return !shared_tiles(packed, workers) && 5ull * packed >= 2ull * crowded;
}

// The packed tiles that are walked apart, a warp each. Launched before
// k_density, which then finds none (a kernel of its own: with this walk in
// k_density, inlined or called, its own tiles take 5-9% longer).
template <bool BATCH>
__global__ void __launch_bounds__(kPackedThreads)
k_density_packed(const __grid_constant__ DevParams P0, const SceneTab T, int n, const float4 *pos,
                 const uint32_t *gcell, const uint32_t *off, const float4 *veval, float *press, uint32_t *hitlist,
                 uint32_t *hitcnt, float4 *pairdata, const CrowdTiles tiles, int workers) {
    follow_previous();
    __shared__ __align__(16) uint32_t s_rows[kPackedThreads / 32][4 * kPackedRow];
    volatile uint32_t *const counters = tiles.counters;
    const uint32_t crowded = counters[0], packed = counters[1];
    if (!walked_apart(crowded, packed, workers)) return;
    for (;;) {
        uint32_t k = 0;
        if (lane_id() == 0) k = atomicAdd(&tiles.counters[3], 1u);
        k = __shfl_sync(0xffffffffu, k, 0);
        if (k >= packed) break;
        packed_tile<BATCH>(P0, T, tile_at(tiles, k, packed), n, pos, gcell, off, veval, press, hitlist, hitcnt, pairdata,
                           s_rows[threadIdx.x >> 5]);
    }
    __syncthreads();
    if (threadIdx.x != 0) return;
    __threadfence();
    if (atomicAdd(&tiles.counters[4], 1u) == gridDim.x - 1) counters[1] = 0;   // every block has read it
}

// The first `workers` blocks take the tiles that the sort's gather listed and
// that are set apart (workers 0: none are), the others 32 slots a warp.
template <bool BATCH>
__global__ void __launch_bounds__(kMaxThreads)
k_density(const __grid_constant__ DevParams P0, const SceneTab T, int n, const float4 *pos,
          const uint32_t *gcell, const uint32_t *off, const float4 *veval,
          float *press, uint32_t *hitlist, uint32_t *hitcnt,
          float4 *pairdata, const CrowdTiles tiles, int workers) {
    follow_previous();
    extern __shared__ __align__(16) uint32_t s_dyn[];
    if ((int)blockIdx.x < workers) {
        __shared__ uint32_t s_next;
        const uint32_t crowded = tiles.counters[0], packed = tiles.counters[1];
        const uint32_t first = shared_tiles(packed, workers) ? packed : 0u;
        const uint32_t count = first + (shared_tiles(crowded, workers) ? crowded : 0u);
        if (count == 0) return;
        for (;;) {
            if (threadIdx.x == 0) s_next = atomicAdd(&tiles.counters[2], 1u);
            __syncthreads();
            const uint32_t k = s_next;
            __syncthreads();
            if (k >= count) return;
            crowded_tile<BATCH>(P0, T, tile_at(tiles, k, first), n, pos, gcell, off, veval, press, hitlist, hitcnt,
                                pairdata, s_dyn);
        }
    }
    const int i = ((int)blockIdx.x - workers) * (int)blockDim.x + (int)threadIdx.x;
    const unsigned lane = lane_id();
    if (i - (int)lane >= n) return;   // whole warp past n
    if (workers) {
        const uint32_t kind = tiles.kind[i >> 5];
        if (kind && shared_tiles(tiles.counters[kind - 1], workers)) return;
    }
    uint32_t *s_warp = s_dyn + (threadIdx.x >> 5) * kWarpWords;
    const uint32_t gc = (i < n) ? gcell[i] : kUndef;
    const bool active = gc != kUndef;
    const DevParams &P = (BATCH && i < n) ? T.params[T.point_scene[i]] : P0;
    Sum s;
    s.p = active ? pos[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    s.sum = 0.0f;
    s.nh = 0;
    s.next = hitlist + list_at(P, i, 0);
    const unsigned act = __ballot_sync(0xffffffffu, active);
    unsigned heads = segment_heads(gc, active);
    const uint32_t before = __shfl_up_sync(0xffffffffu, gc, 1);
    const unsigned cells = __ballot_sync(0xffffffffu, active && (lane == 0 || before != gc));
    if (__popc(cells) <= kMaxCells && __popc(heads) <= kMaxSegments) {
        while (heads) {
            const unsigned seg = next_segment(heads, act);
            const DevParams &PS = BATCH ? T.params[T.point_scene[i - (int)lane + __ffs(seg) - 1]] : P0;
            segment<BATCH>(PS, s, seg, gc, pos, off, s_warp);
        }
    } else if (active) {
        walk<BATCH>(P, s, gc, pos, off);
    }
    if (i < n) finish(P, s, i, active, veval, press, hitcnt, pairdata);
}

size_t rows_smem(int threads) { return (size_t)(threads / 32) * 32 * kRing * sizeof(uint32_t); }

}  // namespace

int fl_density_init() {
    const int most = 32 * kWarpWords * (int)sizeof(uint32_t);
    FL_CUDA_TRY(cudaFuncSetAttribute(k_density<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
    FL_CUDA_TRY(cudaFuncSetAttribute(k_density<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
    const int rows = (int)rows_smem(kMaxThreads);
    FL_CUDA_TRY(cudaFuncSetAttribute(k_density_rows<false, kMaxThreads>, cudaFuncAttributeMaxDynamicSharedMemorySize, rows));
    FL_CUDA_TRY(cudaFuncSetAttribute(k_density_rows<true, kMaxThreads>, cudaFuncAttributeMaxDynamicSharedMemorySize, rows));
    return FL_OK;
}

int fl_density_block(const fl_system *s) { return s->blk_density ? s->blk_density : kDensityThreads; }

static int density_workers(const fl_system *s) { return std::min(kCrowdBlocksPerSm * s->num_sms, (s->n + 31) / 32); }

bool fl_walks_packed_apart(const fl_system *s) {
    return fl_cells_selected(s) && s->D.prune && !shared_tiles((uint32_t)(s->n + 31) / 32, density_workers(s));
}

int fl_launch_density(fl_system *s) {
    if (s->n == 0) return FL_OK;
    if (s->passes == FL_PASSES_POINT_PAIRS && s->D.prune && s->codes_valid) return fl_launch_density_pairs(s);
    // Positions that have moved since the sort (phases called after an advance
    // without a new one read them through the old grid) may be anywhere, or
    // NaN: each point walks alone, as with gridSrch > 2 (in any scene).
    const bool rows = !s->D.prune || !s->codes_valid;
    const int bs = fl_density_block(s);
    if (rows) {
        auto kern = bs <= kRowsThreads ? (s->batched ? k_density_rows<true, kRowsThreads> : k_density_rows<false, kRowsThreads>)
                                       : (s->batched ? k_density_rows<true, kMaxThreads> : k_density_rows<false, kMaxThreads>);
        launch(kern, blocks_for(s->n, bs), bs, rows_smem(bs), s->stream, s->D, fl_scene_tab(s), s->n,
               s->f[F_POS].cur<float4>(), s->f[F_GCELL].cur<uint32_t>(), s->off, s->f[F_VEVAL].cur<float4>(),
               s->f[F_PRESS].cur<float>(), s->hitlist, s->hitcnt, s->pairdata);
    } else {
        const int workers = s->tiles_listed ? density_workers(s) : 0;
        if (workers && fl_walks_packed_apart(s)) {
            auto packed = s->batched ? k_density_packed<true> : k_density_packed<false>;
            launch(packed, kPackedBlocksPerSm * s->num_sms, kPackedThreads, 0, s->stream, s->D, fl_scene_tab(s), s->n,
                   s->f[F_POS].cur<float4>(), s->f[F_GCELL].cur<uint32_t>(), s->off, s->f[F_VEVAL].cur<float4>(),
                   s->f[F_PRESS].cur<float>(), s->hitlist, s->hitcnt, s->pairdata, s->tiles, workers);
            FL_LAUNCH_CHECK("density_packed");
        }
        const size_t smem = (size_t)(bs / 32) * kWarpWords * sizeof(uint32_t);
        auto kern = s->batched ? k_density<true> : k_density<false>;
        launch(kern, workers + blocks_for(s->n, bs), bs, smem, s->stream, s->D, fl_scene_tab(s), s->n,
               s->f[F_POS].cur<float4>(), s->f[F_GCELL].cur<uint32_t>(), s->off, s->f[F_VEVAL].cur<float4>(),
               s->f[F_PRESS].cur<float>(), s->hitlist, s->hitcnt, s->pairdata, s->tiles, workers);
        s->tiles_listed = 0;   // the list is used up
    }
    FL_LAUNCH_CHECK("density");
    s->ran_density_block = bs;
    s->lists_valid = 1;
    return FL_OK;
}

extern "C" int fl_test_density_block(const fl_system *s) {
    if (!s) return fl_fail(FL_ERR_ARG, "fl_test_density_block: null system");
    return s->ran_density_block;
}
