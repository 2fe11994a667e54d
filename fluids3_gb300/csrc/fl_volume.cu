// sampleParticles (fluids4.0/fluid_kernels.cu:263-308): a Gaussian-weighted
// particle count at every voxel of a res.x x res.y x res.z lattice over
// [bmin, bmax), read from the sorted grid. Voxel (x, y, z) sits at
// bmin + (x / res.x, y / res.y, z / res.z) * (bmax - bmin) and writes
// out[(z * res.y + y) * res.x + x] (the reference's final store; its
// out-of-range store uses another order, an upstream slip not kept here);
// voxels outside the scan range read 0.
//
// Two kernels, by how far apart the voxels lie (sample_bricks below):
//
// k_sample_bricks: a warp per brick of 4 x 4 x 2 voxels. It walks the rows of
// cells that its voxels' search blocks cover once, keeps the points in the
// brick's box widened by h, and marks for each voxel which of them count
// (within h, and in the voxel's own search block); each lane then adds its
// own in the reference's order. A thread per voxel over all of its block's
// points, the term behind a branch that some lane nearly always took, was
// bound by issue, and so is this, on half the instructions: 128^3 voxels over
// 250,000 points 273 -> 120 us, 160^3 over 1,000,000 501 -> 279; with the
// 3 x 3 x 3 search block (48 points a voxel) 377 -> 300 and 696 -> 648. Masks
// kept until up to 192 points are staged: drained 32 at a time, the lanes'
// uneven counts cost 10% more; bricks of 4 x 4 x 4, two voxels a lane, were no
// faster.
//
// k_sample_wide: 1 to 32 lanes a voxel, each a part of its points, for lattices
// so coarse that a brick's voxels share few points: 32^3 voxels over 1,000,000
// points 122 us (a thread per voxel as it was), 205 (bricks), 20 (32 lanes).
//
// The reference's exponent, -(sqrt(d2 dsq))^2 / h2, is formed as
// d2 dsq times -1 / h2 (as high and low parts): fewer roundings, no square
// root and no division.
#include <math.h>
#include <type_traits>

#include "fl_internal.h"

namespace {

#include "fl_device.cuh"
#include "fl_step.cuh"
#include "fl_crowd.cuh"

constexpr int kVolumeThreads = 128;

struct Lattice {
    int3 res;
    float3 bmin, bmax;
    float scalar, kern, c_hi, c_lo;   // exponent = t * (c_hi + c_lo), t = dsq * d2
};

__device__ __forceinline__ float voxel_at(int i, int res, float lo, float hi) {
    return lo + ((float)i / (float)res) * (hi - lo);
}

__device__ __forceinline__ float weight(const Lattice &L, float dsq, float d2) {
    const float t = dsq * d2;
    return L.kern * expf(__fmaf_rn(t, L.c_hi, t * L.c_lo));
}

// A voxel's cell on each axis (cell_of), and whether it is in the scan range.
struct VoxelCell {
    int x, y, z;
    bool in;
};
__device__ __forceinline__ VoxelCell voxel_cell(const DevParams &P, float x, float y, float z) {
    VoxelCell c;
    c.x = __float2int_rz((x - P.gridMin.x) * P.gridDelta.x);
    c.y = __float2int_rz((y - P.gridMin.y) * P.gridDelta.y);
    c.z = __float2int_rz((z - P.gridMin.z) * P.gridDelta.z);
    c.in = c.x >= 1 && c.x <= P.gridScanMax.x && c.y >= 1 && c.y <= P.gridScanMax.y && c.z >= 1 && c.z <= P.gridScanMax.z;
    return c;
}

// Cells relative to the brick's first one, 10 bits an axis. cell - first cell
// of a block lies in [0, srch) on every axis exactly when neither the
// difference nor the difference plus (P2 - srch) has a bit at or above P2 in
// any field (P2: the power of two from srch; a negative field has them all,
// and what it borrows from the next field changes nothing then).
__device__ __forceinline__ uint32_t pack_cell(int x, int y, int z) {
    return (uint32_t)x | (uint32_t)y << 10 | (uint32_t)z << 20;
}
constexpr uint32_t kOnes = 1u | 1u << 10 | 1u << 20;
constexpr int kBrickCells = 900;   // cells an axis a brick may span (10 bits)

constexpr int kBrickCap = 192, kBrickWords = kBrickCap / 32;   // points a warp takes at a time
struct BrickShared {
    float4 cand[kBrickCap + 1];        // position, packed cell (one past the last word is read, and not used)
    uint32_t mask[kBrickWords][32];    // per voxel: which of them count
};

// SPARSE: most bricks hold no point, and leave early (20,000 points in a mostly
// empty box, 192^3 voxels: 113 us without, 85 with; a box full of points takes
// 2-5% longer with it).
template <bool SPARSE>
__global__ void __launch_bounds__(kVolumeThreads)
k_sample_bricks(const __grid_constant__ DevParams P, const __grid_constant__ Lattice L, int3 bricks,
                const float4 *__restrict__ pos, const uint32_t *__restrict__ gcell, const uint32_t *__restrict__ off,
                float *__restrict__ out) {
    __shared__ BrickShared s_brick[kVolumeThreads / 32];
    const unsigned lane = lane_id(), below = (1u << lane) - 1u;
    BrickShared &sh = s_brick[threadIdx.x >> 5];
    const uint32_t brick = blockIdx.x * (kVolumeThreads / 32) + (threadIdx.x >> 5);
    const uint32_t brow = brick / (uint32_t)bricks.x;
    const int ix = (int)(brick % (uint32_t)bricks.x) * 4 + (int)(lane & 3u);
    const int iy = (int)(brow % (uint32_t)bricks.y) * 4 + (int)(lane >> 2 & 3u);
    const int iz = (int)(brow / (uint32_t)bricks.y) * 2 + (int)(lane >> 4);   // (past the last brick: past res.z)
    const bool exists = ix < L.res.x && iy < L.res.y && iz < L.res.z;
    const float4 p = make_float4(voxel_at(ix, L.res.x, L.bmin.x, L.bmax.x), voxel_at(iy, L.res.y, L.bmin.y, L.bmax.y),
                                 voxel_at(iz, L.res.z, L.bmin.z, L.bmax.z), 0.0f);
    const VoxelCell c = voxel_cell(P, p.x, p.y, p.z);
    const bool active = exists && c.in;
    const unsigned act = __ballot_sync(0xffffffffu, active);
    float v = 0.0f;
    if (act) {
        const int srch = P.gridSrch;
        const int far = 0x7fffffff;
        const int x0 = __reduce_min_sync(0xffffffffu, active ? c.x : far), x1 = __reduce_max_sync(0xffffffffu, active ? c.x : -far);
        const int y0 = __reduce_min_sync(0xffffffffu, active ? c.y : far), y1 = __reduce_max_sync(0xffffffffu, active ? c.y : -far);
        const int z0 = __reduce_min_sync(0xffffffffu, active ? c.z : far), z1 = __reduce_max_sync(0xffffffffu, active ? c.z : -far);
        const Box box = box_of(p, act);
        const float bx = box.ex + P.band, by = box.ey + P.band, bz = box.ez + P.band;
        // the lane's block begins one cell below its own; cells count from
        // one below the brick's first
        const uint32_t mine = active ? pack_cell(c.x - x0, c.y - y0, c.z - z0) : 0u;
        const uint32_t p2 = srch <= 2 ? 2u : srch <= 4 ? 4u : 8u;
        const uint32_t carry = (p2 - (uint32_t)srch) * kOnes, high = ~((p2 - 1u) * kOnes);
        const float rd2 = active ? P.rd2 : 0.0f, d2 = P.d2;   // (no point counts for an idle lane)
        int cnt = 0;
        auto take = [&]() {   // the cnt points staged: mark, then add each voxel's own
            __syncwarp();
            const int words = (cnt + 31) >> 5;
            for (int w = 0; w < words; w++) {
                const int most = min(32, cnt - 32 * w);
                uint32_t m = 0;
#pragma unroll 4
                for (int e = 0; e < most; e++) {
                    const float4 q = sh.cand[32 * w + e];
                    const float dx = p.x - q.x, dy = p.y - q.y, dz = p.z - q.z;
                    const float dsq = dx * dx + dy * dy + dz * dz;
                    const uint32_t d = __float_as_uint(q.w) - mine;
                    const bool hit = dsq < rd2 && dsq > 0.0f && ((d | (d + carry)) & high) == 0u;
                    m |= (hit ? 1u : 0u) << e;
                }
                sh.mask[w][lane] = m;
            }
            int w = 0;
            uint32_t m = sh.mask[0][lane];
            do {
                const float4 q = sh.cand[32 * w + __clz(__brev(m))];
                const float dx = p.x - q.x, dy = p.y - q.y, dz = p.z - q.z;
                const float t = weight(L, dx * dx + dy * dy + dz * dz, d2);
                v += m ? t : 0.0f;
                m &= m - 1u;
                if (m == 0u && w < words - 1) m = sh.mask[++w][lane];
            } while (m != 0u || w < words - 1);
            cnt = 0;
            __syncwarp();
        };
        int y_end = y1 + srch - 2;
        if constexpr (SPARSE) {   // a look at all rows of cells first, a lane each
            const int zs = z1 - z0 + srch, rows = (y1 - y0 + srch) * zs;
            bool filled = rows > 32;
            if ((int)lane < rows && !filled) {
                const int row = ((y0 - 1 + (int)lane / zs) * P.gridRes.z + z0 - 1 + (int)lane % zs) * P.gridRes.x;
                filled = off[row + x0 - 1] < off[row + x1 + srch - 1];
            }
            if (!__any_sync(0xffffffffu, filled)) y_end = y0 - 2;
        }
        for (int y = y0 - 1; y <= y_end; y++)
            for (int z = z0 - 1; z <= z1 + srch - 2; z++) {
                const int row = (y * P.gridRes.z + z) * P.gridRes.x;
                const uint32_t lo = off[row + x0 - 1], hi = off[row + x1 + srch - 1];
                for (uint32_t jb = lo; jb < hi; jb += 32u) {
                    const uint32_t j = jb + lane;
                    const float4 q = pos[min(j, hi - 1u)];
                    const bool keep = j < hi && fabsf(q.x - box.ox) <= bx && fabsf(q.y - box.oy) <= by && fabsf(q.z - box.oz) <= bz;
                    const unsigned kept = __ballot_sync(0xffffffffu, keep);
                    if (keep) {
                        // its cell in the grid (of the last sort: it may have moved since)
                        const int cx = (int)gcell[j] - row - (x0 - 1);
                        sh.cand[cnt + __popc(kept & below)] =
                            make_float4(q.x, q.y, q.z, __uint_as_float(pack_cell(cx, y - (y0 - 1), z - (z0 - 1))));
                    }
                    cnt += __popc(kept);
                    if (cnt > kBrickCap - 32) take();
                }
            }
        if (cnt) take();
    }
    if (exists) out[((size_t)iz * L.res.y + iy) * L.res.x + ix] = v * L.scalar;
}

template <int LANES>   // a power of two up to 32
__global__ void __launch_bounds__(kVolumeThreads)
k_sample_wide(const __grid_constant__ DevParams P, const __grid_constant__ Lattice L, const float4 *__restrict__ pos,
              const uint32_t *__restrict__ off, float *__restrict__ out) {
    const uint32_t part = threadIdx.x % LANES;
    const uint32_t i = blockIdx.x * (kVolumeThreads / LANES) + threadIdx.x / LANES, line = i / (uint32_t)L.res.x;
    const uint32_t iz = line / (uint32_t)L.res.y;
    const float px = voxel_at((int)(i % (uint32_t)L.res.x), L.res.x, L.bmin.x, L.bmax.x);
    const float py = voxel_at((int)(line % (uint32_t)L.res.y), L.res.y, L.bmin.y, L.bmax.y);
    const float pz = voxel_at((int)iz, L.res.z, L.bmin.z, L.bmax.z);
    const VoxelCell c = voxel_cell(P, px, py, pz);
    const bool exists = iz < (uint32_t)L.res.z;
    float v = 0.0f;
    if (exists && c.in) {
        const int cell = (c.y * P.gridRes.z + c.z) * P.gridRes.x + c.x;
        for (int r = 0; r < P.gridSrch * P.gridSrch; r++) {
            const int at = cell - P.nadj + P.adj[r * P.gridSrch];
            const uint32_t lo = off[at], hi = off[at + P.gridSrch];
            for (uint32_t j = lo + part; j < hi; j += (uint32_t)LANES) {
                const float4 q = pos[j];
                const float dx = px - q.x, dy = py - q.y, dz = pz - q.z;
                const float dsq = dx * dx + dy * dy + dz * dz;
                if (dsq < P.rd2 && dsq > 0.0f) v += weight(L, dsq, P.d2);
            }
        }
    }
#pragma unroll
    for (int d = LANES / 2; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
    if (exists && part == 0) out[i] = v * L.scalar;
}

// Lanes a voxel when not by bricks: as many as leave the chip's threads full
// once (a power of two up to 32). 16^3, 32^3, 48^3 and 64^3 voxels over
// 1,000,000 points in a third of its box: one lane 60, 60, 60, 61 us, 32 lanes
// 20, 29, 48, 88, the rule's 32, 8, 2, 1 lanes 20, 29, 49, 61.
int wide_lanes(long long voxels, int num_sms) {
    int lanes = 1;
    while (lanes < 32 && 2 * lanes * voxels <= 2048LL * num_sms) lanes *= 2;
    return lanes;
}

// Bricks for lattices of at least 20,000 voxels (fewer are too few warps: 16^3
// over the middle of 250,000 points, 0.4 apart) while the brick's
// widened box is no more than 1.1 times a voxel's search block. Both sides
// measured over spacings of 0.15 to 14 world units, 20,000 to 4,000,000 points
// and both search blocks, bricks | lanes, us: gridSrch 2, 64^3 over 250,000
// points, 0.8 apart (0.5 times) 51 | 100; 128^3 over 4,000,000, 2.6 apart (1.3)
// 300 | 360, over 20,000 in a mostly empty box 39 | 38, 96^3, 3.5 apart (2.1)
// 232 | 216; gridSrch 3, 64^3, 0.15 apart (0.86) 41 | 38, 0.8 apart (1.8) 55 |
// 43, 256^3 over 4,000,000, 1.3 apart (2.8) 1,280 | 728.
constexpr long long kBrickVoxels = 20000;
bool sample_bricks(const DevParams &P, const Lattice &L) {
    const float h = sqrtf(P.rd2);
    const float dx = (L.bmax.x - L.bmin.x) / (float)L.res.x, dy = (L.bmax.y - L.bmin.y) / (float)L.res.y,
                dz = (L.bmax.z - L.bmin.z) / (float)L.res.z;
    const float box = (3.0f * fabsf(dx) + 2.0f * h) * (3.0f * fabsf(dy) + 2.0f * h) * (fabsf(dz) + 2.0f * h);
    const float side = (float)P.gridSrch;
    const float block = side * side * side * P.cellw.x * P.cellw.y * P.cellw.z;
    const float most = fmaxf(fmaxf(3.0f * fabsf(dx) / P.cellw.x, 3.0f * fabsf(dy) / P.cellw.y), fabsf(dz) / P.cellw.z);
    return (long long)L.res.x * L.res.y * L.res.z >= kBrickVoxels && box <= 1.1f * block && most < (float)kBrickCells;
}

}  // namespace

int fl_launch_sample_volume(fl_system *s, const int res[3], const float bmin[3], const float bmax[3],
                            float scalar, float gausskern, float h2, float *out) {
    Lattice L;
    L.res = make_int3(res[0], res[1], res[2]);
    L.bmin = make_float3(bmin[0], bmin[1], bmin[2]);
    L.bmax = make_float3(bmax[0], bmax[1], bmax[2]);
    L.scalar = scalar;
    L.kern = gausskern;
    const double c = -1.0 / (double)h2;
    L.c_hi = (float)c;
    L.c_lo = (float)(c - (double)L.c_hi);
    if (sample_bricks(s->D, L)) {
        const int3 bricks = make_int3((res[0] + 3) / 4, (res[1] + 3) / 4, (res[2] + 1) / 2);
        const long long n = (long long)bricks.x * bricks.y * bricks.z;
        // points whose supports fill a twentieth of the box at most
        const float box = fabsf((bmax[0] - bmin[0]) * (bmax[1] - bmin[1]) * (bmax[2] - bmin[2]));
        auto kern = 20.0f * (float)s->n * s->D.rd2 * sqrtf(s->D.rd2) < box ? k_sample_bricks<true> : k_sample_bricks<false>;
        kern<<<blocks_for(n, kVolumeThreads / 32), kVolumeThreads, 0, s->stream>>>(
            s->D, L, bricks, s->f[F_POS].cur<float4>(), s->f[F_GCELL].cur<uint32_t>(), s->off, out);
    } else {
        const long long n = (long long)res[0] * res[1] * res[2];
        auto wide = [&](auto lanes) {
            constexpr int kLanes = decltype(lanes)::value;
            k_sample_wide<kLanes><<<blocks_for(n, kVolumeThreads / kLanes), kVolumeThreads, 0, s->stream>>>(
                s->D, L, s->f[F_POS].cur<float4>(), s->off, out);
        };
        switch (wide_lanes(n, s->num_sms)) {
        case 1: wide(std::integral_constant<int, 1>()); break;
        case 2: wide(std::integral_constant<int, 2>()); break;
        case 4: wide(std::integral_constant<int, 4>()); break;
        case 8: wide(std::integral_constant<int, 8>()); break;
        case 16: wide(std::integral_constant<int, 16>()); break;
        default: wide(std::integral_constant<int, 32>());
        }
    }
    FL_LAUNCH_CHECK("sample_volume");
    return FL_OK;
}
