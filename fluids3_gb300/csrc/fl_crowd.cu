// The force (and advance) of tiles with a point whose pairs overflowed its
// list (computeForce and advanceParticles, fluids4.0/fluid_kernels.cu:180-217,
// 332-420): the force pass lists them and leaves them to this kernel, a
// block per tile at a time (fl_crowd.cuh). The candidates are walked again and
// every term is the reference's, added in its order, so forces are the
// per-point pass's bit for bit.
//
// What it replaced: the overflowed points walked their blocks by themselves,
// a dependent load and a divergent pair a time, while the other lanes of
// their warp waited. Force and advance of a dam break as it collapses:
// 32,768 points after 64 steps (0.9% of the points overflow) 223 -> 77 us,
// after 100 steps (25%, up to 748 pairs) 585 -> 134 us; 65,536 points after
// 160 steps (36%, up to 4,967 pairs) 3,340 -> 570 us. 64% of the issue slots are
// used there; the rest is the first warp's chain of additions and the waits on it.
#include <algorithm>

#include "fl_internal.h"

namespace {

#include "fl_device.cuh"
#include "fl_step.cuh"
#include "fl_crowd.cuh"

constexpr int kCrowdThreads = 512;   // (256: 5-20% slower; 128: half as fast)
constexpr int kCrowdSlots = 8;       // candidates a warp and round
// From this many tiles a multiprocessor in a class (twice as many of the packed
// ones, which differ more), a warp takes each by itself: nothing is lost to the
// adding warp and the waits on it, and there is work for every warp. Force +
// advance, dam break of 1,048,576 points after 110 and 170 steps, shared | alone:
// 1,562 | 944, 12,711 | 7,775 us; of 131,072 after 170 steps (a line at 8 a
// multiprocessor) 2,640 | 5,978 us.
constexpr uint32_t kAloneTiles = 16;
constexpr int kAloneThreads = 128, kAloneBlocksPerSm = 6;
struct ForceShared {               // per warp
    float4 cand[kCrowdSlots][2];              // pair records; the slot in the second's w
    float term[2][kCrowdSlots][3][32];        // per candidate, component and point
    int kept[2];
    int pad[2];
};
static_assert(sizeof(ForceShared) % 16 == 0, "the warps' records stay aligned");

struct ForceArgs {
    CrowdTiles tiles;            // its counters are zero again at the end
    const float *time_dev;       // this step's time
    float dt;
    const float4 *pos_in, *veval_in;
    const float *press;
    const uint32_t *gcell, *off;
    const float4 *pairdata;
    float4 *vel, *force, *pos_out, *veval_out;
    float *host_pos;
    uint32_t *err;
    int moved;                   // the positions are not the sorted ones: no box test
};

// Point i's data, and its results.
__device__ __forceinline__ ForcePoint crowd_point(const DevParams &P, int i, bool active, const ForceArgs &a) {
    ForcePoint fp;
    fp.p = fp.vi = make_float4(0.f, 0.f, 0.f, 0.f);
    fp.di = 1.0f;
    fp.pi = 0.0f;
    fp.f = make_float3(0.f, 0.f, 0.f);
    if (active) {
        fp.p = a.pos_in[i];
        fp.vi = a.veval_in[i];
        fp.di = a.press[i];
        fp.pi = (fp.di - P.prest_dens) * P.pintstiff;
    }
    return fp;
}

template <bool ADVANCE>
__device__ __forceinline__ void finish_point(const DevParams &P, int i, bool active, const ForcePoint &fp,
                                             const ForceArgs &a) {
    if (ADVANCE)
        store_step(P, a.time_dev[0], a.dt, i, active, fp, a.vel, a.force, a.pos_out, a.veval_out, a.err, a.host_pos,
                   a.veval_in);
    else
        a.force[i] = f4(fp.f);
}

template <bool BATCH, bool ADVANCE>
__device__ __forceinline__ void crowded_tile(const DevParams &P0, const SceneTab &T, uint32_t tile, int n,
                                             const ForceArgs &a, ForceShared *s_sh) {
    const unsigned lane = lane_id();
    const int warp = (int)(threadIdx.x >> 5);
    ForceShared &own_sh = s_sh[warp];
    const int i = (int)(tile * 32u + lane);
    const uint32_t gc = (i < n) ? a.gcell[i] : kUndef;
    const bool active = gc != kUndef;
    const DevParams &P = (BATCH && i < n) ? T.params[T.point_scene[i]] : P0;
    ForcePoint fp = crowd_point(P, i, active, a);
    const float4 *const records = after_wait(a.pairdata);
    struct Record {
        float4 q, v;
    };
    const unsigned act = __ballot_sync(0xffffffffu, active);
    unsigned heads = segment_heads(gc, active);
    while (heads) {
        const unsigned seg = next_segment(heads, act);
        const DevParams &PS = BATCH ? T.params[T.point_scene[i - (int)lane + __ffs(seg) - 1]] : P0;
        const Box box = box_of(fp.p, seg);
        const float bx = box.ex + PS.band, by = box.ey + PS.band, bz = box.ez + PS.band;
        crowd_segment<kCrowdSlots>(
            PS, seg, gc, a.off,
            [&](bool ok, uint32_t j) {
                Record d = {make_float4(0.f, 0.f, 0.f, 1.f), make_float4(0.f, 0.f, 0.f, 0.f)};
                if (ok) load_record(records, j, d.q, d.v);
                return d;
            },
            [&](const Record &d) {
                return a.moved || (fabsf(d.q.x - box.ox) <= bx && fabsf(d.q.y - box.oy) <= by && fabsf(d.q.z - box.oz) <= bz);
            },
            [&](int, int e, uint32_t j, const Record &d) {
                own_sh.cand[e][0] = d.q;
                own_sh.cand[e][1] = make_float4(d.v.x, d.v.y, d.v.z, __uint_as_float(j));
            },
            [&](int buf, int kept, RowRange own) {
                for (int e = 0; e < kept; e++) {
                    const float4 q = own_sh.cand[e][0], v = own_sh.cand[e][1];
                    const float dx = fp.p.x - q.x, dy = fp.p.y - q.y, dz = fp.p.z - q.z;
                    const float dsq = dx * dx + dy * dy + dz * dz;
                    const bool hit = dsq < PS.rd2 && dsq > 0.0f && __float_as_uint(v.w) - own.lo < own.len;
                    float3 t = make_float3(0.f, 0.f, 0.f);
                    if (__any_sync(0xffffffffu, hit)) t = pair_term(PS, fp.p, fp.pi, fp.vi, fp.di, q, v, q.w);
                    own_sh.term[buf][e][0][lane] = hit ? t.x : 0.0f;
                    own_sh.term[buf][e][1][lane] = hit ? t.y : 0.0f;
                    own_sh.term[buf][e][2][lane] = hit ? t.z : 0.0f;
                }
                for (int e = kept; e & 3; e++)   // whole groups of four
                    own_sh.term[buf][e][0][lane] = own_sh.term[buf][e][1][lane] = own_sh.term[buf][e][2][lane] = 0.0f;
                if (lane == 0) own_sh.kept[buf] = kept;
            },
            [&](int buf, int w) {
                // a miss adds +0.0, which leaves the sum's bits unchanged (a
                // sum that starts at +0.0 never becomes -0.0)
                const ForceShared &sh = s_sh[w + 1];
                const int kept = sh.kept[buf];
                for (int e = 0; e < kept; e += 4) {
                    float t[4][3];
#pragma unroll
                    for (int u = 0; u < 4; u++)
#pragma unroll
                        for (int k = 0; k < 3; k++) t[u][k] = sh.term[buf][e + u][k][lane];
#pragma unroll
                    for (int u = 0; u < 4; u++) {
                        fp.f.x += t[u][0];
                        fp.f.y += t[u][1];
                        fp.f.z += t[u][2];
                    }
                }
            });
    }
    if (warp == 0 && i < n) finish_point<ADVANCE>(P, i, active, fp, a);
}

// The same by one warp, for when there are tiles for every warp: it stages 32
// candidates a time, marks each lane's pairs among them and adds their terms
// as it goes, without the shared terms, the adding warp and the waits on it.
struct AloneShared {               // per warp
    float4 cand[64][2];            // a ring of pair records; the slot in the second's w
};

template <bool BATCH, bool ADVANCE>
__device__ __forceinline__ void crowded_tile_alone(const DevParams &P0, const SceneTab &T, uint32_t tile, int n,
                                                   const ForceArgs &a, AloneShared &sh) {
    const unsigned lane = lane_id(), below = (1u << lane) - 1u;
    const int i = (int)(tile * 32u + lane);
    const uint32_t gc = (i < n) ? a.gcell[i] : kUndef;
    const bool active = gc != kUndef;
    const DevParams &P = (BATCH && i < n) ? T.params[T.point_scene[i]] : P0;
    ForcePoint fp = crowd_point(P, i, active, a);
    const unsigned act = __ballot_sync(0xffffffffu, active);
    unsigned heads = segment_heads(gc, active);
    while (heads) {
        const unsigned seg = next_segment(heads, act);
        const bool mine = (seg >> lane) & 1u;
        const int first = __ffs(seg) - 1, last = 31 - __clz(seg);
        const DevParams &PS = BATCH ? T.params[T.point_scene[i - (int)lane + first]] : P0;
        const int ca = (int)__shfl_sync(0xffffffffu, gc, first), cb = (int)__shfl_sync(0xffffffffu, gc, last);
        const Box box = box_of(fp.p, seg);
        const float bx = box.ex + PS.band, by = box.ey + PS.band, bz = box.ez + PS.band;
        const int rows = PS.gridSrch * PS.gridSrch;
        const float rd2 = PS.rd2;
        RowRange own = {0u, 0xffffffffu};
        uint32_t head = 0, staged = 0;
        auto drain = [&](uint32_t count) {
            __syncwarp();
            uint32_t m = 0;
            if (mine) {
#pragma unroll 4
                for (uint32_t e = 0; e < count; e++) {
                    const float4 *c = sh.cand[(head + e) & 63u];
                    const float4 q = c[0];
                    const float dx = fp.p.x - q.x, dy = fp.p.y - q.y, dz = fp.p.z - q.z;
                    const float dsq = dx * dx + dy * dy + dz * dz;
                    const bool hit = dsq < rd2 && dsq > 0.0f && __float_as_uint(c[1].w) - own.lo < own.len;
                    m |= (hit ? 1u : 0u) << e;
                }
            }
            while (m) {
                const float4 *c = sh.cand[(head + (uint32_t)__ffs(m) - 1u) & 63u];
                m &= m - 1u;
                add_pair_terms(PS, fp, c[0], c[1], c[0].w);
            }
            head += count;
            __syncwarp();
        };
        for (int r = 0; r < rows; r++) {
            const int at = PS.adj[r * PS.gridSrch] - PS.nadj;
            const uint32_t lo = a.off[ca + at], hi = a.off[cb + at + PS.gridSrch];
            if (ca != cb && mine) {   // points of several cells: each takes its own block's candidates
                own.lo = a.off[(int)gc + at];
                own.len = a.off[(int)gc + at + PS.gridSrch] - own.lo;
            }
            for (uint32_t jb = lo; jb < hi; jb += 32u) {
                const uint32_t j = jb + lane;
                bool keep = j < hi;
                float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
                if (keep) q = a.pairdata[2 * (size_t)j];
                keep = keep && (a.moved || (fabsf(q.x - box.ox) <= bx && fabsf(q.y - box.oy) <= by && fabsf(q.z - box.oz) <= bz));
                const unsigned kept = __ballot_sync(0xffffffffu, keep);
                if (keep) {
                    const float4 v = a.pairdata[2 * (size_t)j + 1];
                    float4 *c = sh.cand[(staged + __popc(kept & below)) & 63u];
                    c[0] = q;
                    c[1] = make_float4(v.x, v.y, v.z, __uint_as_float(j));
                }
                staged += __popc(kept);
                if (staged - head >= 32u) drain(32u);
            }
            if (ca != cb && staged > head) drain(staged - head);   // the next row has other ranges
        }
        if (staged > head) drain(staged - head);
    }
    if (i < n) finish_point<ADVANCE>(P, i, active, fp, a);
}

// Clears the lists once every block has read them: the last one to sign off.
__device__ __forceinline__ void sign_off(const CrowdTiles &t) {
    if (threadIdx.x != 0) return;
    __threadfence();
    if (atomicAdd(&t.counters[4], 1u) == gridDim.x - 1)
        for (int k = 0; k < 5; k++) t.counters[k] = 0;
}

// The tiles of the classes with few (below), a block per tile. `ends`: no
// k_force_alone follows.
template <bool BATCH, bool ADVANCE>
__global__ void __launch_bounds__(kCrowdThreads, BATCH ? 2 : 0)
k_force_crowd(const __grid_constant__ DevParams P0, const SceneTab T, int n, const __grid_constant__ ForceArgs a,
              uint32_t line, bool ends) {
    follow_previous();
    extern __shared__ __align__(16) uint8_t s_dyn[];
    __shared__ uint32_t s_next;
    volatile uint32_t *const counters = a.tiles.counters;
    const uint32_t crowded = counters[0], packed = counters[1];
    if (crowded + packed == 0) return;
    const uint32_t first = packed < 2 * line ? packed : 0u, count = first + (crowded < line ? crowded : 0u);
    for (;;) {
        if (threadIdx.x == 0) s_next = atomicAdd(&a.tiles.counters[2], 1u);
        __syncthreads();
        const uint32_t k = s_next;
        __syncthreads();
        if (k >= count) break;
        crowded_tile<BATCH, ADVANCE>(P0, T, tile_at(a.tiles, k, first), n, a, reinterpret_cast<ForceShared *>(s_dyn));
    }
    if (ends) sign_off(a.tiles);
}

// The other classes' tiles, a warp per tile.
template <bool BATCH, bool ADVANCE>
__global__ void __launch_bounds__(kAloneThreads)
k_force_alone(const __grid_constant__ DevParams P0, const SceneTab T, int n, const __grid_constant__ ForceArgs a,
              uint32_t line) {
    follow_previous();
    __shared__ AloneShared s_sh[kAloneThreads / 32];
    volatile uint32_t *const counters = a.tiles.counters;
    const uint32_t crowded = counters[0], packed = counters[1];
    if (crowded + packed == 0) return;
    const uint32_t first = packed < 2 * line ? 0u : packed, count = first + (crowded < line ? 0u : crowded);
    for (;;) {
        uint32_t k = 0;
        if (lane_id() == 0) k = atomicAdd(&a.tiles.counters[3], 1u);
        k = __shfl_sync(0xffffffffu, k, 0);
        if (k >= count) break;
        crowded_tile_alone<BATCH, ADVANCE>(P0, T, tile_at(a.tiles, k, first), n, a, s_sh[threadIdx.x >> 5]);
    }
    __syncthreads();
    sign_off(a.tiles);
}

constexpr size_t kCrowdSmem = (kCrowdThreads / 32) * sizeof(ForceShared);

}  // namespace

int fl_crowd_init() {
    const int most = (int)kCrowdSmem;
    FL_CUDA_TRY(cudaFuncSetAttribute(k_force_crowd<false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
    FL_CUDA_TRY(cudaFuncSetAttribute(k_force_crowd<false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
    FL_CUDA_TRY(cudaFuncSetAttribute(k_force_crowd<true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
    FL_CUDA_TRY(cudaFuncSetAttribute(k_force_crowd<true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
    return FL_OK;
}

int fl_launch_force_crowd(fl_system *s, bool advance, float dt, float *host_pos) {
    ForceArgs a = {};
    a.tiles = s->over_tiles;
    a.time_dev = s->time_dev + s->time_slot;
    a.dt = dt;
    a.pos_in = s->f[F_POS].cur<float4>();
    a.veval_in = s->f[F_VEVAL].cur<float4>();
    a.press = s->f[F_PRESS].cur<float>();
    a.gcell = s->f[F_GCELL].cur<uint32_t>();
    a.off = s->off;
    a.pairdata = s->pairdata;
    a.vel = s->f[F_VEL].cur<float4>();
    a.force = s->f[F_FORCE].cur<float4>();
    a.pos_out = s->f[F_POS].nxt<float4>();
    a.veval_out = s->f[F_VEVAL].nxt<float4>();
    a.host_pos = host_pos;
    a.err = s->dev_err;
    a.moved = !s->codes_valid;
    const int tiles = (s->n + 31) / 32;
    const uint32_t line = kAloneTiles * (uint32_t)s->num_sms;
    const bool ends = (uint32_t)tiles < line;   // too few points for a class of that many tiles
    auto kern = advance ? (s->batched ? k_force_crowd<true, true> : k_force_crowd<false, true>)
                        : (s->batched ? k_force_crowd<true, false> : k_force_crowd<false, false>);
    launch(kern, std::min(2 * s->num_sms, tiles), kCrowdThreads, kCrowdSmem, s->stream, s->D, fl_scene_tab(s), s->n,
           a, line, ends);
    if (!ends) {
        auto alone = advance ? (s->batched ? k_force_alone<true, true> : k_force_alone<false, true>)
                             : (s->batched ? k_force_alone<true, false> : k_force_alone<false, false>);
        launch(alone, kAloneBlocksPerSm * s->num_sms, kAloneThreads, 0, s->stream, s->D, fl_scene_tab(s), s->n, a,
               line);
    }
    FL_LAUNCH_CHECK("force_crowd");
    return FL_OK;
}
