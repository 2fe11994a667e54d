// A crowded tile (32 consecutive sorted slots whose search blocks hold many
// points) taken by a whole block. Included inside each file's anonymous
// namespace, after fl_device.cuh.
//
// A point's sum is one chain of additions in the reference's pair order, but
// its terms do not depend on one another. So every warp but the first
// evaluates terms (a lane per point, a run of candidates per warp) into
// shared memory, and the first warp adds them, a lane per point, in order,
// while the others evaluate the next candidates. A tile that one warp would
// walk for hundreds of microseconds is shared by all warps of a block, and
// tiles go to whichever block is free.
#pragma once

// Puts a tile on its class's list (one lane calls it).
__device__ __forceinline__ void list_tile(const CrowdTiles &t, uint32_t tile, bool packed) {
    const uint32_t k = atomicAdd(&t.counters[packed ? 1 : 0], 1u);
    t.list[packed ? t.room - 1u - k : k] = tile;
}

// The k-th of `packed` packed tiles followed by the crowded ones.
__device__ __forceinline__ uint32_t tile_at(const CrowdTiles &t, uint32_t k, uint32_t packed) {
    return t.list[k < packed ? t.room - 1u - k : k - packed];
}

// The lane's search-block row: slots [lo, lo + len).
struct RowRange {
    uint32_t lo, len;
};

// Runs of the tile's points that share a walk: consecutive points at most two
// cells apart, in 16 cells. The first cells of a row and the last ones hold no
// points (at least gridSrch + 1 >= 3 of them between two rows or scenes), so
// such points lie in one row of cells. Returns the lanes that begin a run.
__device__ __forceinline__ unsigned segment_heads(uint32_t gc, bool active) {
    const uint32_t prev = __shfl_up_sync(0xffffffffu, active ? gc : kUndef, 1);
    const bool head = active && (lane_id() == 0 || prev == kUndef || gc - prev > 2u || (gc >> 4) != (prev >> 4));
    return __ballot_sync(0xffffffffu, head);
}

// The next run of `heads` (removed from it), as a lane mask.
__device__ __forceinline__ unsigned next_segment(unsigned &heads, unsigned act) {
    const int h0 = __ffs(heads) - 1;
    heads &= heads - 1u;
    const unsigned upto = heads ? (1u << (__ffs(heads) - 1)) - 1u : 0xffffffffu;
    return act & upto & (0xffffffffu << h0);
}

// Centre and half extent of the box of the lanes in `seg`.
struct Box {
    float ox, oy, oz, ex, ey, ez;
};
__device__ __forceinline__ float warp_min(float v) {
    float r;
    asm("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ float warp_max(float v) {
    float r;
    asm("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ Box box_of(float4 p, unsigned seg) {
    const int first = __ffs(seg) - 1;
    const bool mine = (seg >> lane_id()) & 1u;
    const float px = __shfl_sync(0xffffffffu, p.x, first), py = __shfl_sync(0xffffffffu, p.y, first),
                pz = __shfl_sync(0xffffffffu, p.z, first);
    const float vx = mine ? p.x : px, vy = mine ? p.y : py, vz = mine ? p.z : pz;
    const float lx = warp_min(vx), ux = warp_max(vx), ly = warp_min(vy), uy = warp_max(vy), lz = warp_min(vz),
                uz = warp_max(vz);
    Box b;
    b.ox = 0.5f * (lx + ux), b.oy = 0.5f * (ly + uy), b.oz = 0.5f * (lz + uz);
    b.ex = fmaxf(ux - b.ox, b.ox - lx), b.ey = fmaxf(uy - b.oy, b.oy - ly), b.ez = fmaxf(uz - b.oz, b.oz - lz);
    return b;
}

// The candidates of the points in `seg` in the reference's order, PER slots a
// warp and round. All threads of the block call it with the same points.
//   load(ok, j)                 candidate j's data (anything unless ok)
//   near(d)                     whether the box test keeps it
//   put(buf, e, j, d)           candidate e of this warp's round, into shared memory
//   eval(buf, kept, range)      this warp's terms of its candidates; a point takes those in range
//   add(buf, w)                 (first warp) warp w's terms of the round, in order
template <int PER, class Load, class Near, class Put, class Eval, class Add>
__device__ __forceinline__ void crowd_segment(const DevParams &P, unsigned seg, uint32_t gc,
                                              const uint32_t *__restrict__ off, Load load, Near near, Put put,
                                              Eval eval, Add add) {
    const int W = (int)(blockDim.x >> 5), warp = (int)(threadIdx.x >> 5);
    const int evals = W > 1 ? W - 1 : 1, me = W > 1 ? warp - 1 : 0;   // one warp alone does both
    const unsigned lane = lane_id();
    const bool mine = (seg >> lane) & 1u;
    const int first = __ffs(seg) - 1, last = 31 - __clz(seg);
    const int ca = (int)__shfl_sync(0xffffffffu, gc, first), cb = (int)__shfl_sync(0xffffffffu, gc, last);
    const int srch = P.gridSrch;
    int buf = 0;
    for (int r = 0; r < srch * srch; r++) {
        const int at = P.adj[r * srch] - P.nadj;
        const uint32_t lo = off[ca + at], hi = off[cb + at + srch];
        RowRange own = {0u, 0u};
        if (mine) {
            own.lo = off[(int)gc + at];
            own.len = off[(int)gc + at + srch] - own.lo;
        }
        const uint32_t step = (uint32_t)(evals * PER);
        uint32_t j = lo + (uint32_t)(me * PER) + lane;
        const bool loader = me >= 0 && lane < (unsigned)PER;
        auto d = load(loader && j < hi, j);
        for (uint32_t jb = lo; jb < hi; jb += step) {
            if (me >= 0) {
                const bool keep = loader && j < hi && near(d);
                const unsigned kept = __ballot_sync(0xffffffffu, keep);
                if (keep) put(buf, __popc(kept & ((1u << lane) - 1u)), j, d);
                j += step;
                d = load(loader && j < hi, j);
                __syncwarp();
                eval(buf, __popc(kept), own);
                __syncwarp();
            }
            __syncthreads();
            if (warp == 0)
                for (int w = 0; w < evals; w++) add(buf, w);
            buf ^= 1;
        }
    }
    __syncthreads();
}
