// Per-point arithmetic of the step shared by the neighbour passes
// (fl_kernels.cu, fl_density.cu, fl_crowd.cu): packed FP32 helpers, one
// pair's force term and the advance of one point, each in the reference
// kernels' own operation order. Included inside each file's anonymous
// namespace; the files are compiled without FMA contraction, so every
// expression rounds as written.
#pragma once

// ---- packed f32x2 arithmetic (round-to-nearest per element) ---------------
// Each packed operation rounds exactly like its scalar form, but ptxas
// contracts a packed add of two packed products into a packed fused
// multiply-add (measured on GB300, explicit .rn and --fmad=false
// notwithstanding): packed products are added in scalar.
__device__ __forceinline__ uint64_t pk2(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void up2(uint64_t v, float &a, float &b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ uint64_t sub2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}


// A pair record -- (position, density), (evaluated velocity, 0) -- in one
// 256-bit load: with two 128-bit ones the force pass waited on twice the
// requests (1,000,000 points 94 -> 87 us, 250,000 with gridSrch 3 88 -> 73).
// To the compiler the load is a function of its address, free to move (volatile,
// the batched force pass took 56 -> 60 registers and 120 -> 138 us): pairdata
// has to be a pointer got after the wait (after_wait), and no kernel that calls
// this writes the records.
__device__ __forceinline__ void load_record(const float4 *__restrict__ pairdata, uint32_t j, float4 &q, float4 &v) {
    asm("ld.global.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
        : "=f"(q.x), "=f"(q.y), "=f"(q.z), "=f"(q.w), "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
        : "l"(pairdata + 2 * (size_t)j));
}

// The parameters of a pair's force, for a kernel to hold (a batched one would
// read them through the scene table for every pair).
struct PairForceParams {
    float d2, prest_dens, pintstiff, psmoothradius, sim_scale, spikykern, vterm;
    __device__ explicit PairForceParams(const DevParams &P)
        : d2(P.d2), prest_dens(P.prest_dens), pintstiff(P.pintstiff), psmoothradius(P.psmoothradius),
          sim_scale(P.sim_scale), spikykern(P.spikykern), vterm(P.vterm) {}
};

struct ForcePoint {
    float4 p, vi;
    float di, pi;
    float3 f;
};

// One pair's force term on a point at p (pressure term pi, evaluated
// velocity vi, density di) from the neighbour's position q, evaluated
// velocity vj and density dj, in the reference's operation order
// (fluid_kernels.cu:203-210); the pair is known to pass 0 < d^2 < rd2. The
// point's force is the sum of its terms, added component-wise in the
// reference's pair order.
// (Params: DevParams or PairForceParams.)
template <class Params>
__device__ __forceinline__ float3 pair_term(const Params &P, float4 p, float pi, float4 vi, float di, float4 q,
                                            float4 vj, float dj) {
    const float dx = p.x - q.x, dy = p.y - q.y, dz = p.z - q.z;
    const float dsq = dx * dx + dy * dy + dz * dz;
    const float r = sqrtf(dsq * P.d2);
    const float pj = (dj - P.prest_dens) * P.pintstiff;
    const float cr = P.psmoothradius - r;
    const float pterm = P.sim_scale * -0.5f * cr * P.spikykern * (pi + pj) / r;
    const float sx = dx * pterm + (vj.x - vi.x) * P.vterm;
    const float sy = dy * pterm + (vj.y - vi.y) * P.vterm;
    const float sz = dz * pterm + (vj.z - vi.z) * P.vterm;
    const float inv = 1.0f / (di * dj);
    return make_float3((sx * cr) * inv, (sy * cr) * inv, (sz * cr) * inv);
}

__device__ __forceinline__ void add_pair_terms(const DevParams &P, ForcePoint &fp, float4 q, float4 vj,
                                               float dj) {
    const float3 t = pair_term(P, fp.p, fp.pi, fp.vi, fp.di, q, vj, dj);
    fp.f.x += t.x;
    fp.f.y += t.y;
    fp.f.z += t.z;
}

// advanceParticles body (fluids4.0/fluid_kernels.cu:343-419) for an
// in-range point: walls, gravity, limits, leapfrog. `accel` enters as the
// SPH force; returns the new position, velocity and evaluated velocity.
__device__ __forceinline__ void advance_point(const DevParams &P, float time, float dt, float ss,
                                              float3 accel, float3 pos, float3 vel, float3 veval,
                                              float3 &pos_o, float3 &vel_o, float3 &veval_o) {
    accel.x *= P.pmass; accel.y *= P.pmass; accel.z *= P.pmass;
    float diff, adj;
    // Y- wall with slope (cu:356-361)
    diff = P.pradius - (pos.y - (P.bound_min.y + (pos.x - P.bound_min.x) * P.bound_slope)) * ss;
    if (diff > kEpsilon) {
        float3 nrm = make_float3(-P.bound_slope, 1.0f - P.bound_slope, 0.0f);
        adj = P.bound_stiff * diff - P.bound_damp * (nrm.x * veval.x + nrm.y * veval.y + nrm.z * veval.z);
        nrm.x *= adj; nrm.y *= adj; nrm.z *= adj;
        accel.x += nrm.x - veval.x * P.bound_friction;
        accel.y += nrm.y - veval.y * P.bound_friction;
        accel.z += nrm.z - veval.z * P.bound_friction;
    }
    // Y+ (cu:363-368)
    diff = P.pradius - (P.bound_max.y - pos.y) * ss;
    if (diff > kEpsilon) {
        float3 nrm = make_float3(0.0f, -1.0f, 0.0f);
        adj = P.bound_stiff * diff - P.bound_damp * (nrm.x * veval.x + nrm.y * veval.y + nrm.z * veval.z);
        nrm.x *= adj; nrm.y *= adj; nrm.z *= adj;
        accel.x += nrm.x - veval.x * P.bound_friction;
        accel.y += nrm.y - veval.y * P.bound_friction;
        accel.z += nrm.z - veval.z * P.bound_friction;
    }
    // X- moving wall (cu:371-377): stiffness scaled by the wall term. The
    // reference forms `sin(..) * 0.5 + 0.5` and the amplitude product with
    // double literals, so the product is formed in double and rounded once
    // to float, as there (three FP64 operations per point).
    const float wall = (float)(((double)sinf(time * P.bound_wall_freq + pos.z / 400.f) * 0.5 + 0.5) *
                               (double)P.bound_wall_force);
    diff = P.pradius - (pos.x - (P.bound_min.x + wall)) * ss;
    if (diff > kEpsilon) {
        float3 nrm = make_float3(1.0f, 0.0f, 0.0f);
        adj = wall * P.bound_stiff * diff - P.bound_damp * (nrm.x * veval.x + nrm.y * veval.y + nrm.z * veval.z);
        accel.x += nrm.x * adj; accel.y += nrm.y * adj; accel.z += nrm.z * adj;
    }
    // X+ (cu:378-383)
    diff = P.pradius - (P.bound_max.x - pos.x) * ss;
    if (diff > kEpsilon) {
        float3 nrm = make_float3(-1.0f, 0.0f, 0.0f);
        adj = P.bound_stiff * diff - P.bound_damp * (nrm.x * veval.x + nrm.y * veval.y + nrm.z * veval.z);
        accel.x += nrm.x * adj; accel.y += nrm.y * adj; accel.z += nrm.z * adj;
    }
    // Z- (cu:386-391)
    diff = P.pradius - (pos.z - P.bound_min.z) * ss;
    if (diff > kEpsilon) {
        float3 nrm = make_float3(0.0f, 0.0f, 1.0f);
        adj = P.bound_stiff * diff - P.bound_damp * (nrm.x * veval.x + nrm.y * veval.y + nrm.z * veval.z);
        accel.x += nrm.x * adj; accel.y += nrm.y * adj; accel.z += nrm.z * adj;
    }
    // Z+ (cu:392-397)
    diff = P.pradius - (P.bound_max.z - pos.z) * ss;
    if (diff > kEpsilon) {
        float3 nrm = make_float3(0.0f, 0.0f, -1.0f);
        adj = P.bound_stiff * diff - P.bound_damp * (nrm.x * veval.x + nrm.y * veval.y + nrm.z * veval.z);
        accel.x += nrm.x * adj; accel.y += nrm.y * adj; accel.z += nrm.z * adj;
    }
    accel.x += P.gravity.x; accel.y += P.gravity.y; accel.z += P.gravity.z;
    // accel limit (cu:403-406)
    float speed = accel.x * accel.x + accel.y * accel.y + accel.z * accel.z;
    if (speed > P.AL2) {
        const float k = P.AL / sqrtf(speed);
        accel.x *= k; accel.y *= k; accel.z *= k;
    }
    // velocity limit (cu:409-413)
    speed = vel.x * vel.x + vel.y * vel.y + vel.z * vel.z;
    if (speed > P.VL2) {
        const float k = P.VL / sqrtf(speed);
        vel.x *= k; vel.y *= k; vel.z *= k;
    }
    // leapfrog (cu:416-419)
    const float3 vnext = make_float3(accel.x * dt + vel.x, accel.y * dt + vel.y, accel.z * dt + vel.z);
    veval_o = make_float3((vel.x + vnext.x) * 0.5f, (vel.y + vnext.y) * 0.5f, (vel.z + vnext.z) * 0.5f);
    vel_o = vnext;
    const float dts = dt / ss;
    pos_o = make_float3(pos.x + vnext.x * dts, pos.y + vnext.y * dts, pos.z + vnext.z * dts);
}

// The end of the fused step for point i from its force: the force, then walls,
// limits and leapfrog (or, out of range, parked at (-1000, -1000, -1000) with
// zero velocity, cu:339-342). host_pos (fl_run_from_host) also gets the new
// position, packed float x3.
__device__ __forceinline__ void store_step(const DevParams &P, float time, float dt, int i, bool active,
                                           const ForcePoint &fp, float4 *__restrict__ vel, float4 *__restrict__ force,
                                           float4 *__restrict__ pos_out, float4 *__restrict__ veval_out,
                                           uint32_t *__restrict__ err, float *__restrict__ host_pos,
                                           const float4 *__restrict__ veval_in) {
    float3 po = make_float3(-1000.f, -1000.f, -1000.f), vo = make_float3(0.f, 0.f, 0.f);
    if (active) {
        force[i] = f4(fp.f);
        float3 eo;
        advance_point(P, time, dt, P.sim_scale, fp.f, xyz(fp.p), xyz(vel[i]), xyz(fp.vi), po, vo, eo);
        if (!(isfinite(po.x) && isfinite(po.y) && isfinite(po.z))) atomicOr(err, FL_DEV_NONFINITE);
        veval_out[i] = f4(eo);
    } else {
        force[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        veval_out[i] = veval_in[i];
    }
    pos_out[i] = f4(po);
    vel[i] = f4(vo);
    if (host_pos) {
        host_pos[3 * (size_t)i] = po.x;
        host_pos[3 * (size_t)i + 1] = po.y;
        host_pos[3 * (size_t)i + 2] = po.z;
    }
}
