// ss_fuse.cuh — the per-voxel observation and running-average update of
// integrate / deintegrate, shared by the per-frame fuse kernel (ss_grid.cu)
// and the batched re-fusion (ss_refuse.cu), so that a batched re-fusion gives
// bit for bit the volume of the sequential calls.
#pragma once

#include "ss_internal.cuh"

namespace ss {

// The pixel a voxel projects to (getCoordinate, GPUVoxelGrid.h:234-237, and the
// reference's (int) cast, GPUVoxelGrid.cpp:348-349, which picks the pixel half
// a pixel off the projection), in the reference's arithmetic.
static __device__ __noinline__ int project_axis(float p, float f, float z, float c) {
    return __float2int_rz(__fadd_rn(__fdiv_rn(__fmul_rn(p, f), z), c));
}

// The same for two voxels with the quotients from approximate reciprocals (1 ulp)
// where those decide the pixels: an approximate coordinate a and the
// reference's lie within 3 u |p f / z| + 2 u |a| of each other (u = 2^-24; |p f
// / z| <= |a| + |c| and its roundings), below 4e-7 (|a| + |c|), so where a is
// further than 4e-7 (res + 2 + |c|) = 0.5 - decide from every integer they
// truncate alike, or, past res + 2, both lie outside the image. The floor
// comes from an addition of 1.5 2^23 rounded down, and from it the cast, which
// for a negative non-integer is one more; past 2^22 the low bits are a number
// outside any image too. Elsewhere (one coordinate in a thousand at 640 x
// 480), and for infinities and NaN, the division decides: sure is false.
__device__ __forceinline__ float project_decide(int res, float c) {
    return 0.5f - 4.0e-7f * ((float)(res + 2) + fabsf(c));
}
__device__ __forceinline__ void project_axis_pair(f32x2 p, float f, f32x2 rz, float c, float decide, int &p0, int &p1,
                                                  bool &sure0, bool &sure1) {
    auto both = [](float v) { return f2_pack(v, v); };
    const f32x2 big = both(12582912.f);
    const f32x2 a = f2_fma(f2_mul(p, both(f)), rz, both(c)), s = f2_add_down(a, big);
    float s0, s1, t0, t1;
    f2_unpack(s, s0, s1);
    f2_unpack(f2_sub(f2_sub(a, f2_sub(s, big)), both(0.5f)), t0, t1);  // a - floor(a) - 0.5
    sure0 = sure0 && fabsf(t0) < decide;
    sure1 = sure1 && fabsf(t1) < decide;
    p0 = (int)(__float_as_uint(s0) - 0x4B400000u);
    p1 = (int)(__float_as_uint(s1) - 0x4B400000u);
    p0 += (int)((unsigned)p0 >> 31);
    p1 += (int)((unsigned)p1 >> 31);
}

// The observation of integrationCore[Color]Tag / deIntegrationCore[Color]Tag
// (GPUVoxelGrid.cpp:345-469, 516-550) of a lane's four voxels (rows r0 .. r0 +
// 3 of the block at pz: voxel (k, l0 + 4 (r & 1), r >> 1) at row r) in the
// reference's arithmetic: whether a voxel changes, its pixel and observed sdf.
// Voxels 0 and 1, then 2 and 3 go through paired instructions (the same
// roundings), which with the floors in place of conversions took a fusion of
// FP16 517 x 389 from 17 to 15.4 us and a batched re-fusion 10 % of its time.
// The four depth gathers are in flight together.
__device__ __forceinline__ void quad_observe_exact(const GridView &g, const uint16_t *__restrict__ depth, const Mat34 &E,
                                                   const Mat34 &Einv, const F3 &Ez, F3 vm0, F3 pz, int l0, int r0,
                                                   float obs[4], bool ok[4], int pix[4]) {
    auto both = [](float v) { return f2_pack(v, v); };
    const float di = project_decide(g.resi, g.in.ci), dj = project_decide(g.resj, g.in.cj);
    // the voxels' centres: (vm0.x, y[rr & 1], z[rr >> 1])
    const float y[2] = {vm0.y, __fmaf_rn((float)(l0 + 4) + 0.5f, g.vl, pz.y)};
    const float z[2] = {vm0.z, __fmaf_rn((float)((r0 >> 1) + 1) + 0.5f, g.vl, pz.z)};
    F3 q[4];
    int i[4], j[4];
    bool sure[4] = {true, true, true, true};
#pragma unroll
    for (int h = 0; h < 2; h++) {
        F3 &q0 = q[2 * h], &q1 = q[2 * h + 1];
        q0 = xform(Einv, F3{vm0.x, y[0], z[h]});
        q1 = xform(Einv, F3{vm0.x, y[1], z[h]});
        float r0, r1;
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r0) : "f"(q0.z));
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r1) : "f"(q1.z));
        const f32x2 rz = f2_pack(r0, r1);
        project_axis_pair(f2_pack(q0.y, q1.y), g.in.fy, rz, g.in.ci, di, i[2 * h], i[2 * h + 1], sure[2 * h],
                          sure[2 * h + 1]);
        project_axis_pair(f2_pack(q0.x, q1.x), g.in.fx, rz, g.in.cj, dj, j[2 * h], j[2 * h + 1], sure[2 * h],
                          sure[2 * h + 1]);
    }
    if (!(sure[0] && sure[1] && sure[2] && sure[3])) {
#pragma unroll
        for (int rr = 0; rr < 4; rr++)
            if (!sure[rr]) {
                i[rr] = project_axis(q[rr].y, g.in.fy, q[rr].z, g.in.ci);
                j[rr] = project_axis(q[rr].x, g.in.fx, q[rr].z, g.in.cj);
            }
    }
    // -0: the products that feed sums keep their own rounding
    const f32x2 nz = both(__fmul_rn(g.vl, -0.f));
    uint16_t d[4];
    float u[4], v[4];
#pragma unroll
    for (int rr = 0; rr < 4; rr++) {
        ok[rr] = (unsigned)i[rr] < (unsigned)g.resi && (unsigned)j[rr] < (unsigned)g.resj;
        pix[rr] = i[rr] * g.resj + j[rr];
        d[rr] = ok[rr] ? __ldg(depth + pix[rr]) : (uint16_t)0;
        u[rr] = ok[rr] ? __ldg(g.ray_u + j[rr]) : 0.f;
        v[rr] = ok[rr] ? __ldg(g.ray_v + i[rr]) : 0.f;
    }
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int a = 2 * h, b = 2 * h + 1;
        const f32x2 dm = depth_m_pair(d[a], d[b]);
        // getPoint from the grid's quotients
        const f32x2 px = f2_mul(f2_pack(u[a], u[b]), dm), py = f2_mul(f2_pack(v[a], v[b]), dm);
        auto row = [&](int k) {
            return f2_add(f2_add(f2_add(f2_fma(px, both(E.m[k]), nz), f2_fma(py, both(E.m[k + 1]), nz)),
                                 f2_fma(dm, both(E.m[k + 2]), nz)),
                          both(E.m[k + 3]));
        };
        const f32x2 ox = f2_fma(f2_sub(row(0), both(vm0.x)), both(Ez.x), nz);
        const f32x2 oy = f2_fma(f2_sub(row(4), f2_pack(y[0], y[1])), both(Ez.y), nz);
        const f32x2 oz = f2_fma(f2_sub(row(8), both(z[h])), both(Ez.z), nz);
        f2_unpack(f2_add(f2_add(ox, oy), oz), obs[a], obs[b]);
        float d0, d1;
        f2_unpack(dm, d0, d1);
        ok[a] = ok[a] && d0 > g.rmin && fabsf(obs[a]) < g.trunc;
        ok[b] = ok[b] && d1 > g.rmin && fabsf(obs[b]) < g.trunc;
    }
}

// The fast path's observation of a voxel whose pixel holds `depth`: d > rmin,
// and the projective sdf d - q.z within the truncation (q = Einv vm): for a
// rigid E, (E p - vm) . Ez with p the pixel's point at depth d is d - q.z, the
// distance along the camera axis (a voxel behind the camera gets d + |q.z| >
// trunc).
// Two voxels at once, in paired instructions.
__device__ __forceinline__ void observe_fast(const GridView &g, uint16_t depth0, uint16_t depth1, f32x2 qz, f32x2 &sdf,
                                             bool &ok0, bool &ok1) {
    // (float)depth: 2^23 + depth, the 2^23 taken off again
    const f32x2 mm = f2_sub(f2_pack(__uint_as_float(0x4B000000u | depth0), __uint_as_float(0x4B000000u | depth1)),
                            f2_pack(8388608.f, 8388608.f));
    const f32x2 k = f2_pack(1.0e-3f, 1.0e-3f);
    float d0, d1, s0, s1;
    const f32x2 d = f2_mul(mm, k);
    f2_unpack(d, d0, d1);
    sdf = f2_sub(d, qz);
    f2_unpack(sdf, s0, s1);
    ok0 = ok0 && d0 > g.rmin && fabsf(s0) < g.trunc;
    ok1 = ok1 && d1 > g.rmin && fabsf(s1) < g.trunc;
}

// The fast path's observation of a lane's four voxels r0 .. r0 + 3 (r0 even:
// voxel (l0, m0) at vm0, then (l0 + 4, m0), (l0, m0 + 1), (l0 + 4, m0 + 1)).
// Camera-frame points: Einv vm0 and, for the others, the transformed voxel
// steps (ystep: 4 vl along y, zstep: vl along z, from fast_steps) added with
// rounded operations that are never contracted. Pixels: the nearest (the
// reference's truncation picks the pixel half a pixel off the projection, which
// makes frame-to-model tracking drift), with the half pixel of the rounding
// folded into the principal point and the projection from an approximate
// reciprocal (the pixel choice only needs it to ~1 ulp); the floors come from
// additions of 1.5 2^23 rounded down:
// an integer below 2^22 in the sum's low bits, and for everything else
// (infinities and NaN too) a number outside any image. Voxels 0 and 1, then 2
// and 3 go through paired instructions (the same roundings); the four gathers
// are in flight together, and no branch comes before they have arrived. The
// per-frame fusion and the batched re-fusion share it (bit for bit the same
// volume).
__device__ __forceinline__ void quad_observe_fast(const GridView &g, const uint16_t *__restrict__ depth,
                                                  const Mat34 &Einv, const float ystep[3],
                                                  const float zstep[3], F3 vm0, f32x2 obs[2], bool ok[4], int pix[4]) {
    const float ax = fmaf(vm0.x, Einv.m[0], fmaf(vm0.y, Einv.m[1], fmaf(vm0.z, Einv.m[2], Einv.m[3])));
    const float ay = fmaf(vm0.x, Einv.m[4], fmaf(vm0.y, Einv.m[5], fmaf(vm0.z, Einv.m[6], Einv.m[7])));
    const float az = fmaf(vm0.x, Einv.m[8], fmaf(vm0.y, Einv.m[9], fmaf(vm0.z, Einv.m[10], Einv.m[11])));
    auto both = [](float v) { return f2_pack(v, v); };
    auto pair = [](float v, float ystep) { return f2_pack(v, __fadd_rn(v, ystep)); };
    // voxels (0, 1) and (2, 3)
    const f32x2 x[2] = {pair(ax, ystep[0]), pair(__fadd_rn(ax, zstep[0]), ystep[0])};
    const f32x2 y[2] = {pair(ay, ystep[1]), pair(__fadd_rn(ay, zstep[1]), ystep[1])};
    const f32x2 z[2] = {pair(az, ystep[2]), pair(__fadd_rn(az, zstep[2]), ystep[2])};
    uint16_t d[4];
#pragma unroll
    for (int h = 0; h < 2; h++) {
        float qz[2], r[2], fi[2], fj[2];
        f2_unpack(z[h], qz[0], qz[1]);
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r[0]) : "f"(qz[0]));
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r[1]) : "f"(qz[1]));
        const f32x2 rz = f2_pack(r[0], r[1]), big = both(12582912.f);
        f2_unpack(f2_add_down(f2_fma(f2_mul(y[h], both(g.in.fy)), rz, both(g.in.ci + 0.5f)), big), fi[0], fi[1]);
        f2_unpack(f2_add_down(f2_fma(f2_mul(x[h], both(g.in.fx)), rz, both(g.in.cj + 0.5f)), big), fj[0], fj[1]);
#pragma unroll
        for (int u = 0; u < 2; u++) {
            const unsigned i = __float_as_uint(fi[u]) - 0x4B400000u, j = __float_as_uint(fj[u]) - 0x4B400000u;
            const int rr = 2 * h + u;
            pix[rr] = (int)(i * (unsigned)g.resj + j);
            ok[rr] = i < (unsigned)g.resi && j < (unsigned)g.resj;
            d[rr] = ok[rr] ? __ldg(depth + pix[rr]) : (uint16_t)0;
        }
    }
#pragma unroll
    for (int h = 0; h < 2; h++) observe_fast(g, d[2 * h], d[2 * h + 1], z[h], obs[h], ok[2 * h], ok[2 * h + 1]);
}

// x / y for a weight y (1 .. 2^24): x times the approximate reciprocal, as
// __fdividef gives it there without its steps for denormal and huge y.
__device__ __forceinline__ float div_weight(float x, float y) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(y));
    return x * r;
}

// Running-average update of one voxel (sdf, weight) in FP32.
template <bool kDeint, bool kExact>
__device__ __forceinline__ void running_average(float &s, float &w, float obs, float max_weight) {
    if (!kDeint) {
        const float w1 = kExact ? __fadd_rn(w, 1.f) : w + 1.f;
        s = kExact ? __fdiv_rn(__fadd_rn(__fmul_rn(s, w), obs), w1) : div_weight(fmaf(s, w, obs), w1);
        w = (max_weight > 0.f && w1 > max_weight) ? max_weight : w1;
    } else {
        if (w != 1.f) {
            const float w1 = kExact ? __fsub_rn(w, 1.f) : w - 1.f;
            s = kExact ? __fdiv_rn(__fsub_rn(__fmul_rn(s, w), obs), w1) : div_weight(fmaf(s, w, -obs), w1);
            w = w1;
        } else {
            w = 0.f;
            s = 0.f;
        }
    }
}

// min(w, cap) for a weight; a NaN, which only an imported volume holds, stays
// one, as under running_average's comparison.
__device__ __forceinline__ float cap_weight(float w, float cap) {
    float r;
    asm("min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(w), "f"(cap));
    return r;
}

// The fast update of two voxels at once (the same roundings), weights capped.
template <bool kDeint, int kStorage>
__device__ __forceinline__ void running_average_pair(float &s0, float &s1, float &w0, float &w1, f32x2 obs, bool ok0,
                                                     bool ok1, float cap, float trunc, float inv_trunc) {
    const f32x2 w = f2_pack(w0, w1), one = f2_pack(1.f, 1.f);
    const f32x2 v = kDeint ? f2_sub(w, one) : f2_add(w, one);
    float v0, v1, r0, r1, a0, a1;
    f2_unpack(v, v0, v1);
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r0) : "f"(v0));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r1) : "f"(v1));
    const f32x2 a = f2_mul(f2_fma(f2_pack(s0, s1), w, kDeint ? f2_neg(obs) : obs), f2_pack(r0, r1));
    if (kStorage == SS_STORAGE_F16) {  // the value a sequential call would have stored
        f2_unpack(f2_mul(a, f2_pack(inv_trunc, inv_trunc)), a0, a1);
        const float2 h = __half22float2(__floats2half2_rn(a0, a1));
        f2_unpack(f2_mul(f2_pack(h.x, h.y), f2_pack(trunc, trunc)), a0, a1);
    } else {
        f2_unpack(a, a0, a1);
    }
    if (ok0) {
        s0 = kDeint && v0 == 0.f ? 0.f : a0;
        w0 = kDeint ? v0 : cap_weight(v0, cap);
    }
    if (ok1) {
        s1 = kDeint && v1 == 0.f ? 0.f : a1;
        w1 = kDeint ? v1 : cap_weight(v1, cap);
    }
}

template <bool kDeint, bool kExact>
__device__ __forceinline__ void color_average(float &c, float w_old, float obs) {
    if (!kDeint) {
        c = kExact ? __fdiv_rn(__fadd_rn(__fmul_rn(c, w_old), obs), __fadd_rn(w_old, 1.f))
                   : __fdividef(fmaf(c, w_old, obs), w_old + 1.f);
    } else {
        if (w_old != 1.f) {
            c = kExact ? __fdiv_rn(__fsub_rn(__fmul_rn(c, w_old), obs), __fsub_rn(w_old, 1.f))
                       : __fdividef(fmaf(c, w_old, -obs), w_old - 1.f);
        } else {
            c = 0.f;
        }
    }
}

}  // namespace ss
