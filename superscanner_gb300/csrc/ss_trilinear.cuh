// ss_trilinear.cuh — trilinear TSDF sampling and the model-view ray march,
// shared by the raycast (ss_raycast.cu) and its adjoint (ss_raydiff.cu).
#pragma once

#include <climits>

#include "ss_internal.cuh"

namespace ss {

struct TriSample {
    bool valid;
    float f;
    float gx, gy, gz;  // d f / d (world x, y, z)
};

struct BlockCache {
    // this thread's column of a shared-memory table: at [m * stride] the bucket
    // of the block at offset m (bits 1 x, 2 y, 4 z) from a cell's lowest block
    // (cell_finds; eight registers picked by comparisons cost a turn of its
    // loop more than the find)
    int *tab;
    int stride;  // threads of the CTA
    int x = INT_MIN, y = INT_MIN, z = INT_MIN, bucket = -1;  // the last block looked up
    unsigned lookups = 0u;  // hash-table finds issued (cache misses)
    unsigned voxels = 0u;   // voxel words loaded
    __device__ __forceinline__ BlockCache(int *table, int tid, int threads) : tab(table + tid), stride(threads) {}
    // the last sampled cell (its lowest voxel) and its 8 corner values
    int cx = INT_MIN, cy = INT_MIN, cz = INT_MIN;
    bool cok = false;
    float cs[8];
};

template <int kStorage>
__device__ __forceinline__ float2 voxel_sw(const GridView &g, int bucket, int v) {
    const size_t vi = (size_t)bucket * kBlockVoxels + v;
    if (kStorage == SS_STORAGE_F32) {
        return __ldg(g.vox32 + vi);
    } else {
        const uint32_t word = __ldg(g.vox16 + vi);
        return make_float2(__half2float(__ushort_as_half((unsigned short)(word & 0xffffu))) * g.trunc,
                           (float)(word >> 16));
    }
}

// Whether the voxel is observed (its weight positive).
template <int kStorage>
__device__ __forceinline__ bool voxel_seen(const GridView &g, int bucket, int v) {
    const size_t vi = (size_t)bucket * kBlockVoxels + v;
    return kStorage == SS_STORAGE_F32 ? __ldg(&g.vox32[vi].y) > 0.f : __ldg(g.vox16 + vi) > 0xFFFFu;
}

template <bool kSplit = false>
__device__ __forceinline__ int cached_lookup(const GridView &g, BlockCache &c, int bx, int by, int bz) {
    if (bx == c.x && by == c.y && bz == c.z) return c.bucket;
    c.x = bx;
    c.y = by;
    c.z = bz;
    c.lookups++;
    c.bucket = !packable(bx, by, bz) ? -1
               : kSplit              ? table_find_split(g, prime_hash(bx, by, bz))
                                     : table_find(g, prime_hash(bx, by, bz));
    return c.bucket;
}

// Uncached find of a neighbouring block (counted as a lookup).
__device__ __forceinline__ int block_find(const GridView &g, BlockCache &c, int bx, int by, int bz) {
    c.lookups++;
    return packable(bx, by, bz) ? table_find(g, prime_hash(bx, by, bz)) : -1;
}

// The axes along which the cell with lowest voxel (ix, iy, iz) straddles a
// block face, as bits 1 (x), 2 (y), 4 (z): corner k = a + 2 b + 4 c lies in the
// block at offset bits k & cell_straddle from the cell's lowest block.
__device__ __forceinline__ int cell_straddle(int ix, int iy, int iz) {
    return ((ix & 7) == 7 ? 1 : 0) | ((iy & 7) == 7 ? 2 : 0) | ((iz & 7) == 7 ? 4 : 0);
}

// The buckets of a cell's blocks into the table (corner k's block at offset k &
// straddle), the lowest one's being `base`; false where one is missing. A
// straddling cell's further blocks (1, 3 or 7) are
// found one a turn, each lane its own next one: lanes that straddle along
// different axes share the turns (a branch per block cost a warp all seven).
__device__ __forceinline__ bool cell_finds(const GridView &g, int base, int ix, int iy, int iz, int straddle,
                                           BlockCache &c) {
    c.tab[0] = base;
    bool ok = true;
    int m = (0 - straddle) & straddle;  // the first non-empty subset of the straddled axes
    while (m) {
        const int b = block_find(g, c, (ix >> 3) + (m & 1), (iy >> 3) + ((m >> 1) & 1), (iz >> 3) + (m >> 2));
        c.tab[m * c.stride] = b;
        ok &= b >= 0;
        m = ok ? (m - straddle) & straddle : 0;  // the next subset
    }
    return ok;
}

// The bucket of corner k's block, after cell_finds.
__device__ __forceinline__ int cell_bucket(const BlockCache &c, int straddle, int k) {
    return c.tab[(k & straddle) * c.stride];
}

// The voxel of corner k in its block.
__device__ __forceinline__ int cell_voxel(int ix, int iy, int iz, int k) {
    const int vx = ix + (k & 1), vy = iy + ((k >> 1) & 1), vz = iz + (k >> 2);
    return (vx & 7) + 8 * (vy & 7) + 64 * (vz & 7);
}

// The cell's 8 corner values; false where a corner is missing or unobserved.
// The last cell's are kept. One code path for cells in one block and cells
// that straddle, so that the corner loads of a warp whose lanes hold both
// kinds are issued together.
template <int kStorage>
__device__ __forceinline__ bool cell_corners(const GridView &g, int ix, int iy, int iz, BlockCache &c, float *s) {
    if (ix == c.cx && iy == c.cy && iz == c.cz) {  // same cell as the last sample: its corners again
        if (!c.cok) return false;
#pragma unroll
        for (int k = 0; k < 8; k++) s[k] = c.cs[k];
        return true;
    }
    c.cx = ix, c.cy = iy, c.cz = iz, c.cok = false;
    const int base = cached_lookup(g, c, ix >> 3, iy >> 3, iz >> 3);
    const int straddle = cell_straddle(ix, iy, iz);
    if (base < 0 || !cell_finds(g, base, ix, iy, iz, straddle, c)) return false;
    bool ok = true;
    float2 sw[8];
#pragma unroll
    for (int k = 0; k < 8; k++) sw[k] = voxel_sw<kStorage>(g, cell_bucket(c, straddle, k), cell_voxel(ix, iy, iz, k));
    c.voxels += 8;
#pragma unroll
    for (int k = 0; k < 8; k++) {
        ok &= sw[k].y > 0.f;
        s[k] = sw[k].x;
        c.cs[k] = s[k];
    }
    c.cok = ok;
    return ok;
}

template <int kStorage, bool kGrad>
__device__ __forceinline__ TriSample trilinear(const GridView &g, float px, float py, float pz, float inv_vl,
                                               BlockCache &c) {
    TriSample r{false, 0.f, 0.f, 0.f, 0.f};
    const float ux = fmaf(px, inv_vl, -0.5f), uy = fmaf(py, inv_vl, -0.5f), uz = fmaf(pz, inv_vl, -0.5f);
    const float fx0 = floorf(ux), fy0 = floorf(uy), fz0 = floorf(uz);
    const float ax = ux - fx0, ay = uy - fy0, az = uz - fz0;
    float s[8];
    if (!cell_corners<kStorage>(g, (int)fx0, (int)fy0, (int)fz0, c, s)) return r;
    // lerp along x, then y, then z
    const float s00 = fmaf(ax, s[1] - s[0], s[0]), s10 = fmaf(ax, s[3] - s[2], s[2]);
    const float s01 = fmaf(ax, s[5] - s[4], s[4]), s11 = fmaf(ax, s[7] - s[6], s[6]);
    const float s0 = fmaf(ay, s10 - s00, s00), s1 = fmaf(ay, s11 - s01, s01);
    r.valid = true;
    r.f = fmaf(az, s1 - s0, s0);
    if (kGrad) {
        const float dx00 = s[1] - s[0], dx10 = s[3] - s[2], dx01 = s[5] - s[4], dx11 = s[7] - s[6];
        const float dx0 = fmaf(ay, dx10 - dx00, dx00), dx1 = fmaf(ay, dx11 - dx01, dx01);
        r.gx = fmaf(az, dx1 - dx0, dx0) * inv_vl;
        r.gy = fmaf(az, s11 - s01 - (s10 - s00), s10 - s00) * inv_vl;
        r.gz = (s1 - s0) * inv_vl;
    }
    return r;
}

// Regula falsi on a bracket (ta, fa > 0) .. (tb, fb < 0) of the trilinear
// field along the ray: two refinements, then the secant root.
template <int kStorage>
__device__ __forceinline__ float refine_crossing(const GridView &g, float ox, float oy, float oz, float dx, float dy,
                                                 float dz, float ta, float fa, float tb, float fb, BlockCache &cache) {
    const float inv_vl = 1.f / g.vl;
    bool ok = true;
#pragma unroll 1
    for (int r = 0; r < 2; r++) {
        const float tc = ta + (tb - ta) * fa / (fa - fb);
        if (ok) {
            const TriSample q =
                trilinear<kStorage, false>(g, fmaf(tc, dx, ox), fmaf(tc, dy, oy), fmaf(tc, dz, oz), inv_vl, cache);
            ok = q.valid;
            if (ok && q.f > 0.f) {
                ta = tc;
                fa = q.f;
            } else if (ok) {
                tb = tc;
                fb = q.f;
            }
        }
    }
    return ta + (tb - ta) * fa / (fa - fb);
}

constexpr int kRayForward = 0;  // march forward from t0 to t_hi
constexpr int kRaySeek = 1;     // search near a depth hint t0 within [t_lo, t_hi]

// Ray search, one loop with one trilinear sample per iteration for every
// mode, so lanes of a warp in different modes still share the sampling code:
//  forward: in a super-block without allocated blocks, or a block that is not
//    allocated, jump to the exit of its box; an invalid sample (unobserved
//    corner) advances one voxel; a positive one advances max(vl, 0.8 f); a
//    negative one after a positive one brackets the crossing, a negative one
//    without a positive predecessor is a back face (no hit);
//  seek (window [t_lo, t_hi]): one sample at the hint t0; unobserved: no
//    hit; positive: forward from there to t_hi (that sample is the
//    predecessor); negative:
//  back: steps back by max(vl, 0.8 |f|) until a positive sample brackets the
//    crossing (an unobserved sample, or passing t_lo, first: no hit).
// Forward marching ends at t_hi. Every sample or skip counts as one step. A
// bracket is refined by two regula-falsi steps, then the secant root is the
// hit (t).
// Four of five samples of a forward march from the camera are invalid, in runs
// of one-voxel steps. With kAhead a turn first tells, each by one voxel, which
// of the next kAhead points are: a cell's corner nearest to the camera is the
// last to be observed. Only where that corner and the point lie in the block
// of this turn; the other points are sampled as ever. Two points: 200 -> 191
// us (640 x 480, 4 mm), 169 -> 158 (517 x 389, 6 mm); one 170, three 162, six
// 195.
template <int kStorage, int kAhead = 0>
__device__ __forceinline__ bool ray_search(const GridView &g, float ox, float oy, float oz, float dx, float dy,
                                           float dz, float inv_len, int mode, float t0, float t_lo, float t_hi,
                                           int max_steps, int &steps, float &t, BlockCache &cache) {
    constexpr int kBack = 2;
    const float vl = g.vl, inv_vl = 1.f / g.vl, inv_vbl = 1.f / g.vbl;
    const float rdx = 1.f / dx, rdy = 1.f / dy, rdz = 1.f / dz;
    const float sbl = g.vbl * (float)(1 << kSuperShift);
    t = t0;
    bool prev_valid = false, found = false;
    float t_prev = 0.f, f_prev = 0.f;  // forward: last valid sample; back: last (negative) sample
    float ta = 0.f, fa = 0.f, tb = 0.f, fb = 0.f;  // bracket: f(ta) > 0 > f(tb)
    int csx = INT_MIN, csy = INT_MIN, csz = INT_MIN;
    bool cocc = false;
    // one condition ends the loop and no branch inside leaves it: lanes that
    // took such a branch's other side (a skip instead of a sample) would rejoin
    // their warp only behind the loop
    bool go = steps < max_steps && (mode != kRayForward || t < t_hi);
    while (go) {
        float px = fmaf(t, dx, ox), py = fmaf(t, dy, oy), pz = fmaf(t, dz, oz);
        steps++;
        bool skip = false;
        if (mode == kRayForward) {
            const int bx = (int)floorf(px * inv_vbl), by = (int)floorf(py * inv_vbl), bz = (int)floorf(pz * inv_vbl);
            const int sx = bx >> kSuperShift, sy = by >> kSuperShift, sz = bz >> kSuperShift;
            if (sx != csx || sy != csy || sz != csz) {
                csx = sx;
                csy = sy;
                csz = sz;
                cocc = kAhead > 0 ? super_occupied_split(g, sx, sy, sz) : super_occupied(g, sx, sy, sz);
                cache.lookups++;
            }
            const bool empty_super = !cocc;
            skip = empty_super || cached_lookup<(kAhead > 0)>(g, cache, bx, by, bz) < 0;
            if (skip) {
                // exit of the empty super-block's (or block's) box along the ray
                const float box = empty_super ? sbl : g.vbl;
                const int cx = empty_super ? sx : bx, cy = empty_super ? sy : by, cz = empty_super ? sz : bz;
                const float ex = ((float)(cx + (dx > 0.f)) * box - ox) * rdx;
                const float ey = ((float)(cy + (dy > 0.f)) * box - oy) * rdy;
                const float ez = ((float)(cz + (dz > 0.f)) * box - oz) * rdz;
                const float te = fminf(fminf(dx != 0.f ? ex : INFINITY, dy != 0.f ? ey : INFINITY),
                                       dz != 0.f ? ez : INFINITY);
                t = fmaxf(te, t) + 1e-4f * vl * inv_len;
                prev_valid = false;
            }
        }
        if (kAhead > 0 && !skip && mode == kRayForward) {
            float at[kAhead + 1];  // t after so many invalid samples
            bool unseen[kAhead + 1];
            at[0] = t;
            const int bx = floor_int(px * inv_vbl), by = floor_int(py * inv_vbl), bz = floor_int(pz * inv_vbl);
            const int nx = dx > 0.f ? 0 : 1, ny = dy > 0.f ? 0 : 1, nz = dz > 0.f ? 0 : 1;  // the nearest corner
#pragma unroll
            for (int m = 0; m < kAhead; m++) {
                const float x = fmaf(at[m], dx, ox), y = fmaf(at[m], dy, oy), z = fmaf(at[m], dz, oz);
                const int vx = floor_int(fmaf(x, inv_vl, -0.5f)) + nx, vy = floor_int(fmaf(y, inv_vl, -0.5f)) + ny,
                          vz = floor_int(fmaf(z, inv_vl, -0.5f)) + nz;
                unseen[m] = at[m] < t_hi && (vx >> 3) == bx && (vy >> 3) == by && (vz >> 3) == bz &&
                            floor_int(x * inv_vbl) == bx && floor_int(y * inv_vbl) == by && floor_int(z * inv_vbl) == bz;
                if (unseen[m])  // cache.bucket: the block's, looked up above
                    unseen[m] = !voxel_seen<kStorage>(g, cache.bucket, (vx & 7) + 8 * (vy & 7) + 64 * (vz & 7));
                at[m + 1] = fmaf(vl, inv_len, at[m]);
            }
            steps--;  // counted point by point from here
            bool run = true;
#pragma unroll
            for (int m = 0; m < kAhead; m++) {
                run = run && unseen[m] && steps < max_steps;
                if (run) {
                    steps++;
                    t = at[m + 1];
                    prev_valid = false;
                }
            }
            skip = run || !(steps < max_steps && t < t_hi);
            if (!skip) {
                px = fmaf(t, dx, ox), py = fmaf(t, dy, oy), pz = fmaf(t, dz, oz);
                // a point past the block takes a turn of its own
                skip = !(floor_int(px * inv_vbl) == bx && floor_int(py * inv_vbl) == by && floor_int(pz * inv_vbl) == bz);
                if (!skip) steps++;
            }
        }
        bool end = false;
        if (!skip) {
            const TriSample sm = trilinear<kStorage, false>(g, px, py, pz, inv_vl, cache);
            const bool neg = sm.f < 0.f, pos = sm.f > 0.f;
            const float step = fmaxf(vl, 0.8f * fabsf(sm.f));  // of a valid sample, in metres
            if (mode == kRayForward) {
                if (!sm.valid) {
                    prev_valid = false;
                    t = fmaf(vl, inv_len, t);
                } else if (neg) {
                    found = prev_valid && f_prev > 0.f;  // else a back face
                    ta = t_prev;
                    fa = f_prev;
                    tb = t;
                    fb = sm.f;
                    end = true;
                } else {
                    prev_valid = true;
                    t_prev = t;
                    f_prev = sm.f;
                    t = fmaf(step, inv_len, t);
                }
            } else if (!sm.valid) {
                end = true;  // unobserved at the hint (a gap in the band) or on the way back: no hit
            } else if (mode == kRaySeek && sm.f >= 0.f) {
                t_prev = t;
                f_prev = sm.f;
                mode = kRayForward;
                prev_valid = true;
                // a valid sample's corner blocks exist, so the super-block of its
                // point is occupied: the first forward step needs no probe for it
                // (should rounding put the point in a neighbouring block, the march
                // only falls back from a super-block skip to a block skip)
                csx = (int)floorf(px * inv_vbl) >> kSuperShift;
                csy = (int)floorf(py * inv_vbl) >> kSuperShift;
                csz = (int)floorf(pz * inv_vbl) >> kSuperShift;
                cocc = true;
                t = fmaf(step, inv_len, t);
            } else if (mode == kBack && pos) {
                found = true;
                ta = t;
                fa = sm.f;
                tb = t_prev;
                fb = f_prev;
                end = true;
            } else {  // back from a sample behind the surface
                mode = kBack;
                t_prev = t;
                f_prev = sm.f;
                t = fmaf(-step, inv_len, t);
                end = t < t_lo;
            }
        }
        go = !end && steps < max_steps && (mode != kRayForward || t < t_hi);
    }
    if (found) t = refine_crossing<kStorage>(g, ox, oy, oz, dx, dy, dz, ta, fa, tb, fb, cache);
    return found;
}

// One forward ray march from t0 to t_max; returns true on a zero crossing (t = hit depth).
template <int kStorage, int kAhead = 0>
__device__ __forceinline__ bool march(const GridView &g, float ox, float oy, float oz, float dx, float dy, float dz,
                                      float inv_len, float t0, float t_max, int max_steps, int &steps, float &t,
                                      BlockCache &cache) {
    return ray_search<kStorage, kAhead>(g, ox, oy, oz, dx, dy, dz, inv_len, kRayForward, t0, t0, t_max, max_steps, steps,
                                        t, cache);
}

}  // namespace ss
