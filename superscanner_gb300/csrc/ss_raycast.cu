// ss_raycast.cu — reference-semantics raycast (raycastingTag,
// src/VoxelGrid/GPUVoxelGrid.cpp:561-715) and its C-ABI entry point.
//
// One thread per pixel, 32x8 pixel tiles, each warp an 8 x 4 patch of
// neighbouring rays, which stay coherent through the block-skip loop. The unit ray
// table normPcd (createNormPcdTag, :717-722) is recomputed in registers
// instead of being read from a 3.7 MB image.
#include <climits>

#include "ss_grid_impl.cuh"
#include "ss_trilinear.cuh"

namespace ss {

constexpr int kRaycastIterCap = 1 << 20;  // far above the d_max / min-stride bound

struct VoxelRead {
    float sdf, w;
};

template <int kStorage>
__device__ __forceinline__ VoxelRead read_voxel(const GridView &g, int bucket, int v) {
    const size_t vi = (size_t)bucket * kBlockVoxels + v;
    if (kStorage == SS_STORAGE_F32) {
        const float2 sw = __ldg(g.vox32 + vi);
        return {sw.x, sw.y};
    } else {
        const uint32_t word = __ldg(g.vox16 + vi);
        return {__half2float(__ushort_as_half((unsigned short)(word & 0xffffu))) * g.trunc, (float)(word >> 16)};
    }
}

// floor(q) and |q - rint(q)| of q = RN(p rlen), the nearest integer by adding
// 1.5 2^23 (its low bits) and taking it off again: FP32 additions, whose
// latency a march of dependent steps sees, instead of two conversions (the
// block collection, bound by its instructions, keeps the conversions). From
// 2^22 on, where the nearest integer is off, the callers' margins exceed the
// distance it can show.
__device__ __forceinline__ float floor_and_distance(float p, float rlen, float &q, int &out) {
    q = __fmul_rn(p, rlen);
    const float t = __fadd_rn(q, 12582912.f), d = __fsub_rn(q, __fsub_rn(t, 12582912.f));
    out = __float_as_int(t) - 0x4B400000 + (__float_as_int(d) >> 31);
    return fabsf(d);
}

// idx_rule(a, len) by idx_fast's test (rlen = RN(1 / len)); false where that is
// not decisive.
__device__ __forceinline__ bool idx_sure(float a, float rlen, int &out) {
    float q;
    const float d = floor_and_distance(a, rlen, q, out);
    return d > __fmaf_rn(fabsf(q), 3.0e-7f, 3.0e-7f);
}
__device__ __forceinline__ int idx_rule_fast(float a, float len, float rlen) {
    int o;
    return idx_sure(a, rlen, o) ? o : idx_rule(a, len);
}

// The rare ways are functions of their own behind one branch each, and what can
// be selected is selected: a step's time is its chain of instructions and
// branches, each of which parts a warp and rejoins it (with the voxel loop's and
// the table finds' likewise 140 -> 125 us with colour and 132 -> 117 without at
// 640 x 480, 92 -> 80 at 517 x 389, 56 -> 48 at 160 x 120).
static __device__ __noinline__ int3 idx_slow(float px, float py, float pz, float len) {
    return make_int3(idx_rule(px, len), idx_rule(py, len), idx_rule(pz, len));
}

// getVBIndeces (GPUVoxelGrid.h:162-189): the index rule of each coordinate
// (by multiplication where that is provably the IEEE quotient's result).
__device__ __forceinline__ void block_of(const GridView &g, F3 p, int &bx, int &by, int &bz) {
    if (!(idx_sure(p.x, g.rvbl, bx) & idx_sure(p.y, g.rvbl, by) & idx_sure(p.z, g.rvbl, bz))) {
        const int3 b = idx_slow(p.x, p.y, p.z, g.vbl);
        bx = b.x;
        by = b.y;
        bz = b.z;
    }
}

// A voxel's place in its block of 512. Next to a block's face the reference's
// rules can give an axis 8 or -1 (at a negative multiple of the block's edge;
// where the point's distance to the face is lost in its rounding; one pixel of
// ten frames of a room), and so a place up to 73 voxels before the block or 72
// behind it, where the reference reads on in whatever lies there. The grid's
// arrays hold an empty block on either side (ss_grid_create), so such a read
// stays in them; an axis further out (a point too far from the origin for its
// block's voxels) takes its nearest voxel.
__device__ __forceinline__ int voxel_place(int vx, int vy, int vz) {
    const int v = (int)((unsigned)vx + kEdge * (unsigned)vy + kEdge * kEdge * (unsigned)vz);
    if (v >= -kBlockVoxels && v < 2 * kBlockVoxels) return v;
    auto in = [](int a) { return min(max(a, 0), kEdge - 1); };
    return in(vx) + kEdge * in(vy) + kEdge * kEdge * in(vz);
}

// getVinVBIndeces (GPUVoxelGrid.h:192-221): p - vbl * vbInd, then the index rule.
__device__ __forceinline__ int voxel_in_block(const GridView &g, F3 p, int bx, int by, int bz) {
    const F3 q = f3sub(p, F3{__fmul_rn(g.vbl, (float)bx), __fmul_rn(g.vbl, (float)by), __fmul_rn(g.vbl, (float)bz)});
    int vx, vy, vz;
    if (!(idx_sure(q.x, g.rvl, vx) & idx_sure(q.y, g.rvl, vy) & idx_sure(q.z, g.rvl, vz))) {
        const int3 v = idx_slow(q.x, q.y, q.z, g.vl);
        vx = v.x;
        vy = v.y;
        vz = v.z;
    }
    return voxel_place(vx, vy, vz);
}

// Block and voxel of a point at once (block_of, then voxel_in_block). With
// x = p / vl and x at least m = 6 u (|x| + 16) from every integer (u = 2^-24),
// both of the reference's rules see only floor(x): the block quotient x / 8
// lies m / 8 > 5 u (|x / 8| + 1) from every integer (idx_fast's bound), so its
// index is floor(x) >> 3; p - vbl * block, rounded, is off by at most
// u (|x| + 16) vl, so the voxel rule's quotient, within 5 u * 9 of it, truncates
// to floor(x) & 7. q = RN(p RN(1 / vl)) is within 3.02 u |x| of x, so the test
// asks q for 13 u |q| + 268 u. Elsewhere (one point in a thousand at 2 m and 4 mm
// voxels) the two rules decide one after the other.
__device__ __forceinline__ bool voxel_fast(float p, float rvl, int &out) {
    float q;
    const float d = floor_and_distance(p, rvl, q, out);
    return d > __fmaf_rn(fabsf(q), 8.0e-7f, 1.6e-5f);
}
static __device__ __noinline__ int4 voxel_slow(float px, float py, float pz, float vl, float rvl, float vbl, float rvbl) {
    const int bx = idx_rule_fast(px, vbl, rvbl), by = idx_rule_fast(py, vbl, rvbl), bz = idx_rule_fast(pz, vbl, rvbl);
    const F3 q = f3sub(F3{px, py, pz}, F3{__fmul_rn(vbl, (float)bx), __fmul_rn(vbl, (float)by), __fmul_rn(vbl, (float)bz)});
    const int vx = idx_rule_fast(q.x, vl, rvl), vy = idx_rule_fast(q.y, vl, rvl), vz = idx_rule_fast(q.z, vl, rvl);
    return make_int4(bx, by, bz, voxel_place(vx, vy, vz));
}
__device__ __forceinline__ int voxel_of(const GridView &g, F3 p, int &bx, int &by, int &bz) {
    int x, y, z;
    const bool sure = voxel_fast(p.x, g.rvl, x) & voxel_fast(p.y, g.rvl, y) & voxel_fast(p.z, g.rvl, z);
    bx = x >> 3;
    by = y >> 3;
    bz = z >> 3;
    int v = (x & 7) + kEdge * (y & 7) + kEdge * kEdge * (z & 7);
    if (!sure) {
        const int4 r = voxel_slow(p.x, p.y, p.z, g.vl, g.rvl, g.vbl, g.rvbl);
        bx = r.x;
        by = r.y;
        bz = r.z;
        v = r.w;
    }
    return v;
}

// getVoxelMidPoint (GPUVoxelGrid.h:274-278): vb*vbl (float) + (v + 0.5)*vl
// (double), rounded to float; the double sum is exact, so one fmaf matches.
__device__ __forceinline__ F3 voxel_mid(const GridView &g, int v, int bx, int by, int bz) {
    const int vx = v & 7, vy = (v >> 3) & 7, vz = v >> 6;
    return {__fmaf_rn((float)vx + 0.5f, g.vl, __fmul_rn((float)bx, g.vbl)),
            __fmaf_rn((float)vy + 0.5f, g.vl, __fmul_rn((float)by, g.vbl)),
            __fmaf_rn((float)vz + 0.5f, g.vl, __fmul_rn((float)bz, g.vbl))};
}

// Block finds of the reference raycast (UnorderedMap::find of the prime hash,
// GPUVoxelGrid.cpp:590-630). When `skip` holds, a block whose super-block
// holds no allocated block is known to be absent without a table probe: the
// super-block is looked up once per super-block the ray enters. That is exact
// only where no prime-hash collision can make another block answer the find
// (see raycast_ref_kernel).
struct SuperCache {
    int sx = INT_MIN, sy = INT_MIN, sz = INT_MIN;
    bool occ = false;
};

__device__ __forceinline__ int find_block(const GridView &g, int bx, int by, int bz, int &finds, bool skip,
                                          SuperCache &sc) {
    if (skip) {
        const int sx = bx >> kSuperShift, sy = by >> kSuperShift, sz = bz >> kSuperShift;
        if (sx != sc.sx || sy != sc.sy || sz != sc.sz) {
            sc.sx = sx;
            sc.sy = sy;
            sc.sz = sz;
            sc.occ = super_occupied_split(g, sx, sy, sz);
            finds++;
        }
        if (!sc.occ) return -1;
    }
    finds++;
    return table_find_split(g, prime_hash(bx, by, bz));
}

// The shortest difference between two block coordinates with the same prime
// hash (73856093 dx + 19349669 dy + 83492791 dz = 0 mod 2^32, dx, dy, dz not
// all zero) is 951 blocks along some axis (exhaustive search of |dx|, |dy| <=
// 3000 for the dz that solves it): blocks within 950 of each other along
// every axis never share a key.
constexpr int kHashCollisionFree = 950;

template <int kStorage>
__global__ void __launch_bounds__(256, 4) raycast_ref_kernel(GridView g, Mat34 Er, float *__restrict__ out_pcd,
                                                          float *__restrict__ out_col, int iter_cap,
                                                          int patch_shift) {
    // warp w marches a patch of (1 << patch_shift) x 4 pixels, 8 x 4 or, in a small
    // image, 4 x 4 on half its lanes: neighbouring rays in both directions take
    // more similar paths than a 32-pixel row segment (0.351 vs 0.388 ms per call
    // at 640 x 480)
    const int w = threadIdx.y, ln = threadIdx.x;
    const int j = (((blockIdx.x << 2) + (w & 3)) << patch_shift) + (ln & ((1 << patch_shift) - 1));
    const int i = blockIdx.y * blockDim.y + (w >> 2) * 4 + (ln >> patch_shift);
    if (ln >= (4 << patch_shift) || i >= g.resi || j >= g.resj) return;
    const float vl = g.vl, vbl = g.vbl, dtr = g.trunc, dmax = g.d_max;

    const F3 np = f3normalized(get_point(g.in, i, j, 1.0f));
    F3 rv = xform(Er, np);
    const F3 dir = f3sub(rv, F3{Er.m[3], Er.m[7], Er.m[11]});
    float l = 0.1f;
    rv = f3sub(rv, f3smul(__fsub_rn(1.f, l), dir));

    bool done = false, Fn = false, Lp = false;
    int guard = 0, finds = 0, voxels = 0;  // work counters: hash and super-block finds, voxel reads

    // Skip the table probe in empty super-blocks when this ray's blocks and
    // every allocated block (within the super-blocks' bounding box) lie within
    // the collision-free extent: then a find answers only for the block itself.
    bool skip = false;
    {
        const int lo0 = __ldcg(&g.ctr->sb_lo[0]), lo1 = __ldcg(&g.ctr->sb_lo[1]), lo2 = __ldcg(&g.ctr->sb_lo[2]);
        const int hi0 = __ldcg(&g.ctr->sb_hi[0]), hi1 = __ldcg(&g.ctr->sb_hi[1]), hi2 = __ldcg(&g.ctr->sb_hi[2]);
        const float reach = dmax + 2.f * vbl;  // the march ends within d_max plus a step of the start
        const float e[3] = {Er.m[3] + reach * dir.x, Er.m[7] + reach * dir.y, Er.m[11] + reach * dir.z};
        const float c[3] = {Er.m[3], Er.m[7], Er.m[11]};
        const int lo[3] = {lo0, lo1, lo2}, hi[3] = {hi0, hi1, hi2};
        skip = true;
#pragma unroll
        for (int a = 0; a < 3; a++) {
            const float mn = fminf(c[a], e[a]), mx = fmaxf(c[a], e[a]);
            if (!(fabsf(mn) < 1e6f && fabsf(mx) < 1e6f)) skip = false;
            const long long rb_lo = (long long)floorf(mn / vbl) - 1, rb_hi = (long long)floorf(mx / vbl) + 1;
            long long bl = rb_lo, bh = rb_hi;
            if (lo[a] <= hi[a]) {  // allocated blocks lie in super-blocks lo..hi
                bl = min(bl, (long long)lo[a] * 8);
                bh = max(bh, (long long)hi[a] * 8 + 7);
            }
            if (bh - bl > kHashCollisionFree) skip = false;
        }
    }
    SuperCache sc;
    F3 hit{0.f, 0.f, 0.f};
    float cr = 0.f, cg = 0.f, cb = 0.f;

    const F3 sv = f3smul(vl, dir), sb = f3smul(vbl, dir);
    int bx, by, bz;
    block_of(g, rv, bx, by, bz);
    int bucket = l < dmax ? find_block(g, bx, by, bz, finds, skip, sc) : -1;
    // No break leaves these loops: a branch that holds one rejoins its warp
    // only behind the loop, so lanes that took it (a step into another block,
    // say) would march on alone (the loop below with a break behind its find:
    // 1.1 ms a call at 640 x 480); every loop's end is one condition instead.
    // 25 of 32 lanes are then active (16.6 before), and a call went from 0.323
    // to 0.19 ms; with the next block's probe issued before the voxel's value is
    // looked at, and block and voxel from one quotient (voxel_of), to 0.14 ms;
    // with selections for the branches of a step, to 0.12 ms.
    // What is left is the chain of a step's instructions on the longest rays'
    // warps: two voxels a step, the next voxel's value ahead, and four probes
    // of the block skip in flight were slower (0.15, 0.17, 0.15 ms).
    bool go = l < dmax;
    F3 mid{0.f, 0.f, 0.f};
    float half = -1.f;
    while (go) {  // bucket: the find of rv's block
        int count = 0;
        while (bucket < 0 && l < dmax && guard < iter_cap) {
            rv = f3add(rv, sb);
            l = __fadd_rn(l, vbl);
            if (!(fabsf(rv.x - mid.x) < half && fabsf(rv.y - mid.y) < half && fabsf(rv.z - mid.z) < half)) {
                block_of(g, rv, bx, by, bz);
                bucket = find_block(g, bx, by, bz, finds, skip, sc);
                // a point well inside an empty super-block's box lies in it by the index rule too
                half = skip && !sc.occ ? 3.999f * vbl : -1.f;
                mid = F3{(float)(sc.sx * 8 + 4) * vbl, (float)(sc.sy * 8 + 4) * vbl, (float)(sc.sz * 8 + 4) * vbl};
            }
            count++;
            guard++;
        }
        if (l < dmax && count > 0) {
            const float back = __fsub_rn(vbl, dtr);
            rv = f3sub(rv, f3smul(back, dir));
            l = __fsub_rn(l, back);
            block_of(g, rv, bx, by, bz);
            bucket = find_block(g, bx, by, bz, finds, skip, sc);
            while (bucket < 0 && l < dmax && guard < iter_cap) {
                rv = f3add(rv, f3smul(dtr, dir));
                l = __fadd_rn(l, dtr);
                block_of(g, rv, bx, by, bz);
                bucket = find_block(g, bx, by, bz, finds, skip, sc);
                guard++;
            }
        }
        // Voxel steps, through neighbouring allocated blocks in one loop (the
        // reference goes back to its outer loop at every block: GPUVoxelGrid.cpp:633-700;
        // a find that succeeds at once brings it straight back here).
        bool in = l < dmax && guard < iter_cap;
        go = in;
        int v = in ? voxel_in_block(g, rv, bx, by, bz) : 0;
        if (in) in = ++guard < iter_cap;
        while (in) {
            const VoxelRead cv = read_voxel<kStorage>(g, bucket, v);
            voxels++;
            // the next point's block and voxel do not wait for this voxel's value
            const F3 nrv = f3add(rv, sv);
            int nx, ny, nz;
            const int nv = voxel_of(g, nrv, nx, ny, nz);
            const bool same = nx == bx && ny == by && nz == bz;
            // likewise the next block's first probe
            const unsigned long long key = prime_hash(nx, ny, nz);
            const uint32_t home = home_bucket(key, g.mask);
            const unsigned long long k0 = same ? kEmptyKey : __ldg(g.keys + home);
            const bool cross = cv.w > 0 && !(cv.sdf > 0);
            done = cross && Lp;  // a zero crossing, else a back face
            Fn = cross && !Lp;
            Lp = cross ? Lp : cv.w > 0;
            rv.x = cross ? rv.x : nrv.x;
            rv.y = cross ? rv.y : nrv.y;
            rv.z = cross ? rv.z : nrv.z;
            l = cross ? l : __fadd_rn(l, vl);
            bx = cross ? bx : nx;
            by = cross ? by : ny;
            bz = cross ? bz : nz;
            v = cross ? v : nv;
            const bool look = !cross && !same && l < dmax;
            finds += look ? 1 : 0;
            bucket = look ? (k0 == key ? (int)home : -1) : bucket;
            if (look && k0 != key && k0 != kEmptyKey) bucket = table_find_on(g.keys, g.mask, key);
            in = !cross && l < dmax && bucket >= 0;
            guard += in ? 1 : 0;
            in = in && guard < iter_cap;
        }
        go = go && !done && !Fn && l < dmax && guard < iter_cap;
    }
    if (done) {  // zero crossing (GPUVoxelGrid.cpp:655-689) at rv in voxel cv of block (bx, by, bz)
        int v = voxel_in_block(g, rv, bx, by, bz);
        const VoxelRead cv = read_voxel<kStorage>(g, bucket, v);
        const F3 vm_in = voxel_mid(g, v, bx, by, bz);
        rv = f3sub(rv, sv);
        l = __fsub_rn(l, vl);
        int qx, qy, qz;
        block_of(g, rv, qx, qy, qz);
        const int vo = voxel_in_block(g, rv, qx, qy, qz);
        const F3 vm_out = voxel_mid(g, vo, qx, qy, qz);
        const int ob = (qx == bx && qy == by && qz == bz) ? bucket : find_block(g, qx, qy, qz, finds, skip, sc);
        VoxelRead o{0.f, 0.f};
        float orr = 0.f, og = 0.f, obb = 0.f;
        if (ob >= 0) {  // missing block: reads as an empty voxel (reference: value_at(invalid))
            o = read_voxel<kStorage>(g, ob, vo);
            voxels++;
            if (out_col && g.rgb) {
                const float *pl = g.rgb + (size_t)ob * 3 * kBlockVoxels + vo;
                orr = pl[0];
                og = pl[kBlockVoxels];
                obb = pl[2 * kBlockVoxels];
            }
        }
        // x = (w_o*sdf_o/vl + w_i*(1 - sdf_i/vl)) / (w_i + w_o)  (GPUVoxelGrid.cpp:678)
        const float x = __fdiv_rn(
            __fadd_rn(__fdiv_rn(__fmul_rn(o.w, o.sdf), vl), __fmul_rn(cv.w, __fsub_rn(1.f, __fdiv_rn(cv.sdf, vl)))),
            __fadd_rn(cv.w, o.w));
        const F3 p = f3add(vm_out, f3smul(x, f3sub(vm_in, vm_out)));
        const float sproj = __fsub_rn(f3dot(p, dir), f3dot(rv, dir));
        hit = f3add(rv, f3smul(sproj, dir));  // point on the ray (GPUVoxelGrid.cpp:681)
        if (out_col && g.rgb) {
            const float *pl = g.rgb + (size_t)bucket * 3 * kBlockVoxels + v;
            cr = (float)((0.5 * (double)orr + 0.5 * (double)pl[0]) / 255.0);
            cg = (float)((0.5 * (double)og + 0.5 * (double)pl[kBlockVoxels]) / 255.0);
            cb = (float)((0.5 * (double)obb + 0.5 * (double)pl[2 * kBlockVoxels]) / 255.0);
        }
    }
    if (guard >= iter_cap) atomicOr(&g.ctr->status, kStTimeout);
    {  // the warp's work counts, one atomic pair per warp
        const unsigned m = __activemask();
        const unsigned f = __reduce_add_sync(m, (unsigned)finds), vx = __reduce_add_sync(m, (unsigned)voxels);
        if ((threadIdx.x & 31) == __ffs(m) - 1) {
            atomicAdd(&g.ctr->ray_finds, (unsigned long long)f);
            atomicAdd(&g.ctr->ray_voxels, (unsigned long long)vx);
        }
    }
    const size_t pix = (size_t)i * g.resj + j;
    if (!done) hit = F3{0.f, 0.f, 0.f};
    out_pcd[pix * 3 + 0] = hit.x;
    out_pcd[pix * 3 + 1] = hit.y;
    out_pcd[pix * 3 + 2] = hit.z;
    if (out_col) {
        out_col[pix * 3 + 0] = done ? cr : 0.f;
        out_col[pix * 3 + 1] = done ? cg : 0.f;
        out_col[pix * 3 + 2] = done ? cb : 0.f;
    }
}


// ------------------------------------------------------------------------
// Trilinear raycast (the per-frame pipeline's model view): depth, vertex and
// normal maps with at most max_steps march steps per ray.
//
// Ray of pixel (i, j): direction ((j - cj)/fx, (i - ci)/fy, 1) in the camera
// (not normalised, so the ray parameter t is the camera-frame depth). Steps:
//  * the ray point lies in a super-block (8^3 blocks) without any allocated
//    block: jump to the exit of that super-block's box;
//  * the ray point lies in a block that is not allocated: jump to the exit of
//    that block's box (empty-space skip);
//  * the trilinear TSDF sample is invalid (a corner voxel unobserved or in a
//    missing block): advance one voxel;
//  * the sample is positive: advance max(vl, 0.8 f) (f in metres);
//  * the sample is negative after a positive one: zero crossing; two
//    regula-falsi refinements on the bracket, then the hit;
//  * the sample is negative with no positive predecessor: no hit (back face).
// With a depth hint (the frame just fused at this pose, so the same rays), a
// ray whose pixel has depth d searches only [d - margin, d + margin], and
// starts at d: one sample there; in front of the surface (f >= 0) the march
// goes on forward, behind it (f < 0) it steps back by max(vl, 0.8 |f|) until a
// positive sample brackets the crossing (an unobserved sample, or leaving the
// window, first: no hit); an unobserved sample at d (a gap of the band at a
// silhouette) is no hit. A pixel without depth (dropout) takes as d the
// smaller depth of the nearest pixels with depth to its left and right in its
// warp's 32-pixel row segment. Where the fused frame saw d, a crossing
// outside the window contradicts the frame just fused, so the window loses no
// consistent surface; starting at d skips the unobserved voxels in front of
// the band, which a plain march would cross one voxel at a time, and keeps
// the lanes of a warp within a few steps of each other (marching the window
// where the sample at d is unobserved recovers 0.3 % of the hits on the
// synthetic room sequence at 2.3x the warp time).
// Every sample or skip counts as one step. The normal is the normalised
// gradient of the trilinear interpolant at the hit (world frame, pointing
// out of the surface). Outputs: vmap[i][j] = (x, y, z world, depth) and
// nmap[i][j] = (nx, ny, nz, 0); misses are all-zero.
#ifdef SS_RAYCAST_TIMING
// Per-warp SM cycles of the hint, the search (with its refinement) and the
// final sample and stores, and the warps' largest and summed step counts,
// for tuning builds only.
__device__ unsigned long long g_raycast_timing[8];
#define SS_RT_NOW(v) long long v = clock64()
#define SS_RT_ADD(slot, val)                                                                 \
    do {                                                                                     \
        if ((threadIdx.x & 31) == 0) atomicAdd(&g_raycast_timing[slot], (unsigned long long)(val)); \
    } while (0)
extern "C" int ss_debug_raycast_timing(unsigned long long *out, int reset) {
    int e = (int)cudaMemcpyFromSymbol(out, g_raycast_timing, sizeof(g_raycast_timing));
    if (reset) {
        unsigned long long z[8] = {};
        cudaMemcpyToSymbol(g_raycast_timing, z, sizeof(z));
    }
    return e;
}
#else
#define SS_RT_NOW(v)
#define SS_RT_ADD(slot, val) \
    do {                     \
    } while (0)
#endif

template <int kStorage, bool kHint>
__global__ void __launch_bounds__(512, 2) raycast_maps_kernel(GridView g, Mat34 T, const FramePose *__restrict__ pose,
                                                           int max_steps, float t_min, float t_max,
                                                           float4 *__restrict__ vmap, float4 *__restrict__ nmap,
                                                           unsigned long long *__restrict__ counters,
                                                           const uint16_t *__restrict__ hint, float hint_margin,
                                                           Counters *end) {
    // With a hint a warp is a 32-pixel row segment, which a dropout pixel takes
    // its hint from. Without one the rays march all the way, where an 8 x 4 patch
    // keeps together better than a row (240 vs 258 us at 640 x 480, 418 vs 479 us
    // at 1280 x 720; it takes a CTA of a multiple of four rows).
    const bool patch = !kHint && (blockDim.y & 3) == 0;
    const int j = blockIdx.x * 32 + (patch ? (threadIdx.y & 3) * 8 + (threadIdx.x & 7) : threadIdx.x);
    const int i = blockIdx.y * blockDim.y + (patch ? (threadIdx.y >> 2) * 4 + (threadIdx.x >> 3) : threadIdx.y);
    const bool inside = i < g.resi && j < g.resj;
    __shared__ int buckets[8 * 512];
    BlockCache cache(buckets, threadIdx.y * 32 + threadIdx.x, blockDim.y * 32);
    int steps = 0;
    bool hit = false;
    SS_RT_NOW(rt0);
    // Depth hint of this ray: the fused frame's depth at this pixel, or, where
    // that is missing (dropout), the smaller depth of the nearest pixels with
    // depth to its left and right within this warp's 32-pixel row segment.
    unsigned hint_mm = 0;
    if (kHint) {
        const unsigned full = 0xffffffffu;
        const int lane = threadIdx.x & 31;
        const unsigned own = inside ? (unsigned)__ldg(hint + (size_t)i * g.resj + j) : 0u;
        const unsigned have = __ballot_sync(full, own != 0u);
        const unsigned left = have & ((1u << lane) - 1u), right = lane < 31 ? have & (full << (lane + 1)) : 0u;
        const int li = left ? 31 - __clz(left) : lane, ri = right ? __ffs(right) - 1 : lane;
        const unsigned dl = __shfl_sync(full, own, li), dr = __shfl_sync(full, own, ri);
        hint_mm = own ? own : (left && right ? min(dl, dr) : (left ? dl : (right ? dr : 0u)));
    }
    // the hint is the frame's depth, an input; the volume, the pose and the
    // call's counters come from the kernels before this one
    pdl_wait();
    if (end && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0 && threadIdx.y == 0) end_call(end);
    SS_RT_NOW(rt1);
    long long rt2 = 0;
    if (inside) {
    if (pose) {
#pragma unroll
        for (int k = 0; k < 12; k++) T.m[k] = __ldg(&pose->E.m[k]);
    }
    const float dcx = ((float)j - g.in.cj) / g.in.fx, dcy = ((float)i - g.in.ci) / g.in.fy;
    const float dx = fmaf(T.m[0], dcx, fmaf(T.m[1], dcy, T.m[2]));
    const float dy = fmaf(T.m[4], dcx, fmaf(T.m[5], dcy, T.m[6]));
    const float dz = fmaf(T.m[8], dcx, fmaf(T.m[9], dcy, T.m[10]));
    const float ox = T.m[3], oy = T.m[7], oz = T.m[11];
    const float inv_len = rsqrtf(fmaf(dx, dx, fmaf(dy, dy, dz * dz)));  // world length of dt = 1
    const float inv_vl = 1.f / g.vl;

    float t = t_min;
    const float t_hint = (float)hint_mm * 1e-3f - hint_margin;
    if (kHint && t_hint > t_min) {
        // seek from the hint d within [d - margin, d + margin]
        hit = ray_search<kStorage>(g, ox, oy, oz, dx, dy, dz, inv_len, kRaySeek, t_hint + hint_margin, t_hint,
                                   fminf(t_max, t_hint + 2.f * hint_margin), max_steps, steps, t, cache);
    } else {
        hit = march<kStorage>(g, ox, oy, oz, dx, dy, dz, inv_len, t_min, t_max, max_steps, steps, t, cache);
    }
#ifdef SS_RAYCAST_TIMING
    rt2 = clock64();
#endif
    const size_t pix = (size_t)i * g.resj + j;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f), n = make_float4(0.f, 0.f, 0.f, 0.f);
    if (hit) {
        const float px = fmaf(t, dx, ox), py = fmaf(t, dy, oy), pz = fmaf(t, dz, oz);
        const TriSample q = trilinear<kStorage, true>(g, px, py, pz, inv_vl, cache);
        // the sum's order is written out: a compiler's choice of it would move the normal's last bit
        const float gn = q.valid ? sqrtf(fmaf(q.gz, q.gz, fmaf(q.gy, q.gy, __fmul_rn(q.gx, q.gx)))) : 0.f;
        if (gn > 0.f) {
            v = make_float4(px, py, pz, t);
            n = make_float4(q.gx / gn, q.gy / gn, q.gz / gn, 0.f);
        }
    }
    vmap[pix] = v;
    nmap[pix] = n;
    }
#ifdef SS_RAYCAST_TIMING
    {
        const long long rt3 = clock64();
        const unsigned full = 0xffffffffu;
        // lanes outside the image leave rt2 at 0: take the warp's latest search end
        const long long e2 = (long long)__reduce_max_sync(full, (unsigned)(rt2 ? rt2 - rt1 : 0));
        SS_RT_ADD(0, rt1 - rt0);
        SS_RT_ADD(1, e2);
        SS_RT_ADD(2, rt3 - rt1 - e2);
        const unsigned smax = __reduce_max_sync(full, (unsigned)steps), ssum = __reduce_add_sync(full, (unsigned)steps);
        SS_RT_ADD(3, smax);
        SS_RT_ADD(4, ssum);
        SS_RT_ADD(5, 1);
    }
#endif
    if (counters) {  // algorithmic-traffic counters (profiling only), one atomic per warp and field
        const unsigned full = 0xffffffffu;
        const unsigned l = __reduce_add_sync(full, cache.lookups), vx = __reduce_add_sync(full, cache.voxels);
        const unsigned st = __reduce_add_sync(full, (unsigned)steps), h = __reduce_add_sync(full, hit ? 1u : 0u);
        if ((threadIdx.x & 31) == 0) {
            atomicAdd(counters + 0, (unsigned long long)l);
            atomicAdd(counters + 1, (unsigned long long)vx);
            atomicAdd(counters + 2, (unsigned long long)st);
            atomicAdd(counters + 3, (unsigned long long)h);
        }
    }
}

ss_status launch_raycast_maps(ss_grid *g, const Mat34 &T, const FramePose *dpose, int max_steps, float t_min,
                              float t_max, float4 *vmap, float4 *nmap, cudaStream_t s, unsigned long long *counters,
                              const uint16_t *hint, float hint_margin, Counters *end) {
    const int rr = g->lc.raycast_rows;
    const dim3 blk(32, rr), grid((g->p.resj + 31) / 32, (g->p.resi + rr - 1) / rr);
#define SS_RM(ST, HINT)                                                                                             \
    SS_CUDA_TRY(launch_kernel(raycast_maps_kernel<ST, HINT>, grid, blk, 0, s, g->pdl, g->v, T, dpose, max_steps, t_min, \
                              t_max, vmap, nmap, counters, hint, hint_margin, end))
    if (g->p.storage == SS_STORAGE_F32) {
        if (hint)
            SS_RM(SS_STORAGE_F32, true);
        else
            SS_RM(SS_STORAGE_F32, false);
    } else {
        if (hint)
            SS_RM(SS_STORAGE_F16, true);
        else
            SS_RM(SS_STORAGE_F16, false);
    }
#undef SS_RM
    return SS_OK;
}

}  // namespace ss

using namespace ss;

extern "C" ss_status ss_raycast(ss_grid *g, const float extr[16], float *ray_pcd, float *ray_color,
                                ss_stream_t stream) {
    if (!g || !extr || !ray_pcd) return SS_ERR_ARG;
    if (!g->intr_set) return SS_ERR_STATE;
    for (int k = 0; k < 16; k++)
        if (!std::isfinite(extr[k])) return SS_ERR_ARG;
    cudaStream_t s = (cudaStream_t)stream;
    // A warp lasts as long as its longest ray. Where full warps would be no more
    // than four a scheduler, an image ends with its slowest warp, and warps of
    // half the rays wait for fewer: 48 vs 53 us at 160 x 120, 70 vs 71 at
    // 320 x 240. Beyond, the second half of the warps costs issue slots: 84 vs
    // 75 us at 400 x 300, 104 vs 80 at 517 x 389, 160 vs 117 at 640 x 480.
    const int64_t pixels = (int64_t)g->p.resi * g->p.resj;
    const int shift = pixels <= (int64_t)g->num_sms * 4 * 4 * 32 ? 2 : 3;
    const dim3 blk(32, 8), grid((g->p.resj + (4 << shift) - 1) / (4 << shift), (g->p.resi + 7) / 8);
    const Mat34 Er = mat34_from(extr);
    const int cap = g->raycast_cap > 0 ? g->raycast_cap : kRaycastIterCap;
    if (g->p.storage == SS_STORAGE_F32) {
        raycast_ref_kernel<SS_STORAGE_F32><<<grid, blk, 0, s>>>(g->v, Er, ray_pcd, ray_color, cap, shift);
    } else {
        raycast_ref_kernel<SS_STORAGE_F16><<<grid, blk, 0, s>>>(g->v, Er, ray_pcd, ray_color, cap, shift);
    }
    SS_LAUNCH_CHECK();
    return SS_OK;
}

namespace ss {
// Test hook kernel: block and voxel of each point, by voxel_of and by block_of and voxel_in_block.
__global__ void voxel_index_kernel(GridView g, const float *__restrict__ points, int n, int4 *__restrict__ out) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const F3 p{points[3 * k], points[3 * k + 1], points[3 * k + 2]};
    int4 a, b;
    a.w = voxel_of(g, p, a.x, a.y, a.z);
    block_of(g, p, b.x, b.y, b.z);
    b.w = voxel_in_block(g, p, b.x, b.y, b.z);
    out[2 * k] = a;
    out[2 * k + 1] = b;
}
}  // namespace ss

extern "C" ss_status ss_test_voxel_index(const float *points, int32_t n, float voxel, int32_t *out,
                                         ss_stream_t stream) {
    if (n < 0 || (n > 0 && (!points || !out)) || !(voxel > 0.f)) return SS_ERR_ARG;
    if (n == 0) return SS_OK;
    GridView g{};
    g.vl = voxel;
    g.vbl = 8.f * voxel;
    g.rvl = 1.f / g.vl;
    g.rvbl = 1.f / g.vbl;
    voxel_index_kernel<<<(n + 255) / 256, 256, 0, (cudaStream_t)stream>>>(g, points, n, (int4 *)out);
    SS_LAUNCH_CHECK();
    return SS_OK;
}

extern "C" ss_status ss_grid_test_raycast_cap(ss_grid *g, int32_t cap) {
    if (!g || cap < 0) return SS_ERR_ARG;
    g->raycast_cap = cap;
    return SS_OK;
}

extern "C" ss_status ss_raycast_maps(ss_grid *g, const float extr[16], int32_t max_steps, float t_min, float t_max,
                                     const uint16_t *hint_depth, float hint_margin, float *vertex_depth,
                                     float *normal, ss_stream_t stream) {
    if (!g || !extr || !vertex_depth || !normal || max_steps <= 0 || !(t_max > t_min)) return SS_ERR_ARG;
    if (!g->intr_set) return SS_ERR_STATE;
    for (int k = 0; k < 16; k++)
        if (!std::isfinite(extr[k])) return SS_ERR_ARG;
    return launch_raycast_maps(g, mat34_from(extr), nullptr, max_steps, t_min, t_max, (float4 *)vertex_depth,
                               (float4 *)normal, (cudaStream_t)stream, nullptr, hint_depth, hint_margin);
}
