// ss_mesh.cu — triangle mesh of the TSDF's zero level set on the GPU.
//
// The reference meshes the volume on the host: marchingCubesHost
// (GPUVoxelGrid.cpp:200-251) copies every block to the host into an Open3D
// ScalableTSDFVolume and runs its marching cubes. Here the mesh is extracted
// where the volume lives, by marching tetrahedra (a published method: each
// cell of 8 voxel centres is split into the 6 tetrahedra of the Freudenthal
// subdivision along the diagonal from corner 0 to corner 7; the split is the
// same in every cell, so neighbouring cells agree on their shared faces and
// the surface has no cracks; each tetrahedron has 16 sign cases, handled in
// code). A cell counts only where all 8 voxels are observed (weight > 0).
// Vertices lie on tetrahedron edges whose ends change sign (sdf < 0 is
// inside), linearly interpolated; triangles face from negative to positive
// sdf (out of the surface). Output: a triangle soup in world coordinates.
//
// Marching tetrahedra: one CTA per bucket of the hash table (grid-stride;
// empty buckets are skipped by the whole CTA), 256 threads x 2 cells per block;
// the up to 7 neighbouring blocks a block's last row of cells reaches into are
// looked up once per CTA. Each triangle is appended with one atomic on the
// counter. Marching cubes: a warp per block (mesh_mc_kernel).
#include <algorithm>

#include "ss_grid_impl.cuh"
#include "ss_mc_table.h"
#include "ss_trilinear.cuh"

namespace ss {

// The 6 tetrahedra (corner indices n = dx + 2 dy + 4 dz): 0 -> e_a -> e_a + e_b -> 7 for each axis order.
__constant__ int kTet[6][4] = {{0, 1, 3, 7}, {0, 1, 5, 7}, {0, 2, 3, 7}, {0, 2, 6, 7}, {0, 4, 5, 7}, {0, 4, 6, 7}};

struct MeshOut {
    float *tris;                // [cap][9]
    unsigned long long *count;  // total triangles (may exceed cap)
    unsigned long long cap;
};

__device__ __forceinline__ F3 edge_point(const F3 &p, float sp, const F3 &q, float sq) {
    const float t = sp / (sp - sq);
    return F3{fmaf(t, q.x - p.x, p.x), fmaf(t, q.y - p.y, p.y), fmaf(t, q.z - p.z, p.z)};
}

// Appends triangle (a, b, c), flipped if needed so that its normal points
// along dir (from the tetrahedron's inside corners to its outside corners).
__device__ __forceinline__ void emit(const MeshOut &o, F3 a, F3 b, F3 c, const F3 &dir) {
    const float ux = b.x - a.x, uy = b.y - a.y, uz = b.z - a.z, vx = c.x - a.x, vy = c.y - a.y, vz = c.z - a.z;
    const float nx = uy * vz - uz * vy, ny = uz * vx - ux * vz, nz = ux * vy - uy * vx;
    if (nx * dir.x + ny * dir.y + nz * dir.z < 0.f) {
        const F3 t = b;
        b = c;
        c = t;
    }
    const unsigned long long at = atomicAdd(o.count, 1ull);
    if (at >= o.cap) return;
    float *d = o.tris + at * 9;
    d[0] = a.x, d[1] = a.y, d[2] = a.z, d[3] = b.x, d[4] = b.y, d[5] = b.z, d[6] = c.x, d[7] = c.y, d[8] = c.z;
}

__device__ void tetra(const MeshOut &o, const F3 *p, const float *s, const int *t) {
    int in[4], out[4], ni = 0, no = 0;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        if (s[t[k]] < 0.f) in[ni++] = t[k];
        else out[no++] = t[k];
    }
    if (ni == 0 || ni == 4) return;
    F3 ci{0.f, 0.f, 0.f}, co{0.f, 0.f, 0.f};
    for (int k = 0; k < ni; k++) ci = F3{ci.x + p[in[k]].x, ci.y + p[in[k]].y, ci.z + p[in[k]].z};
    for (int k = 0; k < no; k++) co = F3{co.x + p[out[k]].x, co.y + p[out[k]].y, co.z + p[out[k]].z};
    const F3 dir{co.x / no - ci.x / ni, co.y / no - ci.y / ni, co.z / no - ci.z / ni};
    if (ni == 1 || ni == 3) {
        const int a = ni == 1 ? in[0] : out[0];
        const int *r = ni == 1 ? out : in;  // the three other corners
        emit(o, edge_point(p[a], s[a], p[r[0]], s[r[0]]), edge_point(p[a], s[a], p[r[1]], s[r[1]]),
             edge_point(p[a], s[a], p[r[2]], s[r[2]]), dir);
    } else {  // two inside (a, b), two outside (c, d): the quad ac, ad, bd, bc
        const int a = in[0], b = in[1], c = out[0], d = out[1];
        const F3 ac = edge_point(p[a], s[a], p[c], s[c]), ad = edge_point(p[a], s[a], p[d], s[d]);
        const F3 bd = edge_point(p[b], s[b], p[d], s[d]), bc = edge_point(p[b], s[b], p[c], s[c]);
        emit(o, ac, ad, bd, dir);
        emit(o, ac, bd, bc, dir);
    }
}

template <int kStorage>
__global__ void __launch_bounds__(256) mesh_kernel(GridView g, MeshOut o) {
    __shared__ int nb[8];  // bucket of block (bx + (n & 1), by + (n >> 1 & 1), bz + (n >> 2)); -1 missing
    __shared__ int bc[3];
    for (uint32_t bucket = blockIdx.x; bucket <= g.mask; bucket += gridDim.x) {
        const unsigned long long key = g.keys[bucket];
        if (key == kEmptyKey || key == kTombKey) continue;  // uniform over the CTA
        __syncthreads();  // the previous block's cells are done with nb
        if (threadIdx.x == 0) {
            int x, y, z;
            unpack_coords(g.stamp[bucket] & ((1ull << kEpochShift) - 1ull), x, y, z);
            bc[0] = x, bc[1] = y, bc[2] = z;
            nb[0] = (int)bucket;
        }
        __syncthreads();
        if (threadIdx.x >= 1 && threadIdx.x < 8) {
            const int n = threadIdx.x, x = bc[0] + (n & 1), y = bc[1] + ((n >> 1) & 1), z = bc[2] + (n >> 2);
            nb[n] = packable(x, y, z) ? table_find(g, prime_hash(x, y, z)) : -1;
        }
        __syncthreads();
        for (int c = threadIdx.x; c < kBlockVoxels; c += blockDim.x) {
            const int i = c & 7, j = (c >> 3) & 7, k = c >> 6;
            F3 p[8];
            float s[8];
            bool ok = true;
#pragma unroll
            for (int n = 0; n < 8; n++) {
                const int vi = i + (n & 1), vj = j + ((n >> 1) & 1), vk = k + (n >> 2);
                const int b = nb[(vi >> 3) + 2 * (vj >> 3) + 4 * (vk >> 3)];
                if (b < 0) {
                    ok = false;
                    break;
                }
                const float2 sw = voxel_sw<kStorage>(g, b, (vi & 7) + 8 * (vj & 7) + 64 * (vk & 7));
                if (!(sw.y > 0.f)) {
                    ok = false;
                    break;
                }
                s[n] = sw.x;
                // voxel centre (pzero + (index + 0.5) vl, GPUVoxelGrid.cpp:521)
                p[n] = F3{((float)(bc[0] * 8 + vi) + 0.5f) * g.vl, ((float)(bc[1] * 8 + vj) + 0.5f) * g.vl,
                          ((float)(bc[2] * 8 + vk) + 0.5f) * g.vl};
            }
            if (!ok) continue;
#pragma unroll 1
            for (int t = 0; t < 6; t++) tetra(o, p, s, kTet[t]);
        }
    }
}

// ---------------------------------------------------------- marching cubes
// The case table (ss_mc_table.h) in global memory, read through the read-only
// cache (the lanes of a warp hold different cases): per case its number of
// triangles, per triangle its three edges in four bits each.
struct McPacked {
    unsigned char n[256];
    unsigned short tri[256][kMcMaxTris];
};
constexpr McPacked mc_packed() {
    McPacked p{};
    for (int c = 0; c < 256; c++)
        while (p.n[c] < kMcMaxTris && kMcTable.tri[c][3 * p.n[c]] >= 0) {
            const signed char *t = kMcTable.tri[c] + 3 * p.n[c];
            p.tri[c][p.n[c]++] = (unsigned short)(t[0] | t[1] << 4 | t[2] << 8);
        }
    return p;
}
__device__ const McPacked g_mc = mc_packed();

// A table edge runs along x (0, 2, 4, 6), y (1, 3, 5, 7) or z (8..11) from the
// cell corner (bits x, y, z) packed here, four bits an edge: the end with the
// lower coordinate, so the cubes sharing an edge interpolate it alike.
constexpr unsigned long long kMcEdgeCorner = 0x231046540210ull;

// A warp takes 32 buckets at a time from a counter and meshes their live
// blocks one after the other: the block's 512 voxel values and the 217 of its
// neighbours that its last cells reach into go to shared memory (NaN where a
// voxel is unobserved or its block missing), a lane walks two columns of cells
// up, keeping a layer's corners for the next one, and the triangles found are
// listed and written 32 at a time: a lane computes one triangle, the warp
// reserves their places with one atomic and writes the 1152 bytes in order.
// Nothing is synchronised beyond the warp. On a room of 72 k blocks and 6.1 M
// triangles a CTA per bucket with eight global loads a cell and an atomic a
// triangle took 1.03 ms to count and 1.15 ms to write; this counts (kEmit
// false) in 0.11 and writes in 0.29 ms, bound by its instructions (2000 a block,
// half of them the triangles') and the latency between a block's loads.
// Leaving a block without a sign change early was slower (0.14, 0.32 ms: most
// blocks hold one, and the vote waits for every load).
constexpr int kMcWarps = 8;
constexpr int kMcSide = kEdge + 1;                       // voxels of a block's cells per axis
constexpr int kMcVoxels = kMcSide * kMcSide * kMcSide;   // 729
constexpr int kMcList = 31 + 2 * 32 * kMcMaxTris;        // entries left over, and a layer's
constexpr int kMcLayer = kMcSide * kMcSide;

template <int kStorage, bool kEmit>
__global__ void __launch_bounds__(32 * kMcWarps, kEmit ? 4 : 6) mesh_mc_kernel(GridView g, MeshOut o, unsigned *next) {
    constexpr unsigned FULL = 0xffffffffu;
    __shared__ float vox[kMcWarps][kMcVoxels];
    __shared__ unsigned list[kEmit ? kMcWarps : 1][kEmit ? kMcList : 1];  // cell | triangle << 9 | case << 12
    __shared__ float stage[kEmit ? kMcWarps : 1][kEmit ? 32 * 9 : 1];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    float *sv = vox[wid];
    unsigned *sl = list[kEmit ? wid : 0];
    float *ss = stage[kEmit ? wid : 0];
    const unsigned no = 0x7fc0dead;  // a NaN of its own: the value of an unobserved voxel
    const float bad = __uint_as_float(no);
    unsigned long long total = 0;  // kEmit false: this warp's triangles
    const unsigned chunks = (g.mask >> 5) + 1u;
    auto take = [&] {
        unsigned c = 0;
        if (lane == 0) c = atomicAdd(next, 1u);
        return __shfl_sync(FULL, c, 0);
    };
    for (unsigned chunk = take(); chunk < chunks; chunk = take()) {
        const uint32_t mine = chunk * 32u + lane;
        const unsigned long long key = mine <= g.mask ? g.keys[mine] : kEmptyKey;
        unsigned live = __ballot_sync(FULL, key != kEmptyKey && key != kTombKey);
        int cx = 0, cy = 0, cz = 0;
        if ((live >> lane) & 1u) unpack_coords(g.stamp[mine] & ((1ull << kEpochShift) - 1ull), cx, cy, cz);
        while (live) {
            const int src = __ffs(live) - 1;
            live &= live - 1u;
            const int bx = __shfl_sync(FULL, cx, src), by = __shfl_sync(FULL, cy, src), bz = __shfl_sync(FULL, cz, src);
            // lane n < 8: the bucket of the block at offset (n & 1, n >> 1 & 1, n >> 2); -1 missing
            int nb = (int)(chunk * 32u) + src;
            if (lane >= 1 && lane < 8) {
                const int x = bx + (lane & 1), y = by + ((lane >> 1) & 1), z = bz + (lane >> 2);
                nb = packable(x, y, z) ? table_find(g, prime_hash(x, y, z)) : -1;
            }
            __syncwarp();  // the lanes are done with the block before
            const int own = __shfl_sync(FULL, nb, 0);
#pragma unroll
            for (int k = 0; k < kBlockVoxels / 32; k++) {
                const int v = k * 32 + lane;
                const float2 sw = voxel_sw<kStorage>(g, own, v);
                const bool seen = sw.y > 0.f;
                sv[(v & 7) + kMcSide * ((v >> 3) & 7) + kMcLayer * (v >> 6)] = seen ? sw.x : bad;
            }
            // the far faces of the 9 x 9 x 9 voxels: x = 8 (81), y = 8 (72), z = 8 (64)
#pragma unroll
            for (int k = 0; k < 7; k++) {
                const int h = k * 32 + lane;
                int x = 8, y = 8, z = 8;
                if (h < 81) {
                    z = h / 9;
                    y = h - 9 * z;
                } else if (h < 153) {
                    z = (h - 81) >> 3;
                    x = (h - 81) & 7;
                } else {
                    y = ((h - 153) >> 3) & 7;
                    x = (h - 153) & 7;
                }
                const int n = (x >> 3) | (y >> 3) << 1 | (z >> 3) << 2;
                const int b = __shfl_sync(FULL, nb, n);
                if (h < kMcVoxels - kBlockVoxels) {
                    float f = bad;
                    if (b >= 0) {
                        const float2 sw = voxel_sw<kStorage>(g, b, (x & 7) + 8 * (y & 7) + 64 * (z & 7));
                        if (sw.y > 0.f) {
                            f = sw.x;
                        }
                    }
                    sv[x + kMcSide * y + kMcLayer * z] = f;
                }
            }
            __syncwarp();
            // The lane's columns (i, j) and (i, j + 4). A layer's corner bits
            // in the order of the table's lower face: (0,0) (1,0) (1,1) (0,1).
            const int i = lane & 7, j = lane >> 3;
            int listed = 0;
            auto face = [&](int jj, int k, unsigned &bits) {
                const float *q = sv + i + kMcSide * jj + kMcLayer * k;
                const float a = q[0], b = q[1], c = q[kMcSide + 1], d = q[kMcSide];
                bits = (a < 0.f ? 1u : 0u) | (b < 0.f ? 2u : 0u) | (c < 0.f ? 4u : 0u) | (d < 0.f ? 8u : 0u);
                return __float_as_uint(a) != no && __float_as_uint(b) != no && __float_as_uint(c) != no &&
                       __float_as_uint(d) != no;
            };
            auto flush = [&](int n) {  // writes the first n <= 32 listed triangles
                unsigned long long at = 0;
                if (lane == 0) at = atomicAdd(o.count, (unsigned long long)n);
                at = __shfl_sync(FULL, at, 0);
                if (lane < n) {
                    const unsigned e = sl[lane];
                    const int ci = e & 7, cj = (e >> 3) & 7, ck = (e >> 6) & 7;
                    const unsigned tri = __ldg(&g_mc.tri[e >> 12][(e >> 9) & 7]);
#pragma unroll
                    for (int u = 0; u < 3; u++) {
                        const int es = (tri >> (4 * u)) & 15, axis = es < 8 ? es & 1 : 2;
                        const int lo = (int)(kMcEdgeCorner >> (4 * es)) & 7;
                        const int x = ci + (lo & 1), y = cj + ((lo >> 1) & 1), z = ck + (lo >> 2);
                        const float *q = sv + x + kMcSide * y + kMcLayer * z;
                        // voxel centres (pzero + (index + 0.5) vl, GPUVoxelGrid.cpp:521), each rounded
                        auto centre = [&](int v) { return __fmul_rn((float)v + 0.5f, g.vl); };
                        const F3 pa{centre(bx * 8 + x), centre(by * 8 + y), centre(bz * 8 + z)};
                        const F3 pb{axis == 0 ? centre(bx * 8 + x + 1) : pa.x, axis == 1 ? centre(by * 8 + y + 1) : pa.y,
                                    axis == 2 ? centre(bz * 8 + z + 1) : pa.z};
                        const F3 v = edge_point(pa, q[0], pb, q[axis == 0 ? 1 : axis == 1 ? kMcSide : kMcLayer]);
                        ss[9 * lane + 3 * u] = v.x;
                        ss[9 * lane + 3 * u + 1] = v.y;
                        ss[9 * lane + 3 * u + 2] = v.z;
                    }
                }
                __syncwarp();
                if (at < o.cap) {
                    const int floats = 9 * (int)min((unsigned long long)n, o.cap - at);
                    float *d = o.tris + at * 9;
#pragma unroll
                    for (int q = 0; q < 9; q++)
                        if (q * 32 + lane < floats) d[q * 32 + lane] = ss[q * 32 + lane];
                }
                __syncwarp();
            };
            unsigned low0, low1;
            bool ok0 = face(j, 0, low0), ok1 = face(j + 4, 0, low1);
            for (int k = 0; k < kEdge; k++) {
                unsigned high0, high1;
                const bool up0 = face(j, k + 1, high0), up1 = face(j + 4, k + 1, high1);
                const unsigned cs0 = low0 | high0 << 4, cs1 = low1 | high1 << 4;
                const int n0 = ok0 && up0 ? __ldg(g_mc.n + cs0) : 0;
                const int n1 = ok1 && up1 ? __ldg(g_mc.n + cs1) : 0;
                ok0 = up0;
                ok1 = up1;
                low0 = high0;
                low1 = high1;
                if (!kEmit) {
                    total += (unsigned)(n0 + n1);
                    continue;
                }
                if (!__any_sync(FULL, n0 + n1 > 0)) continue;
                int incl = n0 + n1;  // inclusive scan of the lanes' triangles
#pragma unroll
                for (int d = 1; d < 32; d <<= 1) {
                    const int t = __shfl_up_sync(FULL, incl, d);
                    if (lane >= d) incl += t;
                }
                int at = listed + incl - n0 - n1;
                const unsigned cell = i | j << 3 | k << 6;
                for (int t = 0; t < n0; t++) sl[at++] = cell | t << 9 | cs0 << 12;
                for (int t = 0; t < n1; t++) sl[at++] = (cell + 32) | t << 9 | cs1 << 12;
                listed += __shfl_sync(FULL, incl, 31);
                __syncwarp();
                int done = 0;
                while (listed - done >= 32) {
                    sl += done;
                    flush(32);
                    sl -= done;
                    done += 32;
                }
                if (done) {  // the entries left over move to the front
                    const unsigned e = lane < listed - done ? sl[done + lane] : 0u;
                    __syncwarp();
                    sl[lane] = e;
                    listed -= done;
                    __syncwarp();
                }
            }
            if (kEmit && listed > 0) flush(listed);
        }
    }
    if (!kEmit) {
        unsigned t = __reduce_add_sync(FULL, (unsigned)total);  // a warp's triangles: far below 2^32
        if (lane == 0 && t) atomicAdd(o.count, (unsigned long long)t);
    }
}

}  // namespace ss

using namespace ss;

extern "C" ss_status ss_grid_extract_mesh_cubes(ss_grid *g, int64_t max_triangles, float *triangles, int64_t *count,
                                                ss_stream_t stream) {
    if (!g || !count || max_triangles < 0 || (max_triangles > 0 && !triangles)) return SS_ERR_ARG;
    cudaStream_t s = (cudaStream_t)stream;
    if (!g->mesh_count) SS_CUDA_TRY(cudaMalloc(&g->mesh_count, 2 * sizeof(unsigned long long)));
    SS_CUDA_TRY(cudaMemsetAsync(g->mesh_count, 0, 2 * sizeof(unsigned long long), s));
    MeshOut o{triangles, g->mesh_count, (unsigned long long)max_triangles};
    unsigned *next = (unsigned *)(g->mesh_count + 1);
    // as many warps as stay resident (a writing warp holds 5.5 KB of shared memory), no more than chunks of 32 buckets
    const int want = (int)((g->v.mask >> 5) / kMcWarps + 1u);
    const bool emit = max_triangles > 0;
    const int ctas = std::min(g->num_sms * (emit ? 4 : 6), want);
    if (g->p.storage == SS_STORAGE_F32) {
        if (emit)
            mesh_mc_kernel<SS_STORAGE_F32, true><<<ctas, 32 * kMcWarps, 0, s>>>(g->v, o, next);
        else
            mesh_mc_kernel<SS_STORAGE_F32, false><<<ctas, 32 * kMcWarps, 0, s>>>(g->v, o, next);
    } else {
        if (emit)
            mesh_mc_kernel<SS_STORAGE_F16, true><<<ctas, 32 * kMcWarps, 0, s>>>(g->v, o, next);
        else
            mesh_mc_kernel<SS_STORAGE_F16, false><<<ctas, 32 * kMcWarps, 0, s>>>(g->v, o, next);
    }
    SS_LAUNCH_CHECK();
    unsigned long long n = 0;
    SS_CUDA_TRY(cudaMemcpyAsync(&n, g->mesh_count, sizeof(n), cudaMemcpyDeviceToHost, s));
    SS_CUDA_TRY(cudaStreamSynchronize(s));
    *count = (int64_t)n;
    return SS_OK;
}

extern "C" ss_status ss_grid_extract_mesh(ss_grid *g, int64_t max_triangles, float *triangles, int64_t *count,
                                          ss_stream_t stream) {
    if (!g || !count || max_triangles < 0 || (max_triangles > 0 && !triangles)) return SS_ERR_ARG;
    cudaStream_t s = (cudaStream_t)stream;
    if (!g->mesh_count) SS_CUDA_TRY(cudaMalloc(&g->mesh_count, 2 * sizeof(unsigned long long)));
    SS_CUDA_TRY(cudaMemsetAsync(g->mesh_count, 0, sizeof(unsigned long long), s));
    MeshOut o{triangles, g->mesh_count, (unsigned long long)max_triangles};
    const int ctas = g->num_sms * 8;
    if (g->p.storage == SS_STORAGE_F32)
        mesh_kernel<SS_STORAGE_F32><<<ctas, 256, 0, s>>>(g->v, o);
    else
        mesh_kernel<SS_STORAGE_F16><<<ctas, 256, 0, s>>>(g->v, o);
    SS_LAUNCH_CHECK();
    unsigned long long n = 0;
    SS_CUDA_TRY(cudaMemcpyAsync(&n, g->mesh_count, sizeof(n), cudaMemcpyDeviceToHost, s));
    SS_CUDA_TRY(cudaStreamSynchronize(s));
    *count = (int64_t)n;
    return SS_OK;
}
