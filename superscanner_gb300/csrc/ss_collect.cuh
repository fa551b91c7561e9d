// ss_collect.cuh — block collection of one 32 x rows pixel tile
// (depthToPcdTag + vbCollectionTag, GPUVoxelGrid.h:303-307,
// GPUVoxelGrid.cpp:471-514), shared by the per-call collection
// (collect_kernel, ss_grid.cu) and the batched re-fusion's
// (refuse_collect_kernel, ss_refuse.cu). One thread per pixel. Where the cubes
// of the tile's pixels lie in a small box (TileBits, nearly always), the tile's
// blocks are collected as bits of the box; elsewhere in two phases:
//  1. every pixel's candidates, the cube of blocks its truncation band
//     overlaps (GPUVoxelGrid.cpp:485-489), go into a shared-memory hash set,
//     so the tile's candidates are deduplicated on chip: the lanes of a warp
//     are grouped by cube (__match_any_sync on corner and extent; neighbouring
//     pixels mostly share one), and the distinct cubes' blocks are spread
//     over the lanes, 32 per step, each inserted with at most one 32-bit CAS
//     (typically one or two steps per warp instead of one per candidate of a
//     pixel). A key is the block's
//     offset from the camera's block, 10 bits per axis ([-512, 511] blocks,
//     +-16 m at 32 mm blocks); 128 slots per tile row (a tile row at 4 m and
//     4 mm voxels meets about 20 distinct blocks). Most candidates are in the
//     set already, so a plain load of the slot precedes the CAS (shared
//     atomics, not arithmetic, bound this phase). A candidate outside the
//     key range, or one the set cannot place, is visited directly;
//  2. each warp compacts its slice of the set (ballots, no atomics) and
//     visits its distinct blocks; the visits that append a block to the
//     call's list are aggregated per warp.
// The set of allocated blocks is the union of every pixel's candidates, as in
// the reference; only the number of global probes and atomics changes (one
// per distinct block per tile). 8 bytes of shared memory per slot (set and
// per-warp lists; 12 with a tagged set's tags) and 512 bytes per warp for its
// cubes: 6 KB per 4-row tile (8 KB tagged).
//
// A visitor is a callable bool (int bx, int by, int bz, unsigned tag, int
// &bucket): it finds or inserts the block, marks it, and returns true when
// this visit is the one that appends bucket to the list. A tagged set (the
// batched re-fusion's) keeps per slot the OR of the tags (2 bits) of the
// fills that entered the key, so several fills of one tile (a keyframe's two
// phases) share the set and each distinct block is visited once with the tags
// of all of them.
#pragma once

#include "ss_internal.cuh"

namespace ss {

constexpr unsigned kSetEmpty = 0xffffffffu;
constexpr int kSetSlotsPerRow = 128;
constexpr int kSetOff = 512;  // key offsets per axis: [-kSetOff, kSetOff) blocks

// Dynamic shared memory of a tile of `rows` pixel rows (rows warps): the
// set, the per-warp lists, per warp 32 cube entries of 16 bytes, and for a
// tagged set the slots' tags.
inline size_t tile_set_bytes(int rows, bool tagged = false) {
    return (size_t)kSetSlotsPerRow * rows * (tagged ? 3 : 2) * sizeof(unsigned) + (size_t)rows * 32 * sizeof(int4);
}

// The slots' tags of a tagged set (after the cube entries).
__device__ __forceinline__ unsigned *tile_tags(unsigned *cset, int slots) {
    return cset + 2 * slots + blockDim.y * 32 * 4;
}

// The camera's block, about (the origin of the set's keys) of pose E: any
// value works as long as every thread of the tile computes the same one.
__device__ __forceinline__ void camera_block(const GridView &g, const Mat34 &E, int &cbx, int &cby, int &cbz) {
    cbx = (int)floorf(E.m[3] * g.rvbl);
    cby = (int)floorf(E.m[7] * g.rvbl);
    cbz = (int)floorf(E.m[11] * g.rvbl);
}

// One visit outside the tile's set, with its own append.
template <class Visit>
__device__ __forceinline__ void visit_one(const GridView &g, int bx, int by, int bz, unsigned tag, Visit &visit) {
    int bucket = -1;
    if (!visit(bx, by, bz, tag, bucket)) return;
    const int idx = atomicAdd(&g.ctr->list_count, 1);
    if (idx <= (int)g.mask) g.list[idx] = bucket;
    else atomicOr(&g.ctr->status, kStListOverflow);
}

// The camera-frame point of pixel (i, j) (depthToPcdTag, GPUVoxelGrid.h:303-307)
// and whether it takes part (inside the image, z > rmin): the part of a
// pixel's collection that does not depend on the pose.
__device__ __forceinline__ bool tile_point(const GridView &g, const uint16_t *__restrict__ depth, int i, int j, F3 &p) {
    p = F3{0.f, 0.f, 0.f};
    if (!(i < g.resi && j < g.resj)) return false;
    p = get_point_t(g, i, j, depth_m(__ldg(depth + (size_t)i * g.resj + j)));
    return p.z > g.rmin;
}

// The cube of blocks a pixel's truncation band overlaps at pose E
// (GPUVoxelGrid.cpp:485-489): lowest block and extents, all zero extents for a
// pixel that takes no part (p, valid: from tile_point) or whose cube is out of
// range.
struct TileCube {
    int lox, loy, loz, nx, ny, nz;
};
__device__ __forceinline__ TileCube tile_cube(const GridView &g, F3 p, bool valid, const Mat34 &E) {
    TileCube c{0, 0, 0, 0, 0, 0};
    if (valid) {
        const F3 pt = xform(E, p);
        const F3 t{g.trunc, g.trunc, g.trunc};
        const F3 lo = f3sub(pt, t), hi = f3add(pt, t);
        int hix, hiy, hiz;
        block_range(lo, hi, g.vbl, g.rvbl, c.lox, c.loy, c.loz, hix, hiy, hiz);
        c.nx = hix - c.lox + 1;
        c.ny = hiy - c.loy + 1;
        c.nz = hiz - c.loz + 1;
        if (c.nx < 1 || c.ny < 1 || c.nz < 1 || c.nx > 8 || c.ny > 8 || c.nz > 8) {
            atomicOr(&g.ctr->status, kStRange);  // non-finite pose or truncation > 3.5 blocks
            c.nx = c.ny = c.nz = 0;
        }
    }
    return c;
}

// Visits the cnt blocks of a warp's list (packed offsets; tags in the top two
// bits), appending with one atomic per warp step.
template <bool kTagged, class Visit>
__device__ __forceinline__ void tile_visit_list(const GridView &g, const unsigned *wlist, int cnt, int cbx, int cby,
                                                int cbz, Visit &visit) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    __syncwarp();
    for (int base = 0; base < cnt; base += 32) {
        const int e = base + lane;
        bool append = false;
        int bucket = -1;
        if (e < cnt) {
            const unsigned key = wlist[e];
            append = visit(cbx + (int)((key >> 20) & 1023u) - kSetOff, cby + (int)((key >> 10) & 1023u) - kSetOff,
                           cbz + (int)(key & 1023u) - kSetOff, kTagged ? key >> 30 : 1u, bucket);
        }
        const unsigned ap = __ballot_sync(FULL, append);
        if (ap) {
            const int leader = __ffs(ap) - 1;
            int b0 = 0;
            if (lane == leader) b0 = atomicAdd(&g.ctr->list_count, __popc(ap));
            b0 = __shfl_sync(FULL, b0, leader);
            if (append) {
                const int idx = b0 + __popc(ap & lt);
                if (idx <= (int)g.mask) g.list[idx] = bucket;
                else atomicOr(&g.ctr->status, kStListOverflow);
            }
        }
    }
}

// ---- The tile's blocks as bits. The cubes of a tile's pixels mostly lie in a
// small box: with the box's longest side along 16 words at most (two words a
// step where the second side is longer than 4) and 4 x 8 or 8 x 8 blocks of the
// other two sides as a word's bits, a warp ORs its lanes' cubes by one
// reduction a word, and the tile's blocks are the bits of 32 words in shared
// memory (per phase, for a re-fusion). Tiles whose box does not fit (depth
// edges, truncation of many blocks; 2 % of a noisy room's) use the set above.
// Grouping a warp's equal cubes and entering their blocks in the set took most
// of the instructions that bound the collection: noise gives a 32-pixel row ten
// and more distinct cubes. 100 keyframes of 640 x 480 0.99 -> 0.75 ms, a frame of
// 640 x 480 12.8 -> 10.0 us, of 1280 x 720 36 -> 28.6 us.
struct TileBits {
    unsigned box[6];  // lowest x, y, z and 1023 - highest x, y, z: block offsets from the camera's block + kSetOff
    unsigned wide;    // a cube out of the offsets' range
    unsigned bits[2][32];
};

__device__ __forceinline__ void tile_bits_clear(TileBits &t) {
    const int tid = threadIdx.y * blockDim.x + threadIdx.x;
    if (tid < 32) t.bits[0][tid] = t.bits[1][tid] = 0u;
    if (tid < 6) t.box[tid] = 2 * kSetOff;  // empty: lowest > highest
    if (tid == 6) t.wide = 0u;
}

// A cube's corners as offsets (10 bits an axis); hi < lo for an empty one.
struct PackedCube {
    unsigned lo, hi;
};
__device__ __forceinline__ PackedCube tile_pack(const TileCube &c, int cbx, int cby, int cbz, TileBits &t) {
    PackedCube k{0x3fffffffu, 0u};
    if (c.nx) {
        const unsigned x = (unsigned)(c.lox - cbx + kSetOff), y = (unsigned)(c.loy - cby + kSetOff),
                       z = (unsigned)(c.loz - cbz + kSetOff);
        if (max(max(x, y), z) < 2u * kSetOff - 8u) {  // so do the highest blocks, fewer than 8 further
            k.lo = x << 20 | y << 10 | z;
            k.hi = k.lo + ((unsigned)(c.nx - 1) << 20 | (unsigned)(c.ny - 1) << 10 | (unsigned)(c.nz - 1));
        } else {
            t.wide = 1u;
        }
    }
    return k;
}

// Grows the tile's box by the warp's cubes (of both phases: an empty one gives
// the lowest corner's 1023s and the highest's zeros, 1023 from the top).
__device__ __forceinline__ void tile_box(PackedCube k, PackedCube m, TileBits &t) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    unsigned mine = 0u;
#pragma unroll
    for (int a = 0; a < 3; a++) {
        const int sh = 20 - 10 * a;
        const unsigned l = __reduce_min_sync(FULL, min((k.lo >> sh) & 1023u, (m.lo >> sh) & 1023u));
        const unsigned h = __reduce_max_sync(FULL, max((k.hi >> sh) & 1023u, (m.hi >> sh) & 1023u));
        if (lane == a) mine = l;
        if (lane == 3 + a) mine = 1023u - h;
    }
    if (lane < 6) atomicMin(t.box + lane, mine);
}

// How the box lies in the words: the axis (0 x, 1 y, 2 z) along the words, and
// the shifts that take an offset's three axes (word axis, byte axis, bit axis)
// from a packed corner.
struct TileLayout {
    bool fits, empty;
    int sa, sb, sc;                // shifts of the axes in a packed corner
    unsigned a0, b0, c0;           // the box's lowest offsets along them
    int na, two;                   // steps along the words, and words a step - 1
};
__device__ __forceinline__ TileLayout tile_layout(const TileBits &t, int cbx, int cby, int cbz) {
    TileLayout L;
    const int ex = 1024 - (int)(t.box[0] + t.box[3]), ey = 1024 - (int)(t.box[1] + t.box[4]),
              ez = 1024 - (int)(t.box[2] + t.box[5]);
    const int a = ex >= ey && ex >= ez ? 0 : ey >= ez ? 1 : 2, b = a == 0 ? 1 : 0, c = a == 2 ? 1 : 2;
    const int eb = b == 0 ? ex : ey, ec = c == 2 ? ez : ey;
    L.na = a == 0 ? ex : a == 1 ? ey : ez;
    L.sa = 20 - 10 * a;
    L.sb = 20 - 10 * b;
    L.sc = 20 - 10 * c;
    L.a0 = t.box[a];
    L.b0 = t.box[b];
    L.c0 = t.box[c];
    L.two = eb > 4 ? 1 : 0;
    L.empty = ex <= 0 && !t.wide;
    // a warp lists at most 8 words' blocks (tile_flush_words); every offset from
    // the camera's block is a packable coordinate
    constexpr unsigned room = kCoordBias - kSetOff;
    const bool near = (unsigned)cbx + room <= 2 * room && (unsigned)cby + room <= 2 * room && (unsigned)cbz + room <= 2 * room;
    L.fits = !t.wide && near && ex > 0 && L.na <= 16 && eb <= 8 && ec <= 8 && (L.na << L.two) <= 8 * (int)blockDim.y;
    return L;
}

// ORs the warp's cubes into the words of one phase.
__device__ __forceinline__ void tile_fill_bits(PackedCube k, const TileLayout &L, unsigned *words) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const bool any = k.hi >= k.lo;
    const int a0 = any ? (int)(((k.lo >> L.sa) & 1023u) - L.a0) : 31, a1 = any ? (int)(((k.hi >> L.sa) & 1023u) - L.a0) : -1;
    const unsigned b0 = ((k.lo >> L.sb) & 1023u) - L.b0, nb = ((k.hi >> L.sb) & 1023u) - L.b0 - b0;
    const unsigned c0 = ((k.lo >> L.sc) & 1023u) - L.c0, nc = ((k.hi >> L.sc) & 1023u) - L.c0 - c0;
    const unsigned row = any ? ((2u << nc) - 1u) << c0 : 0u;  // a byte's bits
    const unsigned rows = any ? ((2u << nb) - 1u) << b0 : 0u; // which bytes
    // a nibble's bits spread to four bytes' lowest, times the byte
    const unsigned m0 = ((rows & 15u) * 0x00204081u & 0x01010101u) * row;
    const unsigned m1 = ((rows >> 4) * 0x00204081u & 0x01010101u) * row;
    const int first = __reduce_min_sync(FULL, a0), last = __reduce_max_sync(FULL, a1);
    unsigned mine = 0u;
    for (int a = first; a <= last; a++) {
        const bool in = a >= a0 && a <= a1;
        const unsigned o0 = __reduce_or_sync(FULL, in ? m0 : 0u);
        if (lane == a << L.two) mine = o0;
        if (L.two) {
            const unsigned o1 = __reduce_or_sync(FULL, in ? m1 : 0u);
            if (lane == 2 * a + 1) mine = o1;
        }
    }
    if (mine) atomicOr(words + lane, mine);
}

// A listed block: bit `lane` of word w, with its tag.
template <bool kTagged>
__device__ __forceinline__ unsigned tile_bit_key(const TileLayout &L, int w, int lane, unsigned b0, unsigned b1) {
    const unsigned ka = L.a0 + (unsigned)(w >> L.two), kb = L.b0 + (L.two ? 4u * (w & 1) : 0u) + (lane >> 3),
                   kc = L.c0 + (lane & 7);
    const unsigned tag = kTagged ? ((b0 >> lane) & 1u) | ((b1 >> lane) & 1u) << 1 : 0u;
    return ka << L.sa | kb << L.sb | kc << L.sc | tag << 30;
}

// Phase 2 from the bits (after a CTA barrier that follows the fills), list: the
// set's memory. Two ways to share a tile's blocks among its warps:
// - one frame, where the latency of the visits counts: warp w lists the blocks
//   of words w, w + nw, ... and visits them (at most 8 words: 256 entries);
// - a re-fusion's many tiles, where the instructions count: warp w visits the
//   tile's blocks 32 w .. 32 w + 31, in the order of the bits, then those 32 nw
//   further, so that a visit's lanes are full and most warps of a tile have
//   none (100 keyframes 0.86 -> 0.79 ms, but 1 us more for one 517 x 389 frame).
template <class Visit>
__device__ __forceinline__ void tile_flush_words(const GridView &g, const TileBits &t, const TileLayout &L, unsigned *list,
                                                 int nw, int cbx, int cby, int cbz, Visit &visit) {
    const int tid = threadIdx.y * blockDim.x + threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const unsigned lt = (1u << lane) - 1u;
    unsigned *wlist = list + wid * 256;
    int cnt = 0;
    for (int w = wid; w < L.na << L.two; w += nw) {
        const unsigned b = t.bits[0][w];
        if ((b >> lane) & 1u) wlist[cnt + __popc(b & lt)] = tile_bit_key<false>(L, w, lane, b, 0u);
        cnt += __popc(b);
    }
    tile_visit_list<false>(g, wlist, cnt, cbx, cby, cbz, visit);
}

template <class Visit>
__device__ __forceinline__ void tile_flush_tagged(const GridView &g, const TileBits &t, const TileLayout &L, unsigned *list,
                                                  int nw, int cbx, int cby, int cbz, Visit &visit) {
    const unsigned FULL = 0xffffffffu;
    const int tid = threadIdx.y * blockDim.x + threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const unsigned lt = (1u << lane) - 1u;
    const int words = L.na << L.two;
    unsigned *wlist = list + wid * 32;
    int incl = __popc(t.bits[0][lane] | t.bits[1][lane]);  // words past the last are zero
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(FULL, incl, o);
        if (lane >= o) incl += v;
    }
    const int total = __shfl_sync(FULL, incl, 31);
    for (int first = wid * 32; first < total; first += nw * 32) {
        __syncwarp();
        int at = 0;  // the number of the word's first block
        for (int w = __popc(__ballot_sync(FULL, incl <= first)); w < words && at < first + 32; w++) {
            at = w ? __shfl_sync(FULL, incl, w - 1) : 0;
            const unsigned b0 = t.bits[0][w], b1 = t.bits[1][w], b = b0 | b1;
            const int pos = at + __popc(b & lt) - first;
            if (((b >> lane) & 1u) && pos >= 0 && pos < 32) wlist[pos] = tile_bit_key<true>(L, w, lane, b0, b1);
        }
        tile_visit_list<true>(g, wlist, min(total - first, 32), cbx, cby, cbz, visit);
    }
}

// Phase 1 for a pixel of the tile with the cube c of blocks (every thread of
// the CTA calls it; the set, and a tagged set's tags, must be cleared and the
// CTA synced before; fills of a tagged set may follow one another without a
// barrier).
template <bool kTagged, class Visit>
__device__ __forceinline__ void tile_fill_set(const GridView &g, const TileCube &c, unsigned *cset, int slots, int cbx,
                                              int cby, int cbz, unsigned tag, Visit &visit) {
    const unsigned FULL = 0xffffffffu;
    __syncwarp();  // the warp's lanes are done with its cube entries of an earlier fill
    const int lox = c.lox, loy = c.loy, loz = c.loz, nx = c.nx, ny = c.ny, nz = c.nz;
    const int total = nx * ny * nz;
    const int tid = threadIdx.y * blockDim.x + threadIdx.x;
    const int lane = tid & 31, wid = tid >> 5;
    const unsigned lt = (1u << lane) - 1u;
    const uint32_t hmask = (uint32_t)(slots - 1);
    const int hshift = __clz(slots) + 1;  // 32 - log2(slots)
    // Neighbouring pixels mostly share their whole cube of candidates: lanes
    // are grouped by cube (corner and extent), each group's leader enters its
    // cube in the warp's table, and the cubes' blocks are then spread over the
    // lanes, 32 per step. A cube is enumerated over its extents rounded up to
    // powers of two (x outer, z inner), so an item's offsets are shifts and
    // masks; items past an extent are skipped (none while the truncation band
    // spans at most two blocks per axis, the usual case).
    const bool small = abs(lox) < (1 << 16) && abs(loy) < (1 << 16) && abs(loz) < (1 << 16);
    unsigned long long cube = ~0ull - (unsigned long long)lane;  // no cube, or one not grouped: its own key
    if (total > 0 && small)
        cube = ((unsigned long long)(lox & 0x1ffff) << 46) | ((unsigned long long)(loy & 0x1ffff) << 29) |
               ((unsigned long long)(loz & 0x1ffff) << 12) | (unsigned long long)((nx - 1) | (ny - 1) << 4 | (nz - 1) << 8);
    const unsigned peers = __match_any_sync(FULL, cube);
    const bool leader = total > 0 && __ffs(peers) - 1 == lane;
    const unsigned lmask = __ballot_sync(FULL, leader);
    // log2 of the padded extents: 1 -> 0, 2 -> 1, 3-4 -> 2, 5-8 -> 3
    const int ly = 32 - __clz(max(ny - 1, 0)), lz = 32 - __clz(max(nz - 1, 0));
    const int padded = leader ? (1 << (32 - __clz(max(nx - 1, 0)) + ly + lz)) : 0;
    int incl = padded;  // inclusive scan of the leaders' padded block counts
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(FULL, incl, o);
        if (lane >= o) incl += t;
    }
    const int work = __shfl_sync(FULL, incl, 31);
    const int first = incl - padded;  // a leader's first item
    int4 *cubes = reinterpret_cast<int4 *>(cset + 2 * slots) + wid * 32;
    if (leader)
        cubes[__popc(lmask & lt)] =
            make_int4(lox, loy, loz, first << 16 | lz << 11 | ly << 9 | (nz - 1) << 6 | (ny - 1) << 3 | (nx - 1));
    __syncwarp();
    for (int base = 0; base < work; base += 32) {
        // the cube of item w: the leaders that started before this step, plus
        // those starting in it at or before w (one bit per starting item)
        const unsigned starts =
            __reduce_or_sync(FULL, leader && first >= base && first < base + 32 ? 1u << (first - base) : 0u);
        const int before = __popc(__ballot_sync(FULL, leader && first < base));
        const int w = base + lane;
        unsigned key = kSetEmpty;
        bool direct = false;
        int cx = 0, cy = 0, cz = 0;
        if (w < work) {
            const int4 cb = cubes[before + __popc(starts & (0xffffffffu >> (31 - lane))) - 1];
            const int c = w - (cb.w >> 16), sz = (cb.w >> 11) & 3, sy = (cb.w >> 9) & 3;
            const int dz = c & ((1 << sz) - 1), dy = (c >> sz) & ((1 << sy) - 1), dx = c >> (sz + sy);
            if (dx <= (cb.w & 7) && dy <= ((cb.w >> 3) & 7) && dz <= ((cb.w >> 6) & 7)) {
                cx = cb.x + dx;
                cy = cb.y + dy;
                cz = cb.z + dz;
                if (packable(cx, cy, cz)) {
                    const unsigned ox = (unsigned)(cx - cbx + kSetOff), oy = (unsigned)(cy - cby + kSetOff),
                                   oz = (unsigned)(cz - cbz + kSetOff);
                    if (ox < 2u * kSetOff && oy < 2u * kSetOff && oz < 2u * kSetOff) key = (ox << 20) | (oy << 10) | oz;
                    else direct = true;
                } else {
                    atomicOr(&g.ctr->status, kStRange);
                }
            }
        }
        if (direct) visit_one(g, cx, cy, cz, tag, visit);  // outside the key range
        if (key == kSetEmpty) continue;
        // most blocks are already in the set (another warp or step put them
        // there): a plain load finds those without an atomic
        uint32_t h = (key * 0x9E3779B1u) >> hshift;  // the product's top bits (multiplicative hashing)
        int at = -1;
        for (int probe = 0; probe < slots / 2 && at < 0; probe++) {
            h &= hmask;
            unsigned cur = ((volatile unsigned *)cset)[h];
            if (cur == kSetEmpty) cur = atomicCAS(cset + h, kSetEmpty, key);
            if (cur == kSetEmpty || cur == key) at = (int)h;
            h++;
        }
        if (at < 0) {
            visit_one(g, cx, cy, cz, tag, visit);  // set too crowded
        } else if (kTagged) {
            unsigned *tg = tile_tags(cset, slots) + at;
            if ((*(volatile unsigned *)tg & tag) != tag) atomicOr(tg, tag);
        }
    }
}

// Phase 2 (every thread of the CTA calls it after a CTA barrier that follows
// phase 1): warp w compacts slots [w per, (w + 1) per) into its list (a key
// has 30 bits; a tagged set's tag rides in the top two) and visits its
// distinct blocks, appending with one atomic per warp step.
template <bool kTagged, class Visit>
__device__ __forceinline__ void tile_flush_set(const GridView &g, unsigned *cset, int slots, int cbx, int cby,
                                               int cbz, Visit &visit) {
    const unsigned FULL = 0xffffffffu;
    const int tid = threadIdx.y * blockDim.x + threadIdx.x, nthreads = blockDim.x * blockDim.y;
    const int lane = tid & 31, wid = tid >> 5, nw = nthreads >> 5, per = slots / nw;
    const unsigned lt = (1u << lane) - 1u;
    unsigned *wlist = cset + slots + wid * per;
    int cnt = 0;
    for (int r = 0; r < per; r += 32) {
        const unsigned key = cset[wid * per + r + lane];
        const bool present = key != kSetEmpty;
        const unsigned b = __ballot_sync(FULL, present);
        if (present)
            wlist[cnt + __popc(b & lt)] = kTagged ? key | tile_tags(cset, slots)[wid * per + r + lane] << 30 : key;
        cnt += __popc(b);
    }
    tile_visit_list<kTagged>(g, wlist, cnt, cbx, cby, cbz, visit);
}

// Find or insert a block, then stamp it with this call's epoch: the first
// visitor of the epoch appends it (replaces alreadyIntegrated and the
// O(capacity) "Reset booleans" pass); the 64-bit atomicMax on (epoch, packed
// coordinates) also fixes an aliased entry's coordinates canonically (the
// largest packed coordinate of the call). Most visits find the block in its
// home bucket, already stamped by an earlier tile: the home bucket's key and
// stamp (and, with a side array, the block's word of it) are loaded together,
// so such a visit costs one round trip to L2 and no atomic. A stamp that
// already holds this call's value or a larger one would not change, and its
// epoch says "not first", so skipping the atomicMax then changes nothing.
// With a side array (words per bucket `side_stride`), the block's word
// `side_word` gets the bits `side_bit` ORed in (a load first: they are
// usually set; the atomic unless all of them are).
template <bool kSide = false>
__device__ __forceinline__ bool find_and_stamp(const GridView &g, uint32_t epoch, int bx, int by, int bz, int &bucket,
                                               uint32_t *side = nullptr, int side_stride = 0, int side_word = 0,
                                               uint32_t side_bit = 0) {
    const unsigned long long key = prime_hash(bx, by, bz);
    const unsigned long long val = ((unsigned long long)epoch << kEpochShift) | pack_coords(bx, by, bz);
    const uint32_t home = home_bucket(key, g.mask);
    const unsigned long long k0 = ld_relaxed(g.keys + home);
    const unsigned long long s0 = ld_relaxed(g.stamp + home);
    uint32_t m0 = 0;
    if (kSide) m0 = ld_relaxed_u32(side + (size_t)home * side_stride + side_word);
    bool append = false;
    if (k0 == key) {
        bucket = (int)home;
        if (s0 < val) append = (uint32_t)(atomicMax(g.stamp + home, val) >> kEpochShift) != epoch;
    } else {
        bool inserted = false;
        bucket = table_find_or_insert(g, key, &inserted);
        if (inserted) super_insert(g, bx, by, bz);
        if (bucket < 0) return false;
        append = (uint32_t)(atomicMax(g.stamp + bucket, val) >> kEpochShift) != epoch;
        if (kSide) m0 = ld_relaxed_u32(side + (size_t)bucket * side_stride + side_word);
    }
    if (kSide && (m0 & side_bit) != side_bit) atomicOr(side + (size_t)bucket * side_stride + side_word, side_bit);
    return append;
}

}  // namespace ss
