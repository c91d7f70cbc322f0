// world.cu -- mode-P world storage on the device and its upload entry points.
//
// The reference keeps its world in two persistently mapped SSBOs that the host
// writes voxel by voxel (VoxelBrickmap, src/engine/voxel.zig:25-82): a 64^3
// chunk table of brick indices and a pool of 8^3 u32 bricks.  Here the host
// hands over uint8 materials (dense, or one 32^3 chunk at a time) and a kernel
// builds the traversal structures on the device:
//
//   materials  chunk-major; inside a chunk 512 bricks of 64 bytes, brick
//              b = bx + 8*(by + 8*bz), voxel v = x + 4*(y + 4*z) in the brick
//   mask       one u64 per brick, bit v set iff material != 0
//   coarse     one bit per chunk, set iff any brick word of the chunk is != 0
#include <cuda_fp16.h>

#include <algorithm>
#include <cstring>

#include "dist.cuh"
#include "vt_internal.h"

namespace vt {

// One block per chunk, one thread per brick.  src is a dense x-fastest box of
// sdims voxels whose voxel (0,0,0) sits at world voxel `sorg`; world cells
// outside the source box or outside the world read as air.
__global__ void __launch_bounds__(512) k_build_chunks(WorldView w, unsigned long long* mask, unsigned char* mats,
                                                      unsigned long long* coarse, const unsigned char* __restrict__ src,
                                                      int3 sdims, int3 sorg, int3 cfirst, int3 ccount) {
    const int lin = blockIdx.x;
    const int cx = cfirst.x + lin % ccount.x;
    const int cy = cfirst.y + (lin / ccount.x) % ccount.y;
    const int cz = cfirst.z + lin / (ccount.x * ccount.y);
    const unsigned ci = (unsigned)cx + (unsigned)w.cdim[0] * ((unsigned)cy + (unsigned)w.cdim[1] * (unsigned)cz);
    const int b = threadIdx.x;
    const int bx = b & 7, by = (b >> 3) & 7, bz = b >> 6;
    const unsigned wi = ci * 512u + (unsigned)b;
    unsigned long long m = 0ull;
    unsigned packed[16];
#pragma unroll
    for (int z = 0; z < 4; ++z) {
#pragma unroll
        for (int y = 0; y < 4; ++y) {
            unsigned word = 0;
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                const int gx = cx * 32 + bx * 4 + x, gy = cy * 32 + by * 4 + y, gz = cz * 32 + bz * 4 + z;
                const int sx = gx - sorg.x, sy = gy - sorg.y, sz = gz - sorg.z;
                unsigned v = 0;
                if (gx < w.dims[0] && gy < w.dims[1] && gz < w.dims[2] && sx >= 0 && sy >= 0 && sz >= 0 &&
                    sx < sdims.x && sy < sdims.y && sz < sdims.z)
                    v = src[(size_t)sx + (size_t)sdims.x * ((size_t)sy + (size_t)sdims.y * (size_t)sz)];
                word |= v << (8 * x);
                if (v) m |= 1ull << (x + 4 * (y + 4 * z));
            }
            packed[y + 4 * z] = word;
        }
    }
    uint4* dst = reinterpret_cast<uint4*>(mats + (size_t)wi * 64u);
#pragma unroll
    for (int q = 0; q < 4; ++q) dst[q] = make_uint4(packed[4 * q], packed[4 * q + 1], packed[4 * q + 2], packed[4 * q + 3]);
    mask[wi] = m;
    const int any = __syncthreads_or(m != 0ull);
    if (threadIdx.x == 0) {
        const unsigned long long bit = 1ull << (ci & 63u);
        if (any) atomicOr(coarse + (ci >> 6), bit);
        else atomicAnd(coarse + (ci >> 6), ~bit);
    }
}

// VoxelBrickmap.set (voxel.zig:58-61): one voxel, then the chunk's coarse bit.
__global__ void __launch_bounds__(512) k_set_voxel(WorldView w, unsigned long long* mask, unsigned char* mats,
                                                   unsigned long long* coarse, int x, int y, int z, unsigned mat) {
    const unsigned ci = (unsigned)(x >> 5) + (unsigned)w.cdim[0] * ((unsigned)(y >> 5) + (unsigned)w.cdim[1] * (unsigned)(z >> 5));
    const unsigned bi = (unsigned)((x >> 2) & 7) | ((unsigned)((y >> 2) & 7) << 3) | ((unsigned)((z >> 2) & 7) << 6);
    const unsigned vb = (unsigned)(x & 3) | ((unsigned)(y & 3) << 2) | ((unsigned)(z & 3) << 4);
    if (threadIdx.x == 0) {
        const unsigned wi = ci * 512u + bi;
        mats[(size_t)wi * 64u + vb] = (unsigned char)mat;
        if (mat) mask[wi] |= 1ull << vb;
        else mask[wi] &= ~(1ull << vb);
    }
    __syncthreads();
    const int any = __syncthreads_or(mask[ci * 512u + threadIdx.x] != 0ull);
    if (threadIdx.x == 0) {
        const unsigned long long bit = 1ull << (ci & 63u);
        if (any) atomicOr(coarse + (ci >> 6), bit);
        else atomicAnd(coarse + (ci >> 6), ~bit);
    }
}

// Empty-space distances, per direction octant.  For the octant with signs s,
// a weighted Chebyshev distance to the nearest occupied cell ahead is
// separable:
//     min over c' ahead of max(|dx|, w|dy|, |dz|)
//   = min_{dz ahead} max(|dz|, min_{dy ahead} max(w|dy|, min_{dx ahead} max(|dx|, occ(c')))),
// so each field is three one-sided 1-D min-max passes, x, then y, then z.
// The x pass depends on s_x only (2 fields), the y pass on s_x, s_y (4 fields),
// the z pass on all three (8 fields).  Cells outside the grid count as empty.
//
// Chunk level: chunks to chunks, "ahead" meaning 0 <= s_i * d_i <= kDistCap,
// capped at kDistCap + 1.  blockIdx.y is the output field v: bit i of v gives
// the direction of axis i (1: +) for axes 0..axis; the pass reads input field
// v & ((1 << axis) - 1) (pass 0 reads the coarse bits instead).  Fields are
// `stride` bytes apart.  The pass covers the whole chunk grid.
// The window's reads are independent and all in flight at once.
__device__ __forceinline__ void dist_cell(const unsigned long long* coarse, const unsigned char* in, unsigned char* out,
                                          int axis, bool fwd, int CX, int CY, int CZ, unsigned lin) {
    const unsigned p[3] = {lin % (unsigned)CX, (lin / (unsigned)CX) % (unsigned)CY, lin / ((unsigned)CX * (unsigned)CY)};
    const int u = (int)(axis == 0 ? p[0] : (axis == 1 ? p[1] : p[2])), g = axis == 0 ? CX : (axis == 1 ? CY : CZ);
    const int step = (axis == 0 ? 1 : (axis == 1 ? CX : CX * CY)) * (fwd ? 1 : -1);
    int val[kDistCap + 1];
#pragma unroll
    for (int d = 0; d <= kDistCap; ++d) {
        const int q = fwd ? u + d : u - d;
        val[d] = kDistCap + 1;
        if (q >= 0 && q < g) {
            const unsigned idx = (unsigned)((int)lin + d * step);
            val[d] = axis == 0 ? (((coarse[idx >> 6] >> (idx & 63u)) & 1ull) ? 0 : kDistCap + 1) : (int)in[idx];
        }
    }
    int best = kDistCap + 1;
#pragma unroll
    for (int d = 0; d <= kDistCap; ++d) best = min(best, max(d, val[d]));
    out[lin] = (unsigned char)best;
}

// d_changed (null: always run): the pass is skipped when it points to 0, a
// device-side edit that left every coarse bit as it was.
__global__ void k_dist_pass(const unsigned long long* coarse, const unsigned char* in, unsigned char* out, int axis,
                            int CX, int CY, int CZ, size_t stride, const int* d_changed) {
    if (d_changed && !*d_changed) return;
    const unsigned v = blockIdx.y, lin = blockIdx.x * blockDim.x + threadIdx.x;
    if (lin >= (unsigned)CX * (unsigned)CY * (unsigned)CZ) return;
    if (axis > 0) in += (size_t)(v & ((1u << axis) - 1u)) * stride;
    dist_cell(coarse, in, out + (size_t)v * stride, axis, ((v >> axis) & 1u) != 0u, CX, CY, CZ, lin);
}

// The three passes of a small grid in one launch, a block per octant (output
// field), which keeps its own x and y results in shared memory.  Bound: the
// latency of a few dependent rounds of loads.  2048 chunks: 9.1 us against 9.2
// in three launches and the gaps between them; after an edit that changed a
// coarse bit 9.3 us against 36 as one block for all octants, after one that
// changed none (the rule for single voxels) 2.7 against 8.
constexpr int kSmallChunks = 4096;
__global__ void __launch_bounds__(1024) k_dist_small(const unsigned long long* coarse, unsigned char* out, int CX, int CY,
                                                     int CZ, size_t stride, const int* d_changed) {
    if (d_changed && !*d_changed) return;
    __shared__ unsigned char fx[kSmallChunks], fy[kSmallChunks];
    const unsigned n = (unsigned)CX * (unsigned)CY * (unsigned)CZ, v = blockIdx.x;
    for (unsigned i = threadIdx.x; i < n; i += 1024u) dist_cell(coarse, nullptr, fx, 0, (v & 1u) != 0u, CX, CY, CZ, i);
    __syncthreads();
    for (unsigned i = threadIdx.x; i < n; i += 1024u) dist_cell(nullptr, fx, fy, 1, (v & 2u) != 0u, CX, CY, CZ, i);
    __syncthreads();
    for (unsigned i = threadIdx.x; i < n; i += 1024u)
        dist_cell(nullptr, fy, out + (size_t)v * stride, 2, (v & 4u) != 0u, CX, CY, CZ, i);
}

// Brick level, in voxels.  With vertical weight w = 2^shape, brick b has
//     s_w = min(kVoxCap + 1, min over occupied voxels q ahead of b of max(dx, w*dy, dz)),
// where d_i is the number of voxel layers between b's far face on axis i and
// q (0 when q lies within b's extent on that axis) and "ahead" means q is not
// behind b's near face on any axis: b plus s_w - 1 layers beyond its far faces
// across and (s_w - 1) / w layers vertically holds no occupied voxel (s_w = 0:
// b is occupied).  Field o of b stores s_1 for the octants moving +y, and for
// those moving -y the s_w | shape << 6 of the shape with the largest box
// (box_score; the smallest weight on a tie).  Each pass coarsens one axis from
// voxels to bricks:
//   x: X(bx, qy, qz), 2 fields (x direction): layers from brick bx's far x face
//      to the first occupied voxel of row (qy, qz) (read from the mask words);
//   y: Y(bx, by, qz), kYFields fields (y_field: x and y direction, and for -y
//      the shape): min over qy of max(w*dy, X(bx, qy, qz));
//   z: the brick field, 8 fields: min over qz of max(dz, Y(bx, by, qz)), and
//      the shape choice.
// The intermediates are x-fastest arrays: X over (GX bricks, GY*4, GZ*4
// voxels), Y over (GX, GY bricks, GZ*4 voxels).  Each pass covers a box of
// its own output grid, [lo, lo + ext) clipped to the grid (and widened in x to
// whole chunks or groups of four bricks: recomputing a cell that cannot have
// changed gives the value it has); with `d_cell` ({x, y, z, valid, coarse bit
// changed} of an edited voxel in device memory) the box is taken relative to that voxel's brick
// (brick axes) or the brick's first voxel (voxel axes), and skipped when
// !valid.
//
// Bound: the passes are scans over L2-resident bytes.  One byte per thread and
// step was bound by instruction issue (512x256x512 cave world: x 485, y 1111,
// z 804 us).  The x pass now finds first voxels with bit scans of 32-voxel row
// words, and the y and z passes scan four bricks at a time (one 32-bit load,
// 16-bit pair minima and maxima), the four shapes of a downward field in one
// scan; bricks of chunks with open space ahead are not scanned: x 29, y 61, z 64 us
// (42, 108, 126 with every brick scanned).
// The y pass's fields: x direction xs, y direction ys (1: +y) and, for -y,
// the box shape.
constexpr int kYFields = 2 + 2 * kBoxShapes;
__host__ __device__ constexpr int y_field(int xs, int ys, int shape) { return ys ? xs : 2 + xs + 2 * shape; }

// lo relative to the brick of the edited voxel, or in z (voxel layers) to its
// first voxel.
__device__ __forceinline__ int3 edit_origin(int3 lo, const int* d_cell, bool z_voxels) {
    const int bz = d_cell[2] >> 2;
    return make_int3(lo.x + (d_cell[0] >> 2), lo.y + (d_cell[1] >> 2), lo.z + (z_voxels ? 4 * bz : bz));
}

__global__ void k_bdist_x(const unsigned long long* __restrict__ mask, const unsigned long long* __restrict__ coarse,
                          unsigned char* __restrict__ xf, BrickGrid b, int3 lo, int3 ext) {
    int cx, by, qz;
    if (box_item(blockIdx.x * blockDim.x + threadIdx.x, lo, ext, 8, make_int3(b.GX, b.GY, b.GZ * 4), cx, by, qz))
        bdist_x_item<false>(mask, coarse, xf, b, cx, by, qz);
}

// Four bytes (at most 63) as two pairs of 16-bit values with the byte on top:
// bytes 1 and 3 in place, bytes 0 and 2 shifted up.  What lies below the byte
// only breaks ties.  Such values are positive finite halves, whose order is
// that of their bits, so the half-precision pair minimum and maximum (one
// instruction each) apply.
struct Quad {
    unsigned odd, even;
};
__device__ __forceinline__ unsigned pair_min(unsigned a, unsigned b) {
    const __half2 r = __hmin2(*reinterpret_cast<__half2*>(&a), *reinterpret_cast<__half2*>(&b));
    return *reinterpret_cast<const unsigned*>(&r);
}
__device__ __forceinline__ unsigned pair_max(unsigned a, unsigned b) {
    const __half2 r = __hmax2(*reinterpret_cast<__half2*>(&a), *reinterpret_cast<__half2*>(&b));
    return *reinterpret_cast<const unsigned*>(&r);
}
__device__ __forceinline__ unsigned quad_bytes(Quad q) { return (q.odd & 0xFF00FF00u) | ((q.even >> 8) & 0x00FF00FFu); }
// best = min(best, max(dist, v)) in each byte for two layers, of distances d2
// and e2 (dist in both pair bytes).  The integer minimum of three has the same
// order, and takes two layers at once (z pass 68.0 -> 64.4 us, y the same).
__device__ __forceinline__ void quad_take2(Quad& best, unsigned v, unsigned d2, unsigned u, unsigned e2) {
    best.odd = __vimin3_s16x2(best.odd, pair_max(v, d2), pair_max(u, e2));
    best.even = __vimin3_s16x2(best.even, pair_max(v * 256u, d2), pair_max(u * 256u, e2));
}
// The largest of the four.
__device__ __forceinline__ unsigned quad_max(Quad q) {
    const unsigned m = pair_max(q.odd, q.even);
    return max(m & 0xFFFFu, m >> 16) >> 8;
}

// Scans the layers ahead of a brick, four bricks at a time: NF input fields f,
// `step` bytes from one layer to the next, layers 0..3 the brick's own, `count`
// (a multiple of 4) in the grid.  Result k of a field: min over layers of
// max(distance << k, byte), k < NW (NF or NW is 1).  Four layers are in
// flight; a layer whose distance reaches every best cannot lower one, and with
// weight 2^k the distances end at layer 3 + 62 / 2^k.  PREFETCH: the next four
// are on their way before four are used (the z pass, whose loads go to L2: 126
// against 153 us, 18 against 75 us after one edit; the y pass, whose loads hit
// L1, is 8% faster without).
template <int NF, int NW, bool PREFETCH>
__device__ __forceinline__ void scan_layers(const unsigned char* const* f, ptrdiff_t step, int count, Quad* best) {
    static_assert(NF == 1 || NW == 1, "several fields or several weights");
#pragma unroll
    for (int k = 0; k < NF * NW; ++k) best[k].odd = best[k].even = 0x3FFF3FFFu;   // kVoxCap + 1
    static_assert(kVoxCap + 1 == 0x3F, "the cap's byte");
    // the brick's own layers: distance 0, the same for every weight
    unsigned v[NF][4], n[NF][4];
    auto load = [&](unsigned (&to)[NF][4], int t) {
#pragma unroll
        for (int k = 0; k < NF; ++k)
#pragma unroll
            for (int j = 0; j < 4; ++j)
                to[k][j] = __ldg(reinterpret_cast<const unsigned*>(f[k] + (ptrdiff_t)(t + j) * step));
    };
    load(v, 0);
    if (PREFETCH && count > 4) load(n, 4);
#pragma unroll
    for (int k = 0; k < NF; ++k) {
#pragma unroll
        for (int j = 0; j < 4; j += 2) {
            best[k].odd = __vimin3_s16x2(best[k].odd, v[k][j], v[k][j + 1]);
            best[k].even = __vimin3_s16x2(best[k].even, v[k][j] * 256u, v[k][j + 1] * 256u);
        }
#pragma unroll
        for (int s = 1; s < NW; ++s) best[s] = best[0];
    }
    unsigned most = quad_max(best[0]);
#pragma unroll
    for (int k = 1; k < NF; ++k) most = max(most, quad_max(best[k]));
    int t = 4;
    unsigned d2 = 0x01000100u;
#pragma unroll
    for (int weights = NW; weights >= 1; --weights) {   // results 0 .. weights - 1 are still open
        const int end = weights == 1 ? count : min(count, (4 + (kVoxCap >> (weights - 1)) + 3) / 4 * 4);
        // t - 3: the next layer's distance; the other weights end no later
        for (; (unsigned)(t - 3) < most && t < end; t += 4) {
            if (PREFETCH) {
#pragma unroll
                for (int k = 0; k < NF; ++k)
#pragma unroll
                    for (int j = 0; j < 4; ++j) v[k][j] = n[k][j];
                if (t + 4 < count) load(n, t + 4);
            } else {
                load(v, t);
            }
#pragma unroll
            for (int j = 0; j < 4; j += 2) {
                // (distances past the cap, at most 62 + 28, change nothing)
#pragma unroll
                for (int k = 0; k < NF; ++k)
#pragma unroll
                    for (int s = 0; s < weights; ++s)
                        quad_take2(best[k + s], v[k][j], d2 << s, v[k][j + 1], (d2 + 0x01000100u) << s);
                d2 += 0x02000200u;
            }
            most = quad_max(best[0]);
#pragma unroll
            for (int k = 1; k < NF; ++k) most = max(most, quad_max(best[k]));
        }
    }
}

// The chunk distances of the grid (up to date before the brick passes).  From
// a chunk whose distance in an octant is 3 or more the two chunks ahead of it
// on every axis are empty, 64 layers: every brick of it is at the cap, and its
// scans are not run (the sky above a terrain).
struct ChunkDist {
    const unsigned char* d;
    unsigned stride;
    __device__ __forceinline__ bool far(const BrickGrid& b, unsigned oct, int bx, int by, int bz) const {
        const unsigned ci = (unsigned)(bx >> 3) + (unsigned)b.CX * ((unsigned)(by >> 3) + (unsigned)b.CY * (unsigned)(bz >> 3));
        return __ldg(d + oct * stride + ci) >= 3u;
    }
};
constexpr unsigned kAllFar = (unsigned)(kVoxCap + 1) * 0x01010101u;

// One thread: four bricks in x, one field (up) or the four shapes (down).
// blockIdx.y: x direction, y direction << 1.  EDIT: a column group whose values
// change is noted for the z pass.
template <bool EDIT>
__global__ void k_bdist_y(const unsigned char* __restrict__ xf, unsigned char* __restrict__ yf, BrickGrid b, int3 lo,
                          int3 ext, int* __restrict__ d_cell, ChunkDist cd) {
    if (EDIT) {
        if (!d_cell[3]) return;
        lo = edit_origin(lo, d_cell, true);
    }
    const int xs = (int)(blockIdx.y & 1u);
    const bool fwd = (blockIdx.y & 2u) != 0u;
    const int Y = b.GY * 4;
    const int3 g = make_int3(b.GX, b.GY, b.GZ * 4);
    int x4, by, qz;
    if (!box_item(blockIdx.x * blockDim.x + threadIdx.x, lo, ext, 4, g, x4, by, qz)) return;
    const unsigned char* near = xf + (size_t)xs * ((size_t)b.GX * Y * g.z) + (size_t)(4 * x4) +
                                (size_t)b.GX * ((size_t)(fwd ? 4 * by : 4 * by + 3) + (size_t)Y * qz);
    const size_t field = (size_t)g.x * g.y * g.z, cell = (size_t)(4 * x4) + (size_t)g.x * ((size_t)by + (size_t)g.y * qz);
    const unsigned char* const in[1] = {near};
    bool changed = false;
    auto store = [&](int f, unsigned v) {
        unsigned* at = reinterpret_cast<unsigned*>(yf + (size_t)f * field + cell);
        if (EDIT) changed = changed || *at != v;
        *at = v;
    };
    // the scan stays in one layer of z, ahead in both z octants
    const unsigned oct = (unsigned)xs | (fwd ? 2u : 0u);
    const bool far = cd.far(b, oct, 4 * x4, by, qz >> 2) || cd.far(b, oct | 4u, 4 * x4, by, qz >> 2);
    if (fwd) {
        Quad q[1];
        if (!far) scan_layers<1, 1, EDIT>(in, b.GX, Y - 4 * by, q);
        store(y_field(xs, 1, 0), far ? kAllFar : quad_bytes(q[0]));
    } else {
        Quad q[kBoxShapes];
        if (!far) scan_layers<1, kBoxShapes, EDIT>(in, -(ptrdiff_t)b.GX, 4 * by + 4, q);
#pragma unroll
        for (int shape = 0; shape < kBoxShapes; ++shape) store(y_field(xs, 0, shape), far ? kAllFar : quad_bytes(q[shape]));
    }
    if (EDIT && changed) d_cell[kEditColumns + (x4 - max(lo.x, 0) / 4) + kEditGroups * (by - lo.y)] = 1;
}

// One thread: four bricks in x, one octant (blockIdx.y).
// EDIT: only the column groups the y pass changed.
template <bool EDIT>
__global__ void k_bdist_z(const unsigned char* __restrict__ yf, unsigned char* __restrict__ out, BrickGrid b, int3 lo,
                          int3 ext, const int* __restrict__ d_cell, size_t stride, ChunkDist cd) {
    if (EDIT) {
        if (!d_cell[3]) return;
        lo = edit_origin(lo, d_cell, false);
    }
    const unsigned v = blockIdx.y;
    const bool fwd = (v & 4u) != 0u, up = (v & 2u) != 0u;
    const int xs = (int)(v & 1u);
    const int Z = b.GZ * 4;
    int x4, by, bz;
    if (!box_item(blockIdx.x * blockDim.x + threadIdx.x, lo, ext, 4, make_int3(b.GX, b.GY, b.GZ), x4, by, bz)) return;
    if (EDIT && !d_cell[kEditColumns + (x4 - max(lo.x, 0) / 4) + kEditGroups * (by - lo.y)]) return;
    const size_t layer = (size_t)b.GX * b.GY, yfield = layer * Z;
    const unsigned char* near = yf + (size_t)(4 * x4) + (size_t)b.GX * by + layer * (size_t)(fwd ? 4 * bz : 4 * bz + 3);
    const ptrdiff_t step = fwd ? (ptrdiff_t)layer : -(ptrdiff_t)layer;
    const int count = fwd ? Z - 4 * bz : 4 * bz + 4;
    unsigned res = 0u;
    if (cd.far(b, v, 4 * x4, by, bz)) {
        res = kAllFar;   // (shape 0 has the largest box)
    } else if (up) {
        const unsigned char* const in[1] = {near + (size_t)y_field(xs, 1, 0) * yfield};
        Quad q[1];
        scan_layers<1, 1, true>(in, step, count, q);
        res = quad_bytes(q[0]);
    } else {
        const unsigned char* in[kBoxShapes];
#pragma unroll
        for (int shape = 0; shape < kBoxShapes; ++shape) in[shape] = near + (size_t)y_field(xs, 0, shape) * yfield;
        Quad q[kBoxShapes];
        scan_layers<kBoxShapes, 1, true>(in, step, count, q);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            unsigned cell = 0u;
            int best_score = -1;
#pragma unroll
            for (int shape = 0; shape < kBoxShapes; ++shape) {
                const int s = (int)((((i & 1) ? q[shape].odd : q[shape].even) >> ((i >> 1) * 16 + 8)) & 0xFFu);
                const int score = box_score(s, shape);
                if (s != 0 && score > best_score) {   // s is 0 for every shape where the brick is occupied
                    best_score = score;
                    cell = (unsigned)(s | (shape << 6));
                }
            }
            res |= cell << (8 * i);
        }
    }
    *reinterpret_cast<unsigned*>(out + (size_t)v * stride + brick_index(4 * x4, by, bz, b.CX, b.CY)) = res;
}

namespace {

constexpr int kDistThreads = 256;

unsigned dist_blocks(size_t n) { return (unsigned)((n + kDistThreads - 1) / kDistThreads); }

size_t volume(int3 e) { return (size_t)e.x * e.y * e.z; }

// The chunk level over the whole chunk grid (at most a few tens of thousands
// of cells: cheap enough to redo after any edit, and skipped on the device
// after an edit that changed no coarse bit); of a larger grid x into 2 fields
// of tmp, y into the 4 fields after them, z into the 8 output fields.
void chunk_passes(vt_world* w, cudaStream_t st, const int* d_changed) {
    const int CX = w->cdim[0], CY = w->cdim[1], CZ = w->cdim[2];
    const size_t stride = cdist_stride((unsigned)w->nchunks);
    if (w->nchunks <= kSmallChunks) {
        k_dist_small<<<8, 1024, 0, st>>>(w->d_coarse, w->d_cdist, CX, CY, CZ, stride, d_changed);
        return;
    }
    unsigned char* fx = w->d_ctmp;
    unsigned char* fy = w->d_ctmp + 2 * stride;
    const unsigned nb = dist_blocks(w->nchunks);
    k_dist_pass<<<dim3(nb, 2), kDistThreads, 0, st>>>(w->d_coarse, nullptr, fx, 0, CX, CY, CZ, stride, d_changed);
    k_dist_pass<<<dim3(nb, 4), kDistThreads, 0, st>>>(w->d_coarse, fx, fy, 1, CX, CY, CZ, stride, d_changed);
    k_dist_pass<<<dim3(nb, 8), kDistThreads, 0, st>>>(w->d_coarse, fy, w->d_cdist, 2, CX, CY, CZ, stride, d_changed);
}

BrickGrid brick_grid(const vt_world* w) {
    return {w->cdim[0], w->cdim[1], w->cdim[2], w->cdim[0] * 8, w->cdim[1] * 8, w->cdim[2] * 8};
}

// Items of a pass over ext in groups of bricks in x (an aligned group more than
// the box's bricks need).
size_t box_items(int3 ext, int group) { return (size_t)((ext.x + group - 1) / group + 1) * ext.y * ext.z; }

// The brick level, each pass over its own box (x: bricks x brick rows x voxel
// layers, y: bricks x bricks x voxel layers, z: bricks).  The intermediates
// stay valid between calls, which is what lets an edit recompute only the
// boxes it can change.
void brick_passes(vt_world* w, cudaStream_t st, const int3 lo[3], const int3 ext[3]) {
    const BrickGrid b = brick_grid(w);
    const size_t nb = w->nchunks * kBricksPerChunk;
    const ChunkDist cd = {w->d_cdist, cdist_stride((unsigned)w->nchunks)};
    unsigned char* xf = w->d_dtmp;             // 2 fields of 16 bytes per brick
    unsigned char* yf = w->d_dtmp + 32 * nb;   // kYFields fields of 4 bytes per brick
    k_bdist_x<<<dist_blocks(box_items(ext[0], 8)), kDistThreads, 0, st>>>(w->d_mask, w->d_coarse, xf, b, lo[0], ext[0]);
    k_bdist_y<false><<<dim3(dist_blocks(box_items(ext[1], 4)), 4), kDistThreads, 0, st>>>(xf, yf, b, lo[1], ext[1], nullptr,
                                                                                            cd);
    k_bdist_z<false><<<dim3(dist_blocks(box_items(ext[2], 4)), 8), kDistThreads, 0, st>>>(yf, w->d_bdist, b, lo[2], ext[2],
                                                                                          nullptr, nb, cd);
}

// The y and z passes around the voxel of a device-side edit (whose kernel ran
// the x pass): the z pass over the column groups the y pass changed.
void edit_passes(vt_world* w, cudaStream_t st, const int3 lo[3], const int3 ext[3], int* d_cell) {
    const BrickGrid b = brick_grid(w);
    const size_t nb = w->nchunks * kBricksPerChunk;
    const ChunkDist cd = {w->d_cdist, cdist_stride((unsigned)w->nchunks)};
    unsigned char* xf = w->d_dtmp;
    unsigned char* yf = w->d_dtmp + 32 * nb;
    k_bdist_y<true><<<dim3((unsigned)((box_items(ext[1], 4) + 63) / 64), 4), 64, 0, st>>>(xf, yf, b, lo[1], ext[1], d_cell, cd);
    k_bdist_z<true><<<dim3((unsigned)((box_items(ext[2], 4) + 63) / 64), 8), 64, 0, st>>>(yf, w->d_bdist, b, lo[2], ext[2],
                                                                                        d_cell, nb, cd);
}

// After the bricks of box [blo, blo + bext) changed occupancy only these
// cells can change (R bricks: a pass stops before a layer kVoxCap + 1 beyond
// the far face, so it reads at most kVoxCap + 3 layers past the near face,
// which reaches R = (kVoxCap + 3) / 4 bricks away): the x pass in the box
// +- R bricks in x over the edited bricks' voxel rows, the y pass +- R bricks
// in x and y over their voxel layers in z, the z pass +- R bricks on every
// axis.  Recomputing those boxes, in pass order, from the current masks
// leaves every buffer equal to a full rebuild.
void edit_boxes(int3 blo, int3 bext, int3 lo[3], int3 ext[3]) {
    const int R = kEditReach;
    lo[0] = make_int3(blo.x - R, blo.y, 4 * blo.z);
    ext[0] = make_int3(bext.x + 2 * R, bext.y, 4 * bext.z);
    lo[1] = make_int3(blo.x - R, blo.y - R, 4 * blo.z);
    ext[1] = make_int3(bext.x + 2 * R, bext.y + 2 * R, 4 * bext.z);
    lo[2] = make_int3(blo.x - R, blo.y - R, blo.z - R);
    ext[2] = make_int3(bext.x + 2 * R, bext.y + 2 * R, bext.z + 2 * R);
}

}  // namespace

vt_status rebuild_distances(vt_world* w, cudaStream_t st) {
    const int GX = w->cdim[0] * 8, GY = w->cdim[1] * 8, GZ = w->cdim[2] * 8;
    const int3 o = make_int3(0, 0, 0);
    const int3 lo[3] = {o, o, o};
    const int3 ext[3] = {make_int3(GX, GY, 4 * GZ), make_int3(GX, GY, 4 * GZ), make_int3(GX, GY, GZ)};
    chunk_passes(w, st, nullptr);   // before the brick passes, which read them
    brick_passes(w, st, lo, ext);
    VT_CUDA(w->ctx, cudaGetLastError());
    w->dist_dirty = false;
    w->dist_box = false;
    return VT_OK;
}

vt_status update_distances(vt_world* w, cudaStream_t st) {
    if (w->dist_dirty) return rebuild_distances(w, st);
    if (!w->dist_box) return VT_OK;
    const int3 blo = make_int3(w->box_lo[0], w->box_lo[1], w->box_lo[2]);
    const int3 bext = make_int3(w->box_hi[0] - w->box_lo[0] + 1, w->box_hi[1] - w->box_lo[1] + 1,
                                w->box_hi[2] - w->box_lo[2] + 1);
    int3 lo[3], ext[3];
    edit_boxes(blo, bext, lo, ext);
    if (volume(ext[2]) >= w->nchunks * kBricksPerChunk / 2) return rebuild_distances(w, st);
    chunk_passes(w, st, nullptr);   // before the brick passes, which read them
    brick_passes(w, st, lo, ext);
    VT_CUDA(w->ctx, cudaGetLastError());
    w->dist_box = false;
    return VT_OK;
}

vt_status update_distances_at(vt_world* w, int* d_cell, cudaStream_t st) {
    vt_status s = update_distances(w, st);
    if (s || w->dist_dirty) return s;
    int3 lo[3], ext[3];
    edit_boxes(make_int3(0, 0, 0), make_int3(1, 1, 1), lo, ext);
    chunk_passes(w, st, d_cell + kEditCoarse);
    edit_passes(w, st, lo, ext, d_cell);
    VT_CUDA(w->ctx, cudaGetLastError());
    return VT_OK;
}

// Records an edit of the bricks in [lo, hi] (inclusive brick coordinates):
// the distances near them are recomputed before the next use (unless a full
// rebuild is pending anyway).
static void note_edit(vt_world* w, const int lo[3], const int hi[3]) {
    if (w->dist_dirty) return;
    for (int i = 0; i < 3; ++i) {
        if (!w->dist_box || lo[i] < w->box_lo[i]) w->box_lo[i] = lo[i];
        if (!w->dist_box || hi[i] > w->box_hi[i]) w->box_hi[i] = hi[i];
    }
    w->dist_box = true;
}

vt_status world_stage(vt_world* w, size_t bytes, unsigned char** out) {
    if (bytes <= w->stage_bytes) {
        *out = w->d_stage;
        return VT_OK;
    }
    if (w->d_stage) {
        VT_CUDA(w->ctx, cudaDeviceSynchronize());
        vt::dev_free(w->d_stage);
        w->d_stage = nullptr;
        w->stage_bytes = 0;
    }
    VT_CUDA(w->ctx, vt::dev_alloc(&w->d_stage, bytes));
    w->stage_bytes = bytes;
    *out = w->d_stage;
    return VT_OK;
}

// The palette as given, and its channels / 255 (correctly rounded, as the
// shading's table): a hit's albedo is then one 16-byte load.
static cudaError_t upload_palette(vt_world* w, const uint32_t* rgba) {
    unsigned char bytes[kPaletteBytes];
    std::memcpy(bytes, rgba, 256 * sizeof(uint32_t));
    for (int i = 0; i < 1024; ++i) {
        const float v = (float)((rgba[i >> 2] >> (8 * (i & 3))) & 255u) / 255.0f;
        std::memcpy(bytes + 256 * sizeof(uint32_t) + i * sizeof(float), &v, sizeof(float));
    }
    return cudaMemcpy(w->d_palette, bytes, sizeof(bytes), cudaMemcpyHostToDevice);
}

static void free_world(vt_world* w) {
    if (w->d_mask) vt::dev_free(w->d_mask);
    if (w->d_mats) vt::dev_free(w->d_mats);
    if (w->d_coarse) vt::dev_free(w->d_coarse);
    if (w->d_palette) vt::dev_free(w->d_palette);
    if (w->d_stage) vt::dev_free(w->d_stage);
    if (w->d_bdist) vt::dev_free(w->d_bdist);
    if (w->d_cdist) vt::dev_free(w->d_cdist);
    if (w->d_dtmp) vt::dev_free(w->d_dtmp);
    if (w->d_ctmp) vt::dev_free(w->d_ctmp);
    if (w->d_edit) vt::dev_free(w->d_edit);
    if (w->d_entities) vt::dev_free(w->d_entities);
    delete w;
}

}  // namespace vt

using namespace vt;

extern "C" {

vt_status vt_world_create(vt_ctx* ctx, const vt_world_desc* desc, vt_world** out) {
    if (!ctx) return VT_ERR_ARG;
    if (!desc || !out) return fail(ctx, VT_ERR_ARG, "null world descriptor or output");
    *out = nullptr;
    uint64_t cells = 1;
    for (int i = 0; i < 3; ++i) {
        if (desc->dims[i] < 1 || desc->dims[i] > 8192) return fail(ctx, VT_ERR_ARG, "world dims must be in [1, 8192]");
        cells *= (uint64_t)desc->dims[i];
    }
    if (cells >= (1ull << 32)) return fail(ctx, VT_ERR_ARG, "world must hold fewer than 2^32 voxels");
    vt_world* w = new (std::nothrow) vt_world();
    if (!w) return fail(ctx, VT_ERR_OOM, "host allocation failed");
    w->ctx = ctx;
    for (int i = 0; i < 3; ++i) {
        w->dims[i] = desc->dims[i];
        w->cdim[i] = (desc->dims[i] + kChunk - 1) / kChunk;
    }
    w->nchunks = (size_t)w->cdim[0] * w->cdim[1] * w->cdim[2];
    w->ncoarse = (w->nchunks + 63) / 64;
    cudaError_t e;
    if ((e = vt::dev_alloc(&w->d_mask, w->nchunks * kBricksPerChunk * 8)) != cudaSuccess ||
        (e = vt::dev_alloc(&w->d_mats, w->nchunks * (size_t)kChunkBytes)) != cudaSuccess ||
        (e = vt::dev_alloc(&w->d_coarse, w->ncoarse * 8)) != cudaSuccess ||
        (e = vt::dev_alloc(&w->d_palette, kPaletteBytes)) != cudaSuccess ||
        (e = vt::dev_alloc(&w->d_bdist, kOctants * w->nchunks * kBricksPerChunk)) != cudaSuccess ||
        (e = vt::dev_alloc(&w->d_cdist, kOctants * (size_t)cdist_stride((unsigned)w->nchunks))) != cudaSuccess ||
        (e = vt::dev_alloc(&w->d_dtmp, (32 + 4 * kYFields) * w->nchunks * kBricksPerChunk)) != cudaSuccess ||
        (e = vt::dev_alloc(&w->d_ctmp, 6 * (size_t)cdist_stride((unsigned)w->nchunks))) != cudaSuccess ||
        (e = vt::dev_alloc(&w->d_edit, kEditInts * sizeof(int))) != cudaSuccess ||
        (e = vt::dev_alloc(&w->d_entities, kMaxEntities * 6 * sizeof(float))) != cudaSuccess ||
        (e = cudaMemset(w->d_edit, 0, kEditInts * sizeof(int))) != cudaSuccess ||
        (e = cudaMemset(w->d_mask, 0, w->nchunks * kBricksPerChunk * 8)) != cudaSuccess ||
        (e = cudaMemset(w->d_mats, 0, w->nchunks * (size_t)kChunkBytes)) != cudaSuccess ||
        (e = cudaMemset(w->d_coarse, 0, w->ncoarse * 8)) != cudaSuccess) {
        free_world(w);
        return check_cuda(ctx, e, "world allocation");
    }
    uint32_t pal[256];
    vt_default_palette(pal);
    if ((e = upload_palette(w, pal)) != cudaSuccess) {
        free_world(w);
        return check_cuda(ctx, e, "palette upload");
    }
    *out = w;
    return VT_OK;
}

vt_status vt_world_destroy(vt_world* world) {
    if (!world) return VT_ERR_ARG;
    cudaDeviceSynchronize();
    free_world(world);
    return VT_OK;
}

vt_status vt_world_clear(vt_world* w, vt_stream stream) {
    if (!w) return VT_ERR_ARG;
    cudaStream_t s = (cudaStream_t)stream;
    VT_CUDA(w->ctx, cudaMemsetAsync(w->d_mask, 0, w->nchunks * kBricksPerChunk * 8, s));
    VT_CUDA(w->ctx, cudaMemsetAsync(w->d_mats, 0, w->nchunks * (size_t)kChunkBytes, s));
    VT_CUDA(w->ctx, cudaMemsetAsync(w->d_coarse, 0, w->ncoarse * 8, s));
    w->dist_dirty = true;
    return VT_OK;
}

vt_status vt_world_upload_dense(vt_world* w, const uint8_t* h_materials, size_t nbytes, vt_stream stream) {
    if (!w) return VT_ERR_ARG;
    const size_t need = (size_t)w->dims[0] * w->dims[1] * w->dims[2];
    if (!h_materials || nbytes != need) return fail(w->ctx, VT_ERR_ARG, "dense upload needs exactly X*Y*Z bytes");
    unsigned char* stage = nullptr;
    vt_status s = world_stage(w, need, &stage);
    if (s) return s;
    cudaStream_t st = (cudaStream_t)stream;
    VT_CUDA(w->ctx, cudaMemcpyAsync(w->d_stage, h_materials, need, cudaMemcpyHostToDevice, st));
    const int3 sdims = make_int3(w->dims[0], w->dims[1], w->dims[2]);
    k_build_chunks<<<(unsigned)w->nchunks, 512, 0, st>>>(w->view(), w->d_mask, w->d_mats, w->d_coarse, w->d_stage, sdims,
                                                        make_int3(0, 0, 0), make_int3(0, 0, 0),
                                                        make_int3(w->cdim[0], w->cdim[1], w->cdim[2]));
    VT_CUDA(w->ctx, cudaGetLastError());
    w->dist_dirty = true;
    // the staging buffer is reused by the next upload on any stream
    VT_CUDA(w->ctx, cudaStreamSynchronize(st));
    return VT_OK;
}

vt_status vt_world_upload_chunk(vt_world* w, int32_t cx, int32_t cy, int32_t cz, const uint8_t* h_chunk,
                                vt_stream stream) {
    if (!w) return VT_ERR_ARG;
    if (!h_chunk) return fail(w->ctx, VT_ERR_ARG, "null chunk");
    if (cx < 0 || cy < 0 || cz < 0 || cx >= w->cdim[0] || cy >= w->cdim[1] || cz >= w->cdim[2])
        return fail(w->ctx, VT_ERR_ARG, "chunk coordinate out of range");
    unsigned char* stage = nullptr;
    vt_status s = world_stage(w, kChunkBytes, &stage);
    if (s) return s;
    cudaStream_t st = (cudaStream_t)stream;
    VT_CUDA(w->ctx, cudaMemcpyAsync(w->d_stage, h_chunk, kChunkBytes, cudaMemcpyHostToDevice, st));
    k_build_chunks<<<1, 512, 0, st>>>(w->view(), w->d_mask, w->d_mats, w->d_coarse, w->d_stage, make_int3(32, 32, 32),
                                      make_int3(cx * 32, cy * 32, cz * 32), make_int3(cx, cy, cz), make_int3(1, 1, 1));
    VT_CUDA(w->ctx, cudaGetLastError());
    const int blo[3] = {cx * 8, cy * 8, cz * 8}, bhi[3] = {cx * 8 + 7, cy * 8 + 7, cz * 8 + 7};
    note_edit(w, blo, bhi);
    VT_CUDA(w->ctx, cudaStreamSynchronize(st));
    return VT_OK;
}

vt_status vt_world_set_voxel(vt_world* w, int32_t x, int32_t y, int32_t z, uint8_t material, vt_stream stream) {
    if (!w) return VT_ERR_ARG;
    if (x < 0 || y < 0 || z < 0 || x >= w->dims[0] || y >= w->dims[1] || z >= w->dims[2])
        return fail(w->ctx, VT_ERR_ARG, "voxel coordinate out of range");
    k_set_voxel<<<1, 512, 0, (cudaStream_t)stream>>>(w->view(), w->d_mask, w->d_mats, w->d_coarse, x, y, z, material);
    VT_CUDA(w->ctx, cudaGetLastError());
    const int b[3] = {x >> 2, y >> 2, z >> 2};
    note_edit(w, b, b);
    return VT_OK;
}

vt_status vt_world_get_voxel(vt_world* w, int32_t x, int32_t y, int32_t z, uint8_t* material) {
    if (!w) return VT_ERR_ARG;
    if (!material || x < 0 || y < 0 || z < 0 || x >= w->dims[0] || y >= w->dims[1] || z >= w->dims[2])
        return fail(w->ctx, VT_ERR_ARG, "voxel coordinate out of range");
    const unsigned ci = (unsigned)(x >> 5) + (unsigned)w->cdim[0] * ((unsigned)(y >> 5) + (unsigned)w->cdim[1] * (unsigned)(z >> 5));
    const unsigned bi = (unsigned)((x >> 2) & 7) | ((unsigned)((y >> 2) & 7) << 3) | ((unsigned)((z >> 2) & 7) << 6);
    const unsigned vb = (unsigned)(x & 3) | ((unsigned)(y & 3) << 2) | ((unsigned)(z & 3) << 4);
    VT_CUDA(w->ctx, cudaDeviceSynchronize());
    VT_CUDA(w->ctx, cudaMemcpy(material, w->d_mats + ((size_t)ci * 512u + bi) * 64u + vb, 1, cudaMemcpyDeviceToHost));
    return VT_OK;
}

vt_status vt_world_set_palette(vt_world* w, const uint32_t* h_rgba256) {
    if (!w) return VT_ERR_ARG;
    if (!h_rgba256) return fail(w->ctx, VT_ERR_ARG, "null palette");
    VT_CUDA(w->ctx, upload_palette(w, h_rgba256));
    return VT_OK;
}

vt_status vt_world_set_entities(vt_world* w, const float* h_boxes, int32_t n) {
    if (!w) return VT_ERR_ARG;
    if (n < 0 || n > kMaxEntities || (n > 0 && !h_boxes))
        return fail(w->ctx, VT_ERR_ARG, "entity count must be in [0, 1024] with a box list");
    for (int i = 0; i < 6 * n; ++i)
        if (!(h_boxes[i] == h_boxes[i])) return fail(w->ctx, VT_ERR_ARG, "entity box coordinates must not be NaN");
    if (n > 0) VT_CUDA(w->ctx, cudaMemcpy(w->d_entities, h_boxes, (size_t)n * 6 * sizeof(float), cudaMemcpyHostToDevice));
    w->n_entities = n;
    return VT_OK;
}

vt_status vt_world_get_info(const vt_world* w, vt_world_info* info) {
    if (!w || !info) return VT_ERR_ARG;
    std::memset(info, 0, sizeof(*info));
    for (int i = 0; i < 3; ++i) {
        info->dims[i] = w->dims[i];
        info->chunks[i] = w->cdim[i];
    }
    info->mask_bytes = (uint64_t)w->nchunks * kBricksPerChunk * 8;
    info->material_bytes = (uint64_t)w->nchunks * kChunkBytes;
    info->coarse_bytes = (uint64_t)w->ncoarse * 8;
    info->d_mask = w->d_mask;
    info->d_materials = w->d_mats;
    info->d_coarse = w->d_coarse;
    return VT_OK;
}

}  // extern "C"
