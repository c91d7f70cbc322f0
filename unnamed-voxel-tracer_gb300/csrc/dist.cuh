// dist.cuh -- the brick distances' x pass (world.cu has the passes and what
// they compute), shared with the device-side edit, whose block runs it for the
// edited brick's rows.
#pragma once

#include "vt_internal.h"

namespace vt {

__device__ __forceinline__ unsigned brick_index(int bx, int by, int bz, int CX, int CY) {
    const unsigned ci = (unsigned)(bx >> 3) + (unsigned)CX * ((unsigned)(by >> 3) + (unsigned)CY * (unsigned)(bz >> 3));
    return ci * 512u + (unsigned)((bx & 7) | ((by & 7) << 3) | ((bz & 7) << 6));
}

struct BrickGrid {
    int CX, CY, CZ;   // chunks
    int GX, GY, GZ;   // bricks
};

// Item `lin` of the box [lo, lo + ext) whose x axis counts groups of `group`
// bricks (the ones that meet the box): its coordinates, x in groups.  False
// past the box or the grid.
__device__ __forceinline__ bool box_item(unsigned lin, int3 lo, int3 ext, int group, int3 g, int& x, int& y, int& z) {
    const int x0 = max(lo.x, 0) / group, nx = (lo.x + ext.x - 1) / group - x0 + 1;
    if (lo.x + ext.x <= 0 || nx <= 0) return false;
    x = x0 + (int)(lin % (unsigned)nx);
    const unsigned r = lin / (unsigned)nx;
    y = lo.y + (int)(r % (unsigned)ext.y);
    const unsigned rz = r / (unsigned)ext.y;
    if (rz >= (unsigned)ext.z) return false;
    z = lo.z + (int)rz;
    return y >= 0 && z >= 0 && x * group < g.x && y < g.y && z < g.z;
}

// The 8 bricks of a chunk on the 4 voxel rows of brick row by in layer qz,
// both directions.  A row of a chunk is one 32-bit word; the first voxel ahead
// lies in it or in the next two (64 layers, the cap is 63).  The words of a
// chunk whose coarse bit is clear are not read (coarse null: all are).  FRESH:
// the mask was written earlier in this launch, so it is not read through the
// non-coherent cache.
template <bool FRESH>
__device__ __forceinline__ void bdist_x_item(const unsigned long long* mask, const unsigned long long* coarse,
                                             unsigned char* __restrict__ xf, const BrickGrid& b, int cx, int by, int qz) {
    // r[k][y]: row y of chunk cx - 2 + k
    unsigned r[5][4];
#pragma unroll
    for (int k = 0; k < 5; ++k) {
#pragma unroll
        for (int y = 0; y < 4; ++y) r[k][y] = 0u;
        const int c = cx - 2 + k;
        if (c < 0 || c >= b.CX) continue;
        if (coarse) {
            const unsigned ci = (unsigned)c + (unsigned)b.CX * ((unsigned)(by >> 3) + (unsigned)b.CY * (unsigned)(qz >> 5));
            if (!((__ldg(coarse + (ci >> 6)) >> (ci & 63u)) & 1ull)) continue;
        }
        const unsigned short* w = reinterpret_cast<const unsigned short*>(mask + brick_index(8 * c, by, qz >> 2, b.CX, b.CY)) + (qz & 3);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const unsigned v = FRESH ? (unsigned)__ldcg(w + 4 * i) : (unsigned)__ldg(w + 4 * i);   // 16 voxels of brick i: 4 rows of 4
#pragma unroll
            for (int y = 0; y < 4; ++y) r[k][y] |= ((v >> (4 * y)) & 15u) << (4 * i);
        }
    }
    const size_t fsize = (size_t)b.GX * (b.GY * 4) * (b.GZ * 4);
#pragma unroll
    for (int y = 0; y < 4; ++y) {
        unsigned char* row = xf + (size_t)(8 * cx) + (size_t)b.GX * ((size_t)(4 * by + y) + (size_t)(b.GY * 4) * qz);
        unsigned out[2][2] = {{0u, 0u}, {0u, 0u}};
        const unsigned own = r[2][y];
        // layers from the chunk's far face to the first voxel of the next two
        const unsigned ahead = r[3][y] ? (unsigned)__ffs(r[3][y]) : (r[4][y] ? 32u + (unsigned)__ffs(r[4][y]) : 64u);
        const unsigned behind = r[1][y] ? 1u + (unsigned)__clz(r[1][y]) : (r[0][y] ? 33u + (unsigned)__clz(r[0][y]) : 64u);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const bool occ = ((own >> (4 * i)) & 15u) != 0u;
            const unsigned up = i < 7 ? own >> (4 * i + 4) : 0u, down = own & ((1u << (4 * i)) - 1u);
            unsigned f = up ? (unsigned)__ffs(up) : (unsigned)(28 - 4 * i) + ahead;
            unsigned n = down ? (unsigned)(4 * i - 31) + (unsigned)__clz(down) : (unsigned)(4 * i) + behind;
            f = occ ? 0u : min(f, (unsigned)(kVoxCap + 1));
            n = occ ? 0u : min(n, (unsigned)(kVoxCap + 1));
            out[0][i >> 2] |= n << (8 * (i & 3));
            out[1][i >> 2] |= f << (8 * (i & 3));
        }
        *reinterpret_cast<uint2*>(row) = make_uint2(out[0][0], out[0][1]);
        *reinterpret_cast<uint2*>(row + fsize) = make_uint2(out[1][0], out[1][1]);
    }
}

}  // namespace vt
