// world_gen.cu -- scene generation straight into the device world, and the
// dense download of a world.
//
// The reference generates its terrain on the host and writes it voxel by
// voxel into mapped buffers (src/procgen.zig:6-53 through VoxelBrickmap.set,
// src/engine/voxel.zig:58-61).  Here the same seeded generator as the host's
// vt_gen_world (gen_noise.cuh, shared code) runs on the device and writes the
// chunk layout directly: no dense staging grid, no host traffic.  The bytes
// equal vt_gen_world's for every descriptor.
//
//   k_gen_tiles    one block per chunk, one thread per brick: the chunk's
//                  32x32 column heights in shared memory, then 64 cells per
//                  thread (terrain, water, caves), brick word and coarse bit;
//                  the noise in 32 bits from shared lattice tables, decided in
//                  64 bits where 32 cannot
//   k_gen_chunks   the same in 64 bits cell by cell, for noise so fine that a
//                  chunk's lattice tables would not fit
//   k_gen_leaves   one block per tree, one thread per leaf cell
//   k_gen_trunks   one thread per tree, after all leaves (see plant_trees on
//                  why the parallel order gives the sequential bytes)
#include <cmath>
#include <cstring>

#include "gen_noise.cuh"
#include "vt_internal.h"

namespace vt {

namespace {

__device__ __forceinline__ void cell_addr(const WorldView& w, int x, int y, int z, unsigned* wi, unsigned* vb) {
    const unsigned ci = (unsigned)(x >> 5) + (unsigned)w.cdim[0] * ((unsigned)(y >> 5) + (unsigned)w.cdim[1] * (unsigned)(z >> 5));
    const unsigned bi = (unsigned)((x >> 2) & 7) | ((unsigned)((y >> 2) & 7) << 3) | ((unsigned)((z >> 2) & 7) << 6);
    *wi = ci * 512u + bi;
    *vb = (unsigned)(x & 3) | ((unsigned)(y & 3) << 2) | ((unsigned)(z & 3) << 4);
}

// Marks cell (wi, vb) solid in the brick word and its chunk solid in the
// coarse grid.
__device__ __forceinline__ void mark_solid(unsigned long long* mask, unsigned long long* coarse, unsigned wi, unsigned vb) {
    atomicOr(mask + wi, 1ull << vb);
    const unsigned ci = wi >> 9;
    // most trees stand in chunks the terrain marked already
    const unsigned long long bit = 1ull << (ci & 63u);
    if (!(__ldcg(coarse + (ci >> 6)) & bit)) atomicOr(coarse + (ci >> 6), bit);
}

__global__ void __launch_bounds__(512) k_gen_chunks(WorldView w, unsigned long long* mask, unsigned char* mats,
                                                    unsigned long long* coarse, vt_gen_desc d) {
    __shared__ int heights[32 * 32];
    const unsigned ci = blockIdx.x;
    const int cx = (int)(ci % (unsigned)w.cdim[0]);
    const int cy = (int)((ci / (unsigned)w.cdim[0]) % (unsigned)w.cdim[1]);
    const int cz = (int)(ci / ((unsigned)w.cdim[0] * (unsigned)w.cdim[1]));
    for (int c = threadIdx.x; c < 32 * 32; c += blockDim.x) {
        const int gx = cx * 32 + (c & 31), gz = cz * 32 + (c >> 5);
        heights[c] = (gx < w.dims[0] && gz < w.dims[2]) ? gen::height_at(&d, gx, gz) : 0;
    }
    __syncthreads();
    const int water = (int)ceil((double)d.water_level);
    const uint64_t cave_seed = gen::stream_seed(d.seed, gen::kCaves);
    const double cave_freq = 1.0 / (double)d.cave_period;
    const int b = threadIdx.x;
    const int bx = b & 7, by = (b >> 3) & 7, bz = b >> 6;
    unsigned long long m = 0ull;
    unsigned packed[16];
    for (int z = 0; z < 4; ++z) {
        for (int y = 0; y < 4; ++y) {
            unsigned word = 0;
            for (int x = 0; x < 4; ++x) {
                const int lx = bx * 4 + x, lz = bz * 4 + z;
                const int gx = cx * 32 + lx, gy = cy * 32 + by * 4 + y, gz = cz * 32 + lz;
                unsigned v = 0;
                if (gx < w.dims[0] && gy < w.dims[1] && gz < w.dims[2])
                    v = gen::cell_material(&d, gx, gy, gz, heights[lx + 32 * lz], water, cave_seed, cave_freq);
                word |= v << (8 * x);
                if (v) m |= 1ull << (x + 4 * (y + 4 * z));
            }
            packed[y + 4 * z] = word;
        }
    }
    const unsigned wi = ci * 512u + (unsigned)b;
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

// ---------------------------------------------------------------------------
// The generator's noise in 32 bits.
//
// Every material is decided by comparing an fbm value with a number: a cave
// cell by fbm3 > cave_threshold, a column by the floor of base + amplitude *
// fbm2.  The device has two double-precision lanes per SM and cycle, and the
// 64-bit noise of a cave cell costs 48 lattice hashes and about 84 double
// operations, so that the kernel was bound by them (512x256x512 cave world:
// 6.22 ms).  A 32-bit value decides the same comparison unless it lies within
// its error bound of the number; only then is the 64-bit value computed.
// The lattice values a chunk needs (a few hundred) are hashed once into shared
// memory, and the cave noise is interpolated along x once per lattice row.
// The same world now takes 71 us.
//
// Error of the 32-bit values against the real ones, u = 2^-24: a lattice value
// is in [-1, 1) (rounding u / 2); a position is off by at most 2^-28
// (lattice_coord), a weight, whose slope is at most 1.5, by 0.14 u before its one
// rounding and 0.64 u in all; an interpolation a + (b - a) t adds 1.28 u for the
// weight and 1.5 u for its roundings.  Two levels: 6.1 u; the octaves' sum (below
// 2) adds at most u an octave after the first, the division by the amplitudes'
// sum 1.5 u: below 8 u and u an octave.  Three levels: 8.9 u, times 1.5 for the
// two octaves' sum, and 1 u in it: 14.4 u.  Largest found near coordinate 8191,
// 9 million values: caves 4.9 u, heights 4.6 u.  (The 64-bit values' own error is
// below 1e-14.)
constexpr float kUlp = 0x1p-24f, kCaveError = 16.0f * kUlp;

// gen::lattice rounded to 32 bits: the hash as a signed fraction.
__device__ __forceinline__ float lattice32(uint64_t seed, int x, int y, int z) {
    uint64_t h = gen::mix64(seed ^ ((uint64_t)(int64_t)x * 0x9E3779B97F4A7C15ull));
    h = gen::mix64(h ^ ((uint64_t)(int64_t)y * 0xC2B2AE3D27D4EB4Full));
    h = gen::mix64(h ^ ((uint64_t)(int64_t)z * 0x165667B19E3779F9ull));
    return __int2float_rn((int)((unsigned)(h >> 32) ^ 0x80000000u)) * 0x1p-31f;
}

// Lattice cell and interpolation weight of coordinate g (below 2^13) at a
// frequency (below 2^2) rounded to a multiple of 2^-40 (fixed40): the position is
// off by at most 2^13 * 2^-41 = 2^-28, and the noise is continuous across the
// cells.
__device__ __forceinline__ void lattice_coord(int g, long long f, int& cell, float& weight) {
    const long long x = (long long)g * f;
    const unsigned t = (unsigned)((unsigned long long)x >> 8);   // the position in the cell, times 2^32
    cell = (int)(x >> 40);
    // t t (3 - 2 t) in integers
    weight = __uint2float_rn(__umulhi(__umulhi(t, t), 0xC0000000u - (t >> 1))) * 0x1p-30f;
}

__device__ __forceinline__ float lerp32(float a, float b, float t) { return __fmaf_rn(b - a, t, a); }

struct GenArgs {
    vt_gen_desc d;
    double cave_freq;            // 1 / cave_period
    long long height40[16];      // the octaves' frequencies, multiples of 2^-40; [0] 0: heights in 64 bits
    long long cave40[2];
    uint64_t terrain_seed, cave_seed, leaf_seed;
    float norm;                  // 1 / (sum of the octaves' amplitudes)
    float fbm_error;             // of the 32-bit fbm2
    float ceiling;               // no cell at or above it but trees
    int water;
    // shared-memory layout of k_gen_tiles, in floats
    int height_side[16];         // most lattice points a chunk meets on an axis, per octave
    int cave_side[2];
    int cave_floats;             // lattice values; the rows interpolated along x follow them
};

// The 64-bit decisions, out of line: inlined they cost the kernels registers
// (k_gen_tiles 368 bytes of spills) for one column or cell in thousands.
__device__ __noinline__ int height_exact(const vt_gen_desc* d, int x, int z) { return gen::height_at(d, x, z); }
__device__ __noinline__ bool cave_exact(const GenArgs* a, int x, int y, int z) {
    return gen::fbm3(a->cave_seed, (double)x, (double)y, (double)z, a->cave_freq) > (double)a->d.cave_threshold;
}

// The column height from the 32-bit fbm value (gen::height_at's rounding and
// clamps), or in 64 bits where that does not decide the floor.
__device__ __forceinline__ int height_of(const GenArgs& a, float fbm, int x, int z) {
    const float v = __fmaf_rn(a.d.amplitude, fbm, a.d.base_height);
    const float margin = fabsf(a.d.amplitude) * a.fbm_error + fabsf(v) * (4.0f * kUlp);
    const float lo = floorf(v - margin);
    if (!(lo == floorf(v + margin)) || !(fabsf(lo) < 1e6f)) return height_exact(&a.d, x, z);
    int h = (int)lo;
    h = h < a.d.dims[1] - 1 ? h : a.d.dims[1] - 1;
    return h > 1 ? h : 1;
}

// gen::height_at of one column without tables.
__device__ int height_at32(const GenArgs& a, int x, int z) {
    if (!a.height40[0]) return height_exact(&a.d, x, z);
    float sum = 0.0f, amp = 1.0f;
    for (int o = 0; o < a.d.octaves; ++o) {
        int cx, cz;
        float sx, sz;
        lattice_coord(x, a.height40[o], cx, sx);
        lattice_coord(z, a.height40[o], cz, sz);
        const uint64_t seed = a.terrain_seed + (uint64_t)o * gen::kOctaveSalt;
        const float p = lerp32(lattice32(seed, cx, 0, cz), lattice32(seed, cx + 1, 0, cz), sx);
        const float q = lerp32(lattice32(seed, cx, 0, cz + 1), lattice32(seed, cx + 1, 0, cz + 1), sx);
        sum += amp * lerp32(p, q, sz);
        amp *= 0.5f;
    }
    return height_of(a, sum * a.norm, x, z);
}

// gen::tree_site with the 32-bit height.
__device__ bool tree_site32(const GenArgs& a, int t, int* x, int* z, int* h) {
    gen::tree_column(&a.d, t, x, z);
    *h = height_at32(a, *x, *z);
    return *h + 8 < a.d.dims[1];
}

// Bound: issue (63%) and the short phases between barriers.  Cells four in x
// at a time from 16-byte table rows, a layer stored as it is done (71 us on the
// 512x256x512 cave world; one cell at a time with the brick in registers 116 us);
// chunks above every column are cleared at once.
__global__ void __launch_bounds__(512, 2) k_gen_tiles(WorldView w, unsigned long long* mask, unsigned char* mats,
                                                   unsigned long long* coarse, const __grid_constant__ GenArgs a) {
    extern __shared__ __align__(16) float s_gen[];
    __shared__ __align__(16) int heights[32 * 32];
    __shared__ float weight[16][2][32];       // [octave][axis][coordinate]; caves: [octave * 3 + axis][0]
    __shared__ unsigned char cell[16][2][32]; // lattice cell relative to the chunk's first
    __shared__ int first[16][2];              // the chunk's first lattice point
    const unsigned ci = blockIdx.x;
    const int cx = (int)(ci % (unsigned)w.cdim[0]);
    const int cy = (int)((ci / (unsigned)w.cdim[0]) % (unsigned)w.cdim[1]);
    const int cz = (int)(ci / ((unsigned)w.cdim[0] * (unsigned)w.cdim[1]));
    const int tid = threadIdx.x;

    // a chunk above the highest column (fbm is in [-1, 1]) and the water is air
    if (cy > 0 && (float)(cy * 32) >= a.ceiling) {
        uint4* dst = reinterpret_cast<uint4*>(mats + (size_t)ci * kChunkBytes);
#pragma unroll
        for (int q = 0; q < 4; ++q) dst[q * 512 + tid] = make_uint4(0u, 0u, 0u, 0u);
        mask[ci * 512u + (unsigned)tid] = 0ull;
        if (tid == 0) atomicAnd(coarse + (ci >> 6), ~(1ull << (ci & 63u)));
        return;
    }

    // ---- heights
    for (int i = tid; i < a.d.octaves * 64; i += 512) {
        const int o = i >> 6, axis = (i >> 5) & 1, k = i & 31, g0 = (axis ? cz : cx) * 32;
        int c;
        float s;
        lattice_coord(g0 + k, a.height40[o], c, s);
        const int c0 = __shfl_sync(0xFFFFFFFFu, c, 0);   // k is the lane
        weight[o][axis][k] = s;
        cell[o][axis][k] = (unsigned char)(c - c0);
        if (k == 0) first[o][axis] = c0;
    }
    __syncthreads();
    for (int o = 0, base = 0; o < a.d.octaves; ++o) {
        const int n = a.height_side[o];
        const uint64_t seed = a.terrain_seed + (uint64_t)o * gen::kOctaveSalt;
        for (int i = tid; i < n * n; i += 512) s_gen[base + i] = lattice32(seed, first[o][0] + i % n, 0, first[o][1] + i / n);
        base += n * n;
    }
    __syncthreads();
    for (int c = tid; c < 32 * 32; c += 512) {
        const int lx = c & 31, lz = c >> 5, gx = cx * 32 + lx, gz = cz * 32 + lz;
        int h = -1;   // no column
        if (gx < w.dims[0] && gz < w.dims[2]) {
            float sum = 0.0f, amp = 1.0f;
            for (int o = 0, base = 0; o < a.d.octaves; ++o) {
                const int n = a.height_side[o];
                const float* l = s_gen + base + cell[o][0][lx] + n * cell[o][1][lz];
                const float sx = weight[o][0][lx];
                sum += amp * lerp32(lerp32(l[0], l[1], sx), lerp32(l[n], l[n + 1], sx), weight[o][1][lz]);
                amp *= 0.5f;
                base += n * n;
            }
            h = height_of(a, sum * a.norm, gx, gz);
        }
        heights[c] = h;
    }
    __syncthreads();

    // ---- cave tables: per octave the lattice, then its rows along x (fixed
    // lattice y and z) interpolated at the chunk's 32 coordinates
    float* rows = s_gen + a.cave_floats;   // (16-byte aligned)
    if (a.d.caves) {
        for (int i = tid; i < 2 * 96; i += 512) {
            const int o = i / 96, axis = (i % 96) >> 5, k = i & 31, g0 = (axis == 0 ? cx : (axis == 1 ? cy : cz)) * 32;
            int c;
            float s;
            lattice_coord(g0 + k, a.cave40[o], c, s);
            const int c0 = __shfl_sync(0xFFFFFFFFu, c, 0);
            weight[o * 3 + axis][0][k] = s;
            cell[o * 3 + axis][0][k] = (unsigned char)(c - c0);
            if (k == 0) first[o * 3 + axis][0] = c0;
        }
        __syncthreads();
        for (int o = 0, base = 0; o < 2; ++o) {
            const int n = a.cave_side[o];
            const uint64_t seed = a.cave_seed + (uint64_t)o * gen::kOctaveSalt;
            for (int i = tid; i < n * n * n; i += 512)
                s_gen[base + i] = lattice32(seed, first[o * 3][0] + i % n, first[o * 3 + 1][0] + (i / n) % n, first[o * 3 + 2][0] + i / (n * n));
            base += n * n * n;
        }
        __syncthreads();
        for (int o = 0, base = 0, row0 = 0; o < 2; ++o) {
            const int n = a.cave_side[o];
            for (int i = tid; i < n * n * 32; i += 512) {
                const int x = i & 31, r = i >> 5;
                const float* l = s_gen + base + n * r + cell[o * 3][0][x];
                rows[row0 * 32 + i] = lerp32(l[0], l[1], weight[o * 3][0][x]);
            }
            base += n * n * n;
            row0 += n * n;
        }
        __syncthreads();
    }

    // ---- the thread's brick, a layer of 16 cells and one 16-byte store at a
    // time; four cells in x share their loads
    const int bx = tid & 7, by = (tid >> 3) & 7, bz = tid >> 6;
    const int gy0 = cy * 32 + by * 4, water = min(a.water, w.dims[1]);
    const unsigned wi = ci * 512u + (unsigned)tid;
    uint4* dst = reinterpret_cast<uint4*>(mats + (size_t)wi * 64u);
    const float bound = 1.5f * a.d.cave_threshold;   // of noise + noise / 2
    const float margin = kCaveError + 4.0f * kUlp * fabsf(bound);
    const int n0 = a.cave_side[0], n1 = a.cave_side[1];
    unsigned long long m = 0ull;
#pragma unroll 1
    for (int z = 0; z < 4; ++z) {
        const int lz = bz * 4 + z;
        const int4 h4 = *reinterpret_cast<const int4*>(heights + bx * 4 + 32 * lz);
        const int h[4] = {h4.x, h4.y, h4.z, h4.w};
        const int top = max(max(h[0], h[1]), max(h[2], h[3]));
        unsigned word[4] = {0u, 0u, 0u, 0u};
        if (gy0 < top || gy0 < water) {
#pragma unroll
            for (int y = 0; y < 4; ++y) {
                const int gy = gy0 + y;
                unsigned v[4];
#pragma unroll
                for (int x = 0; x < 4; ++x)
                    v[x] = gy < h[x] ? (gy == h[x] - 1 ? 1u : (gy >= h[x] - 4 ? 2u : 3u)) : (gy < water && h[x] > 0 ? 4u : 0u);
                if (a.d.caves && gy > 0 && gy < top) {
                    const int ly = by * 4 + y;
                    const float4* r0 = reinterpret_cast<const float4*>(rows + 32 * (cell[1][0][ly] + n0 * cell[2][0][lz])) + bx;
                    const float4* r1 = reinterpret_cast<const float4*>(rows + 32 * (n0 * n0 + cell[4][0][ly] + n1 * cell[5][0][lz])) + bx;
                    const float4 a00 = r0[0], a10 = r0[8], a01 = r0[8 * n0], a11 = r0[8 * n0 + 8];
                    const float4 b00 = r1[0], b10 = r1[8], b01 = r1[8 * n1], b11 = r1[8 * n1 + 8];
                    const float y0 = weight[1][0][ly], z0 = weight[2][0][lz], y1 = weight[4][0][ly], z1 = weight[5][0][lz];
                    auto noise = [&](float p00, float p10, float p01, float p11, float q00, float q10, float q01, float q11) {
                        const float p = lerp32(lerp32(p00, p10, y0), lerp32(p01, p11, y0), z0);
                        const float q = lerp32(lerp32(q00, q10, y1), lerp32(q01, q11, y1), z1);
                        return __fmaf_rn(0.5f, q, p) - bound;
                    };
                    const float f[4] = {noise(a00.x, a10.x, a01.x, a11.x, b00.x, b10.x, b01.x, b11.x),
                                        noise(a00.y, a10.y, a01.y, a11.y, b00.y, b10.y, b01.y, b11.y),
                                        noise(a00.z, a10.z, a01.z, a11.z, b00.z, b10.z, b01.z, b11.z),
                                        noise(a00.w, a10.w, a01.w, a11.w, b00.w, b10.w, b01.w, b11.w)};
#pragma unroll
                    for (int x = 0; x < 4; ++x) {
                        if (gy >= h[x]) continue;
                        bool cave = f[x] > 0.0f;
                        if (fabsf(f[x]) <= margin) cave = cave_exact(&a, cx * 32 + bx * 4 + x, gy, cz * 32 + lz);
                        if (cave) v[x] = 0u;
                    }
                }
                word[y] = v[0] | (v[1] << 8) | (v[2] << 16) | (v[3] << 24);
                // bit per nonzero byte (materials below 128)
                const unsigned nz = (word[y] + 0x7F7F7F7Fu) & 0x80808080u;
                m |= (unsigned long long)((nz * 0x00204081u) >> 28) << (4 * y + 16 * z);
            }
        }
        dst[z] = make_uint4(word[0], word[1], word[2], word[3]);
    }
    mask[wi] = m;
    const int any = __syncthreads_or(m != 0ull);
    if (tid == 0) {
        const unsigned long long bit = 1ull << (ci & 63u);
        if (any) atomicOr(coarse + (ci >> 6), bit);
        else atomicAnd(coarse + (ci >> 6), ~bit);
    }
}

// Leaf cells of tree blockIdx.x: each kept cell that holds air or water
// becomes 6.  Concurrent trees only ever write 6 over 0 or 4, so a cell
// covered by several trees ends the same whichever comes first.
__global__ void __launch_bounds__(128) k_gen_leaves(WorldView w, unsigned long long* mask, unsigned char* mats,
                                                    unsigned long long* coarse, const __grid_constant__ GenArgs a) {
    __shared__ int site[4];
    const int t = blockIdx.x;
    if (threadIdx.x == 0) site[3] = tree_site32(a, t, &site[0], &site[1], &site[2]) ? 1 : 0;
    __syncthreads();
    const int c = threadIdx.x;
    if (!site[3] || c >= 125) return;
    const int dx = c % 5 - 2, dy = (c / 5) % 5 - 2, dz = c / 25 - 2;
    const int lx = site[0] + dx, ly = site[2] + 5 + dy, lz = site[1] + dz;
    if (lx < 0 || lz < 0 || lx >= w.dims[0] || lz >= w.dims[2] || ly >= w.dims[1]) return;
    if (!gen::leaf_kept(a.leaf_seed, t, dx, dy, dz)) return;
    unsigned wi, vb;
    cell_addr(w, lx, ly, lz, &wi, &vb);
    volatile unsigned char* cell = mats + (size_t)wi * 64u + vb;
    const unsigned char cur = *cell;
    if (cur != 0 && cur != 4) return;
    *cell = 6;
    mark_solid(mask, coarse, wi, vb);
}

// Trunks (material 5 over anything), after every leaf has landed.
__global__ void __launch_bounds__(64) k_gen_trunks(WorldView w, unsigned long long* mask, unsigned char* mats,
                                                    unsigned long long* coarse, const __grid_constant__ GenArgs a) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= a.d.trees) return;
    int x, z, h;
    if (!tree_site32(a, t, &x, &z, &h)) return;
    for (int y = h; y < h + 6; ++y) {
        unsigned wi, vb;
        cell_addr(w, x, y, z, &wi, &vb);
        mats[(size_t)wi * 64u + vb] = 5;
        mark_solid(mask, coarse, wi, vb);
    }
}

// One block per chunk, one thread per brick: the brick's 64 bytes back to the
// x-fastest dense grid (cells outside the world are skipped).
__global__ void __launch_bounds__(512) k_gather_dense(WorldView w, const unsigned char* __restrict__ mats,
                                                      unsigned char* __restrict__ dst) {
    const unsigned ci = blockIdx.x;
    const int cx = (int)(ci % (unsigned)w.cdim[0]);
    const int cy = (int)((ci / (unsigned)w.cdim[0]) % (unsigned)w.cdim[1]);
    const int cz = (int)(ci / ((unsigned)w.cdim[0] * (unsigned)w.cdim[1]));
    const int b = threadIdx.x;
    const int bx = b & 7, by = (b >> 3) & 7, bz = b >> 6;
    const uint4* src = reinterpret_cast<const uint4*>(mats + ((size_t)ci * 512u + (unsigned)b) * 64u);
    unsigned packed[16];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const uint4 v = src[q];
        packed[4 * q] = v.x;
        packed[4 * q + 1] = v.y;
        packed[4 * q + 2] = v.z;
        packed[4 * q + 3] = v.w;
    }
    for (int z = 0; z < 4; ++z)
        for (int y = 0; y < 4; ++y)
            for (int x = 0; x < 4; ++x) {
                const int gx = cx * 32 + bx * 4 + x, gy = cy * 32 + by * 4 + y, gz = cz * 32 + bz * 4 + z;
                if (gx < w.dims[0] && gy < w.dims[1] && gz < w.dims[2])
                    dst[(size_t)gx + (size_t)w.dims[0] * ((size_t)gy + (size_t)w.dims[1] * (size_t)gz)] =
                        (unsigned char)(packed[y + 4 * z] >> (8 * x));
            }
}

// Most dynamic shared memory k_gen_tiles is given (two blocks per SM).
constexpr int kGenSmem = 96 * 1024;

// The kernels' arguments, and the dynamic shared memory of k_gen_tiles; 0
// where its tables would not fit (noise finer than about three voxels) and
// k_gen_chunks generates the cells.
int gen_args(const vt_gen_desc& d, GenArgs& a) {
    std::memset(&a, 0, sizeof(a));
    a.d = d;
    const double freq = 1.0 / (double)d.period;
    a.cave_freq = 1.0 / (double)d.cave_period;
    a.terrain_seed = gen::stream_seed(d.seed, gen::kTerrain);
    a.cave_seed = gen::stream_seed(d.seed, gen::kCaves);
    a.leaf_seed = gen::stream_seed(d.seed, gen::kLeaves);
    a.water = (int)ceil((double)d.water_level);
    const double top = std::fmax((double)d.base_height + std::fabs((double)d.amplitude) + 2.0, (double)a.water + 1.0);
    a.ceiling = top < 1e6 ? (float)top + 1.0f : INFINITY;   // (NaN, too)
    double norm = 0.0, amp = 1.0;
    for (int o = 0; o < d.octaves; ++o, amp *= 0.5) norm += amp;
    a.norm = (float)(1.0 / norm);
    a.fbm_error = (8.0f + (float)d.octaves) * kUlp;
    // 32 coordinates at frequency f meet at most floor(31 f) + 2 cells, one
    // more lattice points
    auto side = [](long long f40) { return (double)((31 * f40) >> 40) + 3.0; };
    auto fixed40 = [](double f, int octave) { return llrint(f * (double)(1 << octave) * 0x1p40); };
    const double finest = freq * (double)(1 << (d.octaves - 1));
    if (!(finest < 2.0)) return 0;
    for (int o = 0; o < d.octaves; ++o) a.height40[o] = fixed40(freq, o);
    if (d.caves && !(a.cave_freq < 1.0)) return 0;
    for (int o = 0; o < 2 && d.caves; ++o) a.cave40[o] = fixed40(a.cave_freq, o);
    double heights = 0.0, caves = 0.0, rows = 0.0;
    for (int o = 0; o < d.octaves; ++o) {
        const double n = side(a.height40[o]);
        a.height_side[o] = (int)n;
        heights += n * n;
    }
    for (int o = 0; o < 2 && d.caves; ++o) {
        const double n = side(a.cave40[o]);
        a.cave_side[o] = (int)n;
        caves += n * n * n;
        rows += n * n;
    }
    const double floats = heights > caves + 3.0 + 32.0 * rows ? heights : caves + 3.0 + 32.0 * rows;
    if (4.0 * floats > (double)kGenSmem) return 0;
    a.cave_floats = ((int)caves + 3) / 4 * 4;
    return (int)floats * 4;
}

}  // namespace

}  // namespace vt

using namespace vt;

extern "C" {

vt_status vt_world_generate(vt_world* w, const vt_gen_desc* desc, vt_stream stream) {
    if (!w) return VT_ERR_ARG;
    if (!desc) return fail(w->ctx, VT_ERR_ARG, "null generator descriptor");
    for (int i = 0; i < 3; ++i)
        if (desc->dims[i] != w->dims[i]) return fail(w->ctx, VT_ERR_ARG, "generator dims must equal the world's dims");
    if (!(desc->period > 0.0f) || !(desc->cave_period > 0.0f) || desc->octaves < 1 || desc->octaves > 16 ||
        desc->trees < 0)
        return fail(w->ctx, VT_ERR_ARG, "generator descriptor out of range");
    cudaStream_t st = (cudaStream_t)stream;
    const WorldView v = w->view();
    GenArgs a;
    const int smem = gen_args(*desc, a);
    if (smem > 0) {
        if (smem > 32 * 1024)
            VT_CUDA(w->ctx, cudaFuncSetAttribute(k_gen_tiles, cudaFuncAttributeMaxDynamicSharedMemorySize, kGenSmem));
        k_gen_tiles<<<(unsigned)w->nchunks, 512, smem, st>>>(v, w->d_mask, w->d_mats, w->d_coarse, a);
    } else {
        k_gen_chunks<<<(unsigned)w->nchunks, 512, 0, st>>>(v, w->d_mask, w->d_mats, w->d_coarse, *desc);
    }
    VT_CUDA(w->ctx, cudaGetLastError());
    if (desc->trees > 0 && w->dims[0] >= 6 && w->dims[2] >= 6) {
        k_gen_leaves<<<(unsigned)desc->trees, 128, 0, st>>>(v, w->d_mask, w->d_mats, w->d_coarse, a);
        VT_CUDA(w->ctx, cudaGetLastError());
        k_gen_trunks<<<(unsigned)((desc->trees + 63) / 64), 64, 0, st>>>(v, w->d_mask, w->d_mats, w->d_coarse, a);
        VT_CUDA(w->ctx, cudaGetLastError());
    }
    w->dist_dirty = true;
    return VT_OK;
}

vt_status vt_world_download_dense(vt_world* w, uint8_t* h_materials, size_t nbytes, vt_stream stream) {
    if (!w) return VT_ERR_ARG;
    const size_t need = (size_t)w->dims[0] * w->dims[1] * w->dims[2];
    if (!h_materials || nbytes != need) return fail(w->ctx, VT_ERR_ARG, "dense download needs exactly X*Y*Z bytes");
    unsigned char* stage = nullptr;
    vt_status s = world_stage(w, need, &stage);
    if (s) return s;
    cudaStream_t st = (cudaStream_t)stream;
    k_gather_dense<<<(unsigned)w->nchunks, 512, 0, st>>>(w->view(), w->d_mats, stage);
    VT_CUDA(w->ctx, cudaGetLastError());
    VT_CUDA(w->ctx, cudaMemcpyAsync(h_materials, stage, need, cudaMemcpyDeviceToHost, st));
    VT_CUDA(w->ctx, cudaStreamSynchronize(st));
    return VT_OK;
}

}  // extern "C"
