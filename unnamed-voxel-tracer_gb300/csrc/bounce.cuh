// bounce.cuh -- bounce rays traced apart from the frame kernel.
//
// Cosine-distributed bounce rays (rng.glsl:41-55) are incoherent: within a
// warp of neighbouring pixels their lengths differ by an order of magnitude,
// so a warp tracing one per lane runs for its longest ray while most lanes
// wait (a step-sequence simulation of a terrain frame puts the useful work at
// a third of the issued work).  With deferral the frame kernel appends each
// hit's bounce ray (origin, direction, pixel) to a queue, with the pixel's
// colour if the ray leaves, and writes the record as if it hit (a coherent
// warp shades both colours for a third of what a pass over the finished pixels
// cost, 126 us of a 4K frame); a persistent kernel traces the queue with
// per-lane refill and recolours the pixels whose ray left.  Every ray is
// walked as in the inline path and the records are identical.
#pragma once

#include "shade.cuh"

namespace vt {

// A queued ray, kept as two arrays of 16 bytes so that a warp's appends and
// reads are whole lines: its origin and the direction's x, then the rest.
// pixel holds the pixel index (below 2^30) and, above it, whether its sun is
// blocked by a voxel (kJobShadowed) or by an entity.
struct __align__(16) BounceHead {
    float o[3];
    float dx;
};
struct __align__(16) BounceTail {
    float dy, dz;
    unsigned pixel;
    unsigned open_rgba;   // the pixel's colour if the ray leaves without a hit
};
struct BounceJob {
    BounceHead head;
    BounceTail tail;
};
static_assert(sizeof(BounceHead) == 16 && sizeof(BounceTail) == 16, "bounce job layout");
constexpr unsigned kJobPixel = (1u << 30) - 1u, kJobShadowed = 1u << 30, kJobEntity = 1u << 31;
static_assert((unsigned long long)kMaxImageSide * kMaxImageSide <= kJobPixel + 1ull, "pixel index and flags share a word");

__device__ __forceinline__ BounceJob bounce_job(const float o[3], const float d[3], unsigned pixel, unsigned flags,
                                                unsigned open_rgba) {
    BounceJob j;
#pragma unroll
    for (int k = 0; k < 3; ++k) j.head.o[k] = o[k];
    j.head.dx = d[0];
    j.tail.dy = d[1];
    j.tail.dz = d[2];
    j.tail.pixel = pixel | ((flags & VT_HIT_SHADOWED) ? kJobShadowed : 0u) | ((flags & VT_HIT_ENTITY) ? kJobEntity : 0u);
    j.tail.open_rgba = open_rgba;
    return j;
}

__device__ __forceinline__ void store_bounce(const FrameParams& f, unsigned slot, const BounceJob& job) {
    reinterpret_cast<BounceHead*>(f.bounce_head)[slot] = job.head;
    reinterpret_cast<BounceTail*>(f.bounce_tail)[slot] = job.tail;
}

// Appends one bounce ray; called by the lanes of a warp that have one, with
// the warp possibly diverged (one atomic per converged group).
__device__ __forceinline__ void append_bounce(const FrameParams& f, const BounceJob& job) {
    const unsigned act = __activemask();
    const unsigned lane = threadIdx.x & 31u;
    const int leader = __ffs(act) - 1;
    unsigned base = 0;
    if ((int)lane == leader) base = atomicAdd(f.bounce_count, (unsigned)__popc(act));
    base = __shfl_sync(act, base, leader);
    const unsigned slot = base + (unsigned)__popc(act & ((1u << lane) - 1u));
    store_bounce(f, slot, job);
}

// ---------------------------------------------------------------------------
// Direction-binned deferral (tuning bounce_sort).  Consecutive queue entries
// then start close together and head the same way, so that the lanes of a
// warp in the trace kernel walk similar paths: every thread of a 256-thread
// frame-kernel block (one 16 x 16-pixel tile) stages its bounce ray in the
// block's shared memory, and at the block's end the block sorts its rays by
// direction class (the cube-map face of the direction and a 4 x 4 cell on
// it, 96 classes) and appends them with one atomic.
constexpr int kStageThreads = 256;  // the frame kernel's block
constexpr unsigned kBins = 96;
constexpr unsigned char kNoBin = 0xFFu;

struct BounceStage {
    BounceJob job[kStageThreads];
    unsigned char bin[kStageThreads];
    unsigned hist[kBins];
    unsigned base;
};

__device__ __forceinline__ BounceStage& bounce_stage() {
    __shared__ BounceStage s;
    return s;
}

__device__ __forceinline__ unsigned direction_bin(const float d[3]) {
    const float ax = fabsf(d[0]), ay = fabsf(d[1]), az = fabsf(d[2]);
    float m = ax, u = d[1], v = d[2], s = d[0];
    unsigned face = 0;
    if (ay > m && ay >= az) {
        m = ay; u = d[0]; v = d[2]; s = d[1]; face = 2;
    } else if (az > m && az > ay) {
        m = az; u = d[0]; v = d[1]; s = d[2]; face = 4;
    }
    if (s < 0.0f) face += 1;
    const float iu = (u / m + 1.0f) * 2.0f, iv = (v / m + 1.0f) * 2.0f;   // [0, 4]
    const unsigned cu = iu >= 3.0f ? 3u : (iu >= 2.0f ? 2u : (iu >= 1.0f ? 1u : 0u));
    const unsigned cv = iv >= 3.0f ? 3u : (iv >= 2.0f ? 2u : (iv >= 1.0f ? 1u : 0u));
    return face * 16u + cu * 4u + cv;
}

// Every thread of the block, before any stage_bounce.
__device__ __forceinline__ void stage_begin() { bounce_stage().bin[threadIdx.x] = kNoBin; }

__device__ __forceinline__ void stage_bounce(const BounceJob& job) {
    BounceStage& st = bounce_stage();
    st.job[threadIdx.x] = job;
    const float d[3] = {job.head.dx, job.tail.dy, job.tail.dz};
    st.bin[threadIdx.x] = (unsigned char)direction_bin(d);
}

// Every thread of the block, at its end: sorts the staged rays by class and
// appends them to the queue (one atomic per block).
__device__ __forceinline__ void stage_flush(const FrameParams& f) {
    BounceStage& st = bounce_stage();
    const unsigned t = threadIdx.x, lane = t & 31u;
    if (t < kBins) st.hist[t] = 0u;
    __syncthreads();
    const unsigned b = st.bin[t];
    // rank within the class: one shared atomic per class and warp
    const unsigned peers = __match_any_sync(0xFFFFFFFFu, b);
    const int leader = __ffs(peers) - 1;
    unsigned wb = 0;
    if ((int)lane == leader && b != kNoBin) wb = atomicAdd(&st.hist[b], (unsigned)__popc(peers));
    wb = __shfl_sync(0xFFFFFFFFu, wb, leader);
    const unsigned rank = wb + (unsigned)__popc(peers & ((1u << lane) - 1u));
    __syncthreads();
    if (t < 32) {
        // exclusive scan of the class counts, 3 per lane
        const unsigned a = st.hist[3 * lane], c1 = st.hist[3 * lane + 1], c2 = st.hist[3 * lane + 2];
        unsigned incl = a + c1 + c2;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned v = __shfl_up_sync(0xFFFFFFFFu, incl, o);
            if ((int)lane >= o) incl += v;
        }
        const unsigned excl = incl - (a + c1 + c2);
        st.hist[3 * lane] = excl;
        st.hist[3 * lane + 1] = excl + a;
        st.hist[3 * lane + 2] = excl + a + c1;
        const unsigned total = __shfl_sync(0xFFFFFFFFu, incl, 31);
        if (lane == 31) st.base = total ? atomicAdd(f.bounce_count, total) : 0u;
    }
    __syncthreads();
    if (b != kNoBin) store_bounce(f, st.base + st.hist[b] + rank, st.job[t]);
}

}  // namespace vt
