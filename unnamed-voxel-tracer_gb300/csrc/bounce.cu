// bounce.cu -- the deferred bounce pass (see bounce.cuh): a persistent
// kernel that traces the queued bounce rays with per-lane refill and recolours
// the pixels whose ray leaves.
#include "bounce.cuh"
#include "launch.cuh"
#include "trace_p.cuh"

namespace vt {

namespace {

constexpr int kBounceBlock = 256;
// a warp takes new rays from the queue once this many of its lanes are idle
// (tuning bounce_refill), and a busy lane makes kActions iterations of the walk
// between two refill checks: 12 and 3 are fastest of 4-16 and 1-4 with the
// forward walk (4K cave frame as first measured 1145 us; 8 and 2: 1182, 16 and
// 4: 1146; refill alone, now: 12 1135 us, 4 1145, 8 1142, 16 1132)
constexpr int kRefill = 12;
constexpr int kActions = 3;

// The walk of one lane.  Both start a ray (kMore: under way; kHit or kMiss: it
// is done already) and advance it by one step.
template <bool FLAT>
struct Walk;

// Walker::step_flat (one code path for jumps and unit steps).
template <>
struct Walk<true> {
    Walker wk;
    __device__ __forceinline__ int start(const WorldView& w, const float o[3], const float d[3], int steps) {
        return wk.start(w, o, d, steps) ? Walker::kMore : Walker::kMiss;
    }
    __device__ __forceinline__ int step(const WorldView& w) {
        TraceHit h;
        return wk.step_flat<true>(w, w.cdist, h);
    }
};

// The forward walk; a ray it does not take (a reciprocal out of its range, a far
// origin) is traced to its end by Walker at the start.
template <>
struct Walk<false> {
    FwdWalk fw;
    __device__ __forceinline__ int start(const WorldView& w, const float o[3], const float d[3], int steps) {
        PRay r;
        pray_init(r, o, d);
        if (ordinary_inv(r.inv) && near_origin(o)) return fw.start(w, r, steps) ? Walker::kMore : Walker::kMiss;
        TraceHit h;
        return trace_fast<false, true, true>(w, w.cdist, r, steps, h) ? Walker::kHit : Walker::kMiss;
    }
    __device__ __forceinline__ int step(const WorldView& w) {
        unsigned wi, vb;
        return fw.step(w, wi, vb);
    }
};

// The record of a pixel whose bounce ray left without a hit: the open colour,
// and the flags without VT_HIT_BOUNCE (the frame kernel wrote it as a hit).
__device__ __forceinline__ void open_pixel(uint4* out, unsigned pixel, unsigned rgba) {
    vt_hit* r = reinterpret_cast<vt_hit*>(out + (pixel & kJobPixel));
    r->rgba = rgba;
    r->flags = (uint8_t)(VT_HIT_PRIMARY | ((pixel & kJobShadowed) ? VT_HIT_SHADOWED : 0u) |
                         ((pixel & kJobEntity) ? VT_HIT_ENTITY : 0u));
}

// Persistent: every warp loops until the queue is drained.  A lane walks one
// ray at a time, kActions iterations of the walk per loop turn.
// Bound: issue slots (78%) at 11.7 lanes an instruction, the lanes of a warp
// being in different phases of unrelated walks; the register cap (4 blocks of
// 64 registers; uncapped 96) hides the lookups' latency.  7 M rays of a 4K
// cave frame: 622 us (601 without chunk jumps and the far test).  Measured
// against 614 then, slower: setting 32 rays up at a time in shared
// memory for idle lanes to take (727 us: the copies cost more instructions
// than the set-ups at few lanes), one code path for jumps and unit steps (568 us
// here, but 11% slower on a 1021x577 frame whose queue is short).
template <bool FLAT>
__global__ void __launch_bounds__(kBounceBlock, 4) k_bounce_trace(WorldView w, const BounceHead* __restrict__ heads,
                                                               const BounceTail* __restrict__ tails,
                                                               const unsigned* __restrict__ counters,
                                                               unsigned* __restrict__ next, uint4* __restrict__ out,
                                                               int max_steps, int refill) {
    const unsigned total = counters[0];
    const unsigned lane = threadIdx.x & 31u;
    const unsigned below = (1u << lane) - 1u;
    Walk<FLAT> wk;
    bool busy = false;
    unsigned job = 0;
    for (;;) {
        const unsigned idle = __ballot_sync(0xFFFFFFFFu, !busy);
        if (idle == 0xFFFFFFFFu || __popc(idle) >= refill) {
            unsigned base = 0;
            if (lane == 0) base = atomicAdd(next, (unsigned)__popc(idle));
            base = __shfl_sync(0xFFFFFFFFu, base, 0);
            if (base >= total && idle == 0xFFFFFFFFu) break;  // drained, and nothing in flight
            if (!busy) {
                job = base + (unsigned)__popc(idle & below);
                if (job < total) {
                    const BounceHead H = heads[job];
                    const BounceTail T = tails[job];
                    const float d[3] = {H.dx, T.dy, T.dz};
                    const int s = wk.start(w, H.o, d, max_steps);
                    busy = s == Walker::kMore;
                    if (s == Walker::kMiss) open_pixel(out, T.pixel, T.open_rgba);
                }
            }
        }
        if (busy) {
            int s = Walker::kMore;
            for (int a = 0; a < kActions && s == Walker::kMore; ++a) s = wk.step(w);
            if (s != Walker::kMore) {
                if (s == Walker::kMiss) open_pixel(out, tails[job].pixel, tails[job].open_rgba);
                busy = false;
            }
        }
    }
}

}  // namespace

vt_status bounce_buffers(vt_ctx* ctx, size_t pixels) {
    if (pixels <= ctx->bounce_capacity) return VT_OK;
    VT_CUDA(ctx, cudaDeviceSynchronize());
    if (ctx->d_bounce_head) vt::dev_free(ctx->d_bounce_head);
    if (ctx->d_bounce_tail) vt::dev_free(ctx->d_bounce_tail);
    ctx->d_bounce_head = nullptr;
    ctx->d_bounce_tail = nullptr;
    ctx->bounce_capacity = 0;
    VT_CUDA(ctx, vt::dev_alloc(&ctx->d_bounce_head, pixels * sizeof(BounceHead)));
    VT_CUDA(ctx, vt::dev_alloc(&ctx->d_bounce_tail, pixels * sizeof(BounceTail)));
    if (!ctx->d_bounce_ctr) VT_CUDA(ctx, vt::dev_alloc(&ctx->d_bounce_ctr, 2 * sizeof(unsigned)));
    if (!ctx->ev_bounce) VT_CUDA(ctx, cudaEventCreateWithFlags(&ctx->ev_bounce, cudaEventDisableTiming));
    ctx->bounce_capacity = pixels;
    return VT_OK;
}

vt_status launch_bounce(vt_ctx* ctx, const vt_world* world, const FrameParams& f, uint4* d_out, cudaStream_t st) {
    const WorldView w = world->view();
    const int flat = ctx->tuning.bounce_walk == 1 ? 1 : 0;
    const int refill = ctx->tuning.bounce_refill > 0 ? ctx->tuning.bounce_refill : kRefill;
    auto k = flat ? k_bounce_trace<true> : k_bounce_trace<false>;
    if (ctx->bounce_blocks[flat] == 0) {
        int nb = 0;
        VT_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k, kBounceBlock, 0));
        ctx->bounce_blocks[flat] = ctx->sm_count * (nb > 0 ? nb : 1);
    }
    cudaAccessPolicyWindow win_storage;
    const cudaAccessPolicyWindow* win = nullptr;  // L2 window over the brick words (tuning l2_persist)
    vt_status s = l2_policy(ctx, world, &win_storage, &win);
    if (s) return s;
    VT_CUDA(ctx, launch_kernel(k, dim3(ctx->bounce_blocks[flat]), dim3(kBounceBlock), 0, st, win, w,
                               (const BounceHead*)ctx->d_bounce_head, (const BounceTail*)ctx->d_bounce_tail,
                               (const unsigned*)ctx->d_bounce_ctr, ctx->d_bounce_ctr + 1, d_out, f.bounce_max_steps,
                               refill));
    // the next deferred frame of this context reuses the queue after this one
    VT_CUDA(ctx, cudaEventRecord(ctx->ev_bounce, st));
    return VT_OK;
}

}  // namespace vt
