// render_pixel.cuh -- one pixel of the render-frame path (primary, shadow and
// bounce rays, shading, the 16-byte record), shared by the single-frame and
// the batched kernels.
#pragma once

#include "bounce.cuh"
#include "shade.cuh"
#include "trace_p.cuh"

namespace vt {

// Whether a frame needs kernels whose shadow rays may be any: a sun direction
// that the forward walk does not take, or a far camera.  A near camera's hits are
// within a cell of the grid: a hit's t is a plane's crossing time inside it, and
// the direction has length 1.  From 2^40 and beyond they may be 2^20 away.  (The
// general walk beside the forward one for every frame: a 16-scene batch 1236 us
// against 1224, a batch with bounce rays 296 against 258.)
inline bool any_shadow(const FrameParams& f) { return !ordinary_inv(f.sun_inv) || !near_origin(f.pos); }

struct PixelCounters {
    unsigned v[kNumCounters];
};

// The instrumented and bounds-checked variants run the three-level model
// traversal (it defines the algorithmic byte counts); the production variant
// runs trace_fast.  Both give identical results.
// NEAR: the caller knows the origin passes near_origin (secondary rays start
// on a hit inside the grid); otherwise the primary ray checks it once.
// SHARE: brick words shared between the lanes of a warp (Walker::brick_word).
template <bool STATS, bool CHECKED, bool MAT, bool NEAR, bool SHARE, class Coarse>
__device__ __forceinline__ bool trace_any(const WorldView& w, const Coarse& coarse, const unsigned char* cd,
                                          const PRay& r, int max_steps, TraceHit& h, TraceCounters& cnt,
                                          unsigned* status) {
    if (STATS || CHECKED) return trace_p<STATS, CHECKED, MAT>(w, coarse, r, max_steps, h, cnt, status);
    if (NEAR || near_origin(r.o)) return trace_fast<MAT, true, true, SHARE>(w, cd, r, max_steps, h);
    return trace_fast<MAT, true, false, SHARE>(w, cd, r, max_steps, h);
}

// The primary ray of a frame whose camera is inside the grid: its cell is the
// frame's (walk_constants).
__device__ __forceinline__ bool trace_primary(const WorldView& w, const FrameParams& f, const PRay& r, TraceHit& h) {
    FwdWalk fw;
    bool go;
    if (f.cam_inside) {   // uniform
        fw.t = 0.0f;
        go = fw.start_cell(w, r, f.cam_c, f.max_steps);
    } else {
        go = fw.start(w, r, f.max_steps);
    }
    return go && fw.finish<true>(w, r, h);
}

// uv: the pixel's screen coordinates (pixel_uv(f, px, py); the frame kernel
// reads them from the frame's screen table or its per-block tables).
// BIN: a deferred bounce ray is staged in the block's shared memory for the
// block's direction-sorted append (stage_flush) instead of appended at once.
// BOUNCE: false leaves the bounce rays' code out (frames without them: the
// kernel's registers and code then serve the walk alone).  ANY: the shadow rays
// may be any (any_shadow).
template <bool STATS, bool CHECKED, class Coarse, bool SHARE = false, bool BIN = false, bool BOUNCE = true,
          bool ANY = true>
__device__ __forceinline__ uint4 render_pixel(const WorldView& w, const Coarse& coarse, const unsigned char* cd,
                                              const FrameParams& f, int px, int py, const PixelUV& uv,
                                              unsigned* status, PixelCounters& pc) {
    float o[3], d[3];
    primary_ray_uv(f, uv, o, d);
    PRay r;
    pray_init(r, o, d);
    TraceHit h;
    TraceCounters cnt;
    constexpr bool kForward = !STATS && !CHECKED && !SHARE;
    const bool hit = kForward && (f.cam_inside || near_origin(r.o)) && ordinary_inv(r.inv)
                         ? trace_primary(w, f, r, h)
                         : trace_any<STATS, CHECKED, true, false, SHARE>(w, coarse, cd, r, f.max_steps, h, cnt, status);
    if (STATS) {
        pc.v[0] += 1;
        pc.v[9] += 16;
    }
    unsigned flags = 0, rgba, voxel = 0xFFFFFFFFu, face = 0xFFu, mat = 0;
    float t = -1.0f;
    float col[4];
    if (hit) {
        flags = VT_HIT_PRIMARY;
        voxel = (unsigned)h.c[0] + (unsigned)w.dims[0] * ((unsigned)h.c[1] + (unsigned)w.dims[1] * (unsigned)h.c[2]);
        t = h.t;
        const int e = h.axis;
        const bool pe = e == 0 ? r.pos[0] : (e == 1 ? r.pos[1] : r.pos[2]);
        face = 2u * (unsigned)e + (pe ? 0u : 1u);
        mat = h.mat;
        const float4 alb = albedo_of(w, mat);
        if (STATS) {
            pc.v[1] += 1;
            pc.v[8] += 1;
        }
        float nrm[3], so[3];
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            nrm[j] = (j == e) ? (pe ? -1.0f : 1.0f) : 0.0f;
            so[j] = __fmaf_rn(r.d[j], t, o[j]);
            if (j == e) so[j] = so[j] + nrm[j] * 0.001f;
        }
        bool shadowed = false;
        if (f.rays & VT_RAYS_SHADOW) {
            if (kForward && (!ANY || ordinary_inv(f.sun_inv))) {
                shadowed = trace_sun<ANY>(w, f.sunw, so, f.shadow_max_steps);
            } else {
                PRay rs;
                pray_init_dir(rs, so, f.sun_d, f.sun_inv);
                TraceHit hs;
                shadowed = trace_any<STATS, CHECKED, false, true, SHARE>(w, coarse, cd, rs, f.shadow_max_steps, hs, cnt, status);
            }
            if (shadowed) flags |= VT_HIT_SHADOWED;
            if (STATS) {
                pc.v[2] += 1;
                pc.v[3] += shadowed ? 1u : 0u;
            }
            if (!shadowed && w.n_entities > 0 && entity_occluded(w, so, f.sun)) {
                shadowed = true;
                flags |= VT_HIT_ENTITY;
            }
        }
        bool bounce_open = false;
        bool deferred = false;
        float bdir[3] = {0.0f, 0.0f, 0.0f};
        if (BOUNCE && (f.rays & VT_RAYS_BOUNCE)) {
            unsigned seed = ((unsigned)px * 1973u + (unsigned)py * 9277u) ^ f.seed;
            cosine_hemisphere(nrm, seed, bdir);
            deferred = !STATS && !CHECKED && f.bounce_head != nullptr;
        }
        if (deferred) {
            // traced by the bounce kernel (bounce.cu).  The record assumes a
            // hit; a ray that leaves turns it into the open colour
            shade_hit(f, alb, e, pe, shadowed, true, bdir, col);
            const unsigned open = f.shade == VT_SHADE_NONE ? __ldg(w.palette + mat) : composite_uv(f, uv, col);
            const BounceJob job = bounce_job(so, bdir, (unsigned)py * (unsigned)f.width + (unsigned)px, flags, open);
            if (BIN) stage_bounce(job);
            else append_bounce(f, job);
            flags |= VT_HIT_BOUNCE;
        } else if (BOUNCE && (f.rays & VT_RAYS_BOUNCE)) {
            PRay rb;
            pray_init(rb, so, bdir);
            TraceHit hb;
            const bool bh = trace_any<STATS, CHECKED, false, true, SHARE>(w, coarse, cd, rb, f.bounce_max_steps, hb, cnt, status);
            if (bh) flags |= VT_HIT_BOUNCE;
            bounce_open = !bh;
            if (STATS) {
                pc.v[4] += 1;
                pc.v[5] += bh ? 1u : 0u;
            }
        }
        shade_hit(f, alb, e, pe, shadowed, bounce_open, bdir, col);
        rgba = f.shade == VT_SHADE_NONE ? __ldg(w.palette + mat) : composite_uv(f, uv, col);
    } else {
        shade_miss(f, d, col);
        rgba = f.shade == VT_SHADE_NONE ? 0u : composite_uv(f, uv, col);
    }
    if (STATS) {
        pc.v[6] += cnt.mask;
        pc.v[7] += cnt.coarse;
        pc.v[10] += cnt.steps;
        pc.v[11] += cnt.iters;
    }
    return make_uint4(voxel, __float_as_uint(t), rgba, face | (mat << 8) | (flags << 16));
}

}  // namespace vt
