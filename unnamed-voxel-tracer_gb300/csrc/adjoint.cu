// adjoint.cu -- differentiable Lambert shading over a fixed hit set.
//
//     c = palette[m] * albedo[v] * (ka + kd * max(0, n . s^) * V),  s^ = s / |s|
//     L = sum (c - target)^2
//     dL/dpalette[m]  = 2 (c - t) * albedo[v] * shade
//     dL/dalbedo[v]   = sum_k 2 (c_k - t_k) * palette[m][k] * shade
//     dL/ds           = (sum_k 2 (c_k - t_k) palette[m][k] albedo[v]) * kd * V * [n . s^ > 0]
//                       * (n - (n . s^) s^) / |s|
//
// The primary hits (voxel, face, material, t) come from vt_render and are held
// fixed; the shadow term V is recomputed here by tracing the shadow ray from
// the hit exactly as the render kernel does (same origin arithmetic, same
// traversal), instead of being stored between passes.  The backward kernel is
// the forward kernel plus the loss and gradient epilogue, one thread per
// pixel.  Palette gradients are summed per warp over the lanes that share a
// material (the warp walks its distinct materials), per block in shared memory,
// then once per block with global atomics; albedo gradients go to global memory
// with one atomic per pixel.
#include <cstring>

#include "shade.cuh"
#include "trace_p.cuh"

namespace vt {

namespace {

constexpr int kAdjBlock = 256;

struct AdjArgs {
    WorldView w;
    const float* pal;
    const float* alb;
    SunWalk sun;                  // the shadow rays
    float sun_raw[3];             // the sun as given (entity boxes)
    float sun_n[3], inv_len;
    float ka, kd;
    int shadow_steps;
    const unsigned char* vis_in;
    unsigned char* vis_out;
    float* loss;
    float* gpal;
    float* galb;
    float* gsun;
    double* sums;                 // 64-bit accumulators of the call, or null
};

// A call's accumulators: 768 palette gradients, the loss and the sun's
// gradient.  Zero between calls: k_shade_sums adds them to the caller's and
// clears them.  (Thousands of blocks adding to one float leave it off by up to
// 1e-5, in one direction where many blocks add the same value.)
constexpr int kGradSums = 772;
static_assert(kGradSums * sizeof(double) <= kShadeSumBytes, "accumulator region");
__device__ __forceinline__ float* grad_sum(const AdjArgs& a, int i) {
    return i < 768 ? a.gpal + i : (i == 768 ? a.loss : a.gsun + (i - 769));
}

// Several views of one world in one launch (blockIdx.z = view): one launch
// instead of one per view, whose tails would leave the GPU partly idle.
constexpr int kMaxViews = 16;
struct ViewP {
    float pos[3];
    float view[16];
    float tan_half_fov;
    int width, height;
    const uint4* hits;
    const float* target;
    float* rgb;
};
struct ViewsArgs {
    AdjArgs a;
    ViewP v[kMaxViews];
};
static_assert(sizeof(ViewsArgs) <= 4096, "the views travel in the kernel parameters");

// Sums of four values over the warp, halving the values with the lanes: the
// sums of a, b, c and d end in lanes 0, 8, 16 and 24 (6 shuffles instead of 20).
__device__ __forceinline__ float warp_sum4(unsigned lane, float a, float b, float c, float d) {
    const bool h16 = (lane & 16u) != 0u, h8 = (lane & 8u) != 0u;
    const float x = (h16 ? c : a) + __shfl_xor_sync(0xFFFFFFFFu, h16 ? a : c, 16);
    const float y = (h16 ? d : b) + __shfl_xor_sync(0xFFFFFFFFu, h16 ? b : d, 16);
    float r = (h8 ? y : x) + __shfl_xor_sync(0xFFFFFFFFu, h8 ? x : y, 8);
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) r += __shfl_xor_sync(0xFFFFFFFFu, r, o);
    return r;
}

// One block: 16x16 pixels.  The forward kernel is the shadow walks; the
// backward one adds the loss and gradients.
//
// A block shades one tile, and blocks start in the order of the views and of
// the tiles in a view: a voxel's albedo gradient is then summed in about that
// order, as by one call per view.  Blocks of four tiles side by side, which
// clear and flush their sums once for four, take 241 us an iteration instead of
// 258, but keep three views of 512x512 in flight at once: a voxel that fills
// much of several views gets 1e4 to 1e5 float addends, whose rounding goes one
// way within a binade, and the gradients of such scenes came out up to 4.6e-4
// from one call per view, where two runs of either differ by up to 9e-5.
//
// Bound: issue slots (forward 79%, 84 us; backward 63%, 147 us, its palette's
// clearing and flushing and its albedo atomics waiting for L2).  An iteration on 16 views of 512x512 took 339 us with the general walk,
// a sum over the warp per value and float atomics for every sum; now 258.
// Register caps: 6 blocks per SM (40 registers); backward with 5 269 us, with 7
// 250, but 2% slower on one view of 1920x1080; forward with 5 2% slower.
// ANY: a sun direction the forward walk does not take (trace_fast).  VIS: the
// shadow term is given, no ray is traced: bound by memory, and a kernel without
// the walk's registers (3840x2160 63.5 us; in the kernel with the walk 88).
template <bool BWD, bool ANY, bool VIS = false>
__global__ void __launch_bounds__(kAdjBlock, 6) k_shade_views(const __grid_constant__ ViewsArgs va) {
    const AdjArgs& a = va.a;
    const ViewP& V = va.v[blockIdx.z];
    __shared__ float s_gpal[BWD ? 768 : 1], s_acc[4];   // palette gradient; loss and sun
    __shared__ float s_col[16], s_row[16];              // ray UVs (shade.cuh, ray_u and ray_v)
    const int x0 = (int)blockIdx.x * 16, y0 = (int)blockIdx.y * 16;
    if (x0 >= V.width || y0 >= V.height) return;  // the view is smaller
    const int warp = threadIdx.x >> 5;
    const unsigned lane = threadIdx.x & 31u;
    const int lx = (warp & 1) * 8 + (int)(lane & 7u), ly = (warp >> 1) * 4 + (int)(lane >> 3);
    const int px = x0 + lx, py = y0 + ly;
    const bool inside = px < V.width && py < V.height;
    const size_t p = inside ? (size_t)py * V.width + px : 0;
    if (BWD) {
        for (int i = threadIdx.x; i < 768; i += kAdjBlock) s_gpal[i] = 0.0f;
        if (threadIdx.x < 4) s_acc[threadIdx.x] = 0.0f;
    }
    if (threadIdx.x < 16) {
        const float u = (((float)(x0 + (int)threadIdx.x) / (float)V.width) * 2.0f) - 1.0f;
        s_col[threadIdx.x] = u * V.tan_half_fov;
    } else if (threadIdx.x >= 128 && threadIdx.x < 144) {
        const float W = (float)V.width, H = (float)V.height;
        float v = (((float)(y0 + (int)threadIdx.x - 128) / H) * 2.0f) - 1.0f;
        v = v * (H / W);
        s_row[threadIdx.x - 128] = v * V.tan_half_fov;
    }
    __syncthreads();
    float lossv = 0.0f, gsun[3] = {0.0f, 0.0f, 0.0f};
    bool hit = false;
    int m = 0;
    unsigned v = 0;
    float c[3] = {0.0f, 0.0f, 0.0f}, shade = 0.0f, albv = 1.0f, ndl_raw = 0.0f, nrm[3] = {0.0f, 0.0f, 0.0f};
    bool lit = false;
    if (inside) {
        const uint4 rec = V.hits[p];
        hit = ((rec.w >> 16) & VT_HIT_PRIMARY) != 0;
        if (hit) {
            v = rec.x;
            const float t = __uint_as_float(rec.y);
            const unsigned face = rec.w & 0xFFu;
            m = (int)((rec.w >> 8) & 0xFFu);
            const int axis = (int)(face >> 1);
            const bool pos = (face & 1u) == 0u;
            // the primary ray (primary_ray_uv) and the shadow origin
            const float u = s_col[lx], w = s_row[ly];
            float q[3], so[3];
#pragma unroll
            for (int j = 0; j < 3; ++j) q[j] = ((u * V.view[j] + w * V.view[4 + j]) + V.view[8 + j]) + V.view[12 + j];
            const float len = __fsqrt_rn((q[0] * q[0] + q[1] * q[1]) + q[2] * q[2]);
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                float d = __fdiv_rn(q[j], len);
                if (d == 0.0f) d = 0.001f;   // map.glsl:85-90
                nrm[j] = (j == axis) ? (pos ? -1.0f : 1.0f) : 0.0f;
                so[j] = __fmaf_rn(d, t, V.pos[j]);
                if (j == axis) so[j] = so[j] + nrm[j] * 0.001f;
            }
            if (VIS) {
                lit = a.vis_in[p] != 0;
            } else {
                bool blocked;
                if (ANY) {
                    PRay rs;
                    pray_init_dir(rs, so, a.sun.d, a.sun.inv);
                    TraceHit hs;
                    blocked = trace_fast<false, true, true>(a.w, a.w.cdist, rs, a.shadow_steps, hs);
                } else {
                    blocked = trace_sun<true>(a.w, a.sun, so, a.shadow_steps);
                }
                lit = !blocked &&
                      !(a.w.n_entities > 0 && entity_occluded(a.w, so, a.sun_raw));
            }
            ndl_raw = dot3(nrm, a.sun_n);
            const float ndl = ndl_raw > 0.0f ? ndl_raw : 0.0f;
            shade = a.ka + a.kd * ndl * (lit ? 1.0f : 0.0f);
            albv = a.alb ? __ldg(a.alb + v) : 1.0f;
#pragma unroll
            for (int k = 0; k < 3; ++k) c[k] = (__ldg(a.pal + 3 * m + k) * albv) * shade;
        }
    }
    if (!BWD) {
        if (inside) {
#pragma unroll
            for (int k = 0; k < 3; ++k) V.rgb[3 * p + k] = c[k];
            if (a.vis_out) a.vis_out[p] = (unsigned char)(hit && lit ? 1 : 0);
        }
        return;
    }

    // ---- loss and gradients
    float g[3] = {0.0f, 0.0f, 0.0f};
    if (inside) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const float diff = c[k] - __ldg(V.target + 3 * p + k);
            g[k] = 2.0f * diff;
            lossv += diff * diff;
        }
    }
    float gp[3] = {0.0f, 0.0f, 0.0f};
    if (hit) {
        float ga = 0.0f, gb = 0.0f;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const float pk = __ldg(a.pal + 3 * m + k);
            gp[k] = g[k] * albv * shade;
            ga += g[k] * pk * shade;
            gb += g[k] * pk * albv;
        }
        if (lit && ndl_raw > 0.0f) {
            const float coef = gb * a.kd * a.inv_len;
#pragma unroll
            for (int k = 0; k < 3; ++k) gsun[k] += coef * (nrm[k] - ndl_raw * a.sun_n[k]);
        }
        // albedo: one global atomic per hit pixel (voxels differ across
        // most of a warp; the L2 absorbs the few repeats)
        if (a.galb) atomicAdd(a.galb + v, ga);
    }
    // palette: one shared-memory atomic per (warp, material, channel).
    // The warp walks its distinct materials (few per warp), no divergence.
    unsigned todo = __ballot_sync(0xFFFFFFFFu, hit);
    while (todo) {
        const int key = __shfl_sync(0xFFFFFFFFu, m, __ffs(todo) - 1);
        const bool mine = hit && m == key;
        todo &= ~__ballot_sync(0xFFFFFFFFu, mine);
        const float s = warp_sum4(lane, mine ? gp[0] : 0.0f, mine ? gp[1] : 0.0f, mine ? gp[2] : 0.0f, 0.0f);
        if ((lane & 7u) == 0u && lane < 24u) atomicAdd(s_gpal + 3 * key + (lane >> 3), s);
    }
    {
        const float s = warp_sum4(lane, lossv, gsun[0], gsun[1], gsun[2]);
        if ((lane & 7u) == 0u) atomicAdd(s_acc + (lane >> 3), s);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < kGradSums; i += kAdjBlock) {
        const float g = i < 768 ? s_gpal[i] : s_acc[i - 768];
        if (g == 0.0f) continue;
        if (a.sums) atomicAdd(a.sums + i, (double)g);
        else atomicAdd(grad_sum(a, i), g);   // (a captured launch may be replayed beside others)
    }
}

// Adds the launches' accumulators to the caller's and clears them.  A launch
// of its own: the last block of the launch before would have to know itself
// the last, and a fence in every block waits for its albedo atomics (139
// against 130 us).
__global__ void __launch_bounds__(kAdjBlock) k_shade_sums(AdjArgs a) {
    for (int i = threadIdx.x; i < kGradSums; i += kAdjBlock) {
        const double g = a.sums[i];
        if (g != 0.0) {
            atomicAdd(grad_sum(a, i), (float)g);
            a.sums[i] = 0.0;
        }
    }
}

// Checks the arguments shared by all views, brings the distances up to date on
// st and fills the shared part of `a` (its frame from `cam`).
vt_status prepare_shade(vt_ctx* ctx, const vt_world* world, const vt_shade_inputs* in, AdjArgs& a, cudaStream_t st) {
    if (!ctx) return VT_ERR_ARG;
    if (!world || !in || !in->d_palette) return fail(ctx, VT_ERR_ARG, "null shading argument");
    if (world->ctx != ctx) return fail(ctx, VT_ERR_ARG, "world belongs to another context");
    const float len2 = (in->sun[0] * in->sun[0] + in->sun[1] * in->sun[1]) + in->sun[2] * in->sun[2];
    if (!(len2 > 0.0f)) return fail(ctx, VT_ERR_ARG, "sun direction must be nonzero");
    {
        vt_status s = update_distances(const_cast<vt_world*>(world), st);
        if (s) return s;
    }
    FrameParams f;
    std::memset(&f, 0, sizeof(f));
    for (int j = 0; j < 3; ++j) f.sun[j] = in->sun[j];
    frame_constants(f);
    a.w = world->view();
    a.pal = in->d_palette;
    a.alb = in->d_albedo;
    for (int j = 0; j < 3; ++j) {
        a.sun_raw[j] = in->sun[j];
        a.sun_n[j] = f.sun_n[j];
    }
    a.sun = sun_walk(f, a.w);
    a.inv_len = 1.0f / sqrtf(len2);
    a.ka = in->ambient;
    a.kd = in->diffuse;
    a.shadow_steps = in->shadow_max_steps;
    return VT_OK;
}

bool camera_size_ok(const vt_camera* cam) {
    return cam->width > 0 && cam->height > 0 && cam->width <= kMaxImageSide && cam->height <= kMaxImageSide;
}

// One of the context's accumulator regions for a call on st, which first waits
// for the call that used the region last (on any stream), or clears it if it is
// the first; the caller records *used after its launches.  None while st is
// being captured: the graph's replays could overlap other launches.
vt_status shade_sums(vt_ctx* ctx, cudaStream_t st, double** sums, cudaEvent_t* used) {
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    VT_CUDA(ctx, cudaStreamIsCapturing(st, &cs));
    if (cs != cudaStreamCaptureStatusNone) return VT_OK;
    const unsigned r = ctx->shade_region % kShadeRegions;
    void* region = static_cast<char*>(ctx->d_shade_sums) + (size_t)r * kShadeSumBytes;
    if (ctx->ev_shade[r]) {
        VT_CUDA(ctx, cudaStreamWaitEvent(st, ctx->ev_shade[r], 0));
    } else {
        VT_CUDA(ctx, cudaMemsetAsync(region, 0, kShadeSumBytes, st));
        VT_CUDA(ctx, cudaEventCreateWithFlags(&ctx->ev_shade[r], cudaEventDisableTiming));
    }
    ++ctx->shade_region;
    *sums = static_cast<double*>(region);
    *used = ctx->ev_shade[r];
    return VT_OK;
}

// n views in launches of up to kMaxViews (the loss and gradients of
// `a` are shared; each view has its hits and its target or output image).
vt_status launch_shade_views(vt_ctx* ctx, const vt_world* world, int32_t n, const vt_camera* cams,
                             const vt_hit* const* d_hits, const vt_shade_inputs* in, const float* const* d_targets,
                             float* const* d_rgb, AdjArgs a, bool bwd, cudaStream_t st) {
    for (int v = 0; v < n; ++v) {
        if (!d_hits[v] || (bwd ? !d_targets[v] : !d_rgb[v])) return fail(ctx, VT_ERR_ARG, "null view buffer");
        if (!camera_size_ok(&cams[v])) return fail(ctx, VT_ERR_ARG, "camera size out of range (1..32768)");
    }
    vt_status s = prepare_shade(ctx, world, in, a, st);
    if (s) return s;
    cudaEvent_t used = nullptr;
    if (bwd) {
        s = shade_sums(ctx, st, &a.sums, &used);
        if (s) return s;
    }
    const bool any = !ordinary_inv(a.sun.inv);
    auto k = bwd ? (any ? k_shade_views<true, true> : k_shade_views<true, false>)
                 : (a.vis_in ? k_shade_views<false, false, true>
                             : (any ? k_shade_views<false, true> : k_shade_views<false, false>));
    ViewsArgs va;
    std::memset(&va, 0, sizeof(va));
    cudaError_t e = cudaSuccess;
    for (int v0 = 0; v0 < n && e == cudaSuccess; v0 += kMaxViews) {
        const int nv = n - v0 < kMaxViews ? n - v0 : kMaxViews;
        int gw = 0, gh = 0;
        for (int i = 0; i < nv; ++i) {
            const vt_camera& c = cams[v0 + i];
            ViewP& V = va.v[i];
            for (int j = 0; j < 3; ++j) V.pos[j] = c.pos[j];
            std::memcpy(V.view, c.view, sizeof(V.view));
            V.tan_half_fov = c.tan_half_fov;
            V.width = c.width;
            V.height = c.height;
            V.hits = reinterpret_cast<const uint4*>(d_hits[v0 + i]);
            V.target = bwd ? d_targets[v0 + i] : nullptr;
            V.rgb = bwd ? nullptr : d_rgb[v0 + i];
            gw = c.width > gw ? c.width : gw;
            gh = c.height > gh ? c.height : gh;
        }
        va.a = a;
        const dim3 grid((gw + 15) / 16, (gh + 15) / 16, nv);
        k<<<grid, kAdjBlock, 0, st>>>(va);
        e = cudaGetLastError();
    }
    if (a.sums) {   // (after a failed launch too: the region is left zero)
        k_shade_sums<<<1, kAdjBlock, 0, st>>>(a);
        const cudaError_t es = cudaGetLastError(), er = cudaEventRecord(used, st);
        if (e == cudaSuccess) e = es != cudaSuccess ? es : er;
    }
    return e == cudaSuccess ? VT_OK : check_cuda(ctx, e, "shading launch");
}

}  // namespace

}  // namespace vt

using namespace vt;

extern "C" {

vt_status vt_shade_forward(vt_ctx* ctx, const vt_world* world, const vt_camera* cam, const vt_hit* d_hits,
                           const vt_shade_inputs* in, const uint8_t* d_vis_in, uint8_t* d_vis_out, float* d_rgb,
                           vt_stream stream) {
    if (!ctx) return VT_ERR_ARG;
    if (!d_rgb) return fail(ctx, VT_ERR_ARG, "null output image");
    AdjArgs a;
    std::memset(&a, 0, sizeof(a));
    a.vis_in = d_vis_in;
    a.vis_out = d_vis_out;
    if (!cam || !d_hits) return fail(ctx, VT_ERR_ARG, "null shading argument");
    return launch_shade_views(ctx, world, 1, cam, &d_hits, in, nullptr, &d_rgb, a, false, (cudaStream_t)stream);
}

vt_status vt_shade_backward(vt_ctx* ctx, const vt_world* world, const vt_camera* cam, const vt_hit* d_hits,
                            const vt_shade_inputs* in, const float* d_target, float* d_loss, float* d_grad_palette,
                            float* d_grad_albedo, float* d_grad_sun, vt_stream stream) {
    if (!ctx) return VT_ERR_ARG;
    if (!d_target || !d_loss || !d_grad_palette || !d_grad_sun)
        return fail(ctx, VT_ERR_ARG, "null target, loss or gradient buffer");
    AdjArgs a;
    std::memset(&a, 0, sizeof(a));
    a.loss = d_loss;
    a.gpal = d_grad_palette;
    a.galb = d_grad_albedo;
    a.gsun = d_grad_sun;
    if (!cam || !d_hits) return fail(ctx, VT_ERR_ARG, "null shading argument");
    return launch_shade_views(ctx, world, 1, cam, &d_hits, in, &d_target, nullptr, a, true, (cudaStream_t)stream);
}

vt_status vt_shade_forward_views(vt_ctx* ctx, const vt_world* world, int32_t n, const vt_camera* cams,
                                 const vt_hit* const* d_hits, const vt_shade_inputs* in, float* const* d_rgb,
                                 vt_stream stream) {
    if (!ctx) return VT_ERR_ARG;
    if (n < 0 || (n > 0 && (!cams || !d_hits || !d_rgb))) return fail(ctx, VT_ERR_ARG, "bad view lists");
    if (n == 0) return VT_OK;
    AdjArgs a;
    std::memset(&a, 0, sizeof(a));
    return launch_shade_views(ctx, world, n, cams, d_hits, in, nullptr, d_rgb, a, false, (cudaStream_t)stream);
}

vt_status vt_shade_backward_views(vt_ctx* ctx, const vt_world* world, int32_t n, const vt_camera* cams,
                                  const vt_hit* const* d_hits, const vt_shade_inputs* in, const float* const* d_targets,
                                  float* d_loss, float* d_grad_palette, float* d_grad_albedo, float* d_grad_sun,
                                  vt_stream stream) {
    if (!ctx) return VT_ERR_ARG;
    if (n < 0 || (n > 0 && (!cams || !d_hits || !d_targets))) return fail(ctx, VT_ERR_ARG, "bad view lists");
    if (!d_loss || !d_grad_palette || !d_grad_sun) return fail(ctx, VT_ERR_ARG, "null loss or gradient buffer");
    if (n == 0) return VT_OK;
    // One launch for up to 16 views (blockIdx.z = view) instead of one per
    // view on concurrent streams.
    AdjArgs a;
    std::memset(&a, 0, sizeof(a));
    a.loss = d_loss;
    a.gpal = d_grad_palette;
    a.galb = d_grad_albedo;
    a.gsun = d_grad_sun;
    return launch_shade_views(ctx, world, n, cams, d_hits, in, d_targets, nullptr, a, true, (cudaStream_t)stream);
}
}  // extern "C"
