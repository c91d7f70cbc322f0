// Test-only: the frame's pixel (render_pixel.cuh) and the shadow walk
// (trace_p.cuh) compiled as host C++, each run under a limit of walk steps and
// with every world read checked against its array, so that a walk that would
// not end, or would read outside its world, is found without a GPU.
#include <math.h>
#include <stdint.h>
#include <string.h>
#include <limits.h>
#include <algorithm>
#include <stdexcept>
#include <vector>

#include <cuda_runtime.h>

using std::max;
using std::min;

struct WalkFault : std::runtime_error {
    using std::runtime_error::runtime_error;
};
static thread_local int64_t steps_left = 0;
#define VT_STEP_HOOK(kind) \
    do { if (--steps_left < 0) throw WalkFault("endless"); } while (0)

// The arrays a read may fall in.
struct Range {
    const char *lo, *hi;
};
static std::vector<Range> ranges;
template <class T> static inline T __ldg(const T* p) {
    for (const Range& r : ranges)
        if ((const char*)p >= r.lo && (const char*)(p + 1) <= r.hi) return *p;
    throw WalkFault("read out of range");
}

// IEEE host equivalents of the intrinsics the headers use.
static inline float __fmaf_rn(float a, float b, float c) { return fmaf(a, b, c); }
static inline float __frcp_rn(float x) { return 1.0f / x; }
static inline float __fmul_rn(float a, float b) { return a * b; }
static inline float __fadd_rn(float a, float b) { return a + b; }
static inline float __fsub_rn(float a, float b) { return a - b; }
static inline float __fdiv_rn(float a, float b) { return a / b; }
static inline float __fsqrt_rn(float a) { return sqrtf(a); }
static inline float __int2float_rn(int k) { return (float)k; }
static inline float __uint2float_rn(unsigned k) { return (float)k; }
static inline float __saturatef(float x) { return x > 0.0f ? (x < 1.0f ? x : 1.0f) : 0.0f; }
static inline unsigned __float_as_uint(float x) { unsigned u; memcpy(&u, &x, 4); return u; }
static inline int __float_as_int(float x) { return (int)__float_as_uint(x); }
static inline float __uint_as_float(unsigned u) { float x; memcpy(&x, &u, 4); return x; }
static inline float __int_as_float(int u) { return __uint_as_float((unsigned)u); }
static inline int __float2int_rd(float x) {
    if (x != x) return 0;
    if (x >= 2147483647.0f) return INT_MAX;
    if (x <= -2147483648.0f) return INT_MIN;
    return (int)floorf(x);
}
static inline unsigned __byte_perm(unsigned a, unsigned b, unsigned s) {
    const uint64_t v = a | ((uint64_t)b << 32);
    unsigned r = 0;
    for (int i = 0; i < 4; ++i) r |= (unsigned)((v >> (8 * ((s >> (4 * i)) & 7u))) & 0xFFu) << (8 * i);
    return r;
}
static inline int __popc(unsigned x) { return __builtin_popcount(x); }
static inline int __ffs(int x) { return __builtin_ffs(x); }
static inline unsigned __activemask() { return 1u; }
template <class T> static inline T __shfl_sync(unsigned, T v, int) { return v; }
template <class T> static inline T __shfl_up_sync(unsigned, T v, int) { return v; }
static inline unsigned __match_any_sync(unsigned, unsigned) { return 1u; }
static inline void __syncthreads() {}
template <class T> static inline T atomicAdd(T* p, T v) { T o = *p; *p += v; return o; }
static inline unsigned atomicOr(unsigned* p, unsigned v) { unsigned o = *p; *p |= v; return o; }
static const struct { unsigned x; } threadIdx = {0};

#include "../../unnamed-voxel-tracer_gb300/csrc/render_pixel.cuh"

namespace {

struct HostWorld {
    vt::WorldView w;
    std::vector<unsigned long long> mask;
    std::vector<unsigned char> mats, bdist, cdist;
    std::vector<unsigned> palette;
    HostWorld(const int32_t dims[3], const uint8_t* dense, const uint8_t* brick, const uint8_t* chunk) {
        memset(&w, 0, sizeof(w));
        for (int i = 0; i < 3; ++i) {
            w.dims[i] = dims[i];
            w.cdim[i] = (dims[i] + 31) / 32;
        }
        const size_t nch = (size_t)w.cdim[0] * w.cdim[1] * w.cdim[2];
        mask.assign(nch * 512, 0ull);
        mats.assign(nch * 32768, 0);
        for (int z = 0; z < dims[2]; ++z)
            for (int y = 0; y < dims[1]; ++y)
                for (int x = 0; x < dims[0]; ++x) {
                    const unsigned char m = dense[(size_t)x + (size_t)dims[0] * ((size_t)y + (size_t)dims[1] * z)];
                    if (!m) continue;
                    const size_t wi = ((size_t)(x >> 5) + w.cdim[0] * ((size_t)(y >> 5) + (size_t)w.cdim[1] * (z >> 5))) * 512 +
                                      (((x >> 2) & 7) | (((y >> 2) & 7) << 3) | (((z >> 2) & 7) << 6));
                    const unsigned vb = (x & 3) | ((y & 3) << 2) | ((z & 3) << 4);
                    mask[wi] |= 1ull << vb;
                    mats[wi * 64 + vb] = m;
                }
        const unsigned cstride = vt::cdist_stride((unsigned)nch);
        bdist.assign(brick, brick + vt::kOctants * nch * 512);
        cdist.assign((size_t)vt::kOctants * cstride, 0);
        for (int o = 0; o < vt::kOctants; ++o) std::copy(chunk + o * nch, chunk + (o + 1) * nch, cdist.begin() + (size_t)o * cstride);
        palette.assign(vt::kPaletteBytes / 4, 0u);
        w.mask = mask.data();
        w.mats = mats.data();
        w.bdist = bdist.data();
        w.cdist = cdist.data();
        w.palette = palette.data();
        w.nwords = (unsigned)(nch * 512);
        w.nchunks = (unsigned)nch;
        w.cstride = cstride;
        ranges.clear();
        auto add = [](const auto& v) { ranges.push_back({(const char*)v.data(), (const char*)(v.data() + v.size())}); };
        add(mask), add(mats), add(bdist), add(cdist), add(palette);
    }
};

// Sun fields of the shadow walk (as sun_walk makes them for a frame).
vt::SunWalk sun_fields(const float sun[3], const vt::WorldView& w) {
    vt::SunWalk s;
    unsigned oct = 0;
    s.flip = 0;
    for (int j = 0; j < 3; ++j) {
        const float d = sun[j] == 0.0f ? 0.001f : sun[j];
        const bool up = d > 0.0f;
        s.d[j] = d;
        s.inv[j] = 1.0f / d;
        s.m[j] = up ? 0 : -1;
        s.side[j] = up ? 1.0f : -1.0f;
        s.off[j] = up ? 1.0f : 0.0f;
        s.ad[j] = fabsf(d);
        s.ai[j] = fabsf(s.inv[j]);
        s.exit[j] = up ? (float)w.dims[j] : 0.0f;
        s.in_hi[j] = (float)(w.dims[j] - 1);
        if (up) oct |= 1u << j;
        else s.flip |= 3u << (2 * j);
    }
    s.field = oct * w.nwords;
    return s;
}

}  // namespace

enum { kEnded = 0, kEndless = 1, kOutOfRange = 2 };

static int fault_of(const WalkFault& e) { return strcmp(e.what(), "endless") ? kOutOfRange : kEndless; }

// Primary and shadow rays of a width x height frame (16 floats of view, row
// major): per pixel {how the walks ended, the record's flags}.
extern "C" void we_frame(const int32_t dims[3], const uint8_t* dense, const uint8_t* brick, const uint8_t* chunk,
                         const float pos[3], const float view[16], float tan_half_fov, int32_t width, int32_t height,
                         const float sun[3], int32_t max_steps, int64_t limit, uint8_t* out) {
    HostWorld hw(dims, dense, brick, chunk);
    vt::FrameParams f;
    memset(&f, 0, sizeof(f));
    bool inside = vt::near_origin(pos);
    for (int j = 0; j < 3; ++j) {
        f.pos[j] = pos[j];
        if (!(pos[j] >= 1.0f && pos[j] <= (float)(dims[j] - 1))) inside = false;
    }
    f.cam_inside = inside ? 1 : 0;
    for (int j = 0; j < 3; ++j) f.cam_c[j] = inside ? floorf(pos[j]) : 0.0f;
    memcpy(f.view, view, sizeof(f.view));
    f.tan_half_fov = tan_half_fov;
    f.width = width;
    f.height = height;
    f.row_end = height;
    f.max_steps = f.shadow_max_steps = max_steps;
    f.sunw = sun_fields(sun, hw.w);
    for (int j = 0; j < 3; ++j) {
        f.sun[j] = sun[j];
        f.sun_d[j] = f.sunw.d[j];
        f.sun_inv[j] = f.sunw.inv[j];
    }
    f.rays = VT_RAYS_PRIMARY | VT_RAYS_SHADOW;
    f.shade = VT_SHADE_NONE;
    const bool any = vt::any_shadow(f);
    for (int y = 0; y < height; ++y)
        for (int x = 0; x < width; ++x) {
            uint8_t* o = out + 2 * ((size_t)y * width + x);
            o[0] = kEnded;
            o[1] = 0;
            steps_left = limit;
            try {
                vt::PixelCounters pc;
                auto pixel = any ? vt::render_pixel<false, false, vt::CoarseGlobal, false, false, false, true>
                                 : vt::render_pixel<false, false, vt::CoarseGlobal, false, false, false, false>;
                const uint4 r = pixel(hw.w, vt::CoarseGlobal{nullptr}, hw.w.cdist, f, x, y, vt::pixel_uv(f, x, y), nullptr, pc);
                o[1] = (uint8_t)(r.w >> 16);
            } catch (const WalkFault& e) {
                o[0] = (uint8_t)fault_of(e);
            }
        }
}

// Shadow rays from n start points: per point {how the shading kernels' walk
// ended, whether it is blocked, the same of trace_fast, the same of the general
// walk, which takes any origin}.
extern "C" void we_shadow(const int32_t dims[3], const uint8_t* dense, const uint8_t* brick, const uint8_t* chunk,
                          const float sun[3], const float* origins, int64_t n, int32_t max_steps, int64_t limit,
                          uint8_t* out) {
    HostWorld hw(dims, dense, brick, chunk);
    const vt::SunWalk s = sun_fields(sun, hw.w);
    for (int64_t i = 0; i < n; ++i) {
        const float* so = origins + 3 * i;
        vt::PRay r;
        vt::pray_init_dir(r, so, s.d, s.inv);
        for (int k = 0; k < 3; ++k) {
            uint8_t* o = out + 6 * i + 2 * k;
            o[0] = kEnded;
            o[1] = 0;
            steps_left = limit;
            vt::TraceHit h;
            try {
                if (k == 0) {
                    o[1] = vt::trace_sun<true>(hw.w, s, so, max_steps);
                } else if (k == 1) {
                    o[1] = vt::trace_fast<false, true, true>(hw.w, hw.w.cdist, r, max_steps, h);
                } else {
                    vt::Walker wk;
                    int st = vt::Walker::kMiss;
                    if (wk.start_ray(hw.w, r, max_steps))
                        while ((st = wk.step<false, true, true>(hw.w, hw.w.cdist, h)) == vt::Walker::kMore) {
                        }
                    o[1] = st == vt::Walker::kHit;
                }
            } catch (const WalkFault& e) {
                o[0] = (uint8_t)fault_of(e);
            }
        }
    }
}
