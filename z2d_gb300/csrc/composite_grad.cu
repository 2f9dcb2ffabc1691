// composite_grad.cu -- the compositor's mask batch with a gradient source.
//
// supersample.zig:171-184 / SurfaceCompositor.run (compositor.zig:302-440)
// with the batch [dst_in(dst = gradient or dithered gradient, src = alpha8
// mask), op] over a whole 4-byte-format or alpha8 surface, integer precision.
// The
// generic composite kernel evaluates such a pixel through out-of-line
// calls and run-time dispatch on every level (source kind, gradient kind,
// interpolation method, operator); here the gradient kind, the
// interpolation space and the presence of a dither are template parameters
// and everything is inlined, so a pixel is its lanes in f32 (grad_f32.cuh;
// where they are undecided, the double-word or f64 offset and the exact
// colour) and the two operators.  Pixel coordinates advance with
// the grid stride instead of being divided out per pixel.  (alpha8, where
// the general kernel's thread draws 16 pixels in turn: 1704 x 86 linear HSL
// with blue noise 66 us, now 25; 1718 x 1347 conic sRGB 144, now 62.)
#include <cuda_runtime.h>

#include <atomic>

#include "z2d_internal.h"

namespace z2dg {

namespace {

constexpr int kGradThreads = 256;

enum : int { kLinRGB = 0, kSRGB = 1, kHSL = 2 };

template <int KIND>
__device__ __forceinline__ float offset_inline(const DevGradient &g, int32_t x, int32_t y) {
    // the kind is known here, so only its evaluation is compiled in
    if ((uint32_t)(x + (1 << 22)) < (1u << 23) && (uint32_t)(y + (1 << 22)) < (1u << 23)) {
        const int32_t mode = g.fz.mode;
        if (mode == kFastVoid) return -1.0f;
        if (mode != kFastNone) {
            const float fx = (float)x + 0.5f, fy = (float)y + 0.5f;
            const bool tf = g.has_tf != 0;
            float t = 0.0f;
            int done;
            if constexpr (KIND == Z2D_GRADIENT_LINEAR) done = fast_linear(g.fz, tf, fx, fy, t);
            else if constexpr (KIND == Z2D_GRADIENT_CONIC) done = fast_conic(g.fz, tf, fx, fy, t);
            else done = fast_radial(g.fz, tf, mode == kFastRadialA0, fx, fy, t);
            if (done) return t;
        }
    }
    return offset_f64_call(g, x, y);
}

// The linear offset inline; the radial and conic evaluations (several
// times its code) out of line, one copy per kind.
template <int KIND>
__device__ __noinline__ float offset_call(const DevGradient &g, int32_t x, int32_t y) {
    return offset_inline<KIND>(g, x, y);
}
template <int KIND>
__device__ __forceinline__ float offset_of(const DevGradient &g, int32_t x, int32_t y) {
    if constexpr (KIND == Z2D_GRADIENT_LINEAR) return offset_inline<KIND>(g, x, y);
    else return offset_call<KIND>(g, x, y);
}
// The source's colour lanes at (x, y): interpolateEncode, or the dithered
// linear colour encoded (Dither.getPixel)
template <int KIND, int METHOD, bool DITH>
__device__ __noinline__ I16 grad_lanes_exact(const DevSrc &s, const DevGradient &g, int32_t x, int32_t y) {
    const Search r = grad_search(g, offset_of<KIND>(g, x, y));
    const RGBf a = stop_prep(g, r.i0), b = stop_prep(g, r.i1);
    // (SRGB.interpolate then toLinearRGB, as interp_encode_prep /
    // interp_linear_prep do, with the gamma out of line)
    if constexpr (!DITH) {
        if constexpr (METHOD == kLinRGB) {
            return interp_encode_prep(Z2D_INTERP_LINEAR_RGB, a, b, r.offset);
        } else if constexpr (METHOD == kSRGB) {
            const RGBf d = rgb_lerp_demul(a, b, r.offset);
            return encode_linear(RGBf{gamma_call(d.r), gamma_call(d.g), gamma_call(d.b), d.a});
        } else {
            return encode_linear(hsl_call(a, b, r.offset, g.method));
        }
    } else {
        RGBf c;
        if constexpr (METHOD == kLinRGB) {
            c = rgb_lerp_demul(a, b, r.offset);
        } else if constexpr (METHOD == kSRGB) {
            const RGBf d = rgb_lerp_demul(a, b, r.offset);
            c = RGBf{gamma_call(d.r), gamma_call(d.g), gamma_call(d.b), d.a};
        } else {
            c = hsl_call(a, b, r.offset, g.method);
        }
        const float m = s.dither_type == Z2D_DITHER_BAYER ? bayer(x, y) : blue_noise(x, y);
        const float scale = 1.0f / (float)((1 << s.dither_scale) - 1);
        return encode_linear(RGBf{fmaxf(0.0f, fminf(c.r + m * scale, 1.0f)), fmaxf(0.0f, fminf(c.g + m * scale, 1.0f)),
                                  fmaxf(0.0f, fminf(c.b + m * scale, 1.0f)), fmaxf(0.0f, fminf(c.a + m * scale, 1.0f))});
    }
}

// The batch's second half for one pixel: dst_in(source lanes, mask), then the
// operator on the destination word.
__device__ __forceinline__ uint32_t grad_composite(int op, uint32_t w, I16 sl, uint32_t m8, int fmt) {
    if (op == Z2D_OP_SRC_OVER && fmt != Z2D_FORMAT_ALPHA8) {  // two channels per 32-bit operation
        const uint32_t L = i16_to_word(sl, word_order(fmt));
        const uint32_t e = div255x2((L & 0x00FF00FFu) * m8), o = div255x2(((L >> 8) & 0x00FF00FFu) * m8);
        return word_src_over(w, e | (o << 8), fmt == Z2D_FORMAT_RGBA || fmt == Z2D_FORMAT_ARGB);
    }
    // IntegerOps.dstIn(d = source, s = mask), then the operator
    const I16 rl = int_op(Z2D_OP_DST_IN, sl, I16{0u, 0u, 0u, m8});
    if (fmt == Z2D_FORMAT_ALPHA8) return int_op_any(op, I16{0u, 0u, 0u, w}, rl).a & 0xFFu;
    return i16_to_word(int_op_any(op, word_to_i16(w, fmt), rl), fmt);
}

// A lane takes a pixel at a time (32 neighbours per warp: coalesced, and the
// body, a few hundred instructions, is compiled once); the pixels whose lanes
// f32 does not decide (grad_f32.cuh) go to the warp's list, 32 of which are
// evaluated exactly at a time: the exact evaluation, several times as long,
// then never runs for one lane with 31 waiting.
template <int KIND, int METHOD, bool DITH>
__global__ void __launch_bounds__(kGradThreads) k_mask_grad(uint8_t *__restrict__ dst, const uint8_t *__restrict__ mask,
                                                           int32_t W, size_t n_px, int32_t fmt, int32_t op,
                                                           const DevSrc src) {
    constexpr uint32_t kAll = 0xffffffffu;
    __shared__ unsigned long long lists[kGradThreads / 32][64];
    const int lane = threadIdx.x & 31;
    unsigned long long *list = lists[threadIdx.x >> 5];
    const DevGradient &g = *src.grad;
    uint32_t *dw = reinterpret_cast<uint32_t *>(dst);
    const int method = METHOD == kLinRGB ? Z2D_INTERP_LINEAR_RGB : METHOD == kSRGB ? Z2D_INTERP_SRGB : src.grad_method;
    const int dither = DITH ? src.dither_type : Z2D_DITHER_NONE;
    const float step = DITH ? dither_step_of(src.dither_scale) : 0.0f;
    const size_t first = (size_t)blockIdx.x * kGradThreads + threadIdx.x;
    const size_t stride = (size_t)gridDim.x * kGradThreads;
    // (x, y) of this thread's first pixel, then advanced by the stride
    // (q rows and r columns)
    int32_t y = (int32_t)(first / (size_t)W), x = (int32_t)(first - (size_t)y * W);
    const int32_t q = (int32_t)(stride / (size_t)W), r = (int32_t)(stride - (size_t)q * W);
    int n = 0;  // pixels in the list
    const bool bytes = fmt == Z2D_FORMAT_ALPHA8;
    auto pixel = [&](size_t p) -> uint32_t { return bytes ? dst[p] : dw[p]; };
    auto put = [&](size_t p, uint32_t v) {
        if (bytes) dst[p] = (uint8_t)v;
        else dw[p] = v;
    };
    auto exact = [&](int at) {
        const size_t p = (size_t)list[at];
        const int32_t py = (int32_t)(p / (size_t)W), px = (int32_t)(p - (size_t)py * W);
        put(p, grad_composite(op, pixel(p), grad_lanes_exact<KIND, METHOD, DITH>(src, g, px, py), mask[p], fmt));
    };
#pragma unroll 1
    for (size_t p0 = first - lane; p0 < n_px; p0 += stride) {
        const size_t p = p0 + lane;
        bool late = false;
        if (p < n_px) {
            const uint32_t w = pixel(p), m8 = __ldcs(mask + p);
            I16 sl;
            if (grad_lanes_f32(KIND, method, dither, step, g, x, y, sl)) put(p, grad_composite(op, w, sl, m8, fmt));
            else late = true;
        }
        const uint32_t m = __ballot_sync(kAll, late);
        if (late) list[n + __popc(m & ((1u << lane) - 1u))] = p;
        n += __popc(m);
        if (n >= 32) {
            __syncwarp();
            n -= 32;
            exact(n + lane);
            __syncwarp();
        }
        y += q;
        if (x >= W - r) {  // (x + r may not fit)
            x -= W - r;
            y++;
        } else {
            x += r;
        }
    }
    __syncwarp();
    if (lane < n) exact(lane);
}

using GradKernel = void (*)(uint8_t *, const uint8_t *, int32_t, size_t, int32_t, int32_t, const DevSrc);

template <int KIND>
GradKernel pick_method(int method, bool dith) {
    if (method == Z2D_INTERP_LINEAR_RGB) return dith ? k_mask_grad<KIND, kLinRGB, true> : k_mask_grad<KIND, kLinRGB, false>;
    if (method == Z2D_INTERP_SRGB) return dith ? k_mask_grad<KIND, kSRGB, true> : k_mask_grad<KIND, kSRGB, false>;
    return dith ? k_mask_grad<KIND, kHSL, true> : k_mask_grad<KIND, kHSL, false>;
}

// Resident blocks per SM of each instantiation (3 kinds x 3 methods x
// dither or not), looked up once: the grid is sized to what fits at once,
// so that no block of the grid-stride loop waits for a second wave.
std::atomic<int> g_grad_occ[3][3][2];

}  // namespace

// The batch [dst_in(gradient source, alpha8 mask), op] on a whole surface of a
// 4-byte format or alpha8 in integer precision; false when J has another
// shape.
bool try_mask_grad(Ctx &c, const CompJob &J, bool whole) {
    if (!whole || J.n_ops != 2 || J.precision != Z2D_PRECISION_INTEGER) return false;
    const CompOp &o0 = J.ops[0], &o1 = J.ops[1];
    if (o0.op != Z2D_OP_DST_IN || o0.src.kind != SRC_SURFACE || o1.dst.kind != SRC_NONE || o1.src.kind != SRC_NONE)
        return false;
    const DevSrc &s = o0.dst;
    bool dith = false;
    if (s.kind == SRC_DITHER) {
        if (s.dither_source != Z2D_DITHER_SRC_GRADIENT ||
            (s.dither_type != Z2D_DITHER_BAYER && s.dither_type != Z2D_DITHER_BLUE_NOISE))
            return false;
        dith = true;
    } else if (s.kind != SRC_GRADIENT) {
        return false;
    }
    if (!s.grad || J.dst.fmt > Z2D_FORMAT_ALPHA8 || o1.op < 0 || o1.op >= Z2D_OP_COUNT) return false;
    if (o0.src.sfc.fmt != Z2D_FORMAT_ALPHA8 || o0.src.sfc.w != J.dst.w || o0.src.sfc.h < J.dst.h) return false;
    if (J.dst.fmt <= Z2D_FORMAT_RGBA && (reinterpret_cast<uintptr_t>(J.dst.data) & 3) != 0) return false;
    const size_t px = (size_t)J.dst.w * J.dst.h;
    const int kind = s.grad_type, method = s.grad_method;
    if (kind < Z2D_GRADIENT_LINEAR || kind > Z2D_GRADIENT_CONIC) return false;
    GradKernel k = kind == Z2D_GRADIENT_LINEAR   ? pick_method<Z2D_GRADIENT_LINEAR>(method, dith)
                   : kind == Z2D_GRADIENT_RADIAL ? pick_method<Z2D_GRADIENT_RADIAL>(method, dith)
                                                 : pick_method<Z2D_GRADIENT_CONIC>(method, dith);
    const int mslot = method == Z2D_INTERP_LINEAR_RGB ? 0 : method == Z2D_INTERP_SRGB ? 1 : 2;
    std::atomic<int> &slot = g_grad_occ[kind - Z2D_GRADIENT_LINEAR][mslot][dith ? 1 : 0];
    int occ = slot.load(std::memory_order_relaxed);
    if (occ <= 0) {
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k, kGradThreads, 0) != cudaSuccess || occ <= 0) occ = 1;
        slot.store(occ, std::memory_order_relaxed);
    }
    size_t blocks = (px + kGradThreads - 1) / kGradThreads;
    const size_t cap = (size_t)c.sm_count * (size_t)occ;
    if (blocks > cap) blocks = cap;
    if (blocks == 0) return true;
    k<<<(unsigned)blocks, kGradThreads, 0, c.stream>>>(J.dst.data, o0.src.sfc.data, J.dst.w, px, J.dst.fmt, o1.op,
                                                      s);
    c.launches++;
    return true;
}

}  // namespace z2dg
