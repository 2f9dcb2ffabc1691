// composite_layer.cu -- one surface composited onto another
// (Surface.composite, src/surface.zig:225-241: SurfaceCompositor.run with one
// surface-source operation), 4-byte formats or alpha8, integer precision, any
// offset.
//
// Bound by memory: 12 bytes a pixel.  The general region kernel divides out
// every pixel's row and reads one pixel at a time through the batch's
// run-time dispatch; here a warp takes 128 neighbouring pixels of a row, four
// per lane 32 apart (eight loads in flight, all coalesced whatever the
// offset's alignment), the operator is a template parameter, and src_over
// works on two channels per 32-bit operation.  2563x1441 RGBA pixels onto
// 3840x2160 (44 MB, in L2): 10.3 us, the region kernel 45; with the L2 written
// over before each call 15.4 and 56.9 (events around the launch, 3 us of them
// their own); 803x701 alpha8 xor 9.3 us a call, the region kernel 10.8.
#include <cuda_runtime.h>

#include <utility>

#include "z2d_internal.h"

namespace z2dg {

namespace {

constexpr int kLayerWarps = 8;
constexpr int kLayerPx = 4;                // pixels per lane
constexpr int kLayerChunk = 32 * kLayerPx;  // pixels of a row per warp

struct LayerArgs {
    uint8_t *dst;         // the region's first pixel
    const uint8_t *src;   // the source's pixel composited there
    int32_t dst_w, src_w; // pixels per surface row
    int32_t line_w, rows;
    int32_t dst_fmt, src_fmt;
    int32_t per_row;      // chunks per row
};

// T: a pixel, a 4-byte format's word or an alpha8 byte.
template <int OP, class T>
__global__ void __launch_bounds__(32 * kLayerWarps) k_layer(const LayerArgs A) {
    const int lane = threadIdx.x & 31;
    const long long chunk = (long long)blockIdx.x * kLayerWarps + (threadIdx.x >> 5);
    const int32_t row = (int32_t)(chunk / A.per_row);
    if (row >= A.rows) return;
    const int32_t x0 = (int32_t)(chunk - (long long)row * A.per_row) * kLayerChunk + lane;
    T *d = reinterpret_cast<T *>(A.dst) + (size_t)A.dst_w * row;
    const T *s = reinterpret_cast<const T *>(A.src) + (size_t)A.src_w * row;
    uint32_t dw[kLayerPx], sw[kLayerPx];
#pragma unroll
    for (int k = 0; k < kLayerPx; k++) {
        const int32_t x = x0 + 32 * k;
        dw[k] = sw[k] = 0u;
        if (x < A.line_w) {
            dw[k] = d[x];
            sw[k] = s[x];
        }
    }
    const bool has_alpha = A.dst_fmt == Z2D_FORMAT_RGBA || A.dst_fmt == Z2D_FORMAT_ARGB;
    const bool src_alpha = A.src_fmt == Z2D_FORMAT_RGBA || A.src_fmt == Z2D_FORMAT_ARGB;
    const bool swap = word_order(A.dst_fmt) != word_order(A.src_fmt);
#pragma unroll
    for (int k = 0; k < kLayerPx; k++) {
        const int32_t x = x0 + 32 * k;
        if (x >= A.line_w) break;
        uint32_t out;
        if constexpr (sizeof(T) == 1) {
            out = int_op(OP, I16{0u, 0u, 0u, dw[k]}, I16{0u, 0u, 0u, sw[k]}).a;
        } else if constexpr (OP == Z2D_OP_SRC_OVER) {
            uint32_t L = swap ? __byte_perm(sw[k], 0u, 0x3012) : sw[k];
            if (!src_alpha) L |= 0xFF000000u;
            out = word_src_over(dw[k], L, has_alpha);
        } else {
            out = i16_to_word(int_op(OP, word_to_i16(dw[k], A.dst_fmt), word_to_i16(sw[k], A.src_fmt)), A.dst_fmt);
        }
        d[x] = (T)out;
    }
}

using LayerKernel = void (*)(const LayerArgs);

template <class T, int... OPS>
LayerKernel layer_kernel(int op, std::integer_sequence<int, OPS...>) {
    static const LayerKernel table[] = {&k_layer<OPS, T>...};
    return table[op];
}

}  // namespace

// One surface-source operation in integer precision between 4-byte formats, or
// from alpha8 to alpha8, whose source covers the whole region; false when J
// has another shape.
bool try_layer(Ctx &c, const CompJob &J) {
    if (J.n_ops != 1 || J.precision != Z2D_PRECISION_INTEGER) return false;
    const CompOp &o = J.ops[0];
    if (o.dst.kind != SRC_NONE || o.src.kind != SRC_SURFACE || o.op < 0 || o.op >= Z2D_OP_COUNT || requires_float(o.op))
        return false;
    const DevSurface &s = o.src.sfc;
    const bool a8 = J.dst.fmt == Z2D_FORMAT_ALPHA8 && s.fmt == Z2D_FORMAT_ALPHA8;
    if (!a8 && (J.dst.fmt > Z2D_FORMAT_RGBA || s.fmt > Z2D_FORMAT_RGBA)) return false;
    const int32_t sx = J.dsx - J.dst_x, sy = J.y0 - J.dst_y;
    if (sx < 0 || sy < 0 || sx + J.line_w > s.w || sy + (J.y1 - J.y0) > s.h) return false;
    if (!a8 && ((reinterpret_cast<uintptr_t>(J.dst.data) | reinterpret_cast<uintptr_t>(s.data)) & 3) != 0) return false;
    LayerArgs A;
    const size_t px = a8 ? 1 : 4;
    A.dst = J.dst.data + px * ((size_t)J.dst.w * J.y0 + J.dsx);
    A.src = s.data + px * ((size_t)s.w * sy + sx);
    A.dst_w = J.dst.w;
    A.src_w = s.w;
    A.line_w = J.line_w;
    A.rows = J.y1 - J.y0;
    A.dst_fmt = J.dst.fmt;
    A.src_fmt = s.fmt;
    A.per_row = row_chunks(J.line_w, kLayerChunk);
    const long long blocks = ((long long)A.per_row * A.rows + kLayerWarps - 1) / kLayerWarps;
    if (blocks > 0x7FFFFFFFll) return false;
    const std::make_integer_sequence<int, Z2D_OP_COUNT> ops{};
    const LayerKernel k = a8 ? layer_kernel<uint8_t>(o.op, ops) : layer_kernel<uint32_t>(o.op, ops);
    k<<<(unsigned)blocks, 32 * kLayerWarps, 0, c.stream>>>(A);
    c.launches++;
    return true;
}

}  // namespace z2dg
