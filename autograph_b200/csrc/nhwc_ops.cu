// Channels-last helpers of the convolution stages (see nhwc_ops.cuh).  Every thread moves
// 16 bytes (8 channels of one pixel); consecutive threads take consecutive channel groups of a
// pixel and then consecutive pixels, so every access of a warp is one contiguous run.
#include "nhwc_ops.cuh"
#include "pool_codes.cuh"

namespace ag {
namespace nhwc {

namespace {

struct Vec8 {
    uint4 raw;
    __device__ __forceinline__ float get(int i) const {
        const uint32_t w = (&raw.x)[i >> 1];
        return __uint_as_float((i & 1) ? (w & 0xffff0000u) : (w << 16));
    }
    __device__ __forceinline__ void set_pair(int j, float a, float b) {
        __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
        (&raw.x)[j] = *reinterpret_cast<uint32_t *>(&h);
    }
};

// FH, FW > 0: the filter size is a compile-time constant (the divisions below become shifts
// and multiplies; with run-time divisors the kernel is bound by them, 173 us against the 25 us
// its 126 MB of stores take at the wide stack's first layer).
template <int FH, int FW>
__global__ void im2col_channels_kernel(const __nv_bfloat16 *__restrict__ x, __nv_bfloat16 *__restrict__ out,
                                       int ic, int ih, int iw, int fh_rt, int fw_rt, int oh, int ow, int cp,
                                       uint32_t per_image) {
    const int fh = FH > 0 ? FH : fh_rt, fw = FW > 0 ? FW : fw_rt;
    const uint32_t groups = (uint32_t)cp / 8;
    const int taps = fh * fw, k = ic * taps;
    const int64_t plane = (int64_t)ih * iw;
    const int64_t b = blockIdx.y;   // one image per grid row: 32-bit index arithmetic inside it
    out += b * (int64_t)per_image * 8;
    // The stride of the loop is a multiple of the groups per pixel, so a thread keeps its channel
    // group: the eight source offsets relative to the pixel are computed once.
    const uint32_t first = blockIdx.x * blockDim.x + threadIdx.x;
    const int g = (int)(first % groups);
    int off[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        const int c = g * 8 + e;
        const int ci = c / taps, r = c - ci * taps;
        const int fi = r / fw, fj = r - fi * fw;
        off[e] = c < k ? (int)(ci * plane) + fi * iw + fj : -1;
    }
    const unsigned short *img = reinterpret_cast<const unsigned short *>(x) + b * ic * plane;
    for (uint32_t i = first; i < per_image; i += gridDim.x * blockDim.x) {
        const uint32_t t = i / groups;
        const uint32_t oy = t / (uint32_t)ow, ox = t - oy * (uint32_t)ow;
        uint32_t wds[4] = {0u, 0u, 0u, 0u};
        if (g * 8 < k) {
            const unsigned short *px = img + oy * (uint32_t)iw + ox;
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const unsigned short v = off[e] >= 0 ? __ldg(px + off[e]) : (unsigned short)0;
                wds[e >> 1] |= (uint32_t)v << ((e & 1) * 16);
            }
        }
        reinterpret_cast<uint4 *>(out)[i] = make_uint4(wds[0], wds[1], wds[2], wds[3]);
    }
}

// The same for the channel pitch of a 64-channel tensor, with the rows a CTA reads staged in shared memory
// and nothing divided per store: the kernel above spends 43 us on 256 x 3 x 64 x 64, 19 us of it stores, in
// index arithmetic and two-byte loads that touch 30 cache lines a warp.
template <int FH, int FW>
__global__ void __launch_bounds__(256)
    im2col_rows_kernel(const __nv_bfloat16 *__restrict__ x, __nv_bfloat16 *__restrict__ out, int ic, int ih, int iw, int oh,
                       int ow, int rows) {
    let_dependents_launch();
    dependency_wait();
    extern __shared__ __align__(16) unsigned short staged[];   // [ic][rows + FH - 1][iw]
    constexpr int taps = FH * FW, groups = 8;
    const int64_t b = blockIdx.y;
    const int y0 = blockIdx.x * rows, ny = min(rows, oh - y0), have = ny + FH - 1, run = have * iw;
    const unsigned short *img = reinterpret_cast<const unsigned short *>(x) + (b * ic * ih + y0) * iw;
    if (iw % 8 == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0) {
        for (int i = threadIdx.x; i < ic * (run / 8); i += 256) {
            const int c = i / (run / 8), r = i - c * (run / 8);
            reinterpret_cast<uint4 *>(staged)[i] = __ldg(reinterpret_cast<const uint4 *>(img + (int64_t)c * ih * iw) + r);
        }
    } else {
        for (int c = 0; c < ic; ++c)
            for (int i = threadIdx.x; i < run; i += 256) staged[c * run + i] = __ldg(img + (int64_t)c * ih * iw + i);
    }
    // a thread keeps its channel group: eight offsets, and the words that hold channels at all
    const int g = threadIdx.x % groups, k = ic * taps;
    int off[8];
    uint32_t keep[4] = {0u, 0u, 0u, 0u};
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        const int c = g * 8 + e, ci = c / taps, r = c - ci * taps;
        off[e] = c < k ? ci * run + r / FW * iw + r % FW : 0;
        if (c < k) keep[e >> 1] |= 0xffffu << ((e & 1) * 16);
    }
    __syncthreads();
    uint4 *q = reinterpret_cast<uint4 *>(out) + (b * oh + y0) * (int64_t)ow * groups + threadIdx.x;
    int ry = threadIdx.x / groups / ow, ox = threadIdx.x / groups - ry * ow;
    while (ry < ny) {
        uint4 o = make_uint4(0u, 0u, 0u, 0u);
        if (g * 8 < k) {
            const unsigned short *px = staged + ry * iw + ox;
            uint32_t v[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) v[e] = px[off[e]];
            o = make_uint4(__byte_perm(v[0], v[1], 0x5410) & keep[0], __byte_perm(v[2], v[3], 0x5410) & keep[1],
                           __byte_perm(v[4], v[5], 0x5410) & keep[2], __byte_perm(v[6], v[7], 0x5410) & keep[3]);
        }
        *q = o;
        q += 256;
        for (ox += 256 / groups; ox >= ow; ox -= ow) ++ry;
    }
}

template <int FH, int FW>
bool launch_im2col_rows(ag_device *dev, const __nv_bfloat16 *x, __nv_bfloat16 *out, int64_t bs, int64_t ic, int64_t ih,
                        int64_t iw, int64_t oh, int64_t ow, int64_t cp) {
    if (cp != 64) return false;
    for (int rows = 16; rows >= 1; rows /= 2) {   // what fits in shared memory without opting in to more
        const int64_t bytes = ic * (rows + FH - 1) * iw * 2;
        if (bytes > 40 * 1024) continue;
        im2col_rows_kernel<FH, FW><<<dim3((unsigned)ceil_div(oh, rows), (unsigned)bs), 256, (size_t)bytes, dev->stream>>>(
            x, out, (int)ic, (int)ih, (int)iw, (int)oh, (int)ow, rows);
        return true;
    }
    return false;
}

// One window's eight channels from p (the window's first pixel) on; returns the pooled values.
__device__ __forceinline__ uint4 pool_window(const __nv_bfloat16 *p, int64_t row, int cp, uint32_t &code) {
    const uint4 raw[4] = {*reinterpret_cast<const uint4 *>(p), *reinterpret_cast<const uint4 *>(p + cp),
                          *reinterpret_cast<const uint4 *>(p + row),
                          *reinterpret_cast<const uint4 *>(p + row + cp)};   // (0,0), (0,1), (1,0), (1,1)
    uint32_t o[4];
    code = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const uint32_t cells[4] = {(&raw[0].x)[j], (&raw[1].x)[j], (&raw[2].x)[j], (&raw[3].x)[j]};
        uint32_t c8;
        o[j] = relu_pool_pair(cells, c8);
        code |= c8 << (8 * j);
    }
    return make_uint4(o[0], o[1], o[2], o[3]);
}

__global__ void relu_pool_kernel(const __nv_bfloat16 *__restrict__ pre, __nv_bfloat16 *__restrict__ y,
                                 uint32_t *__restrict__ codes, int ih, int iw, int ph, int pw, int cp, int64_t total) {
    let_dependents_launch();
    dependency_wait();
    const int groups = cp / 8;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
         i += (int64_t)gridDim.x * blockDim.x) {
        const int g = (int)(i % groups);
        int64_t t = i / groups;
        const int px = (int)(t % pw);
        t /= pw;
        const int py = (int)(t % ph);
        const int64_t b = t / ph;
        uint32_t code;
        const uint4 o = pool_window(pre + ((b * ih + 2 * py) * (int64_t)iw + 2 * px) * cp + g * 8, (int64_t)iw * cp, cp, code);
        if (codes != nullptr) codes[i] = code;
        reinterpret_cast<uint4 *>(y)[i] = o;
    }
}

// CG channels of one image per CTA: their pooled values meet in shared memory as they lie in NCHW, one contiguous run.
// 256 x 29 x 29 x 128: 11 us to channels-last and 13 for the copy that followed, now both in the time of the first.
template <int CG>
__global__ void __launch_bounds__(256)
    relu_pool_nchw_kernel(const __nv_bfloat16 *__restrict__ pre, __nv_bfloat16 *__restrict__ y, uint32_t *__restrict__ codes,
                          int ih, int iw, int ph, int pw, int cp, FastDiv div_pw) {
    let_dependents_launch();
    dependency_wait();
    extern __shared__ __align__(16) unsigned short staged[];   // [CG][ph * pw]
    constexpr int G = CG / 8;
    const int windows = ph * pw, c0 = blockIdx.x * CG;
    const int64_t b = blockIdx.y;
    const __nv_bfloat16 *img = pre + b * ih * iw * (int64_t)cp + c0;
    uint32_t *code_row = codes != nullptr ? codes + (b * windows * cp + c0) / 8 : nullptr;
    for (int i = threadIdx.x; i < windows * G; i += 256) {
        const int g = i % G, win = i / G;
        uint32_t py, px, code;
        div_pw.divmod((uint32_t)win, py, px);
        const uint4 o = pool_window(img + ((int64_t)(2 * py) * iw + 2 * px) * cp + g * 8, (int64_t)iw * cp, cp, code);
        if (code_row != nullptr) code_row[(int64_t)win * (cp / 8) + g] = code;
        unsigned short *dst = staged + g * 8 * windows + win;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            dst[2 * j * windows] = (unsigned short)(&o.x)[j];
            dst[(2 * j + 1) * windows] = (unsigned short)((&o.x)[j] >> 16);
        }
    }
    __syncthreads();
    uint4 *out = reinterpret_cast<uint4 *>(y + (b * cp + c0) * (int64_t)windows);
    for (int i = threadIdx.x; i < windows * G; i += 256) out[i] = reinterpret_cast<const uint4 *>(staged)[i];
}

// The gradient at the four cells of a window's eight channels, from the pooled gradient's words: q is the first cell.
__device__ __forceinline__ void spread_window(const uint32_t (&gw)[4], uint32_t code, __nv_bfloat16 *q, int64_t row_pitch,
                                              int cp) {
    uint32_t w[4][4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        // 0 + dy: the gradient's bits but for a negative zero
        const uint32_t lo = (gw[j] & 0xffffu) == 0x8000u ? 0u : gw[j] & 0xffffu;
        const uint32_t hi = (gw[j] >> 16) == 0x8000u ? 0u : gw[j] & 0xffff0000u;
        const uint32_t cl = (code >> (8 * j)) & 15u, ch = (code >> (8 * j + 4)) & 15u;
#pragma unroll
        for (uint32_t c = 0; c < 4; ++c) w[c][j] = (cl == (c | 4u) ? lo : 0u) | (ch == (c | 4u) ? hi : 0u);
    }
#pragma unroll
    for (int c = 0; c < 4; ++c)
        *reinterpret_cast<uint4 *>(q + (c >> 1) * row_pitch + (c & 1) * cp) = make_uint4(w[c][0], w[c][1], w[c][2], w[c][3]);
}

// Cells no window covers keep the Relu's output.
__device__ __forceinline__ void keep_cells(const __nv_bfloat16 *p, int64_t row, bool has_r1, bool has_c1, __nv_bfloat16 *q,
                                           int64_t row_pitch, int cp) {
    Vec8 v[4], o[4];
    const uint4 zero = make_uint4(0, 0, 0, 0);
    v[0].raw = *reinterpret_cast<const uint4 *>(p);
    v[1].raw = has_c1 ? *reinterpret_cast<const uint4 *>(p + cp) : zero;
    v[2].raw = has_r1 ? *reinterpret_cast<const uint4 *>(p + row) : zero;
    v[3].raw = (has_r1 && has_c1) ? *reinterpret_cast<const uint4 *>(p + row + cp) : zero;
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float x0v = v[c].get(2 * j), x1v = v[c].get(2 * j + 1);
            o[c].set_pair(j, x0v >= 0.f ? x0v : 0.f, x1v >= 0.f ? x1v : 0.f);
        }
    *reinterpret_cast<uint4 *>(q) = o[0].raw;
    if (has_c1) *reinterpret_cast<uint4 *>(q + cp) = o[1].raw;
    if (has_r1) *reinterpret_cast<uint4 *>(q + row_pitch) = o[2].raw;
    if (has_r1 && has_c1) *reinterpret_cast<uint4 *>(q + row_pitch + cp) = o[3].raw;
}

// One thread per (image, window position of the grid that covers every cell, channel group).
__global__ void relu_pool_backward_kernel(const __nv_bfloat16 *__restrict__ pre, const uint32_t *__restrict__ codes,
                                          const __nv_bfloat16 *__restrict__ dy, __nv_bfloat16 *__restrict__ out,
                                          int ih, int iw, int ph, int pw, int cp, int64_t row_pitch,
                                          int64_t image_pitch, int64_t total) {
    let_dependents_launch(kAlwaysEarly);
    dependency_wait();
    const int groups = cp / 8;
    const int wh = (ih + 1) / 2, ww = (iw + 1) / 2;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
         i += (int64_t)gridDim.x * blockDim.x) {
        const int g = (int)(i % groups);
        int64_t t = i / groups;
        const int wx = (int)(t % ww);
        t /= ww;
        const int wy = (int)(t % wh);
        const int64_t b = t / wh;
        const int y0 = 2 * wy, x0 = 2 * wx;
        __nv_bfloat16 *q = out + b * image_pitch + y0 * row_pitch + (int64_t)x0 * cp + g * 8;
        if (wy < ph && wx < pw) {   // a whole window
            const int64_t at = ((b * ph + wy) * (int64_t)pw + wx) * groups + g;
            const uint32_t code = __ldg(codes + at);
            const uint4 gr = __ldg(reinterpret_cast<const uint4 *>(dy) + at);
            const uint32_t gw[4] = {gr.x, gr.y, gr.z, gr.w};
            spread_window(gw, code, q, row_pitch, cp);
        } else {
            keep_cells(pre + ((b * ih + y0) * (int64_t)iw + x0) * cp + g * 8, (int64_t)iw * cp, y0 + 1 < ih, x0 + 1 < iw, q,
                       row_pitch, cp);
        }
    }
}

// The same from an NCHW gradient, CG channels of one image per CTA, with the zero frame around the result.  256 x 29 x 29 x
// 128 with a frame of 2: 13 us for a channels-last copy, 9 for the frame and 17 for the gradient, now one pass.
template <int CG>
__global__ void __launch_bounds__(256)
    relu_pool_backward_nchw_kernel(const __nv_bfloat16 *__restrict__ pre, const uint32_t *__restrict__ codes,
                                   const __nv_bfloat16 *__restrict__ dy, __nv_bfloat16 *__restrict__ framed, int ih, int iw,
                                   int ph, int pw, int cp, int pad_h, int pad_w, FastDiv div_ww, FastDiv div_wp,
                                   FastDiv div_side) {
    let_dependents_launch(kAlwaysEarly);
    dependency_wait();
    extern __shared__ __align__(16) unsigned short staged[];   // [CG][ph * pw]
    constexpr int G = CG / 8;
    const int windows = ph * pw, c0 = blockIdx.x * CG;
    const int64_t b = blockIdx.y;
    const uint4 *src = reinterpret_cast<const uint4 *>(dy + (b * cp + c0) * (int64_t)windows);
    for (int i = threadIdx.x; i < windows * G; i += 256) reinterpret_cast<uint4 *>(staged)[i] = __ldg(src + i);
    const int hp = ih + 2 * pad_h, wp = iw + 2 * pad_w;
    __nv_bfloat16 *out = framed + b * hp * wp * (int64_t)cp + c0;
    // the frame: whole rows above and below, then the sides of the rows between
    const int band = pad_h * wp, frame = 2 * band + 2 * pad_w * ih;
    for (int i = threadIdx.x; i < frame * G; i += 256) {
        const int g = i % G, cell = i / G;
        uint32_t y, x;
        if (cell < 2 * band) {
            div_wp.divmod((uint32_t)cell, y, x);
            if ((int)y >= pad_h) y += ih;
        } else {
            div_side.divmod((uint32_t)(cell - 2 * band), y, x);
            y += pad_h;
            if ((int)x >= pad_w) x += iw;
        }
        *reinterpret_cast<uint4 *>(out + ((int64_t)y * wp + x) * cp + g * 8) = make_uint4(0, 0, 0, 0);
    }
    __syncthreads();
    out += ((int64_t)pad_h * wp + pad_w) * cp;
    const int64_t row_pitch = (int64_t)wp * cp;
    const int ww = (iw + 1) / 2, wh = (ih + 1) / 2;
    const uint32_t *code_row = codes + (b * windows * cp + c0) / 8;
    const __nv_bfloat16 *img = pre != nullptr ? pre + b * ih * iw * (int64_t)cp + c0 : nullptr;
    for (int i = threadIdx.x; i < wh * ww * G; i += 256) {
        const int g = i % G;
        uint32_t wy, wx;
        div_ww.divmod((uint32_t)(i / G), wy, wx);
        const int y0 = 2 * (int)wy, x0 = 2 * (int)wx;
        __nv_bfloat16 *q = out + y0 * row_pitch + (int64_t)x0 * cp + g * 8;
        if ((int)wy < ph && (int)wx < pw) {
            const int win = (int)wy * pw + (int)wx;
            const uint32_t code = __ldg(code_row + (int64_t)win * (cp / 8) + g);
            const unsigned short *v = staged + g * 8 * windows + win;
            uint32_t gw[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) gw[j] = v[2 * j * windows] | ((uint32_t)v[(2 * j + 1) * windows] << 16);
            spread_window(gw, code, q, row_pitch, cp);
        } else {
            keep_cells(img + ((int64_t)y0 * iw + x0) * cp + g * 8, (int64_t)iw * cp, y0 + 1 < ih, x0 + 1 < iw, q, row_pitch, cp);
        }
    }
}

__global__ void zero_frame_kernel(__nv_bfloat16 *framed, int hp, int wp, int pad_h, int pad_w, int cp,
                                  int64_t cells_per_image, int64_t total) {
    let_dependents_launch(kAlwaysEarly);
    dependency_wait();
    const int groups = cp / 8;
    const int64_t band = (int64_t)pad_h * wp;   // cells of the top (and of the bottom) rows
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
         i += (int64_t)gridDim.x * blockDim.x) {
        const int g = (int)(i % groups);
        int64_t t = i / groups;
        const int64_t cell = t % cells_per_image;
        const int64_t b = t / cells_per_image;
        int y, x;
        if (cell < band) {
            y = (int)(cell / wp);
            x = (int)(cell % wp);
        } else if (cell < 2 * band) {
            const int64_t r = cell - band;
            y = hp - pad_h + (int)(r / wp);
            x = (int)(r % wp);
        } else {
            const int64_t r = cell - 2 * band;
            y = pad_h + (int)(r / (2 * pad_w));
            const int k = (int)(r % (2 * pad_w));
            x = k < pad_w ? k : wp - 2 * pad_w + k;
        }
        *reinterpret_cast<uint4 *>(framed + ((b * hp + y) * (int64_t)wp + x) * cp + g * 8) =
            make_uint4(0, 0, 0, 0);
    }
}

inline unsigned grid_for(ag_device *dev, int64_t total) {
    const int64_t want = ceil_div(total, 256);
    const int64_t cap = (int64_t)dev->sm_count * 32;
    return (unsigned)(want < 1 ? 1 : (want > cap ? cap : want));
}

inline bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

}  // namespace

int im2col_channels(ag_device *dev, const __nv_bfloat16 *x, int64_t bs, int64_t ic, int64_t ih,
                    int64_t iw, int fh, int fw, int64_t oh, int64_t ow, int64_t cp,
                    __nv_bfloat16 *out) {
    AG_REQUIRE(cp % 8 == 0 && ic * fh * fw <= cp && aligned16(out), AG_ERR_INVALID,
               "im2col_channels: bad channel pitch or alignment");
    AG_REQUIRE(oh == ih - fh + 1 && ow == iw - fw + 1 && oh > 0 && ow > 0, AG_ERR_SHAPE,
               "im2col_channels: output shape does not match");
    const int64_t per_image = oh * ow * (cp / 8);
    AG_REQUIRE(per_image < (int64_t(1) << 31) && bs <= 65535 && ic * ih * iw < (int64_t(1) << 31), AG_ERR_LIMIT,
               "im2col_channels: image too large");
    AG_REQUIRE(256 % (cp / 8) == 0, AG_ERR_UNSUPPORTED, "im2col_channels: channel pitch must be 64, 128 or 256");
    if (bs == 0) return AG_OK;
    if ((fh == 3 && fw == 3 && launch_im2col_rows<3, 3>(dev, x, out, bs, ic, ih, iw, oh, ow, cp)) ||
        (fh == 5 && fw == 5 && launch_im2col_rows<5, 5>(dev, x, out, bs, ic, ih, iw, oh, ow, cp))) {
        AG_CHECK_LAUNCH();
        return AG_OK;
    }
    // eight pixels per thread, so that the offsets a thread computes up front are used eight times
    const int64_t want = ceil_div(per_image, 256 * 8);
    const dim3 grid((unsigned)(want > 4096 ? 4096 : want), (unsigned)bs);
    if (fh == 3 && fw == 3)
        im2col_channels_kernel<3, 3><<<grid, 256, 0, dev->stream>>>(
            x, out, (int)ic, (int)ih, (int)iw, fh, fw, (int)oh, (int)ow, (int)cp, (uint32_t)per_image);
    else if (fh == 5 && fw == 5)
        im2col_channels_kernel<5, 5><<<grid, 256, 0, dev->stream>>>(
            x, out, (int)ic, (int)ih, (int)iw, fh, fw, (int)oh, (int)ow, (int)cp, (uint32_t)per_image);
    else
        im2col_channels_kernel<0, 0><<<grid, 256, 0, dev->stream>>>(
            x, out, (int)ic, (int)ih, (int)iw, fh, fw, (int)oh, (int)ow, (int)cp, (uint32_t)per_image);
    AG_CHECK_LAUNCH();
    return AG_OK;
}

int relu_pool(ag_device *dev, const __nv_bfloat16 *pre, int64_t bs, int64_t ih, int64_t iw, int64_t cp,
              __nv_bfloat16 *y, uint32_t *codes) {
    AG_REQUIRE(cp % 8 == 0 && aligned16(pre) && aligned16(y), AG_ERR_INVALID,
               "relu_pool: bad channel pitch or alignment");
    AG_REQUIRE(ih >= 2 && iw >= 2, AG_ERR_SHAPE, "relu_pool: window larger than input");
    const int64_t ph = ih / 2, pw = iw / 2;
    const int64_t total = bs * ph * pw * (cp / 8);
    if (total == 0) return AG_OK;
    AG_TRY((launch_dependent(dev, relu_pool_kernel, dim3(grid_for(dev, total)), 256, 0, pre, y, codes, (int)ih, (int)iw,
                             (int)ph, (int)pw, (int)cp, total)));
    return AG_OK;
}

int relu_pool_backward(ag_device *dev, const __nv_bfloat16 *pre, const uint32_t *codes, const __nv_bfloat16 *dy, int64_t bs,
                       int64_t ih, int64_t iw, int64_t cp, __nv_bfloat16 *out, int64_t out_row_pitch,
                       int64_t out_image_pitch) {
    AG_REQUIRE(cp % 8 == 0 && out_row_pitch % 8 == 0 && out_image_pitch % 8 == 0 && aligned16(pre) &&
                   aligned16(dy) && aligned16(out),
               AG_ERR_INVALID, "relu_pool_backward: bad pitch or alignment");
    AG_REQUIRE(ih >= 2 && iw >= 2, AG_ERR_SHAPE, "relu_pool_backward: window larger than input");
    AG_REQUIRE(pre != nullptr || (ih % 2 == 0 && iw % 2 == 0), AG_ERR_INVALID, "relu_pool_backward: odd planes need pre");
    const int64_t total = bs * ((ih + 1) / 2) * ((iw + 1) / 2) * (cp / 8);
    if (total == 0) return AG_OK;
    AG_TRY((launch_dependent(dev, relu_pool_backward_kernel, dim3(grid_for(dev, total)), 256, 0, pre, codes, dy, out,
                             (int)ih, (int)iw, (int)(ih / 2), (int)(iw / 2), (int)cp, out_row_pitch, out_image_pitch,
                             total)));
    return AG_OK;
}

// 64 channels per CTA make whole lines of the channels-last side; 16, or 8, where that leaves SMs without a CTA.
static int channels_per_cta(ag_device *dev, int64_t bs, int64_t c) {
    return bs * (c / 64) >= 2 * dev->sm_count ? 64 : bs * (c / 16) >= dev->sm_count ? 16 : 8;
}

template <class K, class... A>
static int launch_nchw(ag_device *dev, K kernel, int cg, int64_t bs, int64_t c, int64_t windows, const A &...args) {
    const int smem = (int)(cg * windows * 2);
    if (cg == 64) {   // the others stay below 48 KB
        static SmemAllowed allowed;
        AG_TRY(allow_smem(dev, kernel, allowed));
    }
    return launch_dependent(dev, kernel, dim3((unsigned)(c / cg), (unsigned)bs), 256, (size_t)smem, args...);
}

int relu_pool_nchw(ag_device *dev, const __nv_bfloat16 *pre, int64_t bs, int64_t ih, int64_t iw, int64_t c, __nv_bfloat16 *y,
                   uint32_t *codes) {
    const int64_t ph = ih / 2, pw = iw / 2;
    AG_REQUIRE(c % 64 == 0 && aligned16(pre) && aligned16(y), AG_ERR_INVALID, "relu_pool_nchw: bad channels or alignment");
    AG_REQUIRE(ih >= 2 && iw >= 2 && ph * pw <= kMostWindows && bs <= 65535, AG_ERR_SHAPE, "relu_pool_nchw: bad plane");
    if (bs == 0) return AG_OK;
    const int cg = channels_per_cta(dev, bs, c);
    auto kernel = cg == 64 ? relu_pool_nchw_kernel<64> : cg == 16 ? relu_pool_nchw_kernel<16> : relu_pool_nchw_kernel<8>;
    return launch_nchw(dev, kernel, cg, bs, c, ph * pw, pre, y, codes, (int)ih, (int)iw, (int)ph, (int)pw, (int)c, FastDiv((uint32_t)pw));
}

int relu_pool_backward_nchw(ag_device *dev, const __nv_bfloat16 *pre, const uint32_t *codes, const __nv_bfloat16 *dy,
                            int64_t bs, int64_t ih, int64_t iw, int64_t c, int pad_h, int pad_w, __nv_bfloat16 *framed) {
    const int64_t ph = ih / 2, pw = iw / 2;
    AG_REQUIRE(c % 64 == 0 && aligned16(pre) && aligned16(dy) && aligned16(framed), AG_ERR_INVALID,
               "relu_pool_backward_nchw: bad channels or alignment");
    AG_REQUIRE(ih >= 2 && iw >= 2 && ph * pw <= kMostWindows && bs <= 65535, AG_ERR_SHAPE, "relu_pool_backward_nchw: bad plane");
    AG_REQUIRE(pre != nullptr || (ih % 2 == 0 && iw % 2 == 0), AG_ERR_INVALID, "relu_pool_backward_nchw: odd planes need pre");
    if (bs == 0) return AG_OK;
    const int cg = channels_per_cta(dev, bs, c);
    auto kernel = cg == 64 ? relu_pool_backward_nchw_kernel<64>
                : cg == 16 ? relu_pool_backward_nchw_kernel<16> : relu_pool_backward_nchw_kernel<8>;
    return launch_nchw(dev, kernel, cg, bs, c, ph * pw, pre, codes, dy, framed, (int)ih, (int)iw, (int)ph, (int)pw, (int)c, pad_h, pad_w,
                       FastDiv((uint32_t)((iw + 1) / 2)), FastDiv((uint32_t)(iw + 2 * pad_w)),
                       FastDiv((uint32_t)(pad_w > 0 ? 2 * pad_w : 1)));
}

int zero_frame(ag_device *dev, __nv_bfloat16 *framed, int64_t bs, int64_t hp, int64_t wp, int pad_h,
               int pad_w, int64_t cp) {
    AG_REQUIRE(cp % 8 == 0 && aligned16(framed), AG_ERR_INVALID, "zero_frame: bad pitch or alignment");
    const int64_t cells = 2 * (int64_t)pad_h * wp + 2 * (int64_t)pad_w * (hp - 2 * pad_h);
    const int64_t total = bs * cells * (cp / 8);
    if (total <= 0) return AG_OK;
    AG_TRY((launch_dependent(dev, zero_frame_kernel, dim3(grid_for(dev, total)), 256, 0, framed, (int)hp, (int)wp,
                             pad_h, pad_w, (int)cp, cells, total)));
    return AG_OK;
}

}  // namespace nhwc
}  // namespace ag
