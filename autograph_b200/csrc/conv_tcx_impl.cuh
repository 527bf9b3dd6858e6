// Convolutions on the gathered-operand tensor-core engine, for one element type.
#pragma once

#include "gemm_tcx_impl.cuh"

namespace ag {
namespace tcx {

static ConvMap conv_map(int64_t channels, int64_t sh, int64_t sw, int64_t gh, int64_t gw,
                        const ag_conv2_options *o, bool gradient) {
    ConvMap g;
    g.channels = (int)channels;
    g.sh = (int)sh; g.sw = (int)sw;
    g.gw = (int)gw; g.ghw = (int)(gh * gw);
    g.fh = o->filter[0]; g.fw = o->filter[1];
    g.ff = g.fh * g.fw;
    g.st_h = o->stride[0]; g.st_w = o->stride[1];
    g.pad_h = o->padding[0]; g.pad_w = o->padding[1];
    g.dil_h = o->dilation[0]; g.dil_w = o->dilation[1];
    g.gradient = gradient;
    g.always_valid = !gradient && g.pad_h == 0 && g.pad_w == 0;  // gh, gw come from the output rule
    g.ranges = (g.dil_h == 1 || g.fh == 1) && (g.dil_w == 1 || g.fw == 1) && (!gradient || (g.st_h == 1 && g.st_w == 1));
    g.row_ones = 0;
    for (int fi = 0; fi < g.fh; ++fi) g.row_ones |= 1u << (fi * g.fw & 31);
    g.div_ghw = FastDiv((uint32_t)g.ghw);
    g.div_gw = FastDiv((uint32_t)g.gw);
    g.div_fw = FastDiv((uint32_t)g.fw);
    g.div_st_h = FastDiv((uint32_t)g.st_h);
    g.div_st_w = FastDiv((uint32_t)g.st_w);
    g.cp = (g.channels + 7) / 8 * 8;
    g.div_cp = FastDiv((uint32_t)g.cp);
    return g;
}

// A filter bank in the order of ConvRows' k: out[row][tap * cp + c] = w[row * s_row + c * s_c + tap],
// zero for the padding channels.  Without it every 64-k step of every tile would fetch filters at a
// stride of the tap count, one sector per element.
template <class T>
__global__ void repack_kernel(const T *w, T *out, int total, int channels, int cp, int s_row, int s_c,
                              FastDiv div_k, FastDiv div_cp) {
    let_dependents_launch();
    dependency_wait();
    const uint32_t i = blockIdx.x * 256u + threadIdx.x;
    if (i >= (uint32_t)total) return;
    uint32_t row, k, tap, c;
    div_k.divmod(i, row, k);
    div_cp.divmod(k, tap, c);
    out[i] = (int)c < channels ? w[(int)row * s_row + (int)c * s_c + (int)tap] : from_f32<T>(0.f);
}

// A product with the patch matrix of `map` (rows = positions, k = taps x channels) and the filter
// bank w[row * s_row + channel * s_c + tap].
template <class T>
static int patches_times_filters(ag_device *dev, const T *src, const ConvMap &map, int M, const T *w, int N,
                                 int s_row, int s_c, const NchwOut<T> &E) {
    const int K = map.ff * map.cp, total = N * K;
    // One wave of tiles and up to 18 k steps of an input gradient, whose neighbouring rows are neighbouring
    // filters: read in place at the copy's device time, without its launch (forward, 5 x 64 x 22 x 22 -> 128:
    // 27 us in place, 19 copied; input gradient 21.7 and 21.5; 50 steps of 128 channels 5x5 190 and 87).
    // So are they where there is no room for the copy.
    void *ws = nullptr;
    if ((s_row < s_c && K <= 18 * BK && ceil_div(M, BM) * ceil_div(N, 64) <= dev->sm_count) ||
        staging(dev, (size_t)total * sizeof(T), &ws) != AG_OK)
        return gemm<T>(dev, M, N, K, ConvRows<T>{src, map, M}, FilterRows<T>{w, s_row, s_c, map.channels, map.div_cp}, E);
    T *packed = (T *)ws;
    AG_TRY((launch_dependent(dev, repack_kernel<T>, dim3((unsigned)ceil_div(total, 256)), 256, 0, w, packed, total,
                             map.channels, map.cp, s_row, s_c, FastDiv((uint32_t)K), map.div_cp)));
    return gemm<T>(dev, M, N, K, ConvRows<T>{src, map, M}, strided<kVecK>((const T *)packed, K, 1, N), E);
}

// Whether a convolution's patches are better indexed by (channel, tap) than by (tap, channel padded to
// eight): the padding costs more than the table look-ups (6 channels: 8 / 6 of 4 instructions
// per element against 6).  The table packs an offset of at most 26 bits and a sign with the tap; a tap that
// meets the image from far into the padding is at an offset beyond the channel's plane.
static bool few_channels(const ConvMap &g) {
    const int64_t furthest = (int64_t)g.channels * g.sh * g.sw + (int64_t)(g.fh - 1) * g.dil_h * g.sw + (int64_t)(g.fw - 1) * g.dil_w;
    return g.cp * 10 > g.channels * 14 && g.channels * g.ff <= kFewPatch && furthest < (1 << 26);
}

template <class T>
int conv_forward(ag_device *dev, const T *x, int64_t bs, int64_t ic, int64_t ih, int64_t iw,
                 const T *w, int64_t oc, const T *bias, const ag_conv2_options *o, int64_t oh,
                 int64_t ow, bool relu, T *y) {
    const int M = (int)(bs * oh * ow), N = (int)oc, ff = o->filter[0] * o->filter[1];
    NchwOut<T> E{y, bias, N, (int)(oh * ow), FastDiv((uint32_t)(oh * ow)), relu};
    const ConvMap map = conv_map(ic, ih, iw, oh, ow, o, false);
    if (few_channels(map)) {
        const int patch = (int)ic * ff;
        return gemm<T>(dev, M, N, patch, FewRows<T>{x, map, M, patch}, strided<kByRow>(w, patch, 1, N), E);
    }
    return patches_times_filters<T>(dev, x, map, M, w, N, (int)ic * ff, ff, E);
}

constexpr int64_t kTapSums = 1ll << 28;   // f32 values

// dx from the products with every tap: col[c * ff + tap][position of dy] -> dx[b][c][y][x].
template <class T>
__global__ void __launch_bounds__(256)
    taps_to_image_kernel(const float *col, T *dx, ConvMap g, int grid_hw, int64_t positions,
                         int total, FastDiv div_hw, FastDiv div_w, FastDiv div_c) {
    let_dependents_launch();
    dependency_wait();
    const uint32_t i = blockIdx.x * 256u + threadIdx.x;
    if (i >= (uint32_t)total) return;
    uint32_t plane, r, y, x, b, c;
    div_hw.divmod(i, plane, r);
    div_w.divmod(r, y, x);
    div_c.divmod(plane, b, c);
    const float *q = col + (int64_t)c * g.ff * positions + (int64_t)b * grid_hw;
    float s = 0.f;
    for (int fi = 0; fi < g.fh; ++fi) {
        const int ty = (int)y + g.pad_h - fi * g.dil_h;
        uint32_t oy, ry;
        g.div_st_h.divmod((uint32_t)max(ty, 0), oy, ry);
        if (ty < 0 || ry != 0 || oy >= (uint32_t)g.sh) continue;
        for (int fj = 0; fj < g.fw; ++fj) {
            const int tx = (int)x + g.pad_w - fj * g.dil_w;
            uint32_t ox, rx;
            g.div_st_w.divmod((uint32_t)max(tx, 0), ox, rx);
            if (tx < 0 || rx != 0 || ox >= (uint32_t)g.sw) continue;
            s += q[(int64_t)(fi * g.fw + fj) * positions + oy * g.sw + ox];
        }
    }
    dx[i] = from_f32<T>(s);
}

template <class T>
int conv_backward_input(ag_device *dev, const T *w, int64_t oc, int64_t ic, const T *dy, int64_t bs,
                        int64_t ih, int64_t iw, const ag_conv2_options *o, int64_t oh, int64_t ow,
                        T *dx) {
    const int ff = o->filter[0] * o->filter[1];
    const int M = (int)(bs * ih * iw), N = (int)ic;
    const ConvMap map = conv_map(oc, oh, ow, ih, iw, o, true);
    // With few input channels a tile of the patch form is mostly empty columns, and it gathers dy
    // once per tap.  The other order multiplies dy by the filters of every (channel, tap) and adds
    // the taps afterwards, in f32.  Compared by the time of one 128-position tile on an SM: 1.7 us per
    // 64-k step, 34 bytes per ns for the taps' trip through memory (6 channels from 128, 3x3, 132 x 40
    // x 40 f32: 277 us by patches, 92 us by taps).  Beyond 128 (channel, tap) pairs the taps no longer
    // fit L2 at the batch sizes that matter (32 channels from 128, 121 x 27 x 27: 127 and 185 us).
    const int taps_n = N * ff;
    const double by_patches = 1.7 * (double)ceil_div((int64_t)ff * map.cp, 64);
    const double by_taps = 1.7 * (double)(ceil_div(oc, 64) * ceil_div(taps_n, 128)) + 0.03 * taps_n;
    // As many images at a time as have 1 GiB of sums per tap; without room for those, by patches.
    const int64_t image = oh * ow * taps_n, at_once = image < kTapSums ? kTapSums / image : 1;
    const int64_t images = at_once < bs ? at_once : bs;
    void *ws = nullptr;
    if (taps_n <= 128 && 1.3 * by_taps < by_patches && image < (1ll << 31) &&
        staging(dev, sizeof(float) * (size_t)(images * image), &ws) == AG_OK) {
        float *col = (float *)ws;
        ag_conv2_options point = {{1, 1}, {0, 0}, {1, 1}, {1, 1}};
        for (int64_t b = 0; b < bs; b += images) {
            const int64_t n = images < bs - b ? images : bs - b, positions = n * oh * ow;
            AG_TRY(gemm<T>(dev, (int)positions, taps_n, (int)oc,
                           ConvRows<T>{dy + b * oc * oh * ow, conv_map(oc, oh, ow, oh, ow, &point, false), (int)positions},
                           strided<kByRow>(w, 1, taps_n, taps_n), StridedOut<float>{col, 1, positions, 1.f, 0.f}));
            const int total = (int)(n * ic * ih * iw);
            AG_TRY((launch_dependent(dev, taps_to_image_kernel<T>, dim3((unsigned)ceil_div(total, 256)), 256, 0, col,
                                     dx + b * ic * ih * iw, map, (int)(oh * ow), positions, total,
                                     FastDiv((uint32_t)(ih * iw)), FastDiv((uint32_t)iw), FastDiv((uint32_t)ic))));
        }
        return AG_OK;
    }
    NchwOut<T> E{dx, nullptr, N, (int)(ih * iw), FastDiv((uint32_t)(ih * iw)), false};
    return patches_times_filters<T>(dev, dy, map, M, w, N, ff, (int)ic * ff, E);
}

template <class T>
int conv_backward_weight(ag_device *dev, const T *x, int64_t bs, int64_t ic, int64_t ih, int64_t iw,
                         const T *dy, int64_t oc, const ag_conv2_options *o, int64_t oh, int64_t ow,
                         float beta, T *dw) {
    const ConvMap map = conv_map(ic, ih, iw, oh, ow, o, false);
    const int N = (int)oc, K = (int)(bs * oh * ow), hw = (int)(oh * ow);
    if (few_channels(map)) {
        const int patch = (int)ic * map.ff;
        return gemm<T>(dev, patch, N, K, FewCols<T>{{x, map, 0, patch}}, ChannelRows<T>{dy, N, hw, FastDiv((uint32_t)hw)},
                       StridedOut<T>{dw, 1, patch, 1.f, beta});
    }
    const int M = map.ff * map.cp;
    return gemm<T>(dev, M, N, K, ConvCols<T>{x, map, M}, ChannelRows<T>{dy, N, hw, FastDiv((uint32_t)hw)},
                   FilterOut<T>{dw, map.channels, map.ff, map.div_cp, map.cp, beta});
}

}  // namespace tcx
}  // namespace ag
