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
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i >= total) return;
    uint32_t row, k, tap, c;
    div_k.divmod((uint32_t)i, row, k);
    div_cp.divmod(k, tap, c);
    out[i] = (int)c < channels ? w[(int)row * s_row + (int)c * s_c + (int)tap] : from_f32<T>(0.f);
}

// A product with the patch matrix of `map` (rows = positions, k = taps x channels) and the filter
// bank w[row * s_row + channel * s_c + tap].
template <class T>
static int patches_times_filters(ag_device *dev, const T *src, const ConvMap &map, int M, const T *w, int N,
                                 int s_row, int s_c, const NchwOut<T> &E) {
    const int K = map.ff * map.cp, total = N * K;
    void *ws = nullptr;
    AG_TRY(staging(dev, (size_t)total * sizeof(T), &ws));
    T *packed = (T *)ws;
    repack_kernel<T><<<(unsigned)ceil_div(total, 256), 256, 0, dev->stream>>>(
        w, packed, total, map.channels, map.cp, s_row, s_c, FastDiv((uint32_t)K), map.div_cp);
    AG_CHECK_LAUNCH();
    return gemm<T>(dev, M, N, K, ConvRows<T>{src, map, M}, strided<kVecK>((const T *)packed, K, 1, N), E);
}

template <class T>
int conv_forward(ag_device *dev, const T *x, int64_t bs, int64_t ic, int64_t ih, int64_t iw,
                 const T *w, int64_t oc, const T *bias, const ag_conv2_options *o, int64_t oh,
                 int64_t ow, bool relu, T *y) {
    const int M = (int)(bs * oh * ow), N = (int)oc, ff = o->filter[0] * o->filter[1];
    NchwOut<T> E{y, bias, N, (int)(oh * ow), FastDiv((uint32_t)(oh * ow)), relu};
    return patches_times_filters<T>(dev, x, conv_map(ic, ih, iw, oh, ow, o, false), M, w, N, (int)ic * ff, ff, E);
}

template <class T>
int conv_backward_input(ag_device *dev, const T *w, int64_t oc, int64_t ic, const T *dy, int64_t bs,
                        int64_t ih, int64_t iw, const ag_conv2_options *o, int64_t oh, int64_t ow,
                        T *dx) {
    const int ff = o->filter[0] * o->filter[1];
    const int M = (int)(bs * ih * iw), N = (int)ic;
    NchwOut<T> E{dx, nullptr, N, (int)(ih * iw), FastDiv((uint32_t)(ih * iw)), false};
    return patches_times_filters<T>(dev, dy, conv_map(oc, oh, ow, ih, iw, o, true), M, w, N, ff, (int)ic * ff, E);
}

template <class T>
int conv_backward_weight(ag_device *dev, const T *x, int64_t bs, int64_t ic, int64_t ih, int64_t iw,
                         const T *dy, int64_t oc, const ag_conv2_options *o, int64_t oh, int64_t ow,
                         float beta, T *dw) {
    const ConvMap map = conv_map(ic, ih, iw, oh, ow, o, false);
    const int M = map.ff * map.cp, N = (int)oc, K = (int)(bs * oh * ow), hw = (int)(oh * ow);
    return gemm<T>(dev, M, N, K, ConvCols<T>{x, map, M}, ChannelRows<T>{dy, N, hw, FastDiv((uint32_t)hw)},
                   FilterOut<T>{dw, map.channels, map.ff, map.div_cp, map.cp, beta});
}

}  // namespace tcx
}  // namespace ag
