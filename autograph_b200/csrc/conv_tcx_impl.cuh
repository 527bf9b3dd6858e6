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
    g.div_ff = FastDiv((uint32_t)g.ff);
    g.div_fw = FastDiv((uint32_t)g.fw);
    g.div_st_h = FastDiv((uint32_t)g.st_h);
    g.div_st_w = FastDiv((uint32_t)g.st_w);
    return g;
}

template <class T>
int conv_forward(ag_device *dev, const T *x, int64_t bs, int64_t ic, int64_t ih, int64_t iw,
                 const T *w, int64_t oc, const T *bias, const ag_conv2_options *o, int64_t oh,
                 int64_t ow, bool relu, T *y) {
    const int M = (int)(bs * oh * ow), N = (int)oc, K = (int)(ic * o->filter[0] * o->filter[1]);
    ConvRows<T> A{x, conv_map(ic, ih, iw, oh, ow, o, false), M};
    NchwOut<T> E{y, bias, N, (int)(oh * ow), FastDiv((uint32_t)(oh * ow)), relu};
    return gemm<T>(dev, M, N, K, A, strided<T, false>(w, K, 1, N), E);
}

template <class T>
int conv_backward_input(ag_device *dev, const T *w, int64_t oc, int64_t ic, const T *dy, int64_t bs,
                        int64_t ih, int64_t iw, const ag_conv2_options *o, int64_t oh, int64_t ow,
                        T *dx) {
    const int ff = o->filter[0] * o->filter[1];
    const int M = (int)(bs * ih * iw), N = (int)ic, K = (int)(oc * ff);
    ConvRows<T> A{dy, conv_map(oc, oh, ow, ih, iw, o, true), M};
    WeightRows<T> B{w, N, ff, FastDiv((uint32_t)ff)};
    NchwOut<T> E{dx, nullptr, N, (int)(ih * iw), FastDiv((uint32_t)(ih * iw)), false};
    return gemm<T>(dev, M, N, K, A, B, E);
}

template <class T>
int conv_backward_weight(ag_device *dev, const T *x, int64_t bs, int64_t ic, int64_t ih, int64_t iw,
                         const T *dy, int64_t oc, const ag_conv2_options *o, int64_t oh, int64_t ow,
                         float beta, T *dw) {
    // rows = (input channel, tap), the contiguous index of dw [oc][ic * ff]
    const int M = (int)(ic * o->filter[0] * o->filter[1]), N = (int)oc, K = (int)(bs * oh * ow);
    const int hw = (int)(oh * ow);
    ConvCols<T> A{x, conv_map(ic, ih, iw, oh, ow, o, false), M};
    ChannelRows<T> B{dy, N, hw, FastDiv((uint32_t)hw),
                     hw % 8 == 0 && (reinterpret_cast<uintptr_t>(dy) & 15) == 0};
    return gemm<T>(dev, M, N, K, A, B, StridedOut<T>{dw, 1, M, 1.f, beta});
}

}  // namespace tcx
}  // namespace ag
