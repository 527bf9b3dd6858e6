// f32 convolutions on the gathered-operand tensor-core engine.
#include "conv_tcx_impl.cuh"

namespace ag {
namespace tcx {

template int conv_forward<float>(ag_device *, const float *, int64_t, int64_t, int64_t, int64_t, const float *,
                              int64_t, const float *, const ag_conv2_options *, int64_t, int64_t, bool, float *);
template int conv_backward_input<float>(ag_device *, const float *, int64_t, int64_t, const float *, int64_t,
                                     int64_t, int64_t, const ag_conv2_options *, int64_t, int64_t, float *);
template int conv_backward_weight<float>(ag_device *, const float *, int64_t, int64_t, int64_t, int64_t,
                                      const float *, int64_t, const ag_conv2_options *, int64_t, int64_t,
                                      float, float *);

// Against the direct kernels (no padding), us there and here, images x channels x side -> columns: input gradients 484 x 24 x 14 -> 16
// 5 x 5 92 and 38, 213 x 24 x 18 -> 16 3 x 3 26 and 13, 478 x 16 x 10 -> 16 5 x 5 36 and 21, but into few channels, which are padded
// to 16 columns, 1000 x 6 x 12 -> 16 5 x 5 26 and 47, 802 x 6 x 18 -> 8 3 x 3 15 and 26.
bool input_by_rows(ag_device *dev, ag_dtype dtype, int64_t oc, int64_t ic, int64_t bs, int64_t ih, int64_t iw,
                   const ag_conv2_options *o, int64_t oh, int64_t ow) {
    return dtype == AG_F32 && plain(o) && ic >= 12 && conv_input_worth(oc * o->filter[0] * o->filter[1], ic, bs * ih * iw, o) &&
           bs * oc * oh * ow < (1ll << 31) && halo32::takes(dev, input_rows(nullptr, oc, ic, nullptr, bs, ih, iw, o, oh, ow));
}
// Weight gradients 678 x 32 x 30 -> 16 3 x 3 315 and 92, 802 x 16 x 38 -> 8 5 x 5 676 and 154, 107 x 32 x 20 -> 6 3 x 3 50 and 14, 24 x
// 12 x 37 -> 8 5 x 5 25 and 13; few channels are mostly padding (1000 x 1 x 28 -> 6 5 x 5 27 and 104, 553 x 12 x 37 -> 4 5 x 5 70 and
// 102), few channels of a small image fit the direct kernel well (802 x 6 x 18 -> 8 3 x 3 29 and 33, 808 x 8 x 19 -> 20 5 x 5 76 and
// 85).  Its sums are chains of FFMAs: errors against float64 2e-7 to 9e-7 there, 0.8e-7 to 1.3e-7 here.
bool weight_by_rows(ag_dtype dtype, int64_t bs, int64_t ic, int64_t ih, int64_t iw, int64_t oc, const ag_conv2_options *o,
                    int64_t oh, int64_t ow) {
    return dtype == AG_F32 && plain(o) && oc >= 6 && ic * oc >= 64 && (ic >= 12 || ih * iw >= 400) &&
           conv_weight_worth(dtype, ic * o->filter[0] * o->filter[1], oc, bs * oh * ow, o) && bs * oc * oh * ow < (1ll << 31) &&
           halo32::takes_wgrad(weight_rows(nullptr, bs, ic, ih, iw, nullptr, oc, o, oh, ow));
}

}  // namespace tcx
}  // namespace ag
