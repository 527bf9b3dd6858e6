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

}  // namespace tcx
}  // namespace ag
