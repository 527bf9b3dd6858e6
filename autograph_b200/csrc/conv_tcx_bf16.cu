// bf16 convolutions on the gathered-operand tensor-core engine.
#include "conv_tcx_impl.cuh"

namespace ag {
namespace tcx {

template int conv_forward<__nv_bfloat16>(ag_device *, const __nv_bfloat16 *, int64_t, int64_t, int64_t, int64_t, const __nv_bfloat16 *,
                              int64_t, const __nv_bfloat16 *, const ag_conv2_options *, int64_t, int64_t, bool, __nv_bfloat16 *);
template int conv_backward_input<__nv_bfloat16>(ag_device *, const __nv_bfloat16 *, int64_t, int64_t, const __nv_bfloat16 *, int64_t,
                                     int64_t, int64_t, const ag_conv2_options *, int64_t, int64_t, __nv_bfloat16 *);
template int conv_backward_weight<__nv_bfloat16>(ag_device *, const __nv_bfloat16 *, int64_t, int64_t, int64_t, int64_t,
                                      const __nv_bfloat16 *, int64_t, const ag_conv2_options *, int64_t, int64_t,
                                      float, __nv_bfloat16 *);

}  // namespace tcx
}  // namespace ag
