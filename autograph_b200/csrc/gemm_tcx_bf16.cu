// bf16 products that TMA cannot feed, on the gathered-operand tensor-core engine.
#include "gemm_tcx_impl.cuh"

namespace ag {
namespace tcx {

template int gemm_strided<__nv_bfloat16>(ag_device *, int, int, int, float, const __nv_bfloat16 *, int64_t,
                                         int64_t, const __nv_bfloat16 *, int64_t, int64_t, float,
                                         __nv_bfloat16 *, int64_t, int64_t);
template int dense<__nv_bfloat16>(ag_device *, const __nv_bfloat16 *, int, int, const __nv_bfloat16 *, int,
                                  const __nv_bfloat16 *, bool, __nv_bfloat16 *);

}  // namespace tcx
}  // namespace ag
