// f32 products on the gathered-operand tensor-core engine, and the rules that say which
// products the two tensor-core engines for such operands take.
#include <cstdlib>

#include "gemm_tcx_impl.cuh"

namespace ag {
namespace tcx {

static bool enabled() {
    static const bool v = []() {
        const char *e = getenv("AG_TCX");
        return !(e && e[0] == '0');
    }();
    return v;
}

// Against the SIMT engine (B200, device time): f32 390 x 145 x 135 13 us here and 8 us there,
// 300 x 100 x 2000 9.7 and 10.8, 602 x 861 x 163 13 and 32, 1024^3 34 and 83; bf16
// 100 x 256 x 128 8 and 8, 390 x 145 x 135 9 and 18.  A call here costs about 9 us in f32 (slices of
// k, two kernels) whatever the size, so the line is drawn at the multiply-adds the SIMT kernels do
// in that time.
bool gemm_worth(ag_dtype dtype, int64_t m, int64_t k, int64_t n) {
    if (!enabled() || m < 16 || n < 16 || k < 32) return false;
    return (double)m * (double)n * (double)k >= (dtype == AG_F32 ? 3e7 : 4e6);
}

// Against the gathered engine: 1000 x 5000 x 130 f32 33 us packed and 48 us gathered, 1024^3 29 and
// 34 (tn 48), 777 x 1009 x 333 21 and 24, 150 x 8000 x 200 (2.4e8 multiply-adds) 23 and 18.  The
// copy pass and its launch are what a small product cannot amortise.
bool packed_worth(int64_t m, int64_t k, int64_t n) {
    return m >= 128 && n >= 128 && k >= 64 && (double)m * (double)n * (double)k >= 2.5e8;
}

bool conv_worth(ag_dtype dtype, int64_t rows, int64_t cols, int64_t k, const ag_conv2_options *o) {
    (void)dtype;
    return enabled() && o->filter[0] * o->filter[1] <= 32 && rows >= 16 && cols >= 4 && k >= 16;
}

template int gemm_strided<float>(ag_device *, int, int, int, float, const float *, int64_t, int64_t,
                                 const float *, int64_t, int64_t, float, float *, int64_t, int64_t);
template int dense<float>(ag_device *, const float *, int, int, const float *, int, const float *, bool,
                          float *);

}  // namespace tcx
}  // namespace ag
