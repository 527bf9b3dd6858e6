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

// channels x taps and columns of the product, its depth.  Few channels are padded to eight and few
// columns to 32: 1 -> 16 5x5 forward 42 us here and 16 us on the SIMT engine, 3 -> 16 3x3 20 and 10,
// 3 -> 64 28 and 28, 16 -> 16 (8 x 12 x 12) 11 and 21.
bool conv_worth(ag_dtype dtype, int64_t patch, int64_t cols, int64_t positions, const ag_conv2_options *o) {
    (void)dtype;
    return enabled() && o->filter[0] * o->filter[1] <= 32 && patch * cols >= 1024 &&
           positions * patch * cols >= 2000000;
}

// The input gradient, whose engine has a form for few columns (1 <- 16 5x5: 177 us on the SIMT engine).
bool conv_input_worth(int64_t patch, int64_t cols, int64_t positions, const ag_conv2_options *o) {
    return enabled() && o->filter[0] * o->filter[1] <= 32 && patch * cols >= 140 &&
           positions * patch * cols >= 2000000;
}

// The weight gradient: 3 -> 16 3x3 f32 24 us here and 27, 1 -> 16 5x5 52 and 40 (bf16 38 and 60); small
// ones (2.7e6 multiply-adds) 11 and 10.
bool conv_weight_worth(ag_dtype dtype, int64_t patch, int64_t oc, int64_t positions, const ag_conv2_options *o) {
    if (!enabled() || o->filter[0] * o->filter[1] > 32) return false;
    const int64_t macs = positions * patch * oc;
    return dtype == AG_F32 ? patch * oc >= 420 && macs >= 4000000 : patch * oc >= 128 && macs >= 2000000;
}

template int gemm_strided<float>(ag_device *, int, int, int, float, const float *, int64_t, int64_t,
                                 const float *, int64_t, int64_t, float, float *, int64_t, int64_t);
template int dense<float>(ag_device *, const float *, int, int, const float *, int, const float *, bool,
                          float *);

}  // namespace tcx
}  // namespace ag
