// f32 products on the gathered-operand tensor-core engine, and the rules that say which
// products the two tensor-core engines for such operands take.
#include <cstdlib>

#include "gemm_tcx_impl.cuh"

namespace ag {
namespace tcx {

// The slices' ends are ints and round k up.
constexpr int64_t kMostK = 1ll << 30;

static bool enabled() {
    static const bool v = []() {
        const char *e = getenv("AG_TCX");
        return !(e && e[0] == '0');
    }();
    return v;
}

// Against the SIMT engine, m x k x n, us here and there (row-major operands back to back): f32 464 x 16 x 416 7.7 and
// 5.2, 112 x 64 x 2528 7.0 and 6.3, 928 x 2336 x 16 14.0 and 16.5, 300 x 100 x 2000 8.0 and 12.4, 602 x 861 x 163 11.7 and
// 37, 1024^3 34 and 83; bf16 672 x 112 x 96 6.3 and 6.4, 96 x 3120 x 48 7.7 and 16.8, 208 x 624 x 96 7.2 and 14.7.  A
// short k is one launch here, and both engines take 5 to 8 us up to some 1e7 multiply-adds, most of it the launch: the
// lines lie where the SIMT kernels begin to take longer.
// Few rows: 1 to 8 x 25088 x 512 18 us and 68 (bf16 13 and 97), 12 x 100 x 20000 9 and 27.  Few columns: 20000 x 200 x
// 12 25 and 14, 5000 x 2000 x 12 51 and 98.  k below a tile's step: 25088 x 24 x 512 39 and 27,
// f32 1264 x 32 x 4896 22 and 17, 892 x 39 x 7961 24 and 25.
// Beyond k = 128, where the SIMT kernels have no form that stages all of k at once, slices of k win much earlier: f32 16 x
// 1056 x 1088 12.5 and 8.7, 32 x 800 x 64 10.2 and 8.4; bf16 88 x 211 x 97 23 and 8.3, 16 x 496 x 144 17 and 8.3.
bool gemm_worth(ag_dtype dtype, int64_t m, int64_t k, int64_t n) {
    if (!enabled() || k >= kMostK || k < (dtype == AG_F32 ? 40 : 32)) return false;
    const double macs = (double)m * (double)n * (double)k;
    if (m < 16 || n < 16) return macs >= 1e7 && k >= (n < 16 ? 1024 : 64);
    if (k > 128) return macs >= (dtype == AG_F32 ? 2e6 : 3e5);
    return macs >= (dtype == AG_F32 ? 3e7 : 4e6);
}

// Against the gathered engine, m x k x n, us packed and gathered: f32 940 x 589 x 1039 28 and 21, 2401 x 352 x 875 30 and
// 21, 1037 x 438 x 1885 33 and 27, 1584 x 902 x 444 26 and 29, 607 x 1199 x 1072 28 and 37, 391 x 843 x 2387 32 and 45, 808
// x 3023 x 420 31 and 47; bf16 873 x 969 x 1119 22 and 17, 215 x 4559 x 725 21 and 17, 535 x 1481 x 1347 20 and 24, 3821 x
// 2459 x 153 25 and 35.  The copy pass wants some 5e8 multiply-adds, counted by how much of its 256 x 256 tiles the output
// fills (528 columns are 69 % of three tiles), and more of them when k is short, because a tile is then mostly its
// epilogue; bf16, whose gathered tiles take half the time, wants more.  Over 90 drawn products of 1e8 to 3e9 multiply-adds
// these lines are 1.0 % (f32) and 0.7 % (bf16) above always taking the faster engine; 873 x 969 x 1119 is on the wrong side
// of both.
bool packed_worth(ag_dtype dtype, int64_t m, int64_t k, int64_t n) {
    const double fill = ((double)m / (256.0 * ceil_div(m, 256))) * ((double)n / (256.0 * ceil_div(n, 256)));
    const double macs = (double)m * (double)n * (double)k * fill;
    const bool f32 = dtype == AG_F32;
    return m >= 128 && n >= 128 && k >= 64 && macs >= (f32 ? 4.5e8 : 6e8) && macs * (double)k >= (f32 ? 3e11 : 8e11);
}

// The filters are also counted with their channels padded to eight, in an int (repack_kernel).
static bool filters_fit(int64_t patch, int64_t cols, int64_t taps) { return (patch + 7 * taps) * cols < (1ll << 31); }

// patch = channels x taps.  Against the SIMT engine, us here and there (f32 unless said):
//   1024 and more: here.  Below, by what the SIMT tiles are good at:
//   96 columns x 9 (203 x 41 x 41 / 2): 35 and 31, bf16 35 and 52;  32 x 9 (254 x 55 x 55): 124 and 148;
//   32 x 25 (64 x 24 x 24): 10 and 16;  6 x 144 (8 x 40 x 40): 9.4 and 32, bf16 8.3 and 46;
//   16 x 27 (233 x 48 x 48): 77 and 59;  6 x 9 (116 x 35 x 35): 20 and 8;
//   1.8e6 multiply-adds (32 x 27, 21 x 10 x 10): 7 and 4.
bool conv_worth(ag_dtype dtype, int64_t patch, int64_t cols, int64_t positions, const ag_conv2_options *o) {
    const int64_t taps = (int64_t)o->filter[0] * o->filter[1];
    if (!enabled() || taps > 32 || !filters_fit(patch, cols, taps)) return false;
    const int64_t macs = positions * patch * cols;
    if (patch * cols >= 1024) return macs >= 2000000;
    if (macs < 3000000) return false;
    if (dtype == AG_F32) return cols < 32 ? patch >= 96 : cols <= 64 && patch * cols >= 256;
    return cols < 32 ? patch >= 64 : patch * cols >= 256;
}

// The input gradient, whose engine has a form for few columns (SIMT engine: 1 <- 16 5x5 177 us, 3 <- 32 3x3 on
// 21 x 10 x 10 60 us here 10, 1 <- 6 3x3 on 116 x 37 x 37 51 us here 24).
bool conv_input_worth(int64_t patch, int64_t cols, int64_t positions, const ag_conv2_options *o) {
    const int64_t taps = (int64_t)o->filter[0] * o->filter[1];
    return enabled() && taps <= 32 && filters_fit(patch, cols, taps) && positions * patch * cols >= 1000000;
}

// The weight gradient: 1 -> 32 3x3 (254 x 55 x 55) 148 us here and 276, 6 -> 6 3x3 (84 x 60 x 60) 57 and 170; small ones
// (1.1e6 multiply-adds) 11 and 12.
bool conv_weight_worth(ag_dtype, int64_t patch, int64_t oc, int64_t positions, const ag_conv2_options *o) {
    return enabled() && (int64_t)o->filter[0] * o->filter[1] <= 32 && positions < kMostK && positions * patch * oc >= 1000000;
}

template int gemm_strided<float>(ag_device *, int, int, int, float, const float *, int64_t, int64_t,
                                 const float *, int64_t, int64_t, float, float *, int64_t, int64_t);
template int dense<float>(ag_device *, const float *, int, int, const float *, int, const float *, bool,
                          float *);

}  // namespace tcx
}  // namespace ag
