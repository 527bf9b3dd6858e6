// Strided products on the gathered-operand tensor-core engine, for one element type.
#pragma once

#include "gemm_packed.cuh"
#include "gemm_tcx.cuh"
#include "tcx_api.cuh"

namespace ag {
namespace tcx {

template <class T>
static bool rows_aligned(const T *p, int64_t s_row, int64_t s_k) {
    return s_k == 1 && s_row % (int64_t)(16 / sizeof(T)) == 0 &&
           (reinterpret_cast<uintptr_t>(p) & 15) == 0;
}

template <Walk WALK, class T>
static Strided<T, WALK> strided(const T *p, int64_t s_row, int64_t s_k, int rows) {
    return Strided<T, WALK>{p, s_row, s_k, rows};
}

// Calls f with the operand in the walk that its memory asks for.
template <class T, class F>
static int with_operand(const T *p, int64_t s_row, int64_t s_k, int rows, F f) {
    if (rows_aligned(p, s_row, s_k)) return f(strided<kVecK>(p, s_row, s_k, rows));
    if (s_k == 1) return f(strided<kByK>(p, s_row, s_k, rows));
    return f(strided<kByRow>(p, s_row, s_k, rows));
}

// rows of the kernel's tile: the m index of (p, q) below.
template <class T>
static int run(ag_device *dev, int M, int N, int K, const T *p, int64_t p_row, int64_t p_k, const T *q,
               int64_t q_row, int64_t q_k, const StridedOut<T> &E) {
    return with_operand(p, p_row, p_k, M, [&](const auto &A) {
        return with_operand(q, q_row, q_k, N, [&](const auto &B) { return gemm<T>(dev, M, N, K, A, B, E); });
    });
}

template <class T>
constexpr ag_dtype kDtype = sizeof(T) == 4 ? AG_F32 : AG_BF16;

template <class T>
int gemm_strided(ag_device *dev, int m, int k, int n, float alpha, const T *a, int64_t rsa,
                 int64_t csa, const T *b, int64_t rsb, int64_t csb, float beta, T *c, int64_t rsc,
                 int64_t csc) {
    // A warp of the epilogue writes 32 consecutive tile rows: they run along C's contiguous index,
    // so a row-major C is computed as C^T = B^T . A^T.
    const bool a_ok = rsa == 1 || csa == 1, b_ok = rsb == 1 || csb == 1;
    if (a_ok && b_ok && packed_worth(kDtype<T>, m, k, n)) {
        if (csc == 1 && packed::reserve<T>(dev, n, m, k, rsb, csa))
            return packed::gemm<T>(dev, n, m, k, b, csb, rsb, a, rsa, csa, alpha, beta, c, rsc, nullptr, false);
        if (csc != 1 && rsc == 1 && packed::reserve<T>(dev, m, n, k, csa, rsb))
            return packed::gemm<T>(dev, m, n, k, a, rsa, csa, b, csb, rsb, alpha, beta, c, csc, nullptr, false);
    }
    if (csc == 1 && rsc != 1)
        return run<T>(dev, n, m, k, b, csb, rsb, a, rsa, csa, StridedOut<T>{c, csc, rsc, alpha, beta});
    return run<T>(dev, m, n, k, a, rsa, csa, b, csb, rsb, StridedOut<T>{c, rsc, csc, alpha, beta});
}

template <class T>
int dense(ag_device *dev, const T *x, int bs, int inputs, const T *w, int outputs, const T *bias,
          bool relu, T *y) {
    if (packed_worth(kDtype<T>, bs, inputs, outputs) && packed::reserve<T>(dev, outputs, bs, inputs, outputs, 1))
        return packed::gemm<T>(dev, outputs, bs, inputs, w, 1, outputs, x, inputs, 1, 1.f, 0.f, y, outputs,
                               bias, relu);
    const DenseOut<T> E{y, outputs, bias, relu};
    return with_operand(x, (int64_t)inputs, (int64_t)1, bs, [&](const auto &B) {
        return gemm<T>(dev, outputs, bs, inputs, strided<kByRow>(w, 1, outputs, outputs), B, E);
    });
}

}  // namespace tcx
}  // namespace ag
