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

template <class T, bool RF>
static Strided<T, RF> strided(const T *p, int64_t s_row, int64_t s_k, int rows) {
    return Strided<T, RF>{p, s_row, s_k, rows, rows_aligned(p, s_row, s_k)};
}

template <class T>
static int run(ag_device *dev, int M, int N, int K, const T *p, int64_t p_row, int64_t p_k, const T *q,
               int64_t q_row, int64_t q_k, const StridedOut<T> &E) {
    const bool pf = p_k != 1, qf = q_k != 1;
    if (pf && qf)
        return gemm<T>(dev, M, N, K, strided<T, true>(p, p_row, p_k, M), strided<T, true>(q, q_row, q_k, N), E);
    if (pf)
        return gemm<T>(dev, M, N, K, strided<T, true>(p, p_row, p_k, M), strided<T, false>(q, q_row, q_k, N), E);
    if (qf)
        return gemm<T>(dev, M, N, K, strided<T, false>(p, p_row, p_k, M), strided<T, true>(q, q_row, q_k, N), E);
    return gemm<T>(dev, M, N, K, strided<T, false>(p, p_row, p_k, M), strided<T, false>(q, q_row, q_k, N), E);
}

template <class T>
int gemm_strided(ag_device *dev, int m, int k, int n, float alpha, const T *a, int64_t rsa,
                 int64_t csa, const T *b, int64_t rsb, int64_t csb, float beta, T *c, int64_t rsc,
                 int64_t csc) {
    // A warp of the epilogue writes 32 consecutive tile rows: they run along C's contiguous index,
    // so a row-major C is computed as C^T = B^T . A^T.
    const bool a_ok = rsa == 1 || csa == 1, b_ok = rsb == 1 || csb == 1;
    if (a_ok && b_ok && packed_worth(m, k, n)) {
        if (csc == 1)
            return packed::gemm<T>(dev, n, m, k, b, csb, rsb, a, rsa, csa, alpha, beta, c, rsc, nullptr, false);
        if (rsc == 1)
            return packed::gemm<T>(dev, m, n, k, a, rsa, csa, b, csb, rsb, alpha, beta, c, csc, nullptr, false);
    }
    if (csc == 1 && rsc != 1)
        return run<T>(dev, n, m, k, b, csb, rsb, a, rsa, csa, StridedOut<T>{c, csc, rsc, alpha, beta});
    return run<T>(dev, m, n, k, a, rsa, csa, b, csb, rsb, StridedOut<T>{c, rsc, csc, alpha, beta});
}

template <class T>
int dense(ag_device *dev, const T *x, int bs, int inputs, const T *w, int outputs, const T *bias,
          bool relu, T *y) {
    if (packed_worth(bs, inputs, outputs))
        return packed::gemm<T>(dev, outputs, bs, inputs, w, 1, outputs, x, inputs, 1, 1.f, 0.f, y, outputs,
                               bias, relu);
    return gemm<T>(dev, outputs, bs, inputs, strided<T, true>(w, 1, outputs, outputs),
                   strided<T, false>(x, inputs, 1, bs), DenseOut<T>{y, outputs, bias, relu});
}

}  // namespace tcx
}  // namespace ag
