// Large products on operands copied into aligned bf16 planes (gemm_packed.cu).
#pragma once

#include "common.cuh"

namespace ag {
namespace packed {

// C[row + col * ldc] = alpha * sum_k p[row * p_row + k * p_k] * q[col * q_row + k * q_k] + beta * C,
// then the optional bias (per row) and relu of a Dense layer.  One of p_row, p_k and one of q_row,
// q_k must be 1.
template <class T>
int gemm(ag_device *dev, int M, int N, int K, const T *p, int64_t p_row, int64_t p_k, const T *q,
         int64_t q_row, int64_t q_k, float alpha, float beta, T *c, int64_t ldc, const T *bias,
         bool relu);

}  // namespace packed
}  // namespace ag
