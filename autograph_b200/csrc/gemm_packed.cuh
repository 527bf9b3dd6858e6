// Large products on operands copied into aligned bf16 planes (gemm_packed.cu).
#pragma once

#include "common.cuh"

namespace ag {
namespace packed {

// Whether the device has room for the operands' planes, which stay with the device object: up to 4 GiB of them
// at a time.  Without, the gathered engine, which needs none, takes the product.
template <class T>
bool reserve(ag_device *dev, int M, int N, int K, int64_t p_k, int64_t q_k);

// C[row + col * ldc] = alpha * sum_k p[row * p_row + k * p_k] * q[col * q_row + k * q_k] + beta * C,
// then the optional bias (per row) and relu of a Dense layer.  One of p_row, p_k and one of q_row,
// q_k must be 1, and reserve() have returned true.
template <class T>
int gemm(ag_device *dev, int M, int N, int K, const T *p, int64_t p_row, int64_t p_k, const T *q,
         int64_t q_row, int64_t q_k, float alpha, float beta, T *c, int64_t ldc, const T *bias,
         bool relu);

}  // namespace packed
}  // namespace ag
