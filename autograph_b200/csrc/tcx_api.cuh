// Entry points of the tensor-core engines for operands TMA cannot read as they are
// (gemm_tcx.cuh: gathered; gemm_packed.cu: copied into aligned planes first).
#pragma once

#include "common.cuh"

namespace ag {
namespace tcx {

// True when the gathered engine should take C[m,n] = A[m,k] . B[k,n] of this type instead of
// the SIMT engine.
bool gemm_worth(ag_dtype dtype, int64_t m, int64_t k, int64_t n);

// True when such a product is large enough to copy its operands into aligned bf16 planes first.
bool packed_worth(ag_dtype dtype, int64_t m, int64_t k, int64_t n);

// C = alpha * A.B + beta * C on strided views.
template <class T>
int gemm_strided(ag_device *dev, int m, int k, int n, float alpha, const T *a, int64_t rsa,
                 int64_t csa, const T *b, int64_t rsb, int64_t csb, float beta, T *c, int64_t rsc,
                 int64_t csc);

// y = relu?(x . w + bias), row-major contiguous; the product's sums are those of gemm_strided.
template <class T>
int dense(ag_device *dev, const T *x, int bs, int inputs, const T *w, int outputs, const T *bias,
          bool relu, T *y);

// Convolutions (any padding / stride / dilation, at most 32 taps), NCHW.  Sizes as a product: patch =
// channels x taps (of the source that is gathered), cols, positions.
bool conv_worth(ag_dtype dtype, int64_t patch, int64_t cols, int64_t positions, const ag_conv2_options *o);
bool conv_input_worth(int64_t patch, int64_t cols, int64_t positions, const ag_conv2_options *o);
bool conv_weight_worth(ag_dtype dtype, int64_t patch, int64_t oc, int64_t positions,
                       const ag_conv2_options *o);
// f32 gradients that the kernels on pixel rows (conv_halo_f32.cuh) take and are faster at than the direct kernels.
bool input_by_rows(ag_device *dev, ag_dtype dtype, int64_t oc, int64_t ic, int64_t bs, int64_t ih, int64_t iw,
                   const ag_conv2_options *o, int64_t oh, int64_t ow);
bool weight_by_rows(ag_dtype dtype, int64_t bs, int64_t ic, int64_t ih, int64_t iw, int64_t oc, const ag_conv2_options *o,
                    int64_t oh, int64_t ow);

template <class T>
int conv_forward(ag_device *dev, const T *x, int64_t bs, int64_t ic, int64_t ih, int64_t iw,
                 const T *w, int64_t oc, const T *bias, const ag_conv2_options *o, int64_t oh,
                 int64_t ow, bool relu, T *y);
template <class T>
int conv_backward_input(ag_device *dev, const T *w, int64_t oc, int64_t ic, const T *dy, int64_t bs,
                        int64_t ih, int64_t iw, const ag_conv2_options *o, int64_t oh, int64_t ow,
                        T *dx);
template <class T>
int conv_backward_weight(ag_device *dev, const T *x, int64_t bs, int64_t ic, int64_t ih, int64_t iw,
                         const T *dy, int64_t oc, const ag_conv2_options *o, int64_t oh, int64_t ow,
                         float beta, T *dw);

}  // namespace tcx
}  // namespace ag
