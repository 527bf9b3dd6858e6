// Conv2 -> Relu -> MaxPool2 (2 x 2, stride 2) on images of few channels, bf16, as one kernel each way (image_stage.cu).
#pragma once

#include "common.cuh"

namespace ag {
namespace image_stage {

struct Shape {
    int64_t bs, ic, ih, iw, oc;
    int fh, fw;   // padding 0, stride 1, dilation 1
};

// True for 3 x 3 filters on 2 to 4 channels and 5 x 5 on 1 or 2, and 64, 128, 192 or 256 output channels.  The geometries that are
// compiled; others, one channel of 3 x 3 among them, keep the form with patches in memory.
bool takes(const Shape &s);

// y [bs][ph][pw][oc] = max over 2 x 2 windows of relu(conv2(x, w) + bias), x NCHW, an odd last row or column left out
// as the pool does; codes (may be null) [bs][ph][pw][oc / 8] as relu_pool's (nhwc_ops.cuh).
int forward(ag_device *dev, const Shape &s, const __nv_bfloat16 *x, const __nv_bfloat16 *w, const __nv_bfloat16 *bias,
            __nv_bfloat16 *y, uint32_t *codes);

// The gradients of w and (bias) of the bias given dy [bs][ph][pw][oc] and the forward pass's codes, in two steps: f32 sums of
// slices of the batch (partial_floats of them), and their sum.  For even planes (the pool covers all cells).
int64_t partial_floats(ag_device *dev, const Shape &s);
int backward(ag_device *dev, const Shape &s, const __nv_bfloat16 *x, const __nv_bfloat16 *dy, const uint32_t *codes, bool bias,
             float *partial);
int weight_gradient(ag_device *dev, const Shape &s, const float *partial, __nv_bfloat16 *dw);
int bias_gradient(ag_device *dev, const Shape &s, const float *partial, __nv_bfloat16 *db);

}  // namespace image_stage
}  // namespace ag
