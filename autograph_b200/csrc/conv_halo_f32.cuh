// f32 convolutions with stride 1 on the tensor cores, filters resident, one box of pixels per tile (conv_halo_f32.cu).
#pragma once

#include "common.cuh"

namespace ag {
namespace halo32 {

// y[b][n][oy][ox] = sum over (c, fi, fj) of src[b][c][oy + fi - pad_h][ox + fj - pad_w] * w[n * s_row + c * s_c + tap], tap =
// fi * fw + fj, or that counted from the end (reversed: the input gradient's order).
struct Problem {
    const float *src, *w;
    int64_t bs, channels, h, wd;   // source
    int64_t n, oh, ow;
    int fh, fw, pad_h, pad_w;
    int64_t s_row, s_c;
    bool reversed;
};

// Up to 64 channels and columns whose filters fit shared memory beside two boxes; where it is the faster engine.
bool takes(ag_device *dev, const Problem &p);

// With the optional bias and relu of the separate operators.
int run(ag_device *dev, const Problem &p, const float *bias, bool relu, float *y);

// dw[n][c][fi][fj] = beta * dw + sum over (b, oy, ox) of dy[b][n][oy][ox] * x[b][c][oy + fi - pad_h][ox + fj - pad_w].
struct Wgrad {
    const float *x, *dy;
    int64_t bs, channels, h, wd, n, oh, ow;
    int fh, fw, pad_h, pad_w;
};
bool takes_wgrad(const Wgrad &p);
// *taken is false, and nothing was launched, where there is no room for the CTAs' sums.
int run_wgrad(ag_device *dev, const Wgrad &p, float beta, float *dw, bool *taken);

}  // namespace halo32
}  // namespace ag
