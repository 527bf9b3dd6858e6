// LeNet5 inference in bf16 for large batches on the tensor cores (lenet_tiles.cu).
#pragma once

#include "common.cuh"

namespace ag {
namespace lenet_tiles {

// Conv 1 -> 6 5x5, conv 6 -> 16 5x5 (no bias; relu and 2x2 pool after each), dense 256 -> 128 -> 84 -> 10 (relu
// after the first two; biases may be null).
struct Weights {
    const void *conv1, *conv2, *dense[3], *bias[3];
};

// True when a batch of bs images of this device goes to the tile kernel.
bool takes(const ag_device *dev, const void *x, const void *y, int64_t bs);

// x [bs,1,28,28] -> logits y [bs,10], bf16.
int forward(ag_device *dev, const void *x, int64_t bs, const Weights &w, void *y);

}  // namespace lenet_tiles
}  // namespace ag
