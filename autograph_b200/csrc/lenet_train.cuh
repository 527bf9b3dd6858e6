// A training step of LeNet5 (benches/neural-network-benches/src/autograph_backend.rs:70-163) in two
// or three launches (lenet_train.cu).
#pragma once

#include "common.cuh"

namespace ag {
namespace lenet_train {

// Parameters in bucket order: conv 1 -> 6 5x5, conv 6 -> 16 5x5, dense 256 -> 128, 128 -> 84, 84 -> 10,
// bias of the last (off[5] < 0: none).  Element offsets into the flat buckets.
struct Net {
    int64_t off[6];
};

// The optimizer step that follows in the same launch, or only the gradients (update = false).
struct Sgd {
    bool update, use_momentum;
    float lr, momentum;
};

// Forward pass, summed cross-entropy loss (*loss, device-visible), every gradient into `grads` and
// optionally the SGD update of `values` / `velocity`.  x [bs,1,28,28] and t [bs] are device memory or
// pinned host memory.  Nothing synchronises.
int step(ag_device *dev, ag_dtype dtype, const Net &net, const void *x, const uint8_t *t, int64_t bs,
         void *values, void *grads, void *velocity, const Sgd &sgd, float *loss);

}  // namespace lenet_train
}  // namespace ag
