// The one-kernel form of large channels-last BatchNorm layers (batchnorm_grid.cu).
#pragma once

#include "batchnorm_dev.cuh"

namespace musa_b200 {

struct BnGridPlan {
  int tx = 0;   // channel packs per column block; 0: not this form
  int gx = 0;   // column blocks
  int gy = 0;   // CTAs that share the rows of a column block
};

// The plan of a layer (inner == 1, whole 16-byte packs, aligned tensors).
template <typename T, int kMode>
BnGridPlan PlanBnGrid(const Geom& g);

// One cooperative launch; `partial`: [gy][2][channels] floats of scratch.  Returns a
// cudaError_t (cudaErrorCooperativeLaunchTooLarge where the context owns fewer SMs
// than the device has).
template <typename T, int kMode>
int LaunchBnGrid(const BnGridPlan& p, const T* x, const T* dy, T* out, const ApplyArgs& a,
                 float* partial, const Geom& g, cudaStream_t stream);

}  // namespace musa_b200
