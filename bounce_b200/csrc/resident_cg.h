// Shapes and launches of the on-chip MPCG (resident_cg.cuh, resident_cg.cu).
#pragma once

#include <cuda_runtime.h>

#include "cloth_dev.cuh"
#include "resident_shape.h"

namespace b3g {

// The shape of cloth c's solve on the current device.
ResShape resident_shape(const ClothDev& c);
// by_blocks: a cluster sums in the order of the per-iteration kernels, else in
// the cooperative CG's.
cudaError_t launch_resident_cg(const ClothDev& c, const ResShape& s, int dot, bool by_blocks, cudaStream_t st);

}  // namespace b3g
