// Declarations of the auxiliary kernels (JBU, consistency scan, prior
// construction, image preparation).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>
#include "hpm_types.h"

namespace hpm {

cudaError_t launch_jbu(const float* image, int W, int H, const float* sdepth, int sw, int sh, float* out,
                       cudaStream_t st);
cudaError_t launch_jbu_prior(const float* image, int W, int H, const float* sdepth, const float* snormal, int sw,
                             int sh, float* out_depth, float* out_normal, cudaStream_t st);

}  // namespace hpm
