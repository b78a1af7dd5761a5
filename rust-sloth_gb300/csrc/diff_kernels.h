// diff_kernels.h -- launchers of the differentiable shading of a rendered batch.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "batch_kernels.h"

namespace sloth {

constexpr uint32_t kDiffChunk = 2048;   // depth cells (or samples) per block

// blocks[i] = (frame, first depth cell), chunks of kDiffChunk (even) over w*h per frame, for
// both passes.
cudaError_t launch_batch_shade(const BatchDev &b, const int2 *blocks, uint32_t nblocks, const float *vrgb,
                               const float *light, float *rgb, uint2 *vis, cudaStream_t s);
// gpos and gcol (3*nvert floats each) and glight (3) set to zero; any may be null.
cudaError_t launch_clear_gradients(float *gpos, float *gcol, float *glight, uint32_t nvert, cudaStream_t s);
cudaError_t launch_batch_shade_backward(const BatchDev &b, const int2 *blocks, uint32_t nblocks, const float *vrgb,
                                        const float *light, const float *grad_rgb, const uint2 *vis, float *gpos,
                                        float *gcol, float *glight, cudaStream_t s);

}  // namespace sloth
