// Launch interface of the path-replay adjoint renderer (adjoint.cu).
#pragma once
#include <cuda_runtime.h>

#include "pr_internal.h"
#include "render_kernels.h"

namespace pr {

constexpr int kAdjMaterials = 16;  // materials the adjoint pass tracks

// adds dL/dC (3 per material) and dL/dE (3 per material) into d_color and
// d_emission (device, double); scratch of adjoint_scratch_bytes; launches:
// the kernels launched
size_t adjoint_scratch_bytes(const RenderCfg& cfg, int n_mat);
cudaError_t launch_adjoint(const DevScene& S, const RenderCfg& cfg, const float* dl_drgb, int n_mat, void* scratch,
                           double* d_color, double* d_emission, uint32_t* err, unsigned long long* counters,
                           int* launches, cudaStream_t stream);

}  // namespace pr
