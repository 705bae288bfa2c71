// Kerr geodesics, mixed-precision form (PR_KERR_FP32; the templates are in
// kerr_math.cuh): the reference's FP64 Cash-Karp steps with its error
// control near the hole and among the scene geometry; FP32 increments of
// fixed h = 2 steps, added to the FP64 state, only for outbound rays beyond
// max(200 M, scene radius + 2) whose last FP64 error estimate is small; and
// an inbound ray with no radial turning point left reported as captured at
// once.  Compiled with FMA contraction (the FP64 form, kerr.cu, is not).
#include "kerr_math.cuh"

namespace pr {

cudaError_t launch_kerr_trace_fp32(const DevScene& S, const GKerr& K, const double* rays, int64_t n, KerrOut out,
                                   uint32_t* err, unsigned long long* counters, cudaStream_t stream) {
  if (n <= 0) return cudaSuccess;
  kerr_trace_kernel<true><<<geodesic_blocks((unsigned long long)n, sm_count()), 128, 0, stream>>>(S, K, rays, n, out,
                                                                                              err, counters);
  return cudaGetLastError();
}

size_t kerr_scratch_bytes_fp32(const RenderCfg& cfg) { return kerr_bytes(cfg, true); }

cudaError_t launch_kerr_render_fp32(const DevScene& S, const GKerr& K, const RenderCfg& cfg, void* scratch, float* dst,
                                    int accumulate, uint32_t* err, unsigned long long* counters, cudaStream_t stream) {
  const int sms = sm_count();
  for (unsigned long long k = 0, passes = pass_count(cfg); k < passes; k++) {
    KerrFrame F;
    cudaError_t e = kerr_frame(cfg, scratch, true, k, F, stream);
    if (e != cudaSuccess) return e;
    kerr_render_kernel<1><<<geodesic_blocks(F.pass.samples, sms), 128, 0, stream>>>(S, K, cfg, F, err, counters);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    kerr_render_kernel<2><<<geodesic_blocks(F.far_cap, sms), 128, 0, stream>>>(S, K, cfg, F, err, counters);
    e = cudaGetLastError();
    if (e == cudaSuccess) e = launch_sum(cfg, F.pass, dst, accumulate, stream);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

}  // namespace pr
