// Launch interfaces of the render / trace kernels.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "pr_internal.h"

namespace pr {

// Render::Run state for one launch (render.h:1125-1269), prepared on the host.
struct RenderCfg {
  float3 cam_pos, center, screen_x, screen_y;
  float iw, ih, rate, smp;
  float cutoff, sensor;
  int width, height;
  int spp;          // camera samples per pixel in this launch (samples * ss^2)
  int ss;           // supersamples per axis after the tent-filter fold
  int tent;
  int depth, depth_limit;
  int nee, media;
  int flags;
  int max_vertices;
  int chunks;       // sample chunks per pixel (one thread each)
  uint32_t tiles_x, tiles_y;
  uint64_t seed;
  uint64_t sample_offset;
};

// Pixel sums in 64-bit fixed point (2^-40): integer sums do not depend on the
// order in which samples finish.
constexpr float kPixelScaleF = 1099511627776.0f;  // 2^40
constexpr float kPixelInvF = 1.0f / 1099511627776.0f;
#ifdef __CUDACC__
__device__ __forceinline__ void add_pixel(long long* pix, float3 v) {
  unsigned long long* p = reinterpret_cast<unsigned long long*>(pix);
  atomicAdd(p + 0, (unsigned long long)__float2ll_rn(v.x * kPixelScaleF));
  atomicAdd(p + 1, (unsigned long long)__float2ll_rn(v.y * kPixelScaleF));
  atomicAdd(p + 2, (unsigned long long)__float2ll_rn(v.z * kPixelScaleF));
}
#endif
// pixel sums -> float image times the sensor response; accumulate adds to it
cudaError_t launch_resolve(const long long* pix, float* dst, int n3, int accumulate, float sensor, cudaStream_t stream);
// SMs of the current device
inline int sm_count() {
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0)
    sms = 152;
  return sms;
}

cudaError_t launch_megakernel(const DevScene& S, const RenderCfg& cfg, float* out, uint32_t* err,
                              unsigned long long* counters, cudaStream_t stream);
cudaError_t launch_reduce(const float* partial, float* dst, int n3, int chunks, int accumulate, cudaStream_t stream);
// the plain form of scenes without subsurface materials: one kernel and the
// resolve into dst; scratch (plain_scratch_bytes) holds the pixel sums
// and the blocks' path slots
size_t plain_scratch_bytes(const RenderCfg& cfg);
cudaError_t launch_plain(const DevScene& S, const RenderCfg& cfg, void* scratch, float* dst, int accumulate,
                          uint32_t* err, unsigned long long* counters, cudaStream_t stream);
// 8-bit bitmap rows of a float image (output.cu)
cudaError_t launch_to_rgb8(const float* rgb, int width, int height, double gamma_offset, uint8_t* out,
                           cudaStream_t stream);
// Radiance RGBE pixels for the HDR writer (output.cu)
cudaError_t launch_to_rgbe(const float* rgb, int width, int height, uint8_t* out, cudaStream_t stream);
cudaError_t launch_trace_fast(const DevScene& S, const double* rays, int64_t n, int32_t* ent, int32_t* prim, double* t,
                              uint32_t* err, cudaStream_t stream);
cudaError_t launch_first_hit(const DevScene& S, const double* rays, int64_t n, int32_t* ent, int32_t* prim, double* t,
                             uint32_t* err, unsigned long long* counters, cudaStream_t stream);

}  // namespace pr
