// Launch interfaces of the render / trace kernels.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <cstdlib>

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
  int less;         // little device memory is left: smaller passes and pools
};

// A frame whose samples finish in any order (plain form, Kerr and wormhole
// frames): each leaves its radiance in its own place, pixel by pixel, and
// sum_samples adds up a pixel's samples in a fixed order, so the image
// does not depend on the schedule and holds any finite value (sums in fixed
// point wrap or lose what lies outside of their range).  A frame of more
// samples than kPassSamples takes passes of whole pixels.
struct SamplePass {
  float3* sample;              // samples of the pass's pixels, one pixel after another
  unsigned long long* next;    // samples handed out (and the callers' own counters, 256 bytes, zero at the start)
  unsigned long long samples;  // of the pass
  unsigned long long px0;      // its first pixel (scan line order)
};
// 192 MB of samples; PR_PASS_SAMPLES may lower it.  A pass ends on an emptying
// chip: 64 spp of 1024x768 in 3 passes 368.8 ms, some 0.8 less per pass saved
constexpr unsigned long long kPassSamples = 1ull << 24;
inline unsigned long long pass_pixels(const RenderCfg& cfg) {
  const char* e = getenv("PR_PASS_SAMPLES");
  const long long v = e ? strtoll(e, nullptr, 10) : 0;
  const unsigned long long full = cfg.less ? kPassSamples / 16 : kPassSamples;
  const unsigned long long most = v >= 1 && v < (long long)full ? (unsigned long long)v : full;
  const unsigned long long px = (unsigned long long)cfg.width * cfg.height, n = most / (unsigned long long)cfg.spp;
  return n < 1 ? 1 : n < px ? n : px;
}
inline unsigned long long pass_count(const RenderCfg& cfg) {
  const unsigned long long px = (unsigned long long)cfg.width * cfg.height, n = pass_pixels(cfg);
  return (px + n - 1) / n;
}
// a frame's counters and samples, ahead of the callers' own scratch
inline size_t pass_bytes(const RenderCfg& cfg) {
  return 256 + (sizeof(float3) * (size_t)pass_pixels(cfg) * (size_t)cfg.spp + 255) / 256 * 256;
}
// pass k; its counters are zeroed on the stream
inline cudaError_t sample_pass(const RenderCfg& cfg, void* scratch, unsigned long long k, SamplePass& A,
                               cudaStream_t stream) {
  const unsigned long long px = (unsigned long long)cfg.width * cfg.height, n = pass_pixels(cfg);
  A.next = static_cast<unsigned long long*>(scratch);
  A.sample = reinterpret_cast<float3*>(static_cast<char*>(scratch) + 256);
  A.px0 = k * n;
  A.samples = (px - A.px0 < n ? px - A.px0 : n) * (unsigned long long)cfg.spp;
  return cudaMemsetAsync(scratch, 0, 256, stream);
}
// the pass's pixels -> float image times the sensor response; accumulate adds to it
cudaError_t launch_sum(const RenderCfg& cfg, const SamplePass& A, float* dst, int accumulate, cudaStream_t stream);
// pixel and sample of the pass's sample g
__device__ __forceinline__ void pass_sample(const RenderCfg& cfg, const SamplePass& A, uint32_t g, int& x,
                                            int& y, uint32_t& k) {
  const uint32_t p = g / (uint32_t)cfg.spp, px = (uint32_t)A.px0 + p;
  k = g - p * (uint32_t)cfg.spp;
  y = (int)(px / (uint32_t)cfg.width);
  x = (int)(px - (uint32_t)y * (uint32_t)cfg.width);
}
// SMs of the current device
inline int sm_count() {
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0)
    sms = 152;
  return sms;
}
// the SMs that blocks with path slots in device memory are spread over
inline int slot_sms(const RenderCfg& cfg) { return cfg.less ? (sm_count() + 3) / 4 : sm_count(); }

cudaError_t launch_megakernel(const DevScene& S, const RenderCfg& cfg, float* out, uint32_t* err,
                              unsigned long long* counters, cudaStream_t stream);
cudaError_t launch_reduce(const float* partial, float* dst, int n3, int chunks, int accumulate, cudaStream_t stream);
// the plain form of scenes without subsurface materials: one kernel and the
// sum into dst per pass; scratch (plain_scratch_bytes) holds the samples and
// the blocks' path slots
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
