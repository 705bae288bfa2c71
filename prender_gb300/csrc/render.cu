// Plain drop-in renderer: Render::Run's per-sample body (render.h:1203-1385)
// -- camera ray, the whole radiance() branch tree, luminance clamp -- with
// the per-vertex logic of path_logic.cuh, in one kernel and in two shapes:
//
// pt_block: the paths of a block in lock step (block_paths.cuh), every scene
// without subsurface materials; a pixel's samples added up by sum_samples.
//
// pt_megakernel: one thread per (pixel, sample chunk), shadow rays and the
// next segment traced in place, for subsurface scenes (whose frames live on
// the thread's stack) and for pr_render_dev_noalloc (its 16 MiB hold no pool
// of paths).  Each thread sums its samples in order and writes one partial
// image per sample chunk; reduce_chunks adds the chunks in order.
//
// In both the refracted branch of a depth <= 2 glass split waits on a 4-entry
// stack (at most three splits are pending at once: depths 0, 1, 2).
#include <cuda_runtime.h>

#include "path_logic.cuh"
#include "block_paths.cuh"

namespace pr {

// Subsurface continuations whose radiance the reference bounds
// (OVER_RADIANCE_CUT2 / 3): frame f collects its continuation's
// contributions C over all branches inside it; when its last branch ends,
// C (and the vertex's own emission and direct terms E) go to the parent
// unless |C / scale| exceeds the bound, in which case the vertex gave zero.
constexpr int kMaxSssFrames = 16;
struct SssFrames {
  float3 C[kMaxSssFrames], E[kMaxSssFrames], scale[kMaxSssFrames];
  float thr[kMaxSssFrames];
  int parent[kMaxSssFrames], open[kMaxSssFrames];
  int n;
};

__device__ __forceinline__ void frame_add(SssFrames& F, float3& root, int f, float3 x) {
  if (f < 0) root += x;
  else F.C[f] += x;
}

// a branch inside frame f ended (or a child frame closed): close every frame
// that has nothing open left
__device__ __forceinline__ void frame_release(SssFrames& F, float3& root, int f) {
  while (f >= 0) {
    if (--F.open[f] > 0) return;
    const float3 s = F.scale[f], c = F.C[f];
    const float3 q = f3(s.x != 0.0f ? c.x / s.x : 0.0f, s.y != 0.0f ? c.y / s.y : 0.0f, s.z != 0.0f ? c.z / s.z : 0.0f);
    const bool cut = sqrtf(dot(q, q)) > F.thr[f];
    const int p = F.parent[f];
    if (!cut) frame_add(F, root, p, c + F.E[f]);
    f = p;
  }
}

// One camera sample: the whole branch tree of radiance() for one root ray.
template <bool SSS, bool EXT>
__device__ float3 trace_sample(const DevScene& S, const RenderCfg& cfg, float3 o0, float3 d0, uint64_t sample_id,
                               TraceStats& st, uint32_t* err, uint32_t& segs) {
  PathState stack[kSplitStack];
  int sframe[kSplitStack];
  int sp = 0;
  root_path(stack[sp], o0, d0);
  sframe[sp++] = -1;
  float3 L = f3(0, 0, 0);
  SssFrames F;
  F.n = 0;
  while (sp > 0) {
    --sp;
    PathState ps = stack[sp];
    int fr = sframe[sp];
    for (;;) {
      FastHit h;
      segs++;
      const bool hit = fast_closest(S, ps.o, ps.d, h, st, err);
      ShadowReq sh[3];
      int nsh = 0;
      PathState child;
      SssFrameOut fo;
      fo.open = 0;
      const float3 Lb = ps.L;
      const int r = shade<SSS, EXT, EXT>(S, cfg, ps, hit, h, sample_id, sh, nsh, child, err, nullptr, nullptr,
                                         nullptr, SSS ? &fo : nullptr);
      const float3 Lown = ps.L - Lb;
      float3 Lnee = f3(0, 0, 0);
      for (int k = 0; k < nsh; k++) {
        segs++;
        if (!fast_occluded(S, sh[k].o, sh[k].d, sh[k].tmax, st, err)) Lnee += sh[k].contrib;
      }
      if (SSS && fo.open && F.n + fo.open <= kMaxSssFrames) {
        // the branch moves into a new frame (or two nested ones): what it
        // gathered before this vertex belongs outside, the vertex's own terms
        // to the frame, its continuation inside
        const int f = F.n++;
        F.E[f] = Lown + (fo.nee_inner ? f3(0, 0, 0) : Lnee);
        F.C[f] = f3(0, 0, 0);
        F.scale[f] = fo.scale;
        F.thr[f] = fo.thr;
        F.parent[f] = fr;
        F.open[f] = 1;
        frame_add(F, L, fr, Lb);
        int in = f;
        if (fo.open == 2) {
          in = F.n++;
          F.E[in] = f3(0, 0, 0);
          F.C[in] = f3(0, 0, 0);
          F.scale[in] = fo.scale2;
          F.thr[in] = fo.thr2;
          F.parent[in] = f;
          F.open[in] = 1;
        }
        F.C[in] += fo.inner + (fo.nee_inner ? Lnee : f3(0, 0, 0));
        ps.L = f3(0, 0, 0);
        fr = in;  // the parents keep their counts: the branch left, the child frame came
      } else {
        ps.L += Lnee;
        if (SSS && fo.open) ps.L += fo.inner;
      }
      if (r == SHADE_SPLIT) {
        if (sp < kSplitStack) {
          stack[sp] = child;
          sframe[sp++] = fr;
          if (SSS && fr >= 0) F.open[fr]++;
        } else {
          atomicOr(err, PR_DEV_LOOP_CAP);
        }
      }
      if (r == SHADE_END) break;
    }
    if (SSS) {
      frame_add(F, L, fr, ps.L);
      frame_release(F, L, fr);
    } else {
      L += ps.L;
    }
  }
  return L;
}

// the lean form (no subsurface or glossy lobes) at 8 blocks of 128 per SM
// (64 registers, spilling): mesh Cornell box 23.6 -> 24.8 Mpaths/s on GB300;
// the fuller forms keep 3 blocks per SM (168 registers)
template <bool SSS, bool EXT>
__global__ void __launch_bounds__(128, EXT ? 3 : 8) pt_megakernel(DevScene S, RenderCfg cfg, float* __restrict__ out,
                                                     uint32_t* __restrict__ err, unsigned long long* __restrict__ counters) {
  const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t warp = tid >> 5, lane = tid & 31;
  const uint32_t tiles_per_chunk = cfg.tiles_x * cfg.tiles_y;
  const uint32_t chunk = warp / tiles_per_chunk;
  if (chunk >= (uint32_t)cfg.chunks) return;
  const uint32_t tile = warp - chunk * tiles_per_chunk;
  const int x = (int)((tile % cfg.tiles_x) * 8 + (lane & 7));
  const int y = (int)((tile / cfg.tiles_x) * 4 + (lane >> 3));
  TraceStats st{0, 0};
  uint32_t segs = 0, paths = 0;
  if (x < cfg.width && y < cfg.height) {
    const int k0 = (int)(((int64_t)cfg.spp * chunk) / cfg.chunks);
    const int k1 = (int)(((int64_t)cfg.spp * (chunk + 1)) / cfg.chunks);
    float3 acc = f3(0, 0, 0);
    for (int k = k0; k < k1; k++) {
      float3 o, d;
      const uint64_t sample_id = camera_ray(cfg, x, y, cfg.sample_offset + (uint64_t)k, o, d);
      acc += finish_sample(cfg, trace_sample<SSS, EXT>(S, cfg, o, d, sample_id, st, err, segs), err);
      paths++;
    }
    acc = acc * cfg.sensor;
    float* o = out + 3 * ((size_t)chunk * cfg.width * cfg.height + (size_t)(cfg.height - y - 1) * cfg.width + x);
    o[0] = acc.x;
    o[1] = acc.y;
    o[2] = acc.z;
  }
  if (counters) add_counters(counters, paths, segs, st);
}

// sums the per-chunk partial images in chunk order (deterministic) into
// dst; accumulate != 0 adds to what dst holds
__global__ void reduce_chunks(const float* __restrict__ partial, float* __restrict__ dst, int n3, int chunks,
                              int accumulate) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n3) return;
  float s = accumulate ? dst[i] : 0.0f;
  for (int c = 0; c < chunks; c++) s += partial[(size_t)c * n3 + i];
  dst[i] = s;
}

// ---- the plain form without subsurface frames ------------------------------
// Resident blocks take camera samples one by one, pixel by pixel
// (block_paths.cuh), and leave each finished sample in its place of the pass
// (sum_samples adds them up).  Bound by instruction issue and divergence; mesh Cornell
// box 321x243 x 16 spp on GB300 37.7 ms in pt_megakernel, 8.4 here, spheres
// 256x192 x 16 (FP64 sphere tests) 16.8 -> 6.9, Ward 404x248 x 4 22.2 -> 6.1.
// FULL: glossy lobes, other lights, textures; the same shade() instantiations
// as pt_megakernel's, since contraction (and with it a path's last bits)
// differs between instantiations.
struct PlainFrame {
  SamplePass pass;
  uint32_t* item;  // per slot: the pass's sample that its path is (a sample id may wrap past 2^64)
};

template <bool FULL>
struct PlainPaths {
  const DevScene& S;
  const RenderCfg& cfg;
  const PlainFrame& F;
  const BlockPool& P;
  uint32_t* err;
  uint32_t paths;
  bool more;

  __device__ __forceinline__ bool take(bool want, size_t i, PathState& ps) {
    const int lane = threadIdx.x & 31;
    const unsigned int mask = __ballot_sync(0xffffffffu, want && more);
    if (!mask) return false;
    unsigned long long base = 0;
    const int leader = __ffs(mask) - 1;
    if (lane == leader) base = atomicAdd(F.pass.next, (unsigned long long)__popc(mask));
    base = __shfl_sync(0xffffffffu, base, leader);
    if (!((mask >> lane) & 1)) return false;
    const unsigned long long g = base + (unsigned long long)__popc(mask & ((1u << lane) - 1u));
    if (g >= F.pass.samples) {
      more = false;
      return false;
    }
    // a pixel's samples one after another: the first segments of a warp are close together
    F.item[i] = (uint32_t)g;
    int x, y;
    uint32_t k;
    pass_sample(cfg, F.pass, (uint32_t)g, x, y, k);
    float3 o, d;
    P.id[i] = camera_ray(cfg, x, y, cfg.sample_offset + (uint64_t)k, o, d);
    root_path(ps, o, d);
    return true;
  }

  __device__ __forceinline__ void nee(size_t i, PathState& ps, int n, const unsigned char* lit) {
    float3 sum = f3(0, 0, 0);
    for (int k = 0; k < 3; k++)
      if (k < n && lit[k]) {
        const float4 c = P.sh_c[3 * i + k];
        sum += f3(c.x, c.y, c.z);
      }
    ps.L += sum;
  }
  __device__ __forceinline__ void queued(size_t, int, const ShadowReq&) {}

  __device__ __forceinline__ int vertex(size_t i, PathState& ps, int& pending, bool hit, const FastHit& h,
                                        ShadowReq* sh, int& nsh) {
    PathState child;
    const unsigned long long id = P.id[i];
    const uint32_t item = F.item[i];  // with the path's state: read where the path ends, its wait would show
    const int r = shade<false, FULL, FULL>(S, cfg, ps, hit, h, id, sh, nsh, child, err);
    // pending: waiting branches; bit 8: the sample has split
    if (r == SHADE_SPLIT) {
      const int n = pending & 0xFF;
      if (n < kSplitStack) {
        block_push(P, i, n, child, 0);
        if (!(pending & 0x100)) P.root[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        pending = (n + 1) | 0x100;
      } else {
        atomicOr(err, PR_DEV_LOOP_CAP);
      }
    }
    if (r != SHADE_END) return r;
    nsh = 0;
    float3 L = ps.L;
    if (pending & 0x100) {
      const float4 q = P.root[i];
      L = f3(q.x, q.y, q.z) + ps.L;
      const int n = pending & 0xFF;
      if (n > 0) {  // the next branch that waits
        P.root[i] = make_float4(L.x, L.y, L.z, 0.0f);
        block_pop(P, i, n - 1, ps);
        pending--;
        return SHADE_CONTINUE;
      }
    }
    F.pass.sample[item] = finish_sample(cfg, L, err);
    paths++;
    return SHADE_END;
  }
};

template <bool FULL>
__global__ void __launch_bounds__(kBlockThreads, 1)
    pt_block(const __grid_constant__ DevScene S, const __grid_constant__ RenderCfg cfg,
             const __grid_constant__ PlainFrame F, const __grid_constant__ BlockPool P, uint32_t* __restrict__ err,
             unsigned long long* __restrict__ counters) {
  extern __shared__ __align__(16) unsigned char smem[];
  TraceStats st{0, 0};
  uint32_t segs = 0;
  PlainPaths<FULL> drv{S, cfg, F, P, err, 0u, true};
  block_paths(S, P, drv, smem, st, segs, err);
  if (counters) add_counters(counters, drv.paths, segs, st);
}

// Adds up the samples of n pixels from px0 on, g threads a pixel (a power of
// two up to 32, or the whole block), times the sensor response
// (render.h:1405-1409); accumulate != 0 adds to what dst holds.  Each sum is
// two floats (two_add keeps every addition's error): right to some spp 2^-48
// for a few FP32 instructions, where FP64 additions were bound by that pipe
// (1.25 M samples of the mesh Cornell box 321x243: 55 -> 16 us).
constexpr int kSumThreads = 256;
struct Sum3 {
  float s[3], e[3];
};
__device__ __forceinline__ void sum_add(Sum3& a, int c, float s, float e) {
  two_add(a.s[c], a.e[c], s);
  a.e[c] += e;
}
__global__ void __launch_bounds__(kSumThreads)
    sum_samples(const float3* __restrict__ sample, float* __restrict__ dst, int width, int height, uint32_t spp,
                unsigned long long px0, unsigned long long n, uint32_t g, int accumulate, float sensor) {
  __shared__ Sum3 part[kSumThreads / 32];
  const unsigned long long t = (unsigned long long)blockIdx.x * kSumThreads + threadIdx.x, p = t / g;
  const uint32_t l = (uint32_t)(t - p * g);
  Sum3 a = {};
  if (p < n)
    for (uint32_t k = l; k < spp; k += g) {
      const float3 v = sample[p * spp + k];
      sum_add(a, 0, v.x, 0.0f);
      sum_add(a, 1, v.y, 0.0f);
      sum_add(a, 2, v.z, 0.0f);
    }
  for (int off = (int)(g < 32 ? g : 32) / 2; off > 0; off >>= 1)
#pragma unroll
    for (int c = 0; c < 3; c++)
      sum_add(a, c, __shfl_down_sync(0xffffffffu, a.s[c], off), __shfl_down_sync(0xffffffffu, a.e[c], off));
  if (g > 32) {
    if ((threadIdx.x & 31) == 0) part[threadIdx.x / 32] = a;
    __syncthreads();
    for (int w = 1; w < kSumThreads / 32; w++)
      for (int c = 0; c < 3; c++) sum_add(a, c, part[w].s[c], part[w].e[c]);
  }
  if (p >= n || l != 0) return;
  const unsigned long long px = px0 + p, y = px / (unsigned int)width, x = px - y * (unsigned int)width;
  float* o = dst + 3 * ((size_t)(height - 1 - (int)y) * width + (size_t)x);
  for (int c = 0; c < 3; c++) {
    // past the largest float the sum is infinite and its error no number
    const float v = (isfinite(a.s[c]) ? a.s[c] + a.e[c] : a.s[c]) * sensor;
    o[c] = accumulate ? o[c] + v : v;
  }
}

cudaError_t launch_sum(const RenderCfg& cfg, const SamplePass& A, float* dst, int accumulate, cudaStream_t stream) {
  const uint32_t spp = (uint32_t)cfg.spp;
  uint32_t g = 1;  // from 1024 samples a pixel on a block each: a warp alone would take them in 32 or more rounds
  while (g < 32 && 2 * g <= spp) g *= 2;
  if (spp >= 1024) g = kSumThreads;
  const unsigned long long n = A.samples / spp, blocks = (n * g + kSumThreads - 1) / kSumThreads;
  sum_samples<<<(unsigned)blocks, kSumThreads, 0, stream>>>(A.sample, dst, cfg.width, cfg.height, spp, A.px0, n, g,
                                                            accumulate, cfg.sensor);
  return cudaGetLastError();
}

// blocks of the frame's largest pass, for all of its passes
static BlockShape plain_shape(const RenderCfg& cfg) {
  return block_shape(pass_pixels(cfg) * (unsigned long long)cfg.spp, slot_sms(cfg));
}

size_t plain_scratch_bytes(const RenderCfg& cfg) {
  const BlockShape b = plain_shape(cfg);
  const size_t n = (size_t)b.blocks * b.slots;
  return pass_bytes(cfg) + (block_pool_bytes(n) + 255) / 256 * 256 + 4 * n;
}

cudaError_t launch_plain(const DevScene& S, const RenderCfg& cfg, void* scratch, float* dst, int accumulate,
                         uint32_t* err, unsigned long long* counters, cudaStream_t stream) {
  const BlockShape b = plain_shape(cfg);
  const size_t n = (size_t)b.blocks * b.slots, smem = block_shared_bytes(b);
  char* p = static_cast<char*>(scratch) + pass_bytes(cfg);
  BlockPool P = block_pool(p, n);
  P.slots = b.slots;
  P.slots_used = b.used;
  PlainFrame F;
  F.item = reinterpret_cast<uint32_t*>(p + (block_pool_bytes(n) + 255) / 256 * 256);
  for (unsigned long long k = 0, passes = pass_count(cfg); k < passes; k++) {
    cudaError_t e = sample_pass(cfg, scratch, k, F.pass, stream);
    if (e != cudaSuccess) return e;
    if (S.has_glossy || S.n_point_lights > 0 || S.has_tex)
      pt_block<true><<<b.blocks, b.threads, smem, stream>>>(S, cfg, F, P, err, counters);
    else
      pt_block<false><<<b.blocks, b.threads, smem, stream>>>(S, cfg, F, P, err, counters);
    e = cudaGetLastError();
    if (e == cudaSuccess) e = launch_sum(cfg, F.pass, dst, accumulate, stream);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

cudaError_t launch_megakernel(const DevScene& S, const RenderCfg& cfg, float* out, uint32_t* err,
                              unsigned long long* counters, cudaStream_t stream) {
  const uint64_t threads = (uint64_t)cfg.tiles_x * cfg.tiles_y * 32ull * (uint64_t)cfg.chunks;
  const uint32_t blocks = (uint32_t)((threads + 127) / 128);
  // the fuller instantiations (subsurface frames; glossy lobes, parallel /
  // spot / infinity lights, textures) only where needed
  if (S.has_sss) pt_megakernel<true, true><<<blocks, 128, 0, stream>>>(S, cfg, out, err, counters);
  else if (S.has_glossy || S.n_point_lights > 0 || S.has_tex)
    pt_megakernel<false, true><<<blocks, 128, 0, stream>>>(S, cfg, out, err, counters);
  else pt_megakernel<false, false><<<blocks, 128, 0, stream>>>(S, cfg, out, err, counters);
  return cudaGetLastError();
}

cudaError_t launch_reduce(const float* partial, float* dst, int n3, int chunks, int accumulate, cudaStream_t stream) {
  reduce_chunks<<<(n3 + 255) / 256, 256, 0, stream>>>(partial, dst, n3, chunks, accumulate);
  return cudaGetLastError();
}

}  // namespace pr
