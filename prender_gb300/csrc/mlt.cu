// Primary-sample-space Metropolis light transport (Render::RunMLT,
// render.h:363-785; Kelemen, Szirmay-Kalos, Antal and Csonka, "A Simple and
// Robust Mutation Strategy for the Metropolis Light Transport Algorithm",
// 2002) as many independent chains.
//
// A path is a function of its primary samples: the camera takes the first
// six (pixel x, y, the sub-pixel halves, the tent filter's two), and the
// path's first branch the next ones, through the same shade() as the other
// renderers with a sampler that reads them (PssRng); draws past kMltDims
// and those of split branches are fresh in every proposal (an independent,
// symmetric proposal for those coordinates).  A proposal is a large step
// (every coordinate fresh, probability p_large) or a small step (Mutate0 of
// each coordinate, mlt.h:40-53); its values are derived from counter-based
// streams keyed by (chain, iteration, coordinate), so no proposal vector is
// stored: an accepted proposal is written back coordinate by coordinate.
// Each iteration splats the current and the proposed path with Kelemen's
// weights (a + large) / (L_new / b + p_large) and (1 - a) / (L_old / b +
// p_large), times the camera's inverse density W H 4, over the chain's
// length; b is the mean luminance of the bootstrap paths and the chains
// start from bootstrap paths drawn in proportion to their luminance.
#include <algorithm>

#include "block_paths.cuh"
#include "mlt.h"
#include "path_logic.cuh"

namespace pr {
namespace {

constexpr uint32_t kTagFresh = 0x4d4c5401u, kTagMutate = 0x4d4c5402u, kTagStep = 0x4d4c5403u;
constexpr uint32_t kTagExtra = 0x4d4c5500u;   // + branch
constexpr uint32_t kTagStream = 0x4d4c5600u;  // + branch
constexpr uint64_t kLargeBit = 1ull << 62, kSeedBit = 1ull << 63;

// the chains' primary samples (coordinate-major: u[k * chains + chain])
__constant__ float* c_mlt_u;
__constant__ int c_mlt_chains;

__device__ __forceinline__ float u01(uint32_t v) { return (float)(v >> 8) * (1.0f / 16777216.0f); }

__device__ __forceinline__ uint32_t phx(uint64_t seed, uint32_t tag, uint64_t stream, uint32_t k) {
  return philox4x32_10(make_uint4((uint32_t)stream, (uint32_t)(stream >> 32), k, tag),
                       make_uint2((uint32_t)seed, (uint32_t)(seed >> 32)))
      .x;
}

// Mutate0 (mlt.h:40-53): an exponentially distributed step of 1/512 .. 1/16
__device__ __forceinline__ float mutate0(float x, float r) {
  const float s1 = 1.0f / 512.0f, s2 = 1.0f / 16.0f;
  const float dx = s1 / (s1 / s2 + fabsf(2.0f * r - 1.0f)) - s1 / (s1 / s2 + 1.0f);
  if (r < 0.5f) {
    const float x1 = x + dx;
    return x1 < 1.0f ? x1 : x1 - 1.0f;
  }
  const float x1 = x - dx;
  return x1 < 0.0f ? x1 + 1.0f : x1;
}

// coordinate k (< kMltDims) of the proposal (or bootstrap path) `sample`:
// bits 0..61 the stream (chain | iteration << 24, or the bootstrap index),
// bit 62 a large step, bit 63 a bootstrap path
__device__ __forceinline__ float pss_value(uint64_t seed, uint64_t sample, int k) {
  const uint64_t stream = sample & ~kLargeBit;
  if (sample & (kLargeBit | kSeedBit)) return u01(phx(seed, kTagFresh, stream, (uint32_t)k));
  const uint32_t chain = (uint32_t)(sample & 0xFFFFFFu);
  const float cur = c_mlt_u[(size_t)k * c_mlt_chains + chain];
  return mutate0(cur, u01(phx(seed, kTagMutate, stream, (uint32_t)k)));
}

}  // namespace

// shade()'s sampler under MLT: the first branch's draws are primary samples
// 6, 7, ...; the rest fresh per proposal
struct PssRng {
  uint64_t seed, sample;
  uint32_t branch, draws;
  uint32_t vstart, sdraws;  // the vertex's first draw; its stream draws so far
  __device__ __forceinline__ float next() {
    const uint32_t k = draws++;
    if (branch == 0 && k + 6u < (uint32_t)kMltDims) return pss_value(seed, sample, (int)k + 6);
    return u01(phx(seed, kTagExtra + (branch & 0xFFu), sample & ~kLargeBit, k));
  }
  // the light choice and surface NEE point: fresh in every proposal, as the
  // reference's Next01 draws them from its stream under MLT
  __device__ __forceinline__ float next_stream() {
    return u01(phx(seed, kTagStream + (branch & 0xFFu), sample & ~kLargeBit, (vstart << 6) + (sdraws++ & 63u)));
  }
};
__device__ __forceinline__ void rng_at(PssRng& r, uint64_t seed, uint64_t sample, uint32_t branch, uint32_t draws) {
  r.seed = seed;
  r.sample = sample;
  r.branch = branch;
  r.draws = draws;
  r.vstart = draws;
  r.sdraws = 0;
}
__device__ __forceinline__ float rng_stream(PssRng& r) { return r.next_stream(); }
__device__ __forceinline__ uint32_t rng_draws(const PssRng& r) { return r.draws; }

namespace {

__device__ __forceinline__ float luminance(float3 c) { return 0.2126f * c.x + 0.7152f * c.y + 0.0722f * c.z; }

__global__ void mlt_init_kernel(MltCfg m, const int32_t* __restrict__ start, const float4* __restrict__ seed_path,
                                const float* __restrict__ seed_lum, float* __restrict__ u, float4* __restrict__ cur) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= m.chains) return;
  const int s = start[c];
  for (int k = 0; k < kMltDims; k++)
    u[(size_t)k * m.chains + c] = u01(phx(m.seed, kTagFresh, kSeedBit | (uint64_t)s, (uint32_t)k));
  cur[c] = seed_path[s];
  (void)seed_lum;
}

__device__ __forceinline__ void splat(float* acc, int pix, float3 v) {
  atomicAdd(acc + 3 * (size_t)pix, v.x);
  atomicAdd(acc + 3 * (size_t)pix + 1, v.y);
  atomicAdd(acc + 3 * (size_t)pix + 2, v.z);
}

struct MltRun {
  MltCfg m;
  int64_t it0, it1;          // iterations of every chain in this launch (chains)
  unsigned long long* next;  // chains or bootstrap paths handed out
  float* lum;                // bootstrap: luminance and path of each
  float4* path;
  float* u;                  // chains: primary samples, current path, image
  float4* cur;
  float* acc;
  // per slot
  int* chain;
  int64_t* it;
  int* pix;                  // (H - y - 1) W + x of the path under way
};

// The paths of the bootstrap (SEEDS) or of the chains' iterations, on the
// blocks of block_paths.cuh: a slot runs one chain's iterations one after
// another (generate_new_path, render.h:195-357: pixel and sub-pixel from the
// first six primary samples, the tent filter, radiance() over the split
// branches), then takes the next chain.  Bound by the FP64 sphere tests that
// remain and the shading; one chain per thread in nested loops kept 3.7 lanes
// of a warp active (96x72, 8 x 16 mutations a pixel on the sphere Cornell box:
// 64 ms, here 22.6).
template <bool SEEDS>
struct MltPaths {
  const DevScene& S;
  const RenderCfg& cfg;
  const MltRun& R;
  const BlockPool& P;
  uint32_t* err;
  uint32_t paths;
  bool more;
  int accepted;               // this lane's chain took its proposal (or -1)
  unsigned long long sample;  // that proposal

  __device__ __forceinline__ void start(size_t i, unsigned long long sample_, PathState& ps) {
    const uint64_t seed = cfg.seed, sample = sample_;
    int x = (int)(pss_value(seed, sample, 0) * (float)cfg.width);
    int y = (int)(pss_value(seed, sample, 1) * (float)cfg.height);
    x = min(max(x, 0), cfg.width - 1);
    y = min(max(y, 0), cfg.height - 1);
    const int sxx = pss_value(seed, sample, 2) < 0.5f ? 0 : 1;
    const int syy = pss_value(seed, sample, 3) < 0.5f ? 0 : 1;
    const float rr1 = 2.0f * pss_value(seed, sample, 4), rr2 = 2.0f * pss_value(seed, sample, 5);
    const float dx = rr1 < 1.0f ? sqrtf(rr1) - 1.0f : 1.0f - sqrtf(2.0f - rr1);
    const float dy = rr2 < 1.0f ? sqrtf(rr2) - 1.0f : 1.0f - sqrtf(2.0f - rr2);
    const float r1 = (sxx + 0.5f + dx) * 0.5f, r2 = (syy + 0.5f + dy) * 0.5f;
    const float3 sp = cfg.center + cfg.screen_x * ((r1 + x) * cfg.iw - 0.5f) + cfg.screen_y * ((r2 + y) * cfg.ih - 0.5f);
    root_path(ps, cfg.cam_pos, normalize(sp - cfg.cam_pos));
    P.id[i] = sample;
    R.pix[i] = (cfg.height - y - 1) * cfg.width + x;
  }

  __device__ __forceinline__ bool take(bool want, size_t i, PathState& ps) {
    const int lane = threadIdx.x & 31;
    if (!SEEDS) {
      // accepted proposals are written back by the whole warp, one chain at a
      // time: their 64 coordinates took a lane alone as long as half a path
      unsigned int left = __ballot_sync(0xffffffffu, accepted >= 0);
      while (left) {
        const int src = __ffs(left) - 1;
        left &= left - 1;
        const int c = __shfl_sync(0xffffffffu, accepted, src);
        const unsigned long long smp = __shfl_sync(0xffffffffu, sample, src);
        for (int k = lane; k < kMltDims; k += 32) {
          const float v = pss_value(R.m.seed, smp, k);
          R.u[(size_t)k * R.m.chains + c] = v;
        }
      }
      __syncwarp();
      accepted = -1;
    }
    // the slot's chain goes on, or the next one starts
    bool go = false;
    int c = -1;
    int64_t it = R.it0;
    if (!SEEDS && want) {
      c = R.chain[i];
      it = R.it[i] + 1;
      go = c >= 0 && it < R.it1;
    }
    const unsigned int mask = __ballot_sync(0xffffffffu, want && !go && more);
    if (mask) {
      unsigned long long base = 0;
      const int leader = __ffs(mask) - 1;
      if (lane == leader) base = atomicAdd(R.next, (unsigned long long)__popc(mask));
      base = __shfl_sync(0xffffffffu, base, leader);
      if ((mask >> lane) & 1) {
        const unsigned long long g = base + (unsigned long long)__popc(mask & ((1u << lane) - 1u));
        if (g < (unsigned long long)(SEEDS ? R.m.seeds : R.m.chains)) {
          c = (int)g;
          it = R.it0;
          go = true;
        } else {
          more = false;
        }
      }
    }
    if (!want || !go) return false;
    if (SEEDS) {
      R.chain[i] = c;
      start(i, kSeedBit | (uint64_t)c, ps);
    } else {
      R.chain[i] = c;
      R.it[i] = it;
      const uint64_t stream = ((uint64_t)it << 24) | (uint64_t)c;
      const bool large = u01(phx(R.m.seed, kTagStep, stream, 0u)) < R.m.p_large;
      start(i, stream | (large ? kLargeBit : 0ull), ps);
    }
    return true;
  }

  __device__ __forceinline__ void nee(size_t i, PathState& ps, int n, const unsigned char* lit) {
    for (int k = 0; k < 3; k++)
      if (k < n && lit[k]) {
        const float4 c = P.sh_c[3 * i + k];
        ps.L += f3(c.x, c.y, c.z);
      }
  }
  __device__ __forceinline__ void queued(size_t, int, const ShadowReq&) {}

  __device__ __forceinline__ int vertex(size_t i, PathState& ps, int& pending, bool hit, const FastHit& h,
                                        ShadowReq* sh, int& nsh) {
    PathState child;
    const unsigned long long id = P.id[i];
    const int r = shade<false, true, true, PssRng>(S, cfg, ps, hit, h, id, sh, nsh, child, err);
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
    if (!(isfinite(L.x) && isfinite(L.y) && isfinite(L.z))) {
      atomicOr(err, PR_DEV_NONFINITE);
      L = f3(0, 0, 0);
    }
    finish(i, id, L);
    paths++;
    return SHADE_END;
  }

  // a path of radiance F is complete
  __device__ __forceinline__ void finish(size_t i, unsigned long long id, float3 F) {
    const int c = R.chain[i], pix = R.pix[i];
    if (SEEDS) {
      R.lum[c] = luminance(F);
      R.path[c] = make_float4(F.x, F.y, F.z, __int_as_float(pix));
      return;
    }
    const MltCfg& m = R.m;
    const float4 co = R.cur[c];
    const uint64_t stream = id & ~kLargeBit;
    const bool large = (id & kLargeBit) != 0;
    const float accept_r = u01(phx(m.seed, kTagStep, stream, 1u));
    const float3 Fo = f3(co.x, co.y, co.z);
    const float Lnew = luminance(F), Lold = luminance(Fo);
    const float a = Lold > 1.0e-16f ? fminf(1.0f, Lnew / Lold) : 1.0f;
    const float wn = (a + (large ? 1.0f : 0.0f)) / (Lnew / m.b + m.p_large) * m.chain_scale * m.pdf;
    const float wo = (1.0f - a) / (Lold / m.b + m.p_large) * m.chain_scale * m.pdf;
    if (wo > 0.0f && Lold > 0.0f) splat(R.acc, __float_as_int(co.w), Fo * wo);
    if (wn > 0.0f && Lnew > 0.0f) splat(R.acc, pix, F * wn);
    if (accept_r < a) {
      accepted = c;
      sample = id;
      R.cur[c] = make_float4(F.x, F.y, F.z, __int_as_float(pix));
    }
  }
};

template <bool SEEDS>
__global__ void __launch_bounds__(kBlockThreads, 1)
    mlt_paths(const __grid_constant__ DevScene S, const __grid_constant__ RenderCfg cfg,
              const __grid_constant__ MltRun R, const __grid_constant__ BlockPool P, uint32_t* __restrict__ err,
              unsigned long long* __restrict__ counters) {
  extern __shared__ __align__(16) unsigned char smem[];
  TraceStats st{0, 0};
  uint32_t segs = 0;
  MltPaths<SEEDS> drv{S, cfg, R, P, err, 0u, true, -1, 0ull};
  for (int s = threadIdx.x; s < P.slots; s += blockDim.x) R.chain[(size_t)blockIdx.x * P.slots + s] = -1;
  __syncthreads();
  block_paths(S, P, drv, smem, st, segs, err);
  if (counters) add_counters(counters, drv.paths, segs, st);
}

__global__ void mlt_resolve_kernel(const float* __restrict__ acc, float* __restrict__ rgb, int n3, float scale,
                                   int accumulate) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n3) return;
  rgb[i] = (accumulate ? rgb[i] : 0.0f) + acc[i] * scale;
}

// Blocks of 768 threads, one per SM, as soon as they hold four full warps of
// chains: a chain's iterations run for long, so full warps and shared code
// fetches pay at fewer paths than a frame's samples do (block_shape's line).
// Fewer chains are bound by their serial iterations: blocks of 128 then.
BlockShape mlt_shape(unsigned long long n, int sms) {
  if (n < (unsigned long long)sms * 128) return block_shape(n, sms);
  BlockShape b;
  b.threads = kBlockThreads;
  b.blocks = (unsigned int)sms;
  const unsigned long long used = (n + sms - 1) / sms, room = kSlotsPerThread * kBlockThreads;
  b.used = (int)(used < room ? used : room);
  b.slots = (b.used + 15) / 16 * 16;
  return b;
}

template <bool SEEDS>
cudaError_t run_paths(const DevScene& S, const RenderCfg& cfg, MltRun R, unsigned long long n, void* scratch,
                      uint32_t* err, unsigned long long* counters, cudaStream_t stream) {
  const BlockShape b = mlt_shape(n, slot_sms(cfg));
  const size_t slots = (size_t)b.blocks * b.slots;
  char* p = static_cast<char*>(scratch);
  cudaError_t e = cudaMemsetAsync(p, 0, 256, stream);
  if (e != cudaSuccess) return e;
  R.next = reinterpret_cast<unsigned long long*>(p);
  BlockPool P = block_pool(p + 256, slots);
  P.slots = b.slots;
  P.slots_used = b.used;
  p += 256 + (block_pool_bytes(slots) + 255) / 256 * 256;
  R.it = reinterpret_cast<int64_t*>(p);
  R.chain = reinterpret_cast<int*>(R.it + slots);
  R.pix = R.chain + slots;
  mlt_paths<SEEDS><<<b.blocks, b.threads, block_shared_bytes(b), stream>>>(S, cfg, R, P, err, counters);
  return cudaGetLastError();
}

}  // namespace

size_t mlt_scratch_bytes(const RenderCfg& cfg, const MltCfg& m) {
  size_t most = 0;
  for (unsigned long long n : {(unsigned long long)m.seeds, (unsigned long long)m.chains}) {
    const BlockShape b = mlt_shape(n, slot_sms(cfg));
    const size_t slots = (size_t)b.blocks * b.slots;
    most = std::max(most, 512 + block_pool_bytes(slots) + 256 + 16 * slots);
  }
  return most;
}

cudaError_t launch_mlt_seeds(const DevScene& S, const RenderCfg& cfg, const MltCfg& m, float* lum, float4* path,
                             void* scratch, uint32_t* err, unsigned long long* counters, cudaStream_t stream) {
  if (m.seeds <= 0) return cudaSuccess;
  MltRun R{};
  R.m = m;
  R.lum = lum;
  R.path = path;
  return run_paths<true>(S, cfg, R, (unsigned long long)m.seeds, scratch, err, counters, stream);
}

cudaError_t launch_mlt_init(const MltCfg& m, const int32_t* start, const float4* seed_path, const float* seed_lum,
                            float* u, float4* cur, cudaStream_t stream) {
  cudaError_t e = cudaMemcpyToSymbolAsync(c_mlt_u, &u, sizeof(float*), 0, cudaMemcpyHostToDevice, stream);
  if (e == cudaSuccess)
    e = cudaMemcpyToSymbolAsync(c_mlt_chains, &m.chains, sizeof(int), 0, cudaMemcpyHostToDevice, stream);
  if (e != cudaSuccess) return e;
  mlt_init_kernel<<<(m.chains + 127) / 128, 128, 0, stream>>>(m, start, seed_path, seed_lum, u, cur);
  return cudaGetLastError();
}

cudaError_t launch_mlt_chains(const DevScene& S, const RenderCfg& cfg, const MltCfg& m, int64_t it0, int64_t it1,
                              float* u, float4* cur, float* acc, void* scratch, uint32_t* err,
                              unsigned long long* counters, cudaStream_t stream) {
  MltRun R{};
  R.m = m;
  R.it0 = it0;
  R.it1 = it1;
  R.u = u;
  R.cur = cur;
  R.acc = acc;
  return run_paths<false>(S, cfg, R, (unsigned long long)m.chains, scratch, err, counters, stream);
}

cudaError_t launch_mlt_resolve(const float* acc, float* rgb, int n3, float scale, int accumulate, cudaStream_t stream) {
  mlt_resolve_kernel<<<(n3 + 255) / 256, 256, 0, stream>>>(acc, rgb, n3, scale, accumulate);
  return cudaGetLastError();
}

}  // namespace pr
