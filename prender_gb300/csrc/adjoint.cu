// Adjoint of the plain renderer by path replay: gradients of a scalar image
// loss with respect to every material's colour (albedo) and emission.
//
// The caller renders the image with pr_render, forms dL/d(pixel), and calls
// the adjoint with the same camera, parameters and sample range.  The camera
// samples are replayed with the same counter-based streams, so they walk
// exactly the paths of the forward render (Vicini, Speierer and Jakob, "Path
// Replay Backpropagation", SIGGRAPH 2021), and accumulate:
//
//  * colour: every term a branch adds to L after a non-terminal vertex j is
//    proportional to C_{m_j} once (BRDF_Diffuse / Specular / Refraction all
//    scale the continuation and the vertex's next-event terms by the
//    material colour, brdf.h:408-953).  With n_m the number of such
//    vertices of material m and S_m the sum of the branch radiance L
//    recorded right after each of them (before its next-event terms),
//    d L_branch / d C_m = (n_m L_branch - S_m) / C_m per channel.  A glass
//    branch handed back at a split inherits its ancestors' vertices.
//  * emission: shade() reports every emitted term as weight x emission
//    (EmissionTap); next-event terms carry their light's material.
//
// Sampling decisions (Russian roulette, light choice, glass branch choice)
// are held fixed and their probabilities are treated as constants, the
// usual estimator of the derivative of the expectation; the luminance clamp
// of a sample is differentiated exactly.  Scenes with media are
// not supported by this pass; materials are limited to kAdjMaterials.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdlib>

#include "adjoint.h"
#include "block_paths.cuh"

namespace pr {
namespace {

__device__ __forceinline__ float3 safe_div(float3 a, float3 c) {
  return f3(c.x != 0.0f ? a.x / c.x : 0.0f, c.y != 0.0f ? a.y / c.y : 0.0f, c.z != 0.0f ? a.z / c.z : 0.0f);
}

// A pass covers whole warps of the reduction below: a warp is an 8 x 4 pixel
// tile and a sample chunk, each lane sums its pixel's samples [k0, k1) in
// order.  The paths themselves run in any order on resident blocks
// (block_paths.cuh) and leave what the sums need of each sample.
struct AdjointPass {
  uint32_t warp0;            // first warp (chunk * tiles + tile)
  uint32_t kk0;              // first sample of each lane in this pass
  uint32_t kmax;             // samples of each lane in this pass
  int first, last;           // of the passes over these lanes' samples
  unsigned long long items;  // warps * 32 * kmax (sample kk of lane l of warp w: (w 32 + l) kmax + kk)
  unsigned long long* next;  // items handed out
  int n_mat;
  float3* w;                 // per item: dLoss / d(sample radiance); zero where there is no sample
  float3* g_col;             // per item and material: d L / d C_m
  float3* g_em;              // d L / d E_m
  float4* acc;               // per slot and material: sum S_m of the branch, count n_m
  int* anc;                  // per slot: materials of the branch's first three vertices, their number << 24
  unsigned long long* item;  // per slot
  float4* ew;                // 3 per slot: contribution / emission of the queued shadow rays
  float* carry;              // 6 per lane and material: sums carried to the lanes' next pass
};

// pixel and sample of an item; false where the tile or the chunk has none
__device__ __forceinline__ bool adjoint_item(const RenderCfg& cfg, const AdjointPass& A, unsigned long long it, int& x,
                                             int& y, int& k) {
  const uint32_t v = (uint32_t)(it / A.kmax), kk = (uint32_t)(it - (unsigned long long)v * A.kmax);
  const uint32_t warp = A.warp0 + (v >> 5), lane = v & 31;
  const uint32_t tiles = cfg.tiles_x * cfg.tiles_y, chunk = warp / tiles, tile = warp - chunk * tiles;
  x = (int)((tile % cfg.tiles_x) * 8 + (lane & 7));
  y = (int)((tile / cfg.tiles_x) * 4 + (lane >> 3));
  const int k0 = (int)(((int64_t)cfg.spp * chunk) / cfg.chunks);
  const int k1 = (int)(((int64_t)cfg.spp * (chunk + 1)) / cfg.chunks);
  k = k0 + (int)(A.kk0 + kk);
  return x < cfg.width && y < cfg.height && k < k1;
}

struct AdjointPaths {
  const DevScene& S;
  const RenderCfg& cfg;
  const AdjointPass& A;
  const BlockPool& P;
  const float* dl_drgb;
  uint32_t* err;
  uint32_t paths;
  bool more;

  __device__ __forceinline__ void start_branch(size_t i, int anc) {
    float4* acc = A.acc + i * A.n_mat;
    for (int m = 0; m < A.n_mat; m++) acc[m] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    // the branch's radiance all comes after its ancestors' vertices
    for (int k = 0; k < (anc >> 24); k++) acc[(anc >> (8 * k)) & 0xFF].w += 1.0f;
    A.anc[i] = anc;
  }

  __device__ __forceinline__ bool take(bool want, size_t i, PathState& ps) {
    const int lane = threadIdx.x & 31;
    bool got = false;
    for (;;) {
      const unsigned int mask = __ballot_sync(0xffffffffu, want && !got && more);
      if (!mask) return got;
      unsigned long long base = 0;
      const int leader = __ffs(mask) - 1;
      if (lane == leader) base = atomicAdd(A.next, (unsigned long long)__popc(mask));
      base = __shfl_sync(0xffffffffu, base, leader);
      if (!((mask >> lane) & 1)) continue;
      const unsigned long long it = base + (unsigned long long)__popc(mask & ((1u << lane) - 1u));
      if (it >= A.items) {
        more = false;
        continue;
      }
      int x, y, k;
      if (!adjoint_item(cfg, A, it, x, y, k)) continue;
      float3 o, d;
      P.id[i] = camera_ray(cfg, x, y, cfg.sample_offset + (uint64_t)k, o, d);
      root_path(ps, o, d);
      A.item[i] = it;
      start_branch(i, 0);
      got = true;
    }
  }

  __device__ __forceinline__ EmissionTap tap(size_t i) const { return EmissionTap{A.g_em + A.item[i] * A.n_mat, A.n_mat}; }

  __device__ __forceinline__ void nee(size_t i, PathState& ps, int n, const unsigned char* lit) {
    EmissionTap t = tap(i);
    for (int k = 0; k < 3; k++)
      if (k < n && lit[k]) {
        const float4 c = P.sh_c[3 * i + k], e = A.ew[3 * i + k];
        ps.L += f3(c.x, c.y, c.z);
        t.em(__float_as_int(c.w), f3(e.x, e.y, e.z));
      }
  }
  __device__ __forceinline__ void queued(size_t i, int k, const ShadowReq& r) {
    A.ew[3 * i + k] = make_float4(r.ew.x, r.ew.y, r.ew.z, 0.0f);
  }

  __device__ __forceinline__ int vertex(size_t i, PathState& ps, int& pending, bool hit, const FastHit& h,
                                        ShadowReq* sh, int& nsh) {
    PathState child;
    const unsigned long long id = P.id[i];
    EmissionTap t = tap(i);
    const int r = shade<false, false>(S, cfg, ps, hit, h, id, sh, nsh, child, err, nullptr, nullptr, &t);
    int anc = A.anc[i];
    if (r != SHADE_END) {
      // a non-terminal vertex: everything this branch adds from here on scales with its colour
      const int m = S.entf[h.ent].material;
      float4& a = A.acc[i * A.n_mat + m];
      a.w += 1.0f;
      a.x += ps.L.x;
      a.y += ps.L.y;
      a.z += ps.L.z;
      if ((anc >> 24) < 3) {
        anc = (anc & 0xFFFFFF) | (m << (8 * (anc >> 24))) | (((anc >> 24) + 1) << 24);
        A.anc[i] = anc;
      }
    }
    if (r == SHADE_SPLIT) {
      const int n = pending & 0xFF;
      if (n < kSplitStack) {
        block_push(P, i, n, child, anc);
        if (!(pending & 0x100)) P.root[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        pending = (n + 1) | 0x100;
      } else {
        atomicOr(err, PR_DEV_LOOP_CAP);
      }
    }
    if (r != SHADE_END) return r;
    nsh = 0;
    const unsigned long long it = A.item[i];
    for (int m = 0; m < A.n_mat; m++) {
      const float4 a = A.acc[i * A.n_mat + m];
      if (a.w > 0.0f)
        A.g_col[it * A.n_mat + m] += safe_div(ps.L * a.w - f3(a.x, a.y, a.z), ld3(S.mats[m].color));
    }
    float3 L = ps.L;
    if (pending & 0x100) {
      const float4 q = P.root[i];
      L = f3(q.x, q.y, q.z) + ps.L;
      const int n = pending & 0xFF;
      if (n > 0) {  // the next branch that waits
        P.root[i] = make_float4(L.x, L.y, L.z, 0.0f);
        start_branch(i, block_pop(P, i, n - 1, ps));
        pending--;
        return SHADE_CONTINUE;
      }
    }
    // finish_sample: v = L * smp, and above the cutoff v_c = c v / lum(v),
    // whose derivative is (c / lum) (dv - v (W . dv) / lum) with W the
    // luminance weights: the adjoint of the clamp maps delta to
    // (c / lum) (delta - (delta . v / lum) W)
    int x, y, k;
    adjoint_item(cfg, A, it, x, y, k);
    const size_t pix = (size_t)(cfg.height - y - 1) * cfg.width + x;
    const float3 delta = f3(dl_drgb[3 * pix], dl_drgb[3 * pix + 1], dl_drgb[3 * pix + 2]) * cfg.sensor;
    const float3 v = L * cfg.smp;
    float3 w = delta * cfg.smp;
    if (!(isfinite(v.x) && isfinite(v.y) && isfinite(v.z))) {
      w = f3(0, 0, 0);
    } else if (cfg.cutoff > 0.0f) {
      const float3 W = f3(0.2126f, 0.7152f, 0.0722f);
      const float lum = dot(W, v);
      if (lum > cfg.cutoff) w = (delta - W * (dot(delta, v) / lum)) * (cfg.cutoff / lum * cfg.smp);
    }
    A.w[it] = w;
    paths++;
    return SHADE_END;
  }
};

__global__ void __launch_bounds__(kBlockThreads, 1)
    adjoint_paths(const __grid_constant__ DevScene S, const __grid_constant__ RenderCfg cfg,
                  const __grid_constant__ AdjointPass A, const __grid_constant__ BlockPool P,
                  const float* __restrict__ dl_drgb, uint32_t* __restrict__ err,
                  unsigned long long* __restrict__ counters) {
  extern __shared__ __align__(16) unsigned char smem[];
  TraceStats st{0, 0};
  uint32_t segs = 0;
  AdjointPaths drv{S, cfg, A, P, dl_drgb, err, 0u, true};
  block_paths(S, P, drv, smem, st, segs, err);
  if (counters) add_counters(counters, drv.paths, segs, st);
}

// the samples' gradients of a pass: each lane its pixel's samples in order,
// then the warp, then one double atomic per value and warp
__global__ void __launch_bounds__(128) adjoint_reduce(const __grid_constant__ AdjointPass A, double* __restrict__ d_color,
                                                      double* __restrict__ d_emission) {
  const unsigned long long v = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x;
  if ((v >> 5) * 32ull * A.kmax >= A.items) return;  // whole warps leave together
  const int lane = threadIdx.x & 31;
  for (int m = 0; m < A.n_mat; m++) {
    float3 col = f3(0, 0, 0), em = f3(0, 0, 0);
    float* c = A.carry + 6 * (v * A.n_mat + m);
    if (!A.first) {
      col = f3(c[0], c[1], c[2]);
      em = f3(c[3], c[4], c[5]);
    }
    for (uint32_t k = 0; k < A.kmax; k++) {
      const unsigned long long it = v * A.kmax + k;
      const float3 w = A.w[it];
      col += w * A.g_col[it * A.n_mat + m];
      em += w * A.g_em[it * A.n_mat + m];
    }
    if (!A.last) {
      c[0] = col.x;
      c[1] = col.y;
      c[2] = col.z;
      c[3] = em.x;
      c[4] = em.y;
      c[5] = em.z;
      continue;
    }
    const float q6[6] = {col.x, col.y, col.z, em.x, em.y, em.z};
#pragma unroll
    for (int q = 0; q < 6; q++) {
      float a = q6[q];
      for (int off = 16; off > 0; off >>= 1) a += __shfl_down_sync(0xffffffffu, a, off);
      if (lane == 0 && a != 0.0f) atomicAdd((q < 3 ? d_color : d_emission) + 3 * m + (q % 3), (double)a);
    }
  }
}

constexpr size_t kAdjointBytes = 512ull << 20;  // of the samples of one pass (a lane's at most kAdjointLane)
constexpr uint32_t kAdjointLane = 4096;         // PR_ADJOINT_LANE may lower it

uint32_t adjoint_lane() {
  const char* e = getenv("PR_ADJOINT_LANE");
  const long v = e ? strtol(e, nullptr, 10) : 0;
  return v >= 1 && v < (long)kAdjointLane ? (uint32_t)v : kAdjointLane;
}

// warps and samples per lane of a pass, and the scratch it takes
struct AdjointShape {
  uint32_t warps, pass_warps, lane_samples, kmax;  // kmax: a lane's samples in one pass
  BlockShape blocks;                               // of the largest pass, for all of them
  size_t item_bytes, slot_bytes, slots, carry_bytes;
};
AdjointShape adjoint_shape(const RenderCfg& cfg, int n_mat) {
  AdjointShape h;
  h.warps = cfg.tiles_x * cfg.tiles_y * (uint32_t)cfg.chunks;
  h.lane_samples = (uint32_t)((cfg.spp + cfg.chunks - 1) / cfg.chunks);
  h.kmax = std::min(h.lane_samples, adjoint_lane());
  h.item_bytes = sizeof(float3) * (1 + 2 * (size_t)n_mat);
  const size_t per_warp = h.item_bytes * 32 * h.kmax;
  h.pass_warps = (uint32_t)std::max<size_t>(1, std::min<size_t>(h.warps, (cfg.less ? kAdjointBytes / 16 : kAdjointBytes) / per_warp));
  h.blocks = block_shape((unsigned long long)h.pass_warps * 32 * h.kmax, slot_sms(cfg));
  h.slots = (size_t)h.blocks.blocks * h.blocks.slots;
  h.slot_bytes = sizeof(float4) * (n_mat + 3) + 4 + 8;
  h.carry_bytes = h.lane_samples > h.kmax ? (24 * (size_t)n_mat * 32 * h.pass_warps + 255) / 256 * 256 : 0;
  return h;
}

}  // namespace

size_t adjoint_scratch_bytes(const RenderCfg& cfg, int n_mat) {
  const AdjointShape h = adjoint_shape(cfg, n_mat);
  return h.carry_bytes + 256 + (h.item_bytes * h.pass_warps * 32 * h.kmax + 255) / 256 * 256 +
         block_pool_bytes(h.slots) + (h.slot_bytes * h.slots + 255) / 256 * 256 + 256;
}

cudaError_t launch_adjoint(const DevScene& S, const RenderCfg& cfg, const float* dl_drgb, int n_mat, void* scratch,
                           double* d_color, double* d_emission, uint32_t* err, unsigned long long* counters,
                           int* launches, cudaStream_t stream) {
  const AdjointShape h = adjoint_shape(cfg, n_mat);
  const BlockShape& b = h.blocks;
  const size_t n = h.slots;
  *launches = 0;
  for (uint32_t w0 = 0; w0 < h.warps; w0 += h.pass_warps)
    for (uint32_t k0 = 0; k0 < h.lane_samples; k0 += h.kmax) {
      const uint32_t warps = std::min(h.pass_warps, h.warps - w0);
      AdjointPass A;
      A.warp0 = w0;
      A.kk0 = k0;
      A.kmax = std::min(h.kmax, h.lane_samples - k0);
      A.first = k0 == 0;
      A.last = k0 + A.kmax == h.lane_samples;
      A.items = (unsigned long long)warps * 32 * A.kmax;
      A.n_mat = n_mat;
      // the carried sums come first, where every pass finds them: what follows
      // is laid out by this pass's items, fewer in the last one
      A.carry = static_cast<float*>(scratch);
      char* p = static_cast<char*>(scratch) + h.carry_bytes;
      A.next = reinterpret_cast<unsigned long long*>(p);
      A.w = reinterpret_cast<float3*>(p + 256);
      A.g_col = A.w + A.items;
      A.g_em = A.g_col + A.items * n_mat;
      const size_t zero = 256 + h.item_bytes * A.items;
      cudaError_t e = cudaMemsetAsync(p, 0, zero, stream);
      if (e != cudaSuccess) return e;
      p += (zero + 255) / 256 * 256;
      BlockPool P = block_pool(p, n);
      P.slots = b.slots;
      P.slots_used = b.used;
      p += (block_pool_bytes(n) + 255) / 256 * 256;
      A.acc = reinterpret_cast<float4*>(p);
      A.ew = A.acc + n * n_mat;
      A.item = reinterpret_cast<unsigned long long*>(A.ew + 3 * n);
      A.anc = reinterpret_cast<int*>(A.item + n);
      adjoint_paths<<<b.blocks, b.threads, block_shared_bytes(b), stream>>>(S, cfg, A, P, dl_drgb, err, counters);
      e = cudaGetLastError();
      if (e != cudaSuccess) return e;
      adjoint_reduce<<<(warps + 3) / 4, 128, 0, stream>>>(A, d_color, d_emission);
      e = cudaGetLastError();
      if (e != cudaSuccess) return e;
      *launches += 2;
    }
  return cudaSuccess;
}

}  // namespace pr
