// Paths of one thread block in lock step (the plain form): a block keeps a
// pool of path slots in global memory (small enough to stay in the 129 MB L2
// over all blocks) and alternates two phases between barriers:
//
//   shade   every live slot: add the shadow rays that came through, shade the
//           vertex its segment met, queue its shadow rays and its next
//           segment, or end the path and start the next one in its place;
//   trace   the block's warps take the queued rays with dynamic fetch (Aila
//           and Laine, "Understanding the efficiency of ray traversal on
//           GPUs", HPG 2009): a lane whose ray is answered takes the next.
//
// All warps of a block run the same phase, so its code is fetched once for
// many warps: with the phases left to each warp (or nested in each thread)
// instruction fetch was the main stall.  The rays meet the same nodes and
// triangles in the same order as in fast_closest / fast_occluded and each
// path the same shade() calls as in the nested loops, so paths do not change.
#pragma once
#include "path_logic.cuh"

namespace pr {

// idle lanes of a warp that make it fetch rays again
constexpr int kBlockRefill = 12;

// Large frames run one block of 768 threads per SM (80 registers): plain mesh
// Cornell box 321x243 x 16 spp, 5 subdivisions, on GB300 over 256x3 / 384x2 /
// 512x2 / 768x1 / 1024x1 threads x blocks: 9.4 / 9.0 / 9.3 / 8.7 / 9.1 ms
// (one path per thread in nested loops: 37.6); two slots per thread (one 9.2,
// four 10.5 with 512x2, whose slots no longer fit the L2).  A frame of few
// samples is bound by its longest path and the barriers on its way: blocks of
// 128 threads then, six per SM (64x48 x 4 spp spheres: the kernel 1.34 ms with
// large blocks, 1.12 with small ones).
constexpr int kBlockThreads = 768;
constexpr int kSmallBlockThreads = 128;
constexpr int kSlotsPerThread = 2;
struct BlockPool {
  // per slot (block b owns slots [b * slots, (b + 1) * slots))
  float4 *o, *d, *beta, *dpw, *L;  // path state; w lanes: depth, dp, branch, draws, pending branches
  float4* root;                    // radiance of the sample's ended branches
  unsigned long long* id;          // sample id
  float4* hit;                     // t, entity, leaf slot, u
  float* hitv;
  float4* sh_o;                    // origin of the vertex's shadow rays; w: their number
  float4* sh_d;                    // 3 per slot: direction, tmax
  float4* sh_c;                    // 3 per slot: contribution, the light's material
  float4* split;                   // pending glass branches: kSplitStack x 5 per slot
  int slots;                       // per block
  int slots_used;                  // slots of a block that take paths (small frames spread over the blocks)
};

// The block's queues, in dynamic shared memory.
struct BlockShared {
  unsigned int n_ext, n_sh, fetch, pad;  // queued segments and shadow rays, and how many of both are taken
};

// warp-aggregated append of n entries per lane to a shared counter (all lanes)
__device__ __forceinline__ unsigned int block_append(unsigned int* counter, unsigned int n) {
  const int lane = threadIdx.x & 31;
  unsigned int incl = n;
  for (int off = 1; off < 32; off <<= 1) {
    const unsigned int v = __shfl_up_sync(0xffffffffu, incl, off);
    if (lane >= off) incl += v;
  }
  const unsigned int total = __shfl_sync(0xffffffffu, incl, 31);
  unsigned int base = 0;
  if (lane == 31 && total) base = atomicAdd(counter, total);
  base = __shfl_sync(0xffffffffu, base, 31);
  return base + incl - n;
}

__device__ __forceinline__ void block_store(const BlockPool& P, size_t i, const PathState& ps, int pending) {
  P.o[i] = make_float4(ps.o.x, ps.o.y, ps.o.z, __int_as_float(ps.depth));
  P.d[i] = make_float4(ps.d.x, ps.d.y, ps.d.z, __int_as_float(ps.dp));
  P.beta[i] = make_float4(ps.beta.x, ps.beta.y, ps.beta.z, __uint_as_float(ps.branch));
  P.dpw[i] = make_float4(ps.dpw.x, ps.dpw.y, ps.dpw.z, __uint_as_float(ps.draws));
  P.L[i] = make_float4(ps.L.x, ps.L.y, ps.L.z, __int_as_float(pending));
}

__device__ __forceinline__ int block_load(const float4& o, const float4& d, const float4& b, const float4& w,
                                          const float4& l, PathState& ps) {
  ps.o = f3(o.x, o.y, o.z);
  ps.depth = __float_as_int(o.w);
  ps.d = f3(d.x, d.y, d.z);
  ps.dp = __float_as_int(d.w);
  ps.beta = f3(b.x, b.y, b.z);
  ps.branch = __float_as_uint(b.w);
  ps.dpw = f3(w.x, w.y, w.z);
  ps.draws = __float_as_uint(w.w);
  ps.L = f3(l.x, l.y, l.z);
  return __float_as_int(l.w);
}

// the glass branches of slot i that wait (n of them); word: the driver's own
__device__ __forceinline__ void block_push(const BlockPool& P, size_t i, int n, const PathState& c, int word) {
  float4* q = P.split + 5 * (kSplitStack * i + n);
  q[0] = make_float4(c.o.x, c.o.y, c.o.z, __int_as_float(c.depth));
  q[1] = make_float4(c.d.x, c.d.y, c.d.z, __int_as_float(c.dp));
  q[2] = make_float4(c.beta.x, c.beta.y, c.beta.z, __uint_as_float(c.branch));
  q[3] = make_float4(c.dpw.x, c.dpw.y, c.dpw.z, __uint_as_float(c.draws));
  q[4] = make_float4(c.L.x, c.L.y, c.L.z, __int_as_float(word));
}
__device__ __forceinline__ int block_pop(const BlockPool& P, size_t i, int n, PathState& ps) {
  const float4* c = P.split + 5 * (kSplitStack * i + n);
  return block_load(c[0], c[1], c[2], c[3], c[4], ps);
}

// The trace phase: rays [0, n_ext) of extq, then [n_ext, n_ext + n_sh) of shq.
__device__ __forceinline__ void block_trace(const DevScene& S, const BlockPool& P, size_t base, BlockShared& B,
                                            const unsigned short* extq, const unsigned short* shq,
                                            unsigned char* lit, float4* found, TraceStats& st, uint32_t& segs,
                                            uint32_t* err) {
  const int lane = threadIdx.x & 31;
  const unsigned int n_ext = B.n_ext, n = n_ext + B.n_sh;
  const unsigned int warps = blockDim.x / 32;
  // few rays spread over all warps
  const int width = (int)min(32u, (n + warps - 1) / warps);
  TraceLane r;
  lane_start(r, f3(0, 0, 0), f3(0, 0, 1), 0.0f);
  r.any = false;
  WGroup stack[kWStack];
  int item = 0;
  bool busy = false, exhausted = lane >= width;
  for (unsigned int step = 0;; step++) {
    const unsigned int idle = __ballot_sync(0xffffffffu, !busy && !exhausted);
    const unsigned int live = __ballot_sync(0xffffffffu, busy);
    if (idle == 0 && live == 0) break;
    if (step > (1u << 26)) {  // warp-uniform: every lane leaves together
      if (lane == 0) atomicOr(err, PR_DEV_LOOP_CAP);
      break;
    }
    if (idle && (__popc(idle) >= kBlockRefill || live == 0)) {
      const int leader = __ffs(idle) - 1;
      unsigned int first = 0;
      if (lane == leader) first = atomicAdd(&B.fetch, (unsigned int)__popc(idle));
      first = __shfl_sync(0xffffffffu, first, leader);
      if ((idle >> lane) & 1) {
        const unsigned int idx = first + __popc(idle & ((1u << lane) - 1u));
        if (idx < n) {
          busy = true;
          segs++;
          float4 o4, d4;
          r.any = idx >= n_ext;
          if (!r.any) {
            item = extq[idx];
            o4 = P.o[base + item];
            d4 = P.d[base + item];
          } else {
            item = shq[idx - n_ext];
            o4 = P.sh_o[base + (item >> 2)];
            d4 = P.sh_d[3 * (base + (item >> 2)) + (item & 3)];
          }
          lane_start(r, f3(o4.x, o4.y, o4.z), f3(d4.x, d4.y, d4.z), r.any ? d4.w : 3.0e38f);
        } else {
          exhausted = true;
        }
      }
    }
    if (trace_step<TRACE_EITHER>(S, busy, r, stack, found, st, err)) {
      busy = false;
      if (r.any) {
        lit[item] = r.h.ent < 0;
      } else {
        P.hit[base + item] = make_float4(r.h.t, __int_as_float(r.h.ent), __int_as_float(r.h.slot), r.h.u);
        P.hitv[base + item] = r.h.v;
      }
    }
  }
}

// The block's paths.  drv supplies them (take, by all lanes of a warp) and
// shades their vertices:
//   bool take(bool want, size_t slot, PathState& ps)
//   void nee(size_t slot, PathState& ps, int n, const unsigned char* lit)
//        the n shadow rays of the last vertex are answered (lit[k]: ray k came through)
//   void queued(size_t slot, int k, const ShadowReq&)  one of them is queued
//   int vertex(size_t slot, PathState& ps, int& pending, bool hit, const FastHit&, ShadowReq*, int& nsh)
//        SHADE_END if the path (all its branches) ended
template <class D>
__device__ __forceinline__ void block_paths(const DevScene& S, const BlockPool& P, D& drv, unsigned char* smem,
                                            TraceStats& st, uint32_t& segs, uint32_t* err) {
  BlockShared& B = *reinterpret_cast<BlockShared*>(smem);
  float4* found = reinterpret_cast<float4*>(smem + sizeof(BlockShared)) + (threadIdx.x & ~31u);  // warp_triangles
  unsigned short* extq = reinterpret_cast<unsigned short*>(smem + sizeof(BlockShared) + 16 * blockDim.x);
  unsigned short* shq = extq + P.slots;
  unsigned char* lit = reinterpret_cast<unsigned char*>(shq + 3 * P.slots);
  unsigned char* alive = lit + 4 * P.slots;
  const int tid = threadIdx.x, nt = blockDim.x;
  const size_t base = (size_t)blockIdx.x * P.slots;
  for (int s = tid; s < P.slots; s += nt) alive[s] = 0;
  // a small frame's slots go to the warps in turn
  const int warps = nt / 32;
  const bool spread = 2 * P.slots_used <= nt;
  for (unsigned int guard = 0;; guard++) {
    __syncthreads();
    if (tid == 0) {
      B.n_ext = 0;
      B.n_sh = 0;
      B.fetch = 0;
    }
    __syncthreads();
    for (int m = 0; m < P.slots_used; m += nt) {
      const int s = spread ? (tid & 31) * warps + (tid >> 5) : m + tid;
      const bool mine = s < P.slots_used;
      const size_t i = base + s;
      PathState ps;
      int pending = 0, nsh = 0;
      bool go = false;
      ShadowReq req[3];
      req[0].o = f3(0, 0, 0);
      if (mine && alive[s]) {
        const float4 so = P.sh_o[i];
        const float4 h4 = P.hit[i];
        pending = block_load(P.o[i], P.d[i], P.beta[i], P.dpw[i], P.L[i], ps);
        const int had = __float_as_int(so.w);
        if (had) drv.nee(i, ps, had, lit + 4 * s);
        FastHit h;
        h.t = h4.x;
        h.ent = __float_as_int(h4.y);
        h.slot = __float_as_int(h4.z);
        h.u = h4.w;
        h.v = P.hitv[i];
        go = drv.vertex(i, ps, pending, h.ent >= 0, h, req, nsh) != SHADE_END;
      }
      const bool want = mine && !go;
      if (__ballot_sync(0xffffffffu, want)) {
        if (drv.take(want, i, ps)) {
          go = true;
          pending = 0;
          nsh = 0;
        }
      }
      if (mine) {
        alive[s] = go;
        if (go) {
          block_store(P, i, ps, pending);
          P.sh_o[i] = make_float4(req[0].o.x, req[0].o.y, req[0].o.z, __int_as_float(nsh));
          for (int k = 0; k < 3; k++)
            if (k < nsh) {
              P.sh_d[3 * i + k] = make_float4(req[k].d.x, req[k].d.y, req[k].d.z, req[k].tmax);
              P.sh_c[3 * i + k] =
                  make_float4(req[k].contrib.x, req[k].contrib.y, req[k].contrib.z, __int_as_float(req[k].lmat));
              drv.queued(i, k, req[k]);
            }
        }
      }
      const unsigned int qe = block_append(&B.n_ext, go ? 1u : 0u);
      if (go) extq[qe] = (unsigned short)s;
      const unsigned int qs = block_append(&B.n_sh, (unsigned int)nsh);
      for (int k = 0; k < nsh; k++) shq[qs + k] = (unsigned short)(4 * s + k);
    }
    __syncthreads();
    if (B.n_ext == 0) break;
    if (guard > (1u << 24)) {  // block-uniform
      if (tid == 0) atomicOr(err, PR_DEV_LOOP_CAP);
      break;
    }
    block_trace(S, P, base, B, extq, shq, lit, found, st, segs, err);
  }
}

// warp-reduced statistics: paths, segments, nodes visited, triangles tested
__device__ __forceinline__ void add_counters(unsigned long long* counters, uint32_t paths, uint32_t segs,
                                             const TraceStats& st) {
  unsigned long long a = paths, b = segs, c = st.nodes, d = st.tris;
  for (int off = 16; off > 0; off >>= 1) {
    a += __shfl_down_sync(0xffffffffu, a, off);
    b += __shfl_down_sync(0xffffffffu, b, off);
    c += __shfl_down_sync(0xffffffffu, c, off);
    d += __shfl_down_sync(0xffffffffu, d, off);
  }
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(counters + 0, a);
    atomicAdd(counters + 1, b);
    atomicAdd(counters + 2, c);
    atomicAdd(counters + 3, d);
  }
}

// blocks, threads and slots of a frame on a device of sms SMs
struct BlockShape {
  unsigned int blocks;
  int threads, slots, used;
};
inline BlockShape block_shape(unsigned long long samples, int sms) {
  BlockShape b;
  // small: every resident slot would take fewer than two samples
  b.threads = samples < 2ull * sms * kBlockThreads * kSlotsPerThread ? kSmallBlockThreads : kBlockThreads;
  const unsigned long long room = kSlotsPerThread * b.threads;
  const unsigned long long most = (unsigned long long)sms * (kBlockThreads / b.threads);
  unsigned long long used = (samples + most - 1) / most;
  used = used < 16 ? 16 : used > room ? room : used;
  const unsigned long long want = (samples + used - 1) / used;
  b.blocks = (unsigned int)(want < most ? want : most);
  b.used = (int)used;
  b.slots = (b.used + 15) / 16 * 16;
  return b;
}

// bytes of a pool of n slots, and its arrays in a buffer of that size
inline size_t block_pool_bytes(size_t n) { return n * (16 * (5 + 1 + 1 + 1 + 3 + 3 + 5 * kSplitStack) + 8 + 4) + 256; }
inline BlockPool block_pool(void* p, size_t n) {
  BlockPool P;
  float4* f = static_cast<float4*>(p);
  auto take = [&](size_t per) {
    float4* q = f;
    f += per * n;
    return q;
  };
  P.o = take(1);
  P.d = take(1);
  P.beta = take(1);
  P.dpw = take(1);
  P.L = take(1);
  P.root = take(1);
  P.hit = take(1);
  P.sh_o = take(1);
  P.sh_d = take(3);
  P.sh_c = take(3);
  P.split = take(5 * kSplitStack);
  P.id = reinterpret_cast<unsigned long long*>(f);
  P.hitv = reinterpret_cast<float*>(P.id + n);
  P.slots = P.slots_used = 0;
  return P;
}

// dynamic shared memory of block_paths
inline size_t block_shared_bytes(const BlockShape& b) {
  return sizeof(BlockShared) + 16 * (size_t)b.threads + (2 + 6 + 4 + 1) * (size_t)b.slots;
}

}  // namespace pr
