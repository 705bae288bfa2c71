// What the geodesic tracers (kerr_math.cuh, wormhole.cu) share: step control
// and scene-segment decisions that FP32 can settle with room to spare.  The
// kernels are bound by GB300's FP64 pipe (a warp instruction per 64 clocks
// and scheduler, whatever its active lanes; 64 FP32 instructions fit beside
// one), so what does not need FP64 is kept out of it; every value that enters
// a ray's state keeps its FP64 bits.  sincos gives the
// bits of sin and of cos in 24 FP64 instructions instead of 36, a division
// takes 6, a power 85, an arctangent 26, a logarithm 31 (timed on GB300).
// Steps of 192x96 Kerr rays: 51.5 -> 44.8 ms (FP64 instructions an attempt
// 1390 -> 1040).
#pragma once
#include <cuda_runtime.h>

#include "device_common.cuh"
#include "render_kernels.h"

namespace pr {
namespace {

// A double's magnitude rounded towards zero to FP32, by integer operations.
// Tiny values give 0; bad is set for values FP32 does not hold (NaN included).
__device__ __forceinline__ float trunc_f32(double x, bool& bad) {
  const uint32_t hi = (uint32_t)__double2hiint(x) & 0x7FFFFFFFu;
  bad |= hi >= 0x47F00000u;
  return hi < 0x38100000u ? 0.0f
                          : __uint_as_float(((hi - 0x38000000u) << 3) | ((uint32_t)__double2loint(x) >> 29));
}

// max |num[i] / den[i]| (NaN ratios left out), as the reference's loop over
// the exact quotients gives it: only the ratios within 1e-4 of the largest in
// FP32 are divided in FP64 (nearly always one of six)
template <int N>
__device__ __forceinline__ double max_ratio(const double* num, const double* den) {
  float q[N], top = 0.0f;
  bool bad = false;
#pragma unroll
  for (int i = 0; i < N; i++) {
    const float n = trunc_f32(num[i], bad), d = trunc_f32(den[i], bad);
    bad |= !(d > 1.0e-30f && d < 1.0e30f);
    q[i] = __fdividef(n, d);
    top = fmaxf(top, q[i]);
  }
  bad |= !(top > 1.0e-30f && top < 1.0e30f);
  uint32_t left = 0;
#pragma unroll
  for (int i = 0; i < N; i++) left |= (bad || q[i] >= 0.9999f * top) ? 1u << i : 0u;
  double best = 0.0;
  while (left) {
    const int k = __ffs(left) - 1;
    left &= left - 1;
    double n = num[0], d = den[0];
#pragma unroll
    for (int i = 1; i < N; i++)
      if (i == k) {
        n = num[i];
        d = den[i];
      }
    const double t = fabs(n / d);
    if (t > best) best = t;
  }
  return best;
}

// rkqs' next step from the accepted step h and its error, at most cap: the
// power is left out where FP32 shows that it ends above the cap (errmax <
// (0.9 h / cap)^5, with 0.1 % to spare)
__device__ __forceinline__ double next_step(double h, double errmax, double cap) {
  double hnext = 5.0 * h;
  if (errmax > 1.89e-4) {
    bool exact = !(h > 0.0);
    const float q = 0.9f * __fdividef(trunc_f32(h, exact), trunc_f32(cap, exact)), q2 = q * q;
    const float e = trunc_f32(errmax, exact);
    exact = exact || !(e < 0.999f * (q2 * q2 * q));
    hnext = cap;
    if (exact) hnext = 0.9 * h * pow(errmax, -0.2);
  }
  return hnext > cap ? cap : hnext;
}

// What FP32 can say of an accretion disk's alpha test ahead of a segment
struct DiskAlpha {
  const uchar4* tex;  // null: no such disk
  int w, h;
  bool plain;         // no temperature colouring: the test draws wherever the texel is neither clear nor black
  float rms, a2;      // ISCO radius, spin squared
  float pos[3];       // the hole
};

// Whether the segment test from org along dir has to run (-1): FP32, with
// room for its rounding, may show that nothing lies within the distance
// `within` of org -- a hit further on changes nothing, but an accretion
// disk's alpha test draws from its stream wherever the line meets the disk;
// the result is then the number of draws to make (0: none).  One way through
// for all entities: a warp that leaves the loop lane by lane goes on in
// pieces, each of which pays the FP64 step again.
__device__ __forceinline__ int segment_draws(const DevScene& S, dv3 org, dv3 dir, double within, const DiskAlpha& A) {
  const float3 o = f3((float)org.x, (float)org.y, (float)org.z), d = f3((float)dir.x, (float)dir.y, (float)dir.z);
  const float mo = fmaxf(fabsf(o.x), fmaxf(fabsf(o.y), fabsf(o.z)));
  const float dl = sqrtf(dot(d, d));
  const float reach = (float)within * dl;
  const bool unit = fabsf(dl - 1.0f) < 1.0e-6f;
  int draws = 0;
  bool need = false;
  for (int i = 0; i < S.n_ents; i++) {
    const GEntF& e = S.entf[i];
    const float3 w = f3(e.p[0], e.p[1], e.p[2]) - o;
    const float mw = fmaxf(fabsf(w.x), fmaxf(fabsf(w.y), fabsf(w.z)));
    const float tol = 4.0e-6f * (2.0f * mo + mw + reach) + 1.0e-4f;
    if (e.type == PR_ENT_SPHERE) {
      // | |w| - r | > reach + tol, squared: no root.  The test's quadratic has
      // |d| = 1: with another length its roots are not where the line meets the
      // sphere, and a length off by e (FP32 cannot tell 1e-6) moves them by up
      // to sqrt(2 e) of the segment, where the line goes through a small sphere
      const float r = e.radius_eps, q = 1.002f * reach + tol + 1.0e-5f * r, w2 = dot(w, w);
      const float hi = r + q, lo = fmaxf(r - q, 0.0f);
      need = need || !unit || !(w2 > hi * hi * 1.00001f || w2 < lo * lo * 0.99999f);
    } else if (e.type == PR_ENT_UVPLANE || e.type == PR_ENT_CIRCLE) {
      const float3 n = f3(e.n[0], e.n[1], e.n[2]);
      const float nl = sqrtf(dot(n, n)), num = dot(w, n), den = dot(d, n);
      if (e.type == PR_ENT_CIRCLE && A.tex && e.node_base) {
        const float t = num / den, te = 1.1f * (tol * nl + fabsf(t) * 4.0e-6f * dl * nl) / fabsf(den);
        const float3 q = d * t - w;   // the line's point in the disk's plane, from its centre
        const float r = sqrtf(dot(q, q)), re = 1.1f * te * dl + tol + 4.0e-6f * fabsf(t) * dl;
        // the texel as the disk's map finds it (kerr_disk_texel): its angle's
        // cosine and sine are v and u over their length, u and v along the
        // disk's axes over their lengths
        const float3 x = o + d * t - f3(A.pos[0], A.pos[1], A.pos[2]);
        const float x2 = dot(x, x), c = x2 - A.a2;
        const float sr = sqrtf(0.5f * (c + sqrtf(c * c + 4.0f * A.a2 * x.z * x.z)));
        const float rn = (sr - A.rms) / (e.u_length - A.rms);
        const float u = dot(q, f3(e.u[0], e.u[1], e.u[2])), v = dot(q, f3(e.v[0], e.v[1], e.v[2]));
        const float li = rsqrtf(u * u + v * v);
        const float se = 4.0f * re + 1.0e-4f;  // of sr
        // relative error of u and v: that of the point over the axes' scale
        const float ue = re * (fabsf(e.u[0]) + fabsf(e.u[1]) + fabsf(e.u[2]) + fabsf(e.v[0]) + fabsf(e.v[1]) + fabsf(e.v[2]));
        const float fe = 1.0e-4f + 2.0f * (se / (e.u_length - A.rms) + fabsf(rn) * (ue * li + 1.0e-5f));
        const float fx = A.w * (0.5f + rn * v * li), fy = A.h * (0.5f + rn * u * li);
        const float ex = fe * A.w, ey = fe * A.h;
        const bool steep = nl > 0.5f && fabsf(den) > 1.0e-3f * dl;
        // no draw: the plane behind, beside the annulus, inside the ISCO, or off the texture
        const bool none = steep && (t + te < 0.0f || r - re > e.u_length || r + re < e.v_length || sr + se < A.rms ||
                                    fx + ex < -1.0f || fy + ey < -1.0f || fx - ex > A.w || fy - ey > A.h);
        // a draw or a clear or black texel, for certain and beyond the segment
        const bool texel = steep && A.plain && t - te > (float)within && r + re < e.u_length && r - re > e.v_length &&
                           sr - se > A.rms && sr + se < e.u_length && fx - ex > 0.0f && fy - ey > 0.0f &&
                           fx + ex < A.w && fy + ey < A.h && (int)(fx - ex) == (int)(fx + ex) &&
                           (int)(fy - ey) == (int)(fy + ey);
        if (texel && !none) {
          const uchar4 tx = A.tex[(size_t)(int)fy * A.w + (int)fx];
          // alpha = min(a, |colour| / 3) of a colour in 0..1 stays below 0.99
          draws += (tx.w != 0 && (tx.x | tx.y | tx.z) != 0) ? 1 : 0;
        }
        need = need || !(none || texel);
      } else {
        const bool off = fabsf(num) > (reach + tol) * nl && nl > 0.5f;
        const float rr = e.u_length + reach + tol;
        need = need || !(off || (e.type == PR_ENT_CIRCLE && dot(w, w) > rr * rr * 1.00001f));
      }
    } else if (e.type == PR_ENT_POLYGON) {
      // distance to the mesh's bounds along the farthest axis
      const float far = fmaxf(fmaxf(fmaxf(e.u[0] - o.x, o.x - e.v[0]), fmaxf(e.u[1] - o.y, o.y - e.v[1])),
                              fmaxf(e.u[2] - o.z, o.z - e.v[2]));
      need = need || !(far > reach + tol);
    }
  }
  return need ? -1 : draws;
}

// The rays of a warp, 32 at a time.  job: take (a lane's next ray, if any; all
// lanes call it), step (one step of the lanes that run; all lanes call it;
// true where a ray has ended) and ended (true if the lane goes on with
// another ray).  New rays start once all 32 have ended: a start, an exact
// segment test or a retried step costs the FP64 pipe as much with one lane
// active as with 32, and neighbouring rays come to them together.  (Measured
// on the 512x256 accretion frames: refilling the warp at 4 / 8 / 16 / 32
// waiting lanes 176 / 165 / 154 / 145 ms.)
template <class J>
__device__ __forceinline__ void geodesic_warp(J& job) {
  bool busy = false;
  for (;;) {
    const bool want = !busy && job.more;
    if (__ballot_sync(0xffffffffu, want)) busy = job.take(want) || busy;
    if (!__ballot_sync(0xffffffffu, busy)) {
      if (!__ballot_sync(0xffffffffu, job.more)) break;
      continue;
    }
    bool over = false;  // the lane's trace has ended
    while (__ballot_sync(0xffffffffu, busy && !over)) {
      if (job.step(busy && !over)) over = true;
      __syncwarp();
    }
    if (over) busy = job.ended();
    __syncwarp();
  }
}

// Blocks of 128 threads for n rays: a warp per scheduler (four per SM) keeps
// the FP64 pipe busy, and full warps count for more than many; with rays to
// spare two warps per scheduler fill in for each other's other work.
inline unsigned int geodesic_blocks(unsigned long long n, int sms) {
  const unsigned long long want = (n + 127) / 128, one = (unsigned long long)sms;
  const unsigned long long most = n >= 2ull * sms * 256 ? 2 * one : one;
  return (unsigned int)(want < most ? want : most);
}

}  // namespace
}  // namespace pr
