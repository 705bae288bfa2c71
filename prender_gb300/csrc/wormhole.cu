// Wormhole geodesics in FP64 (WormHole.h, scene.cpp:735-925): the Dneg
// wormhole of James, von Tunzelmann, Franklin and Thorne ("Visualizing
// Interstellar's wormhole", Am. J. Phys. 83, 2015) -- radius r(l), the
// geodesic equations (A7) from the initial conditions (A9) in a frame whose
// x axis points from the ray's mouth to the camera, Cash-Karp RK45 with the
// reference's step control, and a straight-segment scene test per step.
// This translation unit is compiled with -fmad=false: every FP64 multiply
// and add rounds on its own in the reference's order (CUDA's sin / cos /
// atan / log / acos may differ from the host libm in the last bit; the
// tests bound the effect on exit directions).
#include "device_common.cuh"
#include "geodesic_math.cuh"
#include "path_logic.cuh"
#include "wormhole.h"

namespace pr {
namespace {

constexpr double kWPi = 3.14159265358979323846264338327950288;

// Cartesian::ToSpherical (vector3d.h:913-939)
__device__ __forceinline__ void w_to_sph(double x, double y, double z, double& r, double& th, double& ph) {
  r = sqrt(x * x + y * y + z * z);
  if (!(r > 1.0e-16)) {
    th = 0;
    ph = 0;
    return;
  }
  const double xx = x / r, yy = y / r, zz = z / r;
  th = acos(zz < -1.0 ? -1.0 : (zz > 1.0 ? 1.0 : zz));
  double phi;
  if (fabs(xx) < 1.0e-6 && fabs(yy) < 1.0e-6) phi = 0.0;
  else phi = atan2(yy, xx);
  if (phi < 0.0) phi += 2.0 * kWPi;
  if (phi >= 2.0 * kWPi) phi = 0.0;
  ph = phi;
}

// Spherical::ToCartesian (vector3d.h:879-887)
__device__ __forceinline__ dv3 w_to_cart(double r, double sint, double cost, double ph) {
  double sinp, cosp;
  sincos(ph, &sinp, &cosp);
  return {r * cosp * sint, r * sinp * sint, r * cost};
}
__device__ __forceinline__ dv3 w_to_cart(double r, double th, double ph) {
  double sint, cost;  // sincos gives the bits of sin and of cos
  sincos(th, &sint, &cost);
  return w_to_cart(r, sint, cost, ph);
}

// Matrix4D * Vector3d (vector3d.h:760-768): the upper 3x3 block
__device__ __forceinline__ dv3 w_mul(const double* m, dv3 v) {
  return {v.x * m[0] + v.y * m[1] + v.z * m[2], v.x * m[4] + v.y * m[5] + v.z * m[6],
          v.x * m[8] + v.y * m[9] + v.z * m[10]};
}

__device__ __forceinline__ dv3 w_normalize(dv3 v) {  // normalize (vector3d.h:162-165)
  const double il = 1.0 / sqrt((v.x * v.x + v.z * v.z) + v.y * v.y);
  return {v.x * il, v.y * il, v.z * il};
}

struct WormRay {
  const GWorm* W;
  const double* mat;  // the frame of the ray's mouth
  const double* inv;
  double l0, theta0, phi0, n_l, n_ph, n_th;
  double b, B2;  // the ray's constants of motion

  __device__ __forceinline__ double r_wh(double l) const {  // WormHole.h:172-180
    const double x = 2.0 * (fabs(l) - W->a) / (kWPi * W->M);
    if (fabs(l) > W->a) return W->Rho + W->M * (x * atan(x) - 0.5 * log(1.0 + x * x));
    return W->Rho;
  }
  // r(l) and dr/dl (:172-193) together: both take the arctangent of the same
  // value (2 (|l| - a) / (pi M), the reference's two spellings of which round alike)
  __device__ __forceinline__ void r_drdl(double l, double& r, double& dr) const {
    if (fabs(l) > W->a) {
      const double x = 2.0 * (fabs(l) - W->a) / (kWPi * W->M);
      const double at = atan(x);
      r = W->Rho + W->M * (x * at - 0.5 * log(1.0 + x * x));
      double sg = 1;
      if (l < 0) sg = -1;
      if (l == 0.0) sg = 0.0;
      dr = (2.0 * at * sg) / kWPi;
    } else {
      r = W->Rho;
      dr = 0;
    }
  }
  // :195-238: Newton's method on r(l) = r from the start point, then from a
  __device__ double rtol(double r, double linit) const {
    const double M = W->M, Rho = W->Rho;
    double x = 2.0 * (fabs(linit) - W->a) / (kWPi * M);
    int stat = -1;
    for (int i = 0; i < 30; i++) {
      const double xi = x;
      x = x - (Rho + M * (x * atan(x) - 0.5 * log(1.0 + x * x)) - r) / (M * atan(x));
      if (fabs(x - xi) < 1.0e-6) {
        stat = 0;
        break;
      }
      if (!isfinite(x)) break;
    }
    double l = x * kWPi * M * 0.5 + W->a;
    if (stat != 0) {
      x = W->a;
      for (int i = 0; i < 30; i++) {
        const double xi = x;
        x = x - (Rho + M * (x * atan(x) - 0.5 * log(1.0 + x * x)) - r) / (M * atan(x));
        if (fabs(x - xi) < 1.0e-6) {
          l = x * kWPi * M * 0.5 + W->a;
          break;
        }
        if (!isfinite(x)) break;
      }
    }
    return (linit < 0) ? -fabs(l) : fabs(l);
  }
  // Setup + initial (WormHole.h:321-428)
  __device__ void start(dv3 org, dv3 dir, double sgn, double* y) {
    const int m = sgn >= 0 ? 0 : 1;
    mat = W->mat[m];
    inv = W->inv[m];
    double pr, pth, pph;
    w_to_sph(org.x - W->pos[m][0], org.y - W->pos[m][1], org.z - W->pos[m][2], pr, pth, pph);
    const dv3 q = w_mul(mat, w_to_cart(pr, pth, pph));
    double qr;
    w_to_sph(q.x, q.y, q.z, qr, theta0, phi0);
    l0 = rtol(qr, sgn * W->a / 2);
    double dr, dth, dph;
    w_to_sph(dir.x, dir.y, dir.z, dr, dth, dph);
    const dv3 rc = w_mul(mat, w_to_cart(dr, dth, dph));
    double rr, th, ph;
    w_to_sph(rc.x, rc.y, rc.z, rr, th, ph);
    const double sint = sin(th);
    const double Nx = sint * cos(ph), Ny = sint * sin(ph), Nz = cos(th);
    n_l = -Nx;
    n_ph = -Ny;
    n_th = Nz;
    y[0] = l0;
    y[1] = theta0;
    y[2] = phi0;
    y[3] = n_l;
    const double r_l0 = r_wh(l0);
    y[4] = r_l0 * n_th;
    b = r_l0 * sin(theta0) * n_ph;
    B2 = r_l0 * r_l0 * (n_th * n_th + n_ph * n_ph);
  }
  // geodesic (WormHole.h:462-488): (A7), with r(l), dr/dl and sin and cos of
  // theta at y given.  b and B2 do not change along the ray: recomputing them
  // in every evaluation (an arctangent, a logarithm and a sine) and r, dr/dl
  // and the sines per use took more than half of the kernel's FP64 work (128x96
  // x 4 spp frame: 192 -> 122 ms with the shared set-up of each step).
  __device__ __forceinline__ void geodesic(const double* y, double r, double dr, double sint, double cost,
                                           double* dydx) const {
    const double r2 = r * r;
    if (fabs(sint) < 1.0e-8) sint = sint > 0.0 ? 1.0e-8 : -1.0e-8;
    const double sint2 = sint * sint;
    const double invr2 = 1.0 / r2;
    dydx[0] = y[3];
    dydx[1] = y[4] * invr2;
    dydx[2] = b * invr2 / sint2;
    dydx[3] = B2 * dr * invr2 / r;
    dydx[4] = (b * b * invr2) * (cost / (sint * sint2));
  }
  __device__ __forceinline__ void geodesic(const double* y, double* dydx) const {
    double r, dr, sint, cost;
    r_drdl(y[0], r, dr);
    sincos(y[1], &sint, &cost);
    geodesic(y, r, dr, sint, cost, dydx);
  }
  // rkstep (WormHole.h:541-612): Cash-Karp, the step negated (traceDir 1)
  __device__ __forceinline__ void rkstep(const double* y, const double* dydx, double h, double* yout, double* yerr) const {
    double ak[5], t1[5], t2[5], t3[5], t4[5], t5[5];
    h *= -1.0;
#pragma unroll
    for (int i = 0; i < 5; i++) {
      const double hd = h * dydx[i], yi = y[i];
      t1[i] = yi + 0.2 * hd;
      t2[i] = yi + (3.0 / 40.0) * hd;
      t3[i] = yi + 0.3 * hd;
      t4[i] = yi - (11.0 / 54.0) * hd;
      t5[i] = yi + (1631.0 / 55296.0) * hd;
      yout[i] = yi + (37.0 / 378.0) * hd;
      yerr[i] = ((37.0 / 378.0) - (2825.0 / 27648.0)) * hd;
    }
    geodesic(t1, ak);
#pragma unroll
    for (int i = 0; i < 5; i++) {
      const double yt = h * ak[i];
      t2[i] += (9.0 / 40.0) * yt;
      t3[i] -= 0.9 * yt;
      t4[i] += 2.5 * yt;
      t5[i] += (175.0 / 512.0) * yt;
    }
    geodesic(t2, ak);
#pragma unroll
    for (int i = 0; i < 5; i++) {
      const double yt = h * ak[i];
      t3[i] += 1.2 * yt;
      t4[i] -= (70.0 / 27.0) * yt;
      t5[i] += (575.0 / 13824.0) * yt;
      yout[i] += (250.0 / 621.0) * yt;
      yerr[i] += ((250.0 / 621.0) - (18575.0 / 48384.0)) * yt;
    }
    geodesic(t3, ak);
#pragma unroll
    for (int i = 0; i < 5; i++) {
      const double yt = h * ak[i];
      t4[i] += (35.0 / 27.0) * yt;
      t5[i] += (44275.0 / 110592.0) * yt;
      yout[i] += (125.0 / 594.0) * yt;
      yerr[i] += ((125.0 / 594.0) - (13525.0 / 55296.0)) * yt;
    }
    geodesic(t4, ak);
#pragma unroll
    for (int i = 0; i < 5; i++) {
      const double yt = h * ak[i];
      t5[i] += (253.0 / 4096.0) * yt;
      yerr[i] -= (277.0 / 14336.0) * yt;
    }
    geodesic(t5, ak);
#pragma unroll
    for (int i = 0; i < 5; i++) {
      const double yt = h * ak[i];
      yout[i] += (512.0 / 1771.0) * yt;
      yerr[i] += ((512.0 / 1771.0) - 0.25) * yt;
    }
  }
  // NextPosition + rkqs (WormHole.h:490-535, :618-683): at most 2000
  // shrinks; returns the next step, at most cap
  __device__ __forceinline__ double next_position(double* y, const double* dydx, double htry, double cap, uint32_t& attempts) const {
    const double escal = 1e11;
    double yscal[5], ytemp[5], yerr[5];
#pragma unroll
    for (int i = 0; i < 5; i++) yscal[i] = fabs(y[i]) + fabs(dydx[i] * htry) + 1.0e-3;
    double h = htry, errmax = 0.0;
    for (int loops = 0; loops < 2000; loops++) {
      attempts++;
      rkstep(y, dydx, h, ytemp, yerr);
      errmax = max_ratio<5>(yerr, yscal);
      errmax *= escal;
      if (errmax <= 1.0) break;
      const double htemp = 0.9 * h / sqrt(sqrt(errmax));
      h *= 0.1;
      if (h >= 0.0) {
        if (htemp > h) h = htemp;
      } else {
        if (htemp < h) h = htemp;
      }
    }
    const double hnext = next_step(h, errmax, cap);
#pragma unroll
    for (int i = 0; i < 5; i++) y[i] = ytemp[i];
    return hnext;
  }
  __device__ __forceinline__ dv3 world(dv3 q, double sgn) const {  // WorldAxisSystem (WormHole.h:430-447)
    const dv3 p = w_mul(inv, q);
    const int m = sgn >= 0 ? 0 : 1;
    return {p.x + W->pos[m][0], p.y + W->pos[m][1], p.z + W->pos[m][2]};
  }
};

struct WormHit {
  int status;  // 1 entity hit, 0 background 1, 3 background 2
  int steps, ent, prim;
  double t;
  dv3 seg_o, dir2;
};

struct WormCount {
  uint32_t steps, attempts, segments;
  uint64_t nodes, tris;
};

// the state of one ray between the steps of intersect_scene__'s loop (scene.cpp:735-925)
struct WormMarch {
  WormRay k;
  double y[5];
  double r, dr, sint, cost;  // r(l), dr/dl, sin and cos of theta at y
  double h_dist, h_step;
  dv3 org1, org2, dir2;      // the polyline's last vertices and direction
  int c;                     // accepted steps
};

__device__ __forceinline__ void worm_start(const GWorm& W, dv3 org, dv3 dir, WormMarch& M, WormHit& out) {
  M.k.W = &W;
  const double sign = sqrt((org.x * org.x + org.z * org.z) + org.y * org.y) > 1000000 ? -1.0 : 1.0;
  M.k.start(org, dir, sign, M.y);
  out.ent = -1;
  out.prim = -1;
  out.t = -1.0;
  M.k.r_drdl(M.y[0], M.r, M.dr);
  sincos(M.y[1], &M.sint, &M.cost);
  M.h_dist = 0.5;
  if (fabs(M.y[0]) < W.a || M.r <= W.Rho) M.h_dist = M.h_dist * 0.15;
  M.h_step = M.h_dist;
  M.org1 = M.org2 = org;
  M.dir2 = dir;
  M.c = 0;
}

// One pass of the loop for the lanes that run (all lanes of the warp call it
// and come together again after the segment test, which few of them need);
// true when the ray's trace has ended
__device__ __forceinline__ bool worm_step(const DevScene& S, const GWorm& W, WormMarch& M, WormHit& out,
                                          WormCount& cnt, uint32_t* err, bool run) {
  bool leave = false, hit = false;
  if (run)
    leave = !(W.max_steps < 0 ? true : M.c < W.max_steps) || fabs(M.y[0]) > 1.0e10 || fabs(M.r) > 1.0e10 ||
            !isfinite(M.y[0]);
  double t = 0.0;
  int ent = -1, prim = -1;
  const bool look = run && !leave;
  cnt.segments += look ? 1u : 0u;
  // all lanes or none: the FP64 test costs the same for one lane as for 32, and
  // a warp that parts here goes on in pieces for the rest of the step, each of
  // which pays the step's FP64 instructions (the 128x96 x 4 spp frame takes 157
  // ms with a branch here, 122 with the vote)
  if (__any_sync(0xffffffffu, look && segment_draws(S, M.org1, M.dir2, M.h_dist, DiskAlpha{}) < 0))
    hit = look && exact_closest(S, M.org1, M.dir2, t, ent, prim, err, cnt.nodes, cnt.tris) && t < M.h_dist;
  __syncwarp();
  if (hit) {
    out.status = 1;
    out.steps = M.c;
    out.ent = ent;
    out.prim = prim;
    out.t = t;
    out.seg_o = M.org1;
    out.dir2 = M.dir2;
  } else if (run && !leave) {
    double dydx[5];
    M.k.geodesic(M.y, M.r, M.dr, M.sint, M.cost, dydx);
    if (fabs(M.h_step) < 1.0e-14) M.h_step = 1.0e-14;
    M.h_step = M.k.next_position(M.y, dydx, M.h_step, M.h_dist, cnt.attempts);
    M.org1 = M.org2;
    M.k.r_drdl(M.y[0], M.r, M.dr);
    sincos(M.y[1], &M.sint, &M.cost);
    M.org2 = M.k.world(w_to_cart(M.r, M.sint, M.cost, M.y[2]), M.y[0]);
    M.dir2 = w_normalize({M.org2.x - M.org1.x, M.org2.y - M.org1.y, M.org2.z - M.org1.z});
    M.c++;
    cnt.steps++;
  } else if (leave) {
    if (W.usr_sign) M.y[0] = W.usr_sign * M.y[0];
    double dr;
    w_to_sph(M.dir2.x, M.dir2.y, M.dir2.z, dr, M.y[1], M.y[2]);
    out.status = M.y[0] >= 0 ? 0 : 3;
    out.steps = M.c;
    out.seg_o = M.org2;
    out.dir2 = M.dir2;
  }
  __syncwarp();
  return hit || leave;
}

// the colour of a ray that ended on a background (scene.cpp:860-920 +
// SphericalMapping::Map, circle.h:92-105)
__device__ float3 worm_background(const GWorm& W, int side, const double* yy, const float* bg) {
  if (!W.tex[side]) return f3(bg[0], bg[1], bg[2]);
  double y1 = yy[1] * W.map_coef[side][0] + W.map_coef[side][1];
  double y2 = yy[2] * W.map_coef[side][2] + W.map_coef[side][3];
  y1 = fmod(y1, kWPi);
  y2 = fmod(y2, 2.0 * kWPi);
  double phi = y2, theta = y1;
  if (phi < 0.0) phi += 2.0 * kWPi;
  if (theta < 0.0) theta = -theta;
  if (!(phi == phi) || !(theta == theta)) return f3(0, 0, 0);
  const int tw = W.tex_w[side], th = W.tex_h[side];
  int x = (int)(phi / (2.0 * kWPi) * tw);
  x = ((x % tw) + tw) % tw;  // in range for any input, NaN included
  int yv = (int)(theta / kWPi * th);
  yv = ((yv % th) + th) % th;
  const unsigned char* t = W.tex[side] + 3 * ((size_t)yv * tw + x);
  const double c = W.tex_coef[side];
  return f3((float)(c * t[0] / 255.0), (float)(c * t[1] / 255.0), (float)(c * t[2] / 255.0));
}

struct WormTraceJob {
  const DevScene& S;
  const GWorm& W;
  const double* rays;
  int64_t n;
  const WormOut& out;
  uint32_t* err;
  WormMarch M;
  WormHit h;
  WormCount c;
  int64_t i;
  bool more;

  __device__ __forceinline__ bool take(bool want) {
    if (!want) return false;
    i += i < 0 ? (int64_t)blockIdx.x * blockDim.x + threadIdx.x + 1 : (int64_t)gridDim.x * blockDim.x;
    if (i >= n) {
      more = false;
      return false;
    }
    const double* r = rays + 6 * i;
    worm_start(W, {r[0], r[1], r[2]}, {r[3], r[4], r[5]}, M, h);
    return true;
  }
  __device__ __forceinline__ bool step(bool run) { return worm_step(S, W, M, h, c, err, run); }
  __device__ __forceinline__ bool ended() {
    if (out.status) out.status[i] = h.status;
    if (out.steps) out.steps[i] = h.steps;
    if (out.hit_entity) out.hit_entity[i] = h.status == 1 ? h.ent : -1;
    if (out.final_y)
      for (int k = 0; k < 3; k++) out.final_y[3 * i + k] = M.y[k];
    if (out.exit_dir) {
      out.exit_dir[3 * i] = h.dir2.x;
      out.exit_dir[3 * i + 1] = h.dir2.y;
      out.exit_dir[3 * i + 2] = h.dir2.z;
    }
    return false;
  }
};

__global__ void __launch_bounds__(128) worm_trace_kernel(const __grid_constant__ DevScene S,
                                                         const __grid_constant__ GWorm W,
                                                         const double* __restrict__ rays, int64_t n,
                                                         const __grid_constant__ WormOut out,
                                                         uint32_t* __restrict__ err,
                                                         unsigned long long* __restrict__ counters) {
  WormTraceJob job{S, W, rays, n, out, err};
  job.c = WormCount{0, 0, 0, 0, 0};
  job.i = -1;
  job.more = true;
  geodesic_warp(job);
  if (counters) {
    const int64_t first = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (first < n) {
      const int64_t stride = (int64_t)gridDim.x * blockDim.x;
      atomicAdd(counters + 0, (unsigned long long)((n - 1 - first) / stride + 1));
    }
    atomicAdd(counters + 1, (unsigned long long)job.c.steps);
    atomicAdd(counters + 2, (unsigned long long)job.c.attempts);
    atomicAdd(counters + 3, (unsigned long long)job.c.segments);
  }
}

// Camera samples of radiance() in a wormhole scene, one path per lane (no
// next-event estimation, no media: every query goes through the wormhole).
// Objects on the far side sit more than 1e6 from the origin (the trace picks
// the mouth by that distance), where a float has a spacing of 0.125 or more:
// the next ray starts at the hit's world position in FP64, as in the
// reference (hitpoint.position), which shade() sees as the local origin 0.
struct WormPathJob {
  const DevScene& S;
  const GWorm& W;
  const RenderCfg& cfg;
  const SamplePass& F;
  uint32_t* err;
  WormMarch M;
  WormHit h;
  WormCount c;
  PathState ps;
  unsigned long long id;
  uint32_t item;  // the pass's sample that the path is (a sample id may wrap past 2^64)
  float3 L;
  int sp;
  uint32_t paths;
  bool more;
  PathState stack[kSplitStack];
  dv3 sorg[kSplitStack];

  __device__ __forceinline__ bool take(bool want) {
    const int lane = threadIdx.x & 31;
    const unsigned int mask = __ballot_sync(0xffffffffu, want);
    const int leader = __ffs(mask) - 1;
    unsigned long long base = 0;
    if (lane == leader) base = atomicAdd(F.next, (unsigned long long)__popc(mask));
    base = __shfl_sync(0xffffffffu, base, leader);
    if (!want) return false;
    const unsigned long long g = base + (unsigned long long)__popc(mask & ((1u << lane) - 1u));
    if (g >= F.samples) {
      more = false;
      return false;
    }
    int x, y;
    uint32_t k;
    pass_sample(cfg, F, (uint32_t)g, x, y, k);
    float3 o, d;
    id = camera_ray(cfg, x, y, cfg.sample_offset + (uint64_t)k, o, d);
    item = (uint32_t)g;
    root_path(ps, o, d);
    L = f3(0, 0, 0);
    sp = 0;
    worm_start(W, {o.x, o.y, o.z}, {d.x, d.y, d.z}, M, h);
    return true;
  }

  __device__ __forceinline__ bool step(bool run) { return worm_step(S, W, M, h, c, err, run); }

  // the ray's trace ended: shade, and go on with the path's next ray or end it
  __device__ __forceinline__ bool ended() {
    FastHit fh;
    Vertex v;
    dv3 pw = {0, 0, 0};  // the hit's world position
    float3 miss = f3(0, 0, 0);
    const bool hit = h.status == 1;
    if (!hit) {
      miss = worm_background(W, h.status == 0 ? 0 : 1, M.y, S.bg);
    } else {
      const GEntity& e = S.ents[h.ent];
      const dv3 o2 = dadd3(h.seg_o, dscale3(h.dir2, 0.000001));
      const dv3 p = {o2.x + h.t * h.dir2.x, o2.y + h.t * h.dir2.y, o2.z + h.t * h.dir2.z};
      float3 n;
      if (e.type == PR_ENT_SPHERE) n = normalize(f3((float)(p.x - e.p[0]), (float)(p.y - e.p[1]), (float)(p.z - e.p[2])));
      else if (e.type == PR_ENT_POLYGON) n = ld3(S.fnorm + 3 * (size_t)(e.face_base + h.prim));
      else n = f3((float)e.normal[0], (float)e.normal[1], (float)e.normal[2]);
      if (e.normal_inverse < 0) n = -n;
      pw = p;
      v.p = f3(0, 0, 0);  // relative to pw
      v.n = n;
      v.ent = h.ent;
      v.mat = e.material;
      v.t = (float)h.t;
      fh.t = (float)h.t;
      fh.ent = h.ent;
      fh.slot = -1;
      fh.u = fh.v = 0.0f;
    }
    ShadowReq sh[3];
    int nsh = 0;
    PathState child;
    const int r = shade(S, cfg, ps, hit, fh, id, sh, nsh, child, err, &v, &miss);
    if (r == SHADE_SPLIT) {
      if (sp < kSplitStack) {
        stack[sp] = child;
        sorg[sp++] = pw;
      } else {
        atomicOr(err, PR_DEV_LOOP_CAP);
      }
    }
    if (r == SHADE_END) {
      L += ps.L;
      if (sp == 0) {
        F.sample[item] = finish_sample(cfg, L, err);
        paths++;
        return false;
      }
      --sp;
      ps = stack[sp];
      pw = sorg[sp];
    }
    worm_start(W, pw, {ps.d.x, ps.d.y, ps.d.z}, M, h);
    return true;
  }
};

__global__ void __launch_bounds__(128) worm_render_kernel(const __grid_constant__ DevScene S,
                                                          const __grid_constant__ GWorm W,
                                                          const __grid_constant__ RenderCfg cfg,
                                                          const __grid_constant__ SamplePass F,
                                                          uint32_t* __restrict__ err,
                                                          unsigned long long* __restrict__ counters) {
  WormPathJob job{S, W, cfg, F, err};
  job.c = WormCount{0, 0, 0, 0, 0};
  job.sp = 0;
  job.paths = 0;
  job.more = true;
  geodesic_warp(job);
  if (counters) {
    unsigned long long a = job.paths, b = job.c.segments, nn = job.c.nodes, tt = job.c.tris;
    for (int off = 16; off > 0; off >>= 1) {
      a += __shfl_down_sync(0xffffffffu, a, off);
      b += __shfl_down_sync(0xffffffffu, b, off);
      nn += __shfl_down_sync(0xffffffffu, nn, off);
      tt += __shfl_down_sync(0xffffffffu, tt, off);
    }
    if ((threadIdx.x & 31) == 0) {
      atomicAdd(counters + 0, a);
      atomicAdd(counters + 1, b);
      atomicAdd(counters + 2, nn);
      atomicAdd(counters + 3, tt);
    }
  }
}

}  // namespace

cudaError_t launch_worm_trace(const DevScene& S, const GWorm& W, const double* rays, int64_t n, WormOut out,
                              uint32_t* err, unsigned long long* counters, cudaStream_t stream) {
  if (n <= 0) return cudaSuccess;
  worm_trace_kernel<<<geodesic_blocks((unsigned long long)n, sm_count()), 128, 0, stream>>>(S, W, rays, n, out, err,
                                                                                        counters);
  return cudaGetLastError();
}

size_t worm_scratch_bytes(const RenderCfg& cfg) { return pass_bytes(cfg); }

cudaError_t launch_worm_render(const DevScene& S, const GWorm& W, const RenderCfg& cfg, void* scratch, float* dst,
                               int accumulate, uint32_t* err, unsigned long long* counters, cudaStream_t stream) {
  for (unsigned long long k = 0, passes = pass_count(cfg); k < passes; k++) {
    SamplePass F;
    cudaError_t e = sample_pass(cfg, scratch, k, F, stream);
    if (e != cudaSuccess) return e;
    worm_render_kernel<<<geodesic_blocks(F.samples, sm_count()), 128, 0, stream>>>(S, W, cfg, F, err, counters);
    e = cudaGetLastError();
    if (e == cudaSuccess) e = launch_sum(cfg, F, dst, accumulate, stream);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

}  // namespace pr
