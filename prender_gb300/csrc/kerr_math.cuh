// Kerr geodesic tracer shared by the FP64 form (kerr.cu, compiled without
// FMA contraction) and the FP32 form (kerr_fast.cu): the Kerr branch of
// intersect_scene (scene.cpp:448-732) with KerrBlackHole's set-up,
// closed-form initial momenta (initial_condition 0), geodesic equations and
// Cash-Karp RK45 step control (KerrBlackHole.h:86-151, :310-440, :471-522,
// :660-852, :1239-1431).
//
// One thread traces one ray.  Each accepted RK step is followed by a
// straight-segment scene test from the previous polyline vertex.  All loops
// are bounded: at most max_steps steps per ray and 40 step-size retries per
// step.
#pragma once
#include <cuda_runtime.h>

#include "geodesic_math.cuh"
#include "kerr.h"
#include "path_logic.cuh"

namespace pr {
namespace {


constexpr double kPi = 3.14159265358979323846;
constexpr double kTwoPi = 6.28318530717958647692;

__device__ __forceinline__ double kclamp(double v, double lo, double hi) {  // Clamp (vector3d.h:236)
  if (v < lo) return lo;
  else if (v > hi) return hi;
  else return v;
}

// Cartesian::ToBoyerLindquist (vector3d.h:941-951)
__device__ __forceinline__ void cart_to_bl(double x, double y, double z, double a, double& r, double& th, double& ph) {
  double r0 = x * x + y * y + z * z;
  const double u = r0 - a * a;
  const double zz = 2. * a * z;
  r0 = sqrt((u + sqrt(u * u + zz * zz)) / 2.);
  th = acos(kclamp(z / r0, -1.0, 1.0));
  double phi = atan2(y / r0, x / r0);
  if (phi < 0.0) phi += kTwoPi;
  if (phi >= kTwoPi) phi = 0.0;
  r = r0;
  ph = phi;
}

// Spherical::ToBoyerLindquist (vector3d.h:888-898): BL (r, theta, phi) ->
// Cartesian.  (sincos gives the bits of sin and of cos for two thirds of the
// FP64 instructions of both.)
__device__ __forceinline__ dv3 bl_to_cart(double r, double sint, double cost, double ph, double a) {
  const double rr = sqrt(r * r + a * a);
  double sinp, cosp;
  sincos(ph, &sinp, &cosp);
  return {rr * cosp * sint, rr * sinp * sint, r * cost};
}
__device__ __forceinline__ dv3 bl_to_cart(double r, double th, double ph, double a) {
  double sint, cost;
  sincos(th, &sint, &cost);
  return bl_to_cart(r, sint, cost, ph, a);
}

// Cartesian::ToSpherical (vector3d.h:900-918), angles only
__device__ __forceinline__ void cart_to_sph(double x, double y, double z, double& th, double& ph) {
  const double r = sqrt(x * x + y * y + z * z);
  double xx, yy, zz;
  if (r > 1.0e-16) {
    xx = x / r;
    yy = y / r;
    zz = z / r;
  } else {
    th = 0;
    ph = 0;
    return;
  }
  th = acos(kclamp(zz, -1.0, 1.0));
  double phi;
  if (fabs(xx) < 1.0e-6 && fabs(yy) < 1.0e-6) phi = 0.0;
  else phi = atan2(yy, xx);
  if (phi < 0.0) phi += 2.0 * kPi;
  if (phi >= 2.0 * kPi) phi = 0.0;
  ph = phi;
}

__device__ __forceinline__ dv3 dnormalize(dv3 v) {  // normalize (vector3d.h): v * (1 / |v|)
  const double l = sqrt((v.x * v.x + v.z * v.z) + v.y * v.y);
  const double il = 1.0 / l;
  return {v.x * il, v.y * il, v.z * il};
}

struct KerrRay {
  double a, a2, M;
  double L, kappa;

  // geodesic (KerrBlackHole.h:1239-1281); the second form is given sin and cos of theta
  __device__ __forceinline__ void geodesic(const double* y, double* dydx) const {
    double sintheta, costheta;
    sincos(y[1], &sintheta, &costheta);
    geodesic(y, sintheta, costheta, dydx);
  }
  __device__ __forceinline__ void geodesic(const double* y, double sintheta, double costheta, double* dydx) const {
    const double r = y[0];
    const double pr = y[4];
    const double ptheta = y[5];
    const double r2 = r * r;
    const double twor = 2.0 * M * r;
    double sin2 = sintheta * sintheta;
    const double cos2 = costheta * costheta;
    const double sigma = r2 + a2 * cos2;
    const double delta = r2 - twor + a2;
    const double sd = sigma * delta;
    const double siginv = 1.0 / sigma;
    const double bot = 1.0 / sd;
    if (fabs(sin2) < 1.0e-16) {
      if (sin2 < 0.0) sin2 = -1.0e-16;
      else sin2 = 1.0e-16;
    }
    dydx[0] = -pr * delta * siginv;
    dydx[1] = -ptheta * siginv;
    dydx[2] = -(twor * a + (sigma - twor) * L / sin2) * bot;
    dydx[3] = -(1.0 + (twor * (r2 + a2) - twor * a * L) * bot);
    dydx[4] = -(((r - 1.0) * (-kappa) + twor * (r2 + a2) - 2.0 * a * L) * bot - 2.0 * pr * pr * (r - 1.0) * siginv);
    dydx[5] = -sintheta * costheta * (L * L / (sin2 * sin2) - a2) * siginv;
  }

  // rkstep (KerrBlackHole.h:1288-1361), traceDir = +1
  __device__ __forceinline__ void rkstep(const double* y, const double* dydx, double h, double* yout,
                                         double* yerr) const {
    double ak[6], t1[6], t2[6], t3[6], t4[6], t5[6];
    h *= 1.0;
#pragma unroll
    for (int i = 0; i < 6; i++) {
      const double hdydx = h * dydx[i];
      const double yi = y[i];
      t1[i] = yi + 0.2 * hdydx;
      t2[i] = yi + (3.0 / 40.0) * hdydx;
      t3[i] = yi + 0.3 * hdydx;
      t4[i] = yi - (11.0 / 54.0) * hdydx;
      t5[i] = yi + (1631.0 / 55296.0) * hdydx;
      yout[i] = yi + (37.0 / 378.0) * hdydx;
      yerr[i] = ((37.0 / 378.0) - (2825.0 / 27648.0)) * hdydx;
    }
    geodesic(t1, ak);
#pragma unroll
    for (int i = 0; i < 6; i++) {
      const double yt = h * ak[i];
      t2[i] += (9.0 / 40.0) * yt;
      t3[i] -= 0.9 * yt;
      t4[i] += 2.5 * yt;
      t5[i] += (175.0 / 512.0) * yt;
    }
    geodesic(t2, ak);
#pragma unroll
    for (int i = 0; i < 6; i++) {
      const double yt = h * ak[i];
      t3[i] += 1.2 * yt;
      t4[i] -= (70.0 / 27.0) * yt;
      t5[i] += (575.0 / 13824.0) * yt;
      yout[i] += (250.0 / 621.0) * yt;
      yerr[i] += ((250.0 / 621.0) - (18575.0 / 48384.0)) * yt;
    }
    geodesic(t3, ak);
#pragma unroll
    for (int i = 0; i < 6; i++) {
      const double yt = h * ak[i];
      t4[i] += (35.0 / 27.0) * yt;
      t5[i] += (44275.0 / 110592.0) * yt;
      yout[i] += (125.0 / 594.0) * yt;
      yerr[i] += ((125.0 / 594.0) - (13525.0 / 55296.0)) * yt;
    }
    geodesic(t4, ak);
#pragma unroll
    for (int i = 0; i < 6; i++) {
      const double yt = h * ak[i];
      t5[i] += (253.0 / 4096.0) * yt;
      yerr[i] -= (277.0 / 14336.0) * yt;
    }
    geodesic(t5, ak);
#pragma unroll
    for (int i = 0; i < 6; i++) {
      const double yt = h * ak[i];
      yout[i] += (512.0 / 1771.0) * yt;
      yerr[i] += ((512.0 / 1771.0) - 0.25) * yt;
    }
  }

  // NextPosition + rkqs (KerrBlackHole.h:471-522, :1366-1431): one accepted
  // step from y (escal 1e11, at most 40 shrinking retries); returns the next
  // step, at most cap
  __device__ __forceinline__ double next_position(double* y, const double* dydx, double htry, double cap,
                                                  uint32_t& attempts, double* errmax_out = nullptr) const {
    double yscal[6];
#pragma unroll
    for (int i = 0; i < 6; i++) yscal[i] = fabs(y[i]) + fabs(dydx[i] * htry) + 1.0e-3;
    const double escal = 1e11;
    double errmax = 0.0, h = htry;
    double yerr[6], ytemp[6];
    for (int loop = 0; loop < 40; loop++) {
      rkstep(y, dydx, h, ytemp, yerr);
      attempts++;
      errmax = max_ratio<6>(yerr, yscal);
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
    if (errmax_out) *errmax_out = errmax;
#pragma unroll
    for (int i = 0; i < 6; i++) y[i] = ytemp[i];
    return hnext;
  }

  // initial2 (KerrBlackHole.h:310-440): momenta, L and kappa from (rdot, thetadot, phidot)
  __device__ __forceinline__ void initial2(double* y0, double* ydot0, double r0, double theta0) {
    y0[3] = 0;
    y0[4] = 0;
    y0[5] = 0;
    double sintheta = sin(theta0);
    const double costheta = cos(theta0);
    const double cos2 = costheta * costheta;
    double sin2 = sintheta * sintheta;
    const double POLE_THRESHOLD = 1e-8;
    if (sin2 < POLE_THRESHOLD * POLE_THRESHOLD) {
      const double sigma = r0 * r0 + a2;
      const double delta = r0 * r0 - 2.0 * M * r0 + a2;
      const double vphi_sin = ydot0[2] * sintheta;
      const double rdot0 = ydot0[0];
      const double thetadot0 = ydot0[1];
      const double energy2 =
          (sigma - 2.0 * r0) * (rdot0 * rdot0 / delta + thetadot0 * thetadot0) + delta * vphi_sin * vphi_sin;
      const double energy = sqrt(fabs(energy2)) + 1e-10;
      y0[4] = rdot0 * sigma / delta / energy;
      y0[5] = thetadot0 * sigma / energy;
      L = 0.0;
      kappa = y0[5] * y0[5] + a2 * sin2;
    } else {
      if (sin2 < 1e-16) {
        sintheta = 1e-16;
        sin2 = 1e-32;
      }
      const double rdot0 = ydot0[0];
      const double thetadot0 = ydot0[1];
      const double r2 = r0 * r0;
      const double sigma = r2 + a2 * cos2;
      const double delta = r2 - 2.0 * M * r0 + a2;
      const double s1 = sigma - 2.0 * r0;
      y0[4] = rdot0 * sigma / delta;
      y0[5] = thetadot0 * sigma;
      const double phidot0 = ydot0[2];
      const double energy2 = s1 * (rdot0 * rdot0 / delta + thetadot0 * thetadot0) + delta * sin2 * phidot0 * phidot0;
      const double energy = sqrt(fabs(energy2)) + 1.0e-10;
      y0[4] = y0[4] / energy;
      y0[5] = y0[5] / energy;
      L = ((sigma * delta * phidot0 - 2.0 * a * r0 * energy) * sin2 / s1) / energy;
      kappa = y0[5] * y0[5] + a2 * sin2 + L * L / sin2;
    }
    geodesic(y0, ydot0);
  }

  // RayToOrdinaryDifferentialEquationInitial, initial_condition 0 (KerrBlackHole.h:720-852)
  __device__ __forceinline__ void initial(dv3 dir, double* y, double* dydx, double r0, double theta0) {
    y[3] = 0;
    y[4] = 0;
    y[5] = 0;
    const double r = y[0], theta = y[1], phi = y[2];
    double theta_obs, phi_obs;
    cart_to_sph(dir.x, dir.y, dir.z, theta_obs, phi_obs);
    const double Phi = phi - phi_obs;
    const double cost = cos(theta);
    const double sintobs = sin(theta_obs);
    const double rr = r * r;
    const double sigma = rr + (a * cost) * (a * cost);
    const double R = sqrt(a2 + rr);
    const double v = -sintobs * cos(Phi);
    const double zdot = 1.;
    const double inv_sigma = 1.0 / sigma;
    const double sint = sin(theta);
    const double rdot0 = zdot * (r * R * v * sint - R * R * cos(theta_obs) * cost) * inv_sigma;
    const double thetadot0 = zdot * (r * sint * cos(theta_obs) + R * v * cost) * inv_sigma;
    double phidot0;
    if (fabs(sint) < 1e-8) phidot0 = 0.0;
    else phidot0 = zdot * sintobs * sin(Phi) / (R * sint);
    dydx[0] = rdot0;
    dydx[1] = thetadot0;
    dydx[2] = phidot0;
    initial2(y, dydx, r0, theta0);
  }
};

// result of one geodesic trace
struct KerrHit {
  int status;      // 0 background, 1 entity hit, 2 event horizon, 4 step underflow, 5 entity ahead at the end
  int steps;
  int ent, prim;   // hit entity / mesh face (status 1 and 5)
  double t;        // hit distance along the last segment
  dv3 seg_o;       // origin of the segment the hit lies on (before the 1e-6 push)
  dv3 dir2;        // last polyline direction
  bool ov;         // status 1 on the accretion disk: its rewritten colour / emission
  float3 ovc, ove;
};

struct KerrCount {
  uint32_t steps, attempts, segments;
  uint64_t nodes, tris;
};

// ---- accretion disk under the black hole (circle.h:240-335) --------------
// calculateLuminance (color.h:47-49)
__device__ __forceinline__ double disk_lum(double x, double y, double z) {
  return 0.2126 * x + 0.7152 * y + 0.0722 * z;
}

// temperatureToRGB (KerrBlackHole.h:1595-1646): the reference's piecewise
// blackbody fit, temperature clamped to 1000..40000 K
__device__ inline void disk_temp_rgb(double temp, double c[3]) {
  temp = kclamp(temp, 1000.0, 40000.0);
  temp /= 100.0;
  double r, g, b;
  if (temp <= 66) r = 255;
  else r = kclamp(329.698727446 * pow(temp - 60, -0.1332047592), 0.0, 255.0);
  if (temp <= 66) g = kclamp(99.4708025861 * log(temp) - 161.1195681661, 0.0, 255.0);
  else g = kclamp(288.1221695283 * pow(temp - 60, -0.0755148492), 0.0, 255.0);
  if (temp >= 66) b = 255;
  else if (temp <= 19) b = 0;
  else b = kclamp(138.5177312231 * log(temp - 10) - 305.0447927307, 0.0, 255.0);
  c[0] = r / 255.0;
  c[1] = g / 255.0;
  c[2] = b / 255.0;
}

// wavelengthToIntensity (relativistic.h:64-81)
__device__ __forceinline__ double disk_wl(double wl, double center) {
  const double diff = wl - center;
  double it = exp(-(diff * diff) / (2.0 * 100.0 * 100.0));
  if (wl < 380.0 || wl > 750.0) it *= (wl < 380.0) ? exp(-(380.0 - wl) / 50.0) : exp(-(wl - 750.0) / 50.0);
  return it;
}

// applyDopplerShiftFull (relativistic.h:84-170): beaming D^4 blended with a
// wavelength shift of the three channels by the effect strength, in [0, 1]
__device__ inline void disk_doppler(double c[3], double d, double effect) {
  const double lam[3] = {700.0, 546.1, 435.8};
  const double f = 1.0 + (d - 1.0) * effect;
  double wl[3] = {0.0, 0.0, 0.0};
#pragma unroll
  for (int src = 0; src < 3; src++) {
    const double w = lam[src] / f;
#pragma unroll
    for (int dst = 0; dst < 3; dst++) wl[dst] += c[src] * disk_wl(w, lam[dst]);
  }
  const double it = d * d * d * d;
#pragma unroll
  for (int k = 0; k < 3; k++) {
    const double sh = kclamp(wl[k], 0, 1) * effect + (c[k] * it) * (1.0 - effect);
    c[k] = kclamp(sh, 0, 1);
  }
}

// The deterministic part of the disk branch at world point p: false where
// the disk is not there (inside the horizon or the ISCO, beyond its radius,
// off the texture); else colour, emission and alpha (circle.h:244-322).
// In two parts: the texel with its temperature and alpha, which decide whether
// the hit counts, and the Doppler shift (most of the work) of a hit that does.
__device__ inline bool kerr_disk_texel(const GKerr& K, const GEntity& e, dv3 p, double col[3], double em[3],
                                       double& alp) {
  const double rx = p.x - K.pos[0], ry = p.y - K.pos[1], rz = p.z - K.pos[2];
  double sr, sth, sph;
  cart_to_bl(rx, ry, rz, K.a, sr, sth, sph);
  if (sr < K.Rhor || sr > e.radius || !(sr >= K.Rmstable)) return false;
  // the base UVPlane's (u, v) of the hit (plane.h:228-229)
  const dv3 rel = dsub3(p, ldd3(e.p));
  const double u = ddot(rel, ldd3(e.du_axis)) / e.du_len;
  const double v = ddot(rel, ldd3(e.dv_axis)) / e.dv_len;
  // DiscMapping::MapUV (circle.h:53-77), rMin = ISCO, disk_r = the disk radius
  const double theta = atan2(u / sr, v / sr);
  const double rn = (sr - K.Rmstable) / (e.radius - K.Rmstable);
  const double fx = K.disk_w * 0.5 + K.disk_w * rn * cos(theta);
  const double fy = K.disk_h * 0.5 + K.disk_h * rn * sin(theta);
  // the int conversion truncates toward zero: in range iff -1 < f < size
  if (!(fx > -1.0 && fx < (double)K.disk_w) || !(fy > -1.0 && fy < (double)K.disk_h)) return false;
  const uchar4 t = K.disk_tex[(size_t)(int)fy * K.disk_w + (int)fx];
  const double tmp_r = sqrt((rx * rx + rz * rz) + ry * ry);
  col[0] = t.x / 255.0;
  col[1] = t.y / 255.0;
  col[2] = t.z / 255.0;
  if (K.use_temp) {
    // accretionDiskTemperatureGeom (KerrBlackHole.h:1565-1593), then
    // adjustToSourceLuminance (color.h:51-74) to 0..255 integer levels
    double temp = 0.0;
    if (tmp_r > K.Rmstable) {
      const double mdot = 0.1 * ((4.0 * kPi * 1.67262192369e-27) / (0.1 * 6.6524587158e-29));
      double inner = 1.0 - sqrt(K.Rmstable / tmp_r);
      if (inner < 0) inner = 0;
      temp = pow(mdot / (tmp_r * tmp_r * tmp_r) * inner, 0.25);
    }
    double tc[3];
    disk_temp_rgb(temp, tc);
    const double want = disk_lum(col[0], col[1], col[2]);
    const double cur = disk_lum(tc[0], tc[1], tc[2]);
    if (cur == 0.0) {
      const double v0 = (double)(int)kclamp((double)(int)round(want / 0.2126), 0, 255);
      col[0] = col[1] = col[2] = v0;
    } else {
      const double sc = want / cur;
#pragma unroll
      for (int k = 0; k < 3; k++) col[k] = kclamp((double)(int)round(tc[k] * sc), 0, 255);
    }
  }
#pragma unroll
  for (int k = 0; k < 3; k++) em[k] = e.disk_em[k] * col[k];
  alp = t.w / 255.0;
  const double cl = sqrt((col[0] * col[0] + col[2] * col[2]) + col[1] * col[1]) / 3.0;
  if (cl < alp) alp = cl;  // std::min(alpha, |colour| / 3)
  return true;
}

__device__ inline void kerr_disk_shift(const GKerr& K, dv3 p, double col[3], double em[3]) {
  const double rx = p.x - K.pos[0], ry = p.y - K.pos[1], rz = p.z - K.pos[2];
  const double tmp_r = sqrt((rx * rx + rz * rz) + ry * ry);
  // the disk's orbital velocity (getDiskVelocity about +z with sign -1,
  // KerrBlackHole.h:1507-1531) scaled to the circular-orbit speed seen by a
  // locally non-rotating observer (circle.h:292-302)
  double vx = 0.0, vy = 0.0, vz = 0.0;
  if (!(tmp_r < 1e-6)) {
    const double vm = sqrt(1.0 / tmp_r);
    double dx = 0.0 * rz - 1.0 * ry, dy = 1.0 * rx - 0.0 * rz, dz = 0.0 * ry - 0.0 * rx;
    const double il = 1.0 / sqrt((dx * dx + dz * dz) + dy * dy);
    dx *= il;
    dy *= il;
    dz *= il;
    const double sg = vm * -1.0;
    vx = dx * sg;
    vy = dy * sg;
    vz = dz * sg;
  }
  const double a = K.a;
  const double omg = 1.0 / (pow(tmp_r, 3.0 / 2.0) + a);
  const double delt = tmp_r * tmp_r - 2.0 * tmp_r + a * a;
  const double A = pow(tmp_r, 4.0) + a * a * tmp_r * tmp_r + 2.0 * a * a * tmp_r;
  const double o = 2.0 * a * tmp_r / A;
  {
    const double il = 1.0 / sqrt((vx * vx + vz * vz) + vy * vy);
    const double m = omg - o, den = tmp_r * tmp_r * sqrt(delt);
    vx = ((vx * il) * m) * A;
    vy = ((vy * il) * m) * A;
    vz = ((vz * il) * m) * A;
    if (den == 0.0) {  // Vector3d::operator/ by zero (vector3d.h:67-75)
      vx = vy = vz = 1.0;
    } else {
      vx /= den;
      vy /= den;
      vz /= den;
    }
  }
  // calculateDopplerFactorFromObserver (KerrBlackHole.h:1534-1562)
  double dop = 1.0;
  {
    double wx = p.x - K.observer[0], wy = p.y - K.observer[1], wz = p.z - K.observer[2];
    const double iw = 1.0 / sqrt((wx * wx + wz * wz) + wy * wy);
    wx *= iw;
    wy *= iw;
    wz *= iw;
    const double beta = sqrt((vx * vx + vz * vz) + vy * vy);
    if (!(beta < 1e-6)) {
      const double ib = 1.0 / beta;
      const double cos_t = (wx * (vx * ib) + wz * (vz * ib)) + wy * (vy * ib);
      const double gamma = 1.0 / sqrt(1.0 - beta * beta);
      dop = 1.0 / (gamma * (1.0 - beta * cos_t));
    }
  }
  disk_doppler(col, dop, K.doppler_effect);
  disk_doppler(em, dop, K.doppler_effect);
}

__device__ inline bool kerr_disk_shade(const GKerr& K, const GEntity& e, dv3 p, double col[3], double em[3],
                                       double& alp) {
  if (!kerr_disk_texel(K, e, p, col, em, alp)) return false;
  kerr_disk_shift(K, p, col, em);
  return true;
}

constexpr double kSegment = 2.0;  // h_dist: the longest step, and how far a segment test looks

// exact_closest hook of the Kerr tracer: a disk_map disk is there only where
// its texture is and its alpha test passes; the closest hit on it carries the
// rewritten colour and emission.  The alpha test draws from its own stream
// (the reference draws it from the scene's generator, scene_env.h:213, :306).
struct KerrDiskShading {
  const GKerr* K;
  Rng* rng;
  bool cand, ov;
  float3 cc, ce, oc, oe;
  __device__ __forceinline__ void begin() { ov = false; }
  __device__ __forceinline__ bool circle(const GEntity& e, dv3 p, double t) {
    cand = false;
    if (!e.kerr_disk || !K->disk_tex) return true;
    double col[3], em[3], alp;
    if (!kerr_disk_texel(*K, e, p, col, em, alp)) return false;
    if (alp == 0.0) return false;
    if (alp < 0.99 && alp <= (double)rng->next()) return false;
    if (t < kSegment) kerr_disk_shift(*K, p, col, em);  // a hit beyond the segment is not kept
    cand = true;
    cc = f3((float)col[0], (float)col[1], (float)col[2]);
    ce = f3((float)em[0], (float)em[1], (float)em[2]);
    return true;
  }
  __device__ __forceinline__ void best(const GEntity& e) {
    ov = e.type == PR_ENT_CIRCLE && cand;
    oc = cc;
    oe = ce;
  }
};

__device__ __forceinline__ DiskAlpha disk_alpha(const GKerr& K) {
  return DiskAlpha{K.disk_tex, K.disk_w, K.disk_h, K.use_temp == 0, K.rms_f, K.a2_f, {K.pos_f[0], K.pos_f[1], K.pos_f[2]}};
}

// the key of the alpha-test stream: the render seed mixed with the disk seed
__device__ __forceinline__ uint64_t disk_stream_key(uint64_t seed, const GKerr& K) {
  return seed ^ (K.disk_seed * 0x9E3779B97F4A7C15ull);
}
constexpr uint32_t kDiskBranch = 0xFFFFFFFFu;  // counter lane of the alpha-test stream

// ======================================================================
// Mixed-precision form (pr_kerr.precision = PR_KERR_FP32).  GB300 runs FP32
// at 64x its FP64 rate.  This form keeps the reference's FP64 step (the same
// step control, so the same step sequence and polyline) wherever the
// integration needs it -- near the hole, at polar and radial turning points
// -- and switches to FP32 only where the reference's step is known to be the
// capped h = 2 accepted at the first attempt:
//  * far field: once a ray is outbound (dr/dlambda > 0), beyond
//    max(kFarRadius, scene radius + 2), with the last FP64 step's error
//    estimate below kFarErrmax (the estimate only falls further out), every
//    further step is h = 2 computed in FP32 and added to the FP64 state (the
//    reference accepts exactly these steps: errmax << 0.59 keeps hnext above
//    the cap); no segment test is needed there, nothing of the scene is
//    ahead of an outbound ray beyond the scene radius;
//  * capture: a ray inbound inside the innermost scene geometry whose radial
//    potential R(r) = ((r^2 + a^2) - a L)^2 - Delta (kappa - 2 a L) stays
//    positive down to the horizon has no turning point left; the reference
//    steps it on until its step size underflows (status 4, "no hit"), this
//    form reports that outcome at once.
// Status, steps to the far field, hits and exit directions follow the FP64
// form; the FP32 far-field steps differ from the reference's in rounding only.
// ======================================================================
constexpr double kFarRadius = 200.0;  // M
constexpr double kFarErrmax = 1.0e-3;
constexpr double kPoleSin2 = 1.0e-4;

struct KerrRayF {
  float a, a2, M;
  float L, kappa;

  // geodesic (KerrBlackHole.h:1239-1281) in FP32
  __device__ __forceinline__ void geodesic(const float* y, float* dydx) const {
    const float r = y[0], pr = y[4], ptheta = y[5];
    const float r2 = r * r;
    const float twor = 2.0f * M * r;
    float sintheta, costheta;
    sincosf(y[1], &sintheta, &costheta);
    float sin2 = sintheta * sintheta;
    const float cos2 = costheta * costheta;
    const float sigma = r2 + a2 * cos2;
    const float delta = r2 - twor + a2;
    const float siginv = 1.0f / sigma;
    const float bot = 1.0f / (sigma * delta);
    if (fabsf(sin2) < 1.0e-16f) sin2 = 1.0e-16f;
    const float r2a2 = r2 + a2;
    dydx[0] = -pr * delta * siginv;
    dydx[1] = -ptheta * siginv;
    dydx[2] = -(twor * a + (sigma - twor) * L / sin2) * bot;
    dydx[3] = -(1.0f + (twor * r2a2 - twor * a * L) * bot);
    dydx[4] = -(((r - 1.0f) * (-kappa) + twor * r2a2 - 2.0f * a * L) * bot - 2.0f * pr * pr * (r - 1.0f) * siginv);
    dydx[5] = -sintheta * costheta * (L * L / (sin2 * sin2) - a2) * siginv;
  }

  // one Cash-Karp step of size h in FP32, as increments dy = y_out - y
  __device__ __forceinline__ void step(const float* y, const float* dydx, float h, float* dy) const {
    float ak[6], t[6], k1[6], k2[6], k3[6], k4[6], k6[6];
#pragma unroll
    for (int i = 0; i < 6; i++) {
      k1[i] = h * dydx[i];
      t[i] = y[i] + 0.2f * k1[i];
    }
    geodesic(t, ak);
#pragma unroll
    for (int i = 0; i < 6; i++) {
      k2[i] = h * ak[i];
      t[i] = y[i] + (3.0f / 40.0f) * k1[i] + (9.0f / 40.0f) * k2[i];
    }
    geodesic(t, ak);
#pragma unroll
    for (int i = 0; i < 6; i++) {
      k3[i] = h * ak[i];
      t[i] = y[i] + 0.3f * k1[i] - 0.9f * k2[i] + 1.2f * k3[i];
    }
    geodesic(t, ak);
#pragma unroll
    for (int i = 0; i < 6; i++) {
      k4[i] = h * ak[i];
      t[i] = y[i] - (11.0f / 54.0f) * k1[i] + 2.5f * k2[i] - (70.0f / 27.0f) * k3[i] + (35.0f / 27.0f) * k4[i];
    }
    geodesic(t, ak);
#pragma unroll
    for (int i = 0; i < 6; i++) {
      const float k5 = h * ak[i];
      t[i] = y[i] + (1631.0f / 55296.0f) * k1[i] + (175.0f / 512.0f) * k2[i] + (575.0f / 13824.0f) * k3[i] +
             (44275.0f / 110592.0f) * k4[i] + (253.0f / 4096.0f) * k5;
    }
    geodesic(t, ak);
#pragma unroll
    for (int i = 0; i < 6; i++) {
      k6[i] = h * ak[i];
      dy[i] = (37.0f / 378.0f) * k1[i] + (250.0f / 621.0f) * k3[i] + (125.0f / 594.0f) * k4[i] +
              (512.0f / 1771.0f) * k6[i];
    }
  }
};

// R(r) of the radial motion (E = 1): ((r^2 + a^2) - a L)^2 - Delta (kappa - 2 a L),
// where the reference's kappa = p_theta^2 + a^2 sin^2 + L^2 / sin^2 = Q + L^2 + a^2
__device__ __forceinline__ double radial_potential(double r, double a, double L, double kappa) {
  const double w = r * r + a * a - a * L;
  const double delta = r * r - 2.0 * r + a * a;
  return w * w - delta * (kappa - 2.0 * a * L);
}

// no turning point between the horizon and r: R > 0 on a fine grid of [r+, r].
// FP32 decides where R's sign clears its rounding (all but rays within about
// 1e-5 of critical), FP64 the rest.
__device__ __forceinline__ bool no_turning_point(double r, double rplus, double a, double L, double kappa) {
  const int n = 64;
  {
    const float rp = (float)rplus, dr = (float)(r - rplus), af = (float)a, aL = (float)(a * L);
    const float q = (float)(kappa - 2.0 * a * L), a2 = af * af;
    bool clear = true;
    for (int i = 0; i <= n; i++) {
      const float rr = rp + dr * ((float)i / n), r2 = rr * rr;
      const float w = r2 + a2 - aL, delta = r2 - 2.0f * rr + a2;
      const float R = w * w - delta * q;
      // the sums' terms, and R's change over the rounding of rr
      const float m = r2 + a2 + fabsf(aL), e = 1.0e-5f * (m * m + (r2 + 2.0f * rr + a2) * fabsf(q));
      if (R < -e) return false;
      clear = clear && R > e;
    }
    if (clear) return true;
  }
  for (int i = 0; i <= n; i++) {
    const double rr = rplus + (r - rplus) * (double)i / n;
    if (!(radial_potential(rr, a, L, kappa) > 0.0)) return false;
  }
  return true;
}

// ---- the march of one ray ---------------------------------------------------
// The state between the steps of the reference's loop (scene.cpp:448-732)
struct KerrMarch {
  KerrRay k;
  double y[6];
  double sint, cost;     // of y[1] (not kept up in the far field)
  double h_step, errmax;
  dv3 org1, org2, dir2;  // the polyline's last vertices and direction
  double yprev[3];       // mixed form: the state before the last step
  int c;                 // accepted steps
  bool far_mode;         // mixed form: in the far field
  bool capture_checked;
};

// Set-up of a ray; false if it starts inside the horizon (out says so)
__device__ __forceinline__ bool kerr_start(const GKerr& K, dv3 org, dv3 dir, KerrMarch& M, KerrHit& out) {
  M.k = KerrRay{K.a, K.a2, K.M, 0.0, 0.0};
  const dv3 rel = {org.x - K.pos[0], org.y - K.pos[1], org.z - K.pos[2]};  // Setup (KerrBlackHole.h:153-166)
  double r0, th0, ph0;
  cart_to_bl(rel.x, rel.y, rel.z, K.a, r0, th0, ph0);
  M.y[0] = r0;
  M.y[1] = th0;
  M.y[2] = ph0;
  M.y[3] = 0;
  M.y[4] = 0;
  M.y[5] = 0;
  out.steps = 0;
  out.ov = false;
  out.ent = -1;
  out.prim = -1;
  out.t = -1.0;
  out.dir2 = dir;
  out.seg_o = org;
  if (r0 < K.Rhor) {
    out.status = 2;
    return false;
  }
  double dydx[6];
  M.k.initial(dir, M.y, dydx, r0, th0);
  sincos(M.y[1], &M.sint, &M.cost);
  M.h_step = kSegment;
  M.errmax = 1.0;
  M.org1 = M.org2 = org;
  M.dir2 = dir;
  for (int i = 0; i < 3; i++) M.yprev[i] = M.y[i];
  M.c = 0;
  M.far_mode = false;
  M.capture_checked = false;
  return true;
}

// The end of the loop: the polyline's last vertex looks straight on
template <class HS>
__device__ __forceinline__ void kerr_finish(const DevScene& S, const GKerr& K, KerrMarch& M, KerrHit& out,
                                            KerrCount& cnt, uint32_t* err, HS& hs) {
  if (M.far_mode) {
    // the polyline's last vertex and chord, in FP64, from the last two states
    const dv3 q1 = bl_to_cart(M.yprev[0], M.yprev[1], M.yprev[2], K.a);
    const dv3 q2 = bl_to_cart(M.y[0], M.y[1], M.y[2], K.a);
    M.org2 = {q2.x + K.pos[0], q2.y + K.pos[1], q2.z + K.pos[2]};
    M.dir2 = dnormalize({q2.x - q1.x, q2.y - q1.y, q2.z - q1.z});
  }
  out.steps = M.c;
  out.dir2 = M.dir2;
  out.seg_o = M.org2;
  double t;
  int ent, prim;
  cnt.segments++;
  if (exact_closest_hs(S, M.org2, M.dir2, t, ent, prim, err, cnt.nodes, cnt.tris, hs)) {
    out.status = 5;
    out.ent = ent;
    out.prim = prim;
    out.t = t;
  } else {
    out.status = 0;
  }
}

// One pass of the reference's loop outside the far field, for the lanes that
// run; true when the ray's trace has ended.  SYNC: all lanes of the warp call
// it together, and the warp comes together again after the parts that few
// lanes take.  look: with the segment test (not on the step that leaves the far field).
template <bool FAST, bool SYNC, class HS>
__device__ __forceinline__ bool kerr_step(const DevScene& S, const GKerr& K, KerrMarch& M, KerrHit& out,
                                          KerrCount& cnt, uint32_t* err, HS& hs, bool capture_shortcut, bool run,
                                          bool look) {
  bool leave = run && M.c >= K.max_steps, done = false, hit = false;
  double t = 0.0;
  int ent = -1, prim = -1;
  look = look && run && !leave;
  int draws = 0;
  if (look) draws = segment_draws(S, M.org1, M.dir2, kSegment, disk_alpha(K));
  cnt.segments += look ? 1u : 0u;
  for (int i = 0; i < draws; i++) (void)hs.rng->next();
  if (draws < 0)  // the exact test makes its own draws
    hit = exact_closest_hs(S, M.org1, M.dir2, t, ent, prim, err, cnt.nodes, cnt.tris, hs) && t < kSegment;
  if (SYNC) __syncwarp();
  if (hit) {
    // hit point of intersect_scene_: (org1 + 1e-6 dir2) + t dir2
    const dv3 o2 = dadd3(M.org1, dscale3(M.dir2, 0.000001));
    const dv3 p = {o2.x + t * M.dir2.x, o2.y + t * M.dir2.y, o2.z + t * M.dir2.z};
    double sr, sth, sph;
    cart_to_bl(p.x - K.pos[0], p.y - K.pos[1], p.z - K.pos[2], K.a, sr, sth, sph);
    out.steps = M.c;
    out.dir2 = M.dir2;
    out.seg_o = M.org1;
    if (sr < K.Rhor) {
      out.status = 2;
    } else {
      out.status = 1;
      out.ent = ent;
      out.prim = prim;
      out.t = t;
      out.ov = hs.ov;
      out.ovc = hs.oc;
      out.ove = hs.oe;
    }
    done = true;
  } else if (run && !leave) {
    double dydx[6];
    M.k.geodesic(M.y, M.sint, M.cost, dydx);
    if (fabs(M.h_step) < 1.0e-10) {
      out.status = 4;
      out.steps = M.c;
      out.dir2 = M.dir2;
      done = true;
    }
    if (FAST && !done) {
      if (capture_shortcut && !M.capture_checked && dydx[0] < 0.0 && M.y[0] < K.scene_inner) {
        // inbound inside all scene geometry: captured if no turning point is
        // left.  The reference ends such a ray with a step underflow (status 4)
        // or inside the horizon (2); the shortcut reports 4, so it is taken only
        // where the two look alike
        M.capture_checked = true;
        if (no_turning_point(M.y[0], K.M + sqrt(K.M * K.M - K.a2), K.a, M.k.L, M.k.kappa)) {
          out.status = 4;
          out.steps = M.c;
          out.dir2 = M.dir2;
          done = true;
        }
      }
      for (int i = 0; i < 3; i++) M.yprev[i] = M.y[i];
    }
    if (!done) {
      const double r_before = M.y[0];
      M.h_step = M.k.next_position(M.y, dydx, M.h_step, kSegment, cnt.attempts, &M.errmax);
      if (M.y[0] < K.Rhor) {
        out.status = 2;
        out.steps = M.c;
        out.dir2 = M.dir2;
        done = true;
      } else {
        M.org1 = M.org2;
        sincos(M.y[1], &M.sint, &M.cost);
        const dv3 q = bl_to_cart(M.y[0], M.sint, M.cost, M.y[2], K.a);
        M.org2 = {q.x + K.pos[0], q.y + K.pos[1], q.z + K.pos[2]};
        M.dir2 = dnormalize({M.org2.x - M.org1.x, M.org2.y - M.org1.y, M.org2.z - M.org1.z});
        if (FAST && M.y[0] > fmax(kFarRadius, K.scene_radius + 2.0) && M.y[0] > r_before && M.errmax < kFarErrmax &&
            M.h_step == kSegment && M.sint * M.sint >= kPoleSin2)
          M.far_mode = true;
        M.c++;
        cnt.steps++;
        // optional early exit (not in the reference): far out and receding
        leave = K.escape_radius > 0.0 && M.y[0] > K.escape_radius && M.y[0] > r_before;
      }
    }
  }
  if (SYNC) __syncwarp();
  if (leave) {
    kerr_finish(S, K, M, out, cnt, err, hs);
    done = true;
  }
  return done;
}

// background map lookup of an escaped ray (scene.cpp:711-727; SphericalMapping::Map, circle.h:92-105)
__device__ __forceinline__ float3 kerr_background(const GKerr& K, const double* yy, const float* bg) {
  if (!K.texture) return f3(bg[0], bg[1], bg[2]);
  double y1 = yy[1] * K.map_coef[0] + K.map_coef[1];
  double y2 = yy[2] * K.map_coef[2] + K.map_coef[3];
  y1 = fmod(y1, kPi);
  y2 = fmod(y2, 2.0 * kPi);
  double phi = y2, theta = y1;
  if (phi < 0.0) phi += 2.0 * kPi;
  if (theta < 0.0) theta = -theta;
  int x = (int)(phi / (2.0 * kPi) * K.tex_w);
  x = ((x % K.tex_w) + K.tex_w) % K.tex_w;  // in range for any input, NaN included
  int yv = (int)(theta / kPi * K.tex_h);
  yv = ((yv % K.tex_h) + K.tex_h) % K.tex_h;
  const unsigned char* t = K.texture + 3 * ((size_t)yv * K.tex_w + x);
  return f3((float)(K.texture_coef * t[0] / 255.0), (float)(K.texture_coef * t[1] / 255.0),
            (float)(K.texture_coef * t[2] / 255.0));
}

template <class T>
__device__ __forceinline__ T warp_sum(T v) {
  for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
  return v;
}

__device__ __forceinline__ void flush_counts(const KerrCount& c, uint32_t rays, unsigned long long* counters) {
  if (!counters) return;
  const unsigned long long a = warp_sum<unsigned long long>(rays), b = warp_sum<unsigned long long>(c.steps),
                           d = warp_sum<unsigned long long>(c.attempts),
                           e = warp_sum<unsigned long long>(c.segments);
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(counters + 0, a);
    atomicAdd(counters + 1, b);
    atomicAdd(counters + 2, d);
    atomicAdd(counters + 3, e);
  }
}


// One step in the far field (FP32 increments to the FP64 state); true when
// the ray's trace has ended.  A pole ahead ends the far field: then the step
// is the reference's (kerr_step without its segment test).
template <class HS>
__device__ __forceinline__ bool kerr_far_step(const DevScene& S, const GKerr& K, KerrMarch& M, KerrHit& out,
                                              KerrCount& cnt, uint32_t* err, HS& hs, bool capture_shortcut) {
  if (M.c >= K.max_steps) {
    kerr_finish(S, K, M, out, cnt, err, hs);
    return true;
  }
  const float stf = sinf((float)M.y[1]);
  if (stf * stf < (float)kPoleSin2) {
    M.far_mode = false;
    sincos(M.y[1], &M.sint, &M.cost);
    return kerr_step<true, false>(S, K, M, out, cnt, err, hs, capture_shortcut, true, false);
  }
  const double r_before = M.y[0];
  for (int i = 0; i < 3; i++) M.yprev[i] = M.y[i];
  const KerrRayF kf{(float)K.a, (float)K.a2, (float)K.M, (float)M.k.L, (float)M.k.kappa};
  float yf[6], df[6], dy[6];
#pragma unroll
  for (int i = 0; i < 6; i++) yf[i] = (float)M.y[i];
  kf.geodesic(yf, df);
  kf.step(yf, df, (float)kSegment, dy);
#pragma unroll
  for (int i = 0; i < 6; i++) M.y[i] += (double)dy[i];
  cnt.attempts++;
  M.h_step = kSegment;
  M.c++;
  cnt.steps++;
  if (K.escape_radius > 0.0 && M.y[0] > K.escape_radius && M.y[0] > r_before) {
    kerr_finish(S, K, M, out, cnt, err, hs);
    return true;
  }
  return false;
}

// Rays of a batch (KerrOut), one per lane: a lane whose ray has ended takes
// the next one
template <bool FAST>
struct KerrTraceJob {
  const DevScene& S;
  const GKerr& K;
  const double* rays;
  int64_t n;
  const KerrOut& out;
  uint32_t* err;
  unsigned long long* next;  // rays handed out beyond each lane's first
  KerrMarch M;
  KerrHit h;
  KerrCount c;
  Rng drng;
  int64_t i;
  uint32_t rays_done;
  bool more, ended_at_start;

  __device__ __forceinline__ bool take(bool want) {
    const int lane = threadIdx.x & 31;
    const unsigned int mask = __ballot_sync(0xffffffffu, want);
    unsigned long long base = 0;
    if (i < 0) {  // the first ray of every lane
      base = (unsigned long long)blockIdx.x * blockDim.x + (threadIdx.x & ~31);
    } else {
      const int leader = __ffs(mask) - 1;
      if (lane == leader) base = atomicAdd(next, (unsigned long long)__popc(mask)) + (unsigned long long)gridDim.x * blockDim.x;
      base = __shfl_sync(0xffffffffu, base, leader);
    }
    if (!want) return false;
    i = (int64_t)(base + (unsigned long long)__popc(mask & ((1u << lane) - 1u)));
    if (i >= n) {
      more = false;
      return false;
    }
    const double* r = rays + 6 * i;
    drng.init(disk_stream_key(0, K), (uint64_t)i, kDiskBranch);
    if (!kerr_start(K, {r[0], r[1], r[2]}, {r[3], r[4], r[5]}, M, h)) ended_at_start = true;
    return true;
  }
  __device__ __forceinline__ bool step(bool run) {
    KerrDiskShading hs{&K, &drng};
    const bool far = FAST && run && M.far_mode && !ended_at_start;
    bool done = run && ended_at_start;
    done |= kerr_step<FAST, true>(S, K, M, h, c, err, hs, true, run && !far && !ended_at_start, true);
    if (far) done = kerr_far_step(S, K, M, h, c, err, hs, true);
    return done;
  }
  __device__ __forceinline__ bool ended() {
    ended_at_start = false;
    if (out.status) out.status[i] = h.status;
    if (out.steps) out.steps[i] = h.steps;
    if (out.final_bl) {
      out.final_bl[3 * i] = M.y[0];
      out.final_bl[3 * i + 1] = M.y[1];
      out.final_bl[3 * i + 2] = M.y[2];
    }
    if (out.exit_dir) {
      out.exit_dir[3 * i] = h.dir2.x;
      out.exit_dir[3 * i + 1] = h.dir2.y;
      out.exit_dir[3 * i + 2] = h.dir2.z;
    }
    if (out.hit_entity) out.hit_entity[i] = h.ent;
    if (out.hit_t) out.hit_t[i] = h.t;
    rays_done++;
    return false;
  }
};

template <bool FAST>
__global__ void __launch_bounds__(128) kerr_trace_kernel(const __grid_constant__ DevScene S,
                                                         const __grid_constant__ GKerr K,
                                                         const double* __restrict__ rays, int64_t n,
                                                         const __grid_constant__ KerrOut out,
                                                         uint32_t* __restrict__ err,
                                                         unsigned long long* __restrict__ counters) {
  KerrTraceJob<FAST> job{S, K, rays, n, out, err, counters + kKerrNextCounter};
  job.c = KerrCount{0, 0, 0, 0, 0};
  job.i = -1;
  job.rays_done = 0;
  job.more = true;
  job.ended_at_start = false;
  geodesic_warp(job);
  flush_counts(job.c, job.rays_done, counters);
}

// A path in the far field, handed from the near kernel of the mixed form to
// the far one
struct KerrFar {
  double y[6], yprev[3], L, kappa, h_step, errmax;
  dv3 org2, dir2;
  unsigned long long id;
  Rng drng;
  PathState ps;
  float3 root;
  uint32_t item;
  int c;
  int capture_checked;
};

struct KerrFrame {
  SamplePass pass;  // next: [0] samples handed out, [1] far records written, [2] far records taken
  KerrFar* far;     // mixed form
  unsigned long long far_cap;
};

// Camera samples of radiance() in a Kerr scene, one path per lane (no
// next-event estimation, no media: every query is a geodesic, as
// intersect_scene makes it).  PHASE 0: the FP64 form; 1: the mixed form's
// near field, which hands a path that reaches the far field on; 2: its far
// field, from those records.  A step near the hole costs the FP64 pipe what
// fifty far steps cost the FP32 ones; side by side in a warp each waited for
// the other.
template <int PHASE>
struct KerrPathJob {
  static constexpr bool FAST = PHASE != 0;
  const DevScene& S;
  const GKerr& K;
  const RenderCfg& cfg;
  const KerrFrame& F;
  uint32_t* err;
  KerrMarch M;
  KerrHit h;
  KerrCount c;
  Rng drng;  // the accretion disk's alpha tests of this camera sample
  PathState ps;
  unsigned long long id;
  uint32_t item;  // the pass's sample that the path is (a sample id may wrap past 2^64)
  float3 L;
  int sp;
  uint32_t paths;
  bool more, ended_at_start;
  PathState stack[kSplitStack];

  // a captured ray's colour: black (horizon) or BACKGROUND (step underflow)
  // are the same only on a black background
  __device__ __forceinline__ bool shortcut() const { return S.bg[0] == 0.0f && S.bg[1] == 0.0f && S.bg[2] == 0.0f; }

  __device__ __forceinline__ void start_ray() {
    ended_at_start = !kerr_start(K, {ps.o.x, ps.o.y, ps.o.z}, {ps.d.x, ps.d.y, ps.d.z}, M, h);
  }

  __device__ __forceinline__ bool take(bool want) {
    const int lane = threadIdx.x & 31;
    const unsigned int mask = __ballot_sync(0xffffffffu, want);
    const int leader = __ffs(mask) - 1;
    unsigned long long base = 0;
    if (lane == leader) base = atomicAdd(F.pass.next + (PHASE == 2 ? 2 : 0), (unsigned long long)__popc(mask));
    base = __shfl_sync(0xffffffffu, base, leader);
    if (!want) return false;
    const unsigned long long g = base + (unsigned long long)__popc(mask & ((1u << lane) - 1u));
    sp = 0;
    if (PHASE == 2) {
      const unsigned long long n = F.pass.next[1] < F.far_cap ? F.pass.next[1] : F.far_cap;
      if (g >= n) {
        more = false;
        return false;
      }
      const KerrFar& f = F.far[g];
      for (int q = 0; q < 6; q++) M.y[q] = f.y[q];
      for (int q = 0; q < 3; q++) M.yprev[q] = f.yprev[q];
      M.k = KerrRay{K.a, K.a2, K.M, f.L, f.kappa};
      M.h_step = f.h_step;
      M.errmax = f.errmax;
      M.org1 = M.org2 = f.org2;
      M.dir2 = f.dir2;
      M.c = f.c;
      M.far_mode = true;
      M.capture_checked = f.capture_checked != 0;
      M.sint = M.cost = 0.0;
      h.steps = 0;
      h.ov = false;
      h.ent = -1;
      h.prim = -1;
      h.t = -1.0;
      id = f.id;
      item = f.item;
      drng = f.drng;
      ps = f.ps;
      L = f.root;
      ended_at_start = false;
      return true;
    }
    if (g >= F.pass.samples) {
      more = false;
      return false;
    }
    int x, y;
    uint32_t k;
    pass_sample(cfg, F.pass, (uint32_t)g, x, y, k);
    float3 o, d;
    id = camera_ray(cfg, x, y, cfg.sample_offset + (uint64_t)k, o, d);
    item = (uint32_t)g;
    root_path(ps, o, d);
    drng.init(disk_stream_key(cfg.seed, K), id, kDiskBranch);
    L = f3(0, 0, 0);
    start_ray();
    return true;
  }

  __device__ __forceinline__ bool step(bool run) {
    KerrDiskShading hs{&K, &drng};
    const bool far = FAST && run && M.far_mode && !ended_at_start;
    bool done = run && ended_at_start;
    done |= kerr_step<FAST, true>(S, K, M, h, c, err, hs, FAST && shortcut(), run && !far && !ended_at_start, true);
    if (PHASE == 1) {
      // newly in the far field (or started a step there: no room in the list)
      if (run && !done && M.far_mode) {
        unsigned long long at = F.far_cap;
        if (!far && sp == 0) at = atomicAdd(F.pass.next + 1, 1ull);
        if (at < F.far_cap) {
          KerrFar& f = F.far[at];
          for (int q = 0; q < 6; q++) f.y[q] = M.y[q];
          for (int q = 0; q < 3; q++) f.yprev[q] = M.yprev[q];
          f.L = M.k.L;
          f.kappa = M.k.kappa;
          f.h_step = M.h_step;
          f.errmax = M.errmax;
          f.org2 = M.org2;
          f.dir2 = M.dir2;
          f.c = M.c;
          f.capture_checked = M.capture_checked;
          f.id = id;
          f.item = item;
          f.drng = drng;
          f.ps = ps;
          f.root = L;
          h.status = -1;  // handed on
          done = true;
        }
      }
    }
    if (far) done = kerr_far_step(S, K, M, h, c, err, hs, shortcut());
    return done;
  }

  // the ray's trace ended: shade, and go on with the path's next ray or end it
  __device__ __forceinline__ bool ended() {
    if (PHASE == 1 && h.status == -1) return false;
    FastHit fh;
    Vertex v;
    float3 miss = f3(0, 0, 0), ovr[2];
    bool has_ovr = false;
    const bool hit = h.status == 1;
    if (!hit) {
      if (h.status == 0) miss = kerr_background(K, M.y, S.bg);
      else if (h.status != 2) miss = f3(S.bg[0], S.bg[1], S.bg[2]);
    } else {
      // the vertex the straight-ray tracer would build from the last segment
      const GEntity& e = S.ents[h.ent];
      const dv3 o2 = dadd3(h.seg_o, dscale3(h.dir2, 0.000001));
      const dv3 p = {o2.x + h.t * h.dir2.x, o2.y + h.t * h.dir2.y, o2.z + h.t * h.dir2.z};
      float3 n;
      if (e.type == PR_ENT_SPHERE) {
        n = normalize(f3((float)(p.x - e.p[0]), (float)(p.y - e.p[1]), (float)(p.z - e.p[2])));
      } else if (e.type == PR_ENT_POLYGON) {
        n = ld3(S.fnorm + 3 * (size_t)(e.face_base + h.prim));
      } else {
        n = f3((float)e.normal[0], (float)e.normal[1], (float)e.normal[2]);
      }
      if (e.normal_inverse < 0) n = -n;
      v.p = f3((float)p.x, (float)p.y, (float)p.z);
      v.n = n;
      v.ent = h.ent;
      v.mat = e.material;
      v.t = (float)h.t;
      if (h.ov) {  // the accretion disk's own colour and emission at this point
        has_ovr = true;
        ovr[0] = h.ovc;
        ovr[1] = h.ove;
      }
      fh.t = (float)h.t;
      fh.ent = h.ent;
      fh.slot = -1;
      fh.u = fh.v = 0.0f;
    }
    ShadowReq sh[3];
    int nsh = 0;
    PathState child;
    const int r = shade(S, cfg, ps, hit, fh, id, sh, nsh, child, err, &v, &miss, nullptr, nullptr,
                        has_ovr ? ovr : nullptr);
    if (r == SHADE_SPLIT) {
      if (sp < kSplitStack) stack[sp++] = child;
      else atomicOr(err, PR_DEV_LOOP_CAP);
    }
    if (r == SHADE_END) {
      L += ps.L;
      if (sp == 0) {
        F.pass.sample[item] = finish_sample(cfg, L, err);
        paths++;
        return false;
      }
      ps = stack[--sp];
    }
    start_ray();
    return true;
  }
};

template <int PHASE>
__global__ void __launch_bounds__(128) kerr_render_kernel(const __grid_constant__ DevScene S,
                                                          const __grid_constant__ GKerr K,
                                                          const __grid_constant__ RenderCfg cfg,
                                                          const __grid_constant__ KerrFrame F,
                                                          uint32_t* __restrict__ err,
                                                          unsigned long long* __restrict__ counters) {
  KerrPathJob<PHASE> job{S, K, cfg, F, err};
  job.c = KerrCount{0, 0, 0, 0, 0};
  job.sp = 0;
  job.paths = 0;
  job.more = true;
  job.ended_at_start = false;
  geodesic_warp(job);
  flush_counts(job.c, job.paths, counters);
}

// scratch of a frame: the samples of a pass, then the far records
inline unsigned long long kerr_far_cap(const RenderCfg& cfg) {
  const unsigned long long n = pass_pixels(cfg) * (unsigned long long)cfg.spp;
  const unsigned long long most = cfg.less ? 1ull << 15 : 1ull << 19;  // beyond that the near kernel goes on itself
  return n < most ? n : most;
}
inline size_t kerr_bytes(const RenderCfg& cfg, bool far) {
  return pass_bytes(cfg) + (far ? sizeof(KerrFar) * (size_t)kerr_far_cap(cfg) : 0);
}
// pass k of a frame (its counters are zeroed)
inline cudaError_t kerr_frame(const RenderCfg& cfg, void* scratch, bool far, unsigned long long k, KerrFrame& F,
                              cudaStream_t stream) {
  F.far = far ? reinterpret_cast<KerrFar*>(static_cast<char*>(scratch) + pass_bytes(cfg)) : nullptr;
  F.far_cap = far ? kerr_far_cap(cfg) : 0;
  return sample_pass(cfg, scratch, k, F.pass, stream);
}

}  // namespace
}  // namespace pr
