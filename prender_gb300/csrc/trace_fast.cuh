// FP32 closest-hit and any-hit queries used while rendering.
//
// Traversal of the render path's compressed 8-wide trees (WNode) per thread
// with a small local stack of node groups: children visited near to far by
// their octant slots, each child box culled against the current closest hit,
// leaves tested as soon as their node is visited.
// Spheres that FP32 bounds cannot rule out take the reference's FP64 test
// (its 1e5-radius walls cancel catastrophically in FP32); planes and
// triangles are FP32.
#pragma once
#include "device_common.cuh"

namespace pr {

struct FastHit {
  float t;
  int ent;
  int slot;   // leaf slot of the triangle (meshes), -1 otherwise
  float u, v; // barycentrics of the triangle hit
};

struct TraceStats {
  uint32_t nodes;
  uint32_t tris;
};

__device__ __forceinline__ bool fast_tri(const float4* __restrict__ T, float3 o, float3 d, float tmax, float& t, float& bu,
                                         float& bv) {
  const float4 A = __ldg(T), B = __ldg(T + 1), C = __ldg(T + 2);
  const float3 v0 = f3(A.x, A.y, A.z);
  const float3 e1 = f3(B.x, B.y, B.z) - v0, e2 = f3(C.x, C.y, C.z) - v0;
  const float3 p = cross(d, e2);
  const float det = dot(e1, p);
  if (fabsf(det) <= 1.0e-7f) return false;  // det eps of CheckIntersection2 (polygon.h:98)
  const float inv = 1.0f / det;
  const float3 tv = o - v0;
  const float u = dot(tv, p) * inv;
  if (u < 0.0f || u > 1.0f) return false;
  const float3 q = cross(tv, e1);
  const float v = dot(d, q) * inv;
  if (v < 0.0f || u + v > 1.0f) return false;
  const float tt = dot(e2, q) * inv;
  if (!(tt > 0.0f) || !(tt < tmax)) return false;
  t = tt;
  bu = u;
  bv = v;
  return true;
}

// Ray data of the wide traversal
struct WRay {
  float3 o, d, inv;
  int oct;  // sign bits of d (bit a: negative along axis a)
};

__device__ __forceinline__ float3 safe_inv(float3 d) {
  const float big = 1.0e30f;
  return f3(d.x != 0.0f ? 1.0f / d.x : copysignf(big, d.x), d.y != 0.0f ? 1.0f / d.y : copysignf(big, d.y),
            d.z != 0.0f ? 1.0f / d.z : copysignf(big, d.z));
}

__device__ __forceinline__ WRay make_wray(float3 o, float3 d) {
  WRay r;
  r.o = o;
  r.d = d;
  r.inv = safe_inv(d);
  r.oct = (d.x < 0.0f ? 1 : 0) | (d.y < 0.0f ? 2 : 0) | (d.z < 0.0f ? 4 : 0);
  return r;
}

// two FP32 values in one register pair: Blackwell's packed fma / add
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float a, float b) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float o[2]) { asm("mov.b64 {%0, %1}, %2;" : "=f"(o[0]), "=f"(o[1]) : "l"(v)); }
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
// bytes k and k + 1 of w as exact floats (0x4B0000qq is 2^23 + qq)
__device__ __forceinline__ f32x2 qbytes2(uint32_t w, int k) {
  return add2(pack2(__uint_as_float(__byte_perm(w, 0x4B000000u, 0x7440u + (uint32_t)k)),
                    __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7441u + (uint32_t)k))),
              pack2(-8388608.0f, -8388608.0f));
}

// three-input minimum / maximum (one instruction on sm_100 and later)
__device__ __forceinline__ float fmax3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
__device__ __forceinline__ float fmin3(float a, float b, float c) {
  float d;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

// bit i of m moves to bit i ^ x (x in 0..7)
__device__ __forceinline__ uint32_t permute_xor8(uint32_t m, int x) {
  if (x & 1) m = ((m & 0x55u) << 1) | ((m >> 1) & 0x55u);
  if (x & 2) m = ((m & 0x33u) << 2) | ((m >> 2) & 0x33u);
  if (x & 4) m = ((m & 0x0Fu) << 4) | ((m >> 4) & 0x0Fu);
  return m;
}

// Node group of the wide traversal: the node index of the first inner child,
// the node's inner-child mask and the not yet visited inner children that the
// ray hit, in traversal order (bit i: slot i ^ oct)
struct WGroup {
  int base;
  uint32_t bits;  // hits | imask << 8
};

// One wide node against the ray (slab test of its eight quantised child
// boxes against [0, tmax)): the group of its hit inner children and the
// mask of its hit leaves' triangles (bit k: triangle slot tri_base + k).
__device__ __forceinline__ void wnode_visit(const WNode* __restrict__ n, const WRay& r, float tmax, WGroup& g,
                                            uint32_t& tri_mask, int& tri_base) {
  const float4 a = __ldg(reinterpret_cast<const float4*>(n));
  const int4 b = __ldg(reinterpret_cast<const int4*>(n) + 1);
  const uint4 c = __ldg(reinterpret_cast<const uint4*>(n) + 2);  // qlo_x, qlo_y
  const uint4 d = __ldg(reinterpret_cast<const uint4*>(n) + 3);  // qlo_z, qhi_x
  const uint4 e = __ldg(reinterpret_cast<const uint4*>(n) + 4);  // qhi_y, qhi_z
  const uint32_t em = __float_as_uint(a.w);
  // plane q of axis x at distance (p + q 2^e - o) / d = q sx + bx.  (Folding
  // the bytes' 2^23 bias into bx saves the subtraction but rounds bx by up
  // to half a grid step, which needs a step of margin around every box:
  // measured on GB300, twice the triangle tests per shadow ray and no gain.)
  const float sx = __uint_as_float((em & 0xFFu) << 23) * r.inv.x;
  const float sy = __uint_as_float(((em >> 8) & 0xFFu) << 23) * r.inv.y;
  const float sz = __uint_as_float(((em >> 16) & 0xFFu) << 23) * r.inv.z;
  const float bx = (a.x - r.o.x) * r.inv.x;
  const float by = (a.y - r.o.y) * r.inv.y;
  const float bz = (a.z - r.o.z) * r.inv.z;
  const f32x2 sx2 = pack2(sx, sx), sy2 = pack2(sy, sy), sz2 = pack2(sz, sz);
  const f32x2 bx2 = pack2(bx, bx), by2 = pack2(by, by), bz2 = pack2(bz, bz);
  // near and far planes per axis: the low planes are near for a positive direction
  const bool nx = r.oct & 1, ny = r.oct & 2, nz = r.oct & 4;
  const uint32_t nx0 = nx ? d.z : c.x, nx1 = nx ? d.w : c.y, fx0 = nx ? c.x : d.z, fx1 = nx ? c.y : d.w;
  const uint32_t ny0 = ny ? e.x : c.z, ny1 = ny ? e.y : c.w, fy0 = ny ? c.z : e.x, fy1 = ny ? c.w : e.y;
  const uint32_t nz0 = nz ? e.z : d.x, nz1 = nz ? e.w : d.y, fz0 = nz ? d.x : e.z, fz1 = nz ? d.y : e.w;
  // two children per packed FP32 instruction: the kernel is bound by
  // instruction issue, and fma / add on f32x2 round as the scalar ones do
  uint32_t hits = 0;
#pragma unroll
  for (int s = 0; s < 8; s += 2) {
    const int k = s & 3;
    float tnx[2], tfx[2], tny[2], tfy[2], tnz[2], tfz[2];
    unpack2(fma2(qbytes2(s < 4 ? nx0 : nx1, k), sx2, bx2), tnx);
    unpack2(fma2(qbytes2(s < 4 ? fx0 : fx1, k), sx2, bx2), tfx);
    unpack2(fma2(qbytes2(s < 4 ? ny0 : ny1, k), sy2, by2), tny);
    unpack2(fma2(qbytes2(s < 4 ? fy0 : fy1, k), sy2, by2), tfy);
    unpack2(fma2(qbytes2(s < 4 ? nz0 : nz1, k), sz2, bz2), tnz);
    unpack2(fma2(qbytes2(s < 4 ? fz0 : fz1, k), sz2, bz2), tfz);
#pragma unroll
    for (int j = 0; j < 2; j++) {
      const float tn = fmax3(tnx[j], tny[j], fmaxf(tnz[j], 0.0f));
      const float tf = fmin3(tfx[j], tfy[j], fminf(tfz[j], tmax));
      hits |= (tn <= tf) ? (1u << (s + j)) : 0u;
    }
  }
  const uint32_t imask = em >> 24;
  uint32_t tm = 0;
  for (uint32_t leaves = hits & ~imask; leaves; leaves &= leaves - 1u) {
    const uint32_t m = __byte_perm((uint32_t)b.z, (uint32_t)b.w, __ffs(leaves) - 1u) & 0xFFu;
    tm |= (m >> 5) << (m & 31u);
  }
  g.base = b.x;
  g.bits = permute_xor8(hits & imask, r.oct) | imask << 8;
  tri_mask = tm;
  tri_base = b.y;
}

// the next child of a group (its lowest pending hit); clears it
__device__ __forceinline__ int wgroup_next(WGroup& g, int oct) {
  const int i = __ffs(g.bits & 0xFFu) - 1;
  g.bits &= ~(1u << i);
  const int s = i ^ oct;
  return g.base + __popc((g.bits >> 8) & ((1u << s) - 1u));
}

// the root of a mesh as a group with one pending child
__device__ __forceinline__ WGroup wgroup_root(int root, int oct) {
  WGroup g;
  g.base = root;
  g.bits = (1u << oct) | (1u << 8);  // pending bit oct is slot 0, the only inner child
  return g;
}

// Wide-BVH closest hit (ANY = false) or any hit below tmax (ANY = true):
// children are visited near to far by the slot order, each node's leaf
// triangles tested as soon as the node is visited.
template <bool ANY>
__device__ __forceinline__ bool fast_qbvh(const DevScene& S, const GEntF& e, const WRay& r, float& tbest, int& slot,
                                          float& bu, float& bv, TraceStats& st, uint32_t* err) {
  WGroup stack[kWStack];
  int sp = 0;
  WGroup g = wgroup_root(e.node_base, r.oct);
  bool hit = false;
  int guard = 0;
  while (true) {
    if ((g.bits & 0xFFu) == 0) {
      if (sp == 0) break;
      g = stack[--sp];
    }
    if (++guard > (1 << 22)) { atomicOr(err, PR_DEV_LOOP_CAP); break; }
    const int child = wgroup_next(g, r.oct);
    if (g.bits & 0xFFu) {
      if (sp >= kWStack) { atomicOr(err, PR_DEV_STACK_OVERFLOW); return hit; }
      stack[sp++] = g;
    }
    st.nodes++;
    uint32_t tm;
    int tb;
    wnode_visit(S.rnodes + child, r, tbest, g, tm, tb);
    while (tm) {
      const int k = __ffs(tm) - 1;
      tm &= tm - 1u;
      st.tris++;
      float t, uu, vv;
      if (fast_tri(S.rtris + 3 * (size_t)(tb + k), r.o, r.d, tbest, t, uu, vv)) {
        tbest = t;
        slot = tb + k;
        bu = uu;
        bv = vv;
        hit = true;
        if (ANY) return true;
      }
    }
  }
  return hit;
}

// FP64 sphere distance of an FP32 ray; threshold PS_EPS as in sphere.h:80-87
__device__ __forceinline__ bool sphere_t64(const GEntity& e, float3 o, float3 d, double& tt) {
  const double px = e.p[0] - (double)o.x, py = e.p[1] - (double)o.y, pz = e.p[2] - (double)o.z;
  const double b = px * (double)d.x + py * (double)d.y + pz * (double)d.z;
  const double D4 = b * b - (px * px + py * py + pz * pz) + e.radius * e.radius;
  if (D4 < 0.0) return false;
  const double s = sqrt(D4);
  const double t1 = b - s, t2 = b + s;
  if (t1 < kEps && t2 < kEps) return false;
  tt = (t1 > kEps) ? t1 : t2;
  return true;
}

// t is the FP32 distance, rest what it rounded off (t + rest is the FP64
// distance to ~2^-48: the hit point is rebuilt from it, since the FP32
// distance alone is up to half an ulp of t off -- 1.5e-5 beyond t = 256, as
// much as the origin offset of the next ray near a coordinate of zero)
__device__ __forceinline__ bool fast_sphere(const GEntity& e, float3 o, float3 d, float tmax, float& t, float& rest) {
  double tt;
  if (!sphere_t64(e, o, d, tt) || !(tt < (double)tmax)) return false;
  // a hemisphere keeps the hit only on its y >= y_centre half (sphere.h:98-103)
  if (e.hemisphere && (double)o.y + tt * (double)d.y - e.p[1] < 0.0) return false;
  t = (float)tt;
  rest = (float)(tt - (double)t);
  return true;
}

// UVPlane::intersect semantics in FP32 (plane.h:86-110, :220-239): the
// extent check compares u / |U| against |U| (the reference's own rule).
__device__ __forceinline__ bool fast_uvplane(const GEntF& e, float3 o, float3 d, float tmax, float& t) {
  const float s = e.normal_inverse < 0 ? -1.0f : 1.0f;
  const float3 n = f3(e.n[0] * s, e.n[1] * s, e.n[2] * s);
  const float dd = dot(d, n);
  if (fabsf(dd) < 1.0e-14f) return false;
  const float3 org = f3(e.p[0], e.p[1], e.p[2]);
  const float tt = dot(org - o, n) / dd;
  if (!(tt > 0.0f) || !(tt < tmax)) return false;
  const float3 rel = (o + d * tt) - org;
  const float ul = e.u_length, vl = e.v_length;
  const float u = dot(rel, f3(e.u[0], e.u[1], e.u[2])) / ul;
  const float v = dot(rel, f3(e.v[0], e.v[1], e.v[2])) / vl;
  if (u < 0.0f || u > ul || v < 0.0f || v > vl) return false;
  t = tt;
  return true;
}

// Circle::intersect in FP32 (circle.h:177-200): plane test, then the annulus
// (u_length = radius, v_length = inner radius)
__device__ __forceinline__ bool fast_circle(const GEntF& e, float3 o, float3 d, float tmax, float& t) {
  const float3 n = f3(e.n[0], e.n[1], e.n[2]);
  const float dd = dot(d, n);
  if (fabsf(dd) < 1.0e-14f) return false;
  const float3 org = f3(e.p[0], e.p[1], e.p[2]);
  const float tt = dot(org - o, n) / dd;
  if (!(tt > 0.0f) || !(tt < tmax)) return false;
  const float3 rel = (o + d * tt) - org;
  const float r2 = dot(rel, rel);
  if (r2 > e.u_length * e.u_length || r2 < e.v_length * e.v_length) return false;
  t = tt;
  return true;
}

// ---- spheres without FP64 ---------------------------------------------
// GB300 issues one FP64 warp instruction per 16 clocks and SM (64 per
// scheduler) whatever number of lanes is active, so the nine FP64 sphere
// tests of a ray in the sphere Cornell box, not memory, bound such scenes
// (FP64 pipe 85 % busy).  The FP64 test is kept for the spheres that can
// still be the answer; the others are ruled out in FP32 with error bounds:
// along the ray the test solves F(t) = t^2 + 2 b t + c = 0, with b = d.(o-C)
// and c = |o-C|^2 - r^2.  From an anchor A (the centre, or for a sphere much
// larger than the scene the point of its surface nearest to the scene, which
// keeps the cancellation out of c) with w = o - A and q = A - C:
//   b = d.w + d.q,  c = w.w + 2 w.q + c0,  c0 = |q|^2 - r^2.
// A is a float triple exactly; q and c0 carry FP32 high and low parts
// (GEntF::v / n, u_length / v_length).  kSphErr = 16 rounding units bounds
// each sum's error relative to its terms' magnitudes.
constexpr float kSphErr = 1.0e-6f;
constexpr float kSphNear = 1.0e-5f;  // above the test's own threshold of 1e-6

struct SphF {
  float b, c, eb, ec;  // coefficients and their error bounds
};

__device__ __forceinline__ SphF sph_coeffs(const GEntF& e, float3 o, float3 d, float dmax) {
  const float3 w = o - f3(e.u[0], e.u[1], e.u[2]), q = f3(e.v[0], e.v[1], e.v[2]);
  const float m = fabsf(w.x) + fabsf(w.y) + fabsf(w.z), Q = fabsf(q.x) + fabsf(q.y) + fabsf(q.z);
  SphF f;
  f.b = dot(d, w) + dot(d, q);
  f.c = dot(w, w) + 2.0f * dot(w, q) + e.u_length;
  f.eb = kSphErr * (m + Q) * dmax;
  f.ec = kSphErr * (m * m + 2.0f * m * Q + fabsf(e.u_length));
  return f;
}
__device__ __forceinline__ float sph_val(const SphF& f, float t) { return fmaf(t, t + 2.0f * f.b, f.c); }
__device__ __forceinline__ float sph_err(const SphF& f, float t) {
  return f.ec + 2.0f * t * f.eb + kSphErr * (t * (t + 2.0f * fabsf(f.b)) + fabsf(f.c));
}

// c to about 1e-13 of its terms (two-float sums and products: Dekker 1971,
// Knuth; the products' errors by fma), for an origin on the sphere itself
// (where a ray that just left it starts), whose c FP32 cannot tell from 0
__device__ __forceinline__ void two_add(float& s, float& e, float x) {
  const float t = __fadd_rn(s, x), z = __fsub_rn(t, s);
  e += __fadd_rn(__fsub_rn(s, __fsub_rn(t, z)), __fsub_rn(x, z));
  s = t;
}
__device__ __forceinline__ float sph_c_refined(const GEntF& e, float3 o) {
  float s = e.u_length, err = e.v_length;
  const float oo[3] = {o.x, o.y, o.z};
#pragma unroll
  for (int a = 0; a < 3; a++) {
    const float A = e.u[a];
    float w = oo[a], wl = 0.0f;  // w + wl = o - A exactly
    two_add(w, wl, -A);
    float y = w, yl = wl + 2.0f * e.n[a];  // y + yl = w + 2 q
    two_add(y, yl, 2.0f * e.v[a]);
    const float p = __fmul_rn(w, y);
    two_add(s, err, p);
    err += fmaf(w, y, -p) + (w * yl + wl * y);
  }
  return s + err;
}

// rules sphere e out: no hit of it can lie below the limit T
__device__ __forceinline__ bool sph_reject(const SphF& f, float T) {
  const float v = sph_val(f, T), ev = sph_err(f, T);
  if (f.c < -f.ec) return v < -ev;  // the origin is inside: the exit lies beyond T
  if (f.c > f.ec) {
    if (f.b > f.eb) return true;  // outside and behind
    const float D = f.b * f.b - f.c;
    if (D < -(2.0f * fabsf(f.b) * f.eb + f.eb * f.eb + f.ec + kSphErr * f.b * f.b)) return true;  // passes by
    return v > ev && T < -f.b - f.eb;  // the entry lies beyond T
  }
  return false;
}

// the same for an origin on the sphere: the near root lies below the test's
// threshold (so the far one would be returned) and the far one beyond T
__device__ __forceinline__ bool sph_reject_surface(const GEntF& e, const SphF& f, float3 o, float T) {
  const float c = sph_c_refined(e, o);
  // error of c (1e-12 of its terms), and half of F(1e-6) - c = 2 b 1e-6 as room
  const float room = 1.0e-6f * fabsf(f.b) - 1.0e-6f * f.ec;
  if (!(room > 0.0f)) return false;
  if (f.b > f.eb) return c > -room;  // leaving outward: both roots below 1e-6
  if (f.b < -f.eb) return c < room && sph_val(f, T) < -sph_err(f, T);
  return false;
}

// an upper bound of sphere e's hit distance, where it is certain to be hit
// (the caller excludes hemispheres); 3e38 where it is not
__device__ __forceinline__ float sph_upper(const SphF& f) {
  const float D = f.b * f.b - f.c;
  if (!(D > 0.0f)) return 3.0e38f;
  const float s = sqrtf(D);
  const float vn = sph_val(f, kSphNear), en = sph_err(f, kSphNear);
  if (f.c < -f.ec) {
    const float t = (f.b <= 0.0f ? s - f.b : __fdividef(-f.c, f.b + s)) * 1.001f + 1.0e-3f;
    return (vn < -en && sph_val(f, t) > sph_err(f, t)) ? t : 3.0e38f;
  }
  if (f.c > f.ec && f.b < -f.eb) {
    const float t = __fdividef(f.c, s - f.b) * 1.001f + 1.0e-3f;
    return (vn > en && sph_val(f, t) < -sph_err(f, t)) ? t : 3.0e38f;
  }
  return 3.0e38f;
}

// The run of consecutive spheres of the entity list from i on (i moves past
// it): the closest one below h.t, as the FP64 test of each in list order
// finds it.  Spheres ruled out by the FP32 bounds lie beyond a certain hit
// of another one (by more than a float rounding), so leaving them out does
// not change which sphere wins nor its distance.
__device__ __forceinline__ void sphere_run_closest(const DevScene& S, int& i, float3 o, float3 d, FastHit& h) {
  const int first = i;
  const float dmax = fmaxf(1.0f, fmaxf(fabsf(d.x), fmaxf(fabsf(d.y), fabsf(d.z))));
  unsigned long long left = 0;  // spheres not ruled out (bit: index in the run)
  float T = h.t;
  for (; i < S.n_ents && S.entf[i].type == PR_ENT_SPHERE; i++) {
    const GEntF& e = S.entf[i];
    const SphF f = sph_coeffs(e, o, d, dmax);
    if (sph_reject(f, T)) continue;
    left |= 1ull << (i - first);
    if (!e.node_base) T = fminf(T, sph_upper(f));  // node_base: a hemisphere
  }
  while (left) {
    const int k = first + __ffsll((long long)left) - 1;
    left &= left - 1;
    const GEntF& e = S.entf[k];
    const SphF f = sph_coeffs(e, o, d, dmax);
    const float Tk = fminf(T, h.t);
    if (sph_reject(f, Tk) || (fabsf(f.c) <= f.ec && sph_reject_surface(e, f, o, Tk))) continue;
    float t, rest;
    if (fast_sphere(S.ents[k], o, d, h.t, t, rest) && t < h.t) {
      h.t = t;
      h.ent = k;
      h.slot = -1;
      h.u = rest;
      h.v = 0.0f;
    }
  }
}

// the run's any-hit query: a sphere hit below tmax, or -1
__device__ __forceinline__ int sphere_run_any(const DevScene& S, int& i, float3 o, float3 d, float tmax) {
  const float dmax = fmaxf(1.0f, fmaxf(fabsf(d.x), fmaxf(fabsf(d.y), fabsf(d.z))));
  const int first = i;
  unsigned long long left = 0;
  int found = -1;
  for (; i < S.n_ents && S.entf[i].type == PR_ENT_SPHERE; i++) {
    const GEntF& e = S.entf[i];
    const SphF f = sph_coeffs(e, o, d, dmax);
    if (sph_reject(f, tmax)) continue;
    if (!e.node_base && sph_upper(f) < tmax) found = i;
    left |= 1ull << (i - first);
  }
  if (found >= 0) return found;
  while (left) {
    const int k = first + __ffsll((long long)left) - 1;
    left &= left - 1;
    const GEntF& e = S.entf[k];
    const SphF f = sph_coeffs(e, o, d, dmax);
    if (fabsf(f.c) <= f.ec && sph_reject_surface(e, f, o, tmax)) continue;
    float t, rest;
    if (fast_sphere(S.ents[k], o, d, tmax, t, rest)) return k;
  }
  return -1;
}

// ---- persistent traversal: one ray per lane, advanced step by step ---------
enum : int { TRACE_CLOSEST = 0, TRACE_ANY = 1, TRACE_EITHER = 2 };

struct TraceLane {
  WRay ray;
  float tmax;    // current closest (closest hit) or the ray's limit (any hit)
  int ent;       // next entity of the list to test (the current mesh while in_mesh)
  int sp;        // node groups on the traversal stack
  bool in_mesh;  // inside the traversal of mesh 'ent'
  bool any;      // TRACE_EITHER: an any-hit ray
  WGroup g;      // the current node group
  FastHit h;
};

__device__ __forceinline__ void lane_start(TraceLane& r, float3 o, float3 d, float tmax) {
  r.ray = make_wray(o, d);
  r.tmax = tmax;
  r.ent = 0;
  r.sp = 0;
  r.in_mesh = false;
  r.g.base = 0;
  r.g.bits = 0;
  r.h.t = tmax;
  r.h.ent = -1;
  r.h.slot = -1;
  r.h.u = r.h.v = 0.0f;
}

// The bounds of a whole mesh against the ray (GEntF::u, v: the root's child
// boxes together): a mesh missed here costs 20 instructions instead of a
// node visit.  The bounds hold the padded root box, so no triangle is lost.
__device__ __forceinline__ bool mesh_bounds_hit(const GEntF& e, const WRay& r, float tmax) {
  const float x0 = (e.u[0] - r.o.x) * r.inv.x, x1 = (e.v[0] - r.o.x) * r.inv.x;
  const float y0 = (e.u[1] - r.o.y) * r.inv.y, y1 = (e.v[1] - r.o.y) * r.inv.y;
  const float z0 = (e.u[2] - r.o.z) * r.inv.z, z1 = (e.v[2] - r.o.z) * r.inv.z;
  const float tn = fmax3(fminf(x0, x1), fminf(y0, y1), fmaxf(fminf(z0, z1), 0.0f));
  const float tf = fmin3(fmaxf(x0, x1), fmaxf(y0, y1), fminf(fmaxf(z0, z1), tmax));
  return tn <= tf;
}

// One step of a ray, in three parts: trace_visit goes through the other
// entities up to the next mesh the ray may meet (if it is not in one) and
// visits one node of that mesh; warp_triangles tests the triangles of the
// leaves that the warp's rays hit there; trace_next leaves a finished mesh.
// True when the ray is answered (any hit: h.ent >= 0 means occluded).
// tm, tb: the node's triangles to test (bit k: triangle slot tb + k).
template <int MODE>
__device__ __forceinline__ bool trace_visit(const DevScene& S, TraceLane& r, WGroup* stack, TraceStats& st,
                                            uint32_t* err, uint32_t& tm, int& tb) {
  const bool any = MODE == TRACE_ANY || (MODE == TRACE_EITHER && r.any);
  if (!r.in_mesh) {
    while (r.ent < S.n_ents) {
      const int i = r.ent;
      const GEntF& e = S.entf[i];
      if (e.type == PR_ENT_POLYGON) {
        if (mesh_bounds_hit(e, r.ray, r.tmax)) {
          r.g = wgroup_root(e.node_base, r.ray.oct);
          r.sp = 0;
          r.in_mesh = true;
          break;
        }
        r.ent++;
        continue;
      }
      if (e.type == PR_ENT_SPHERE) {
        if (any) {
          r.h.ent = sphere_run_any(S, r.ent, r.ray.o, r.ray.d, r.tmax);
          if (r.h.ent >= 0) return true;
        } else {
          sphere_run_closest(S, r.ent, r.ray.o, r.ray.d, r.h);
          r.tmax = r.h.t;
        }
        continue;
      }
      float t = r.tmax;
      bool got = false;
      if (e.type == PR_ENT_UVPLANE) got = fast_uvplane(e, r.ray.o, r.ray.d, r.tmax, t);
      else if (e.type == PR_ENT_CIRCLE) got = fast_circle(e, r.ray.o, r.ray.d, r.tmax, t);
      r.ent++;
      if (any && got) {  // the test itself keeps t below the limit
        r.h.ent = i;
        return true;
      }
      if (got && t < r.tmax) {
        r.h.ent = i;
        r.h.slot = -1;
        r.h.u = r.h.v = 0.0f;
        r.tmax = t;
        r.h.t = t;
      }
    }
    if (!r.in_mesh) return true;  // past the last entity
  }
  if ((r.g.bits & 0xFFu) == 0) r.g = stack[--r.sp];  // stacked groups always hold a pending child
  const int child = wgroup_next(r.g, r.ray.oct);
  if (r.g.bits & 0xFFu) {
    if (r.sp >= kWStack) {
      atomicOr(err, PR_DEV_STACK_OVERFLOW);
      return true;
    }
    stack[r.sp++] = r.g;
  }
  st.nodes++;
  wnode_visit(S.rnodes + child, r.ray, r.tmax, r.g, tm, tb);
  return false;
}

// The triangles of a step (tm, tb of every lane; none where tm is 0), spread
// over the warp: a node visit leaves 1.25 triangles a ray on average but many
// on some, and tested by their own lanes they were more than half of the
// traversal's instructions at some six lanes each.  Lane j takes the j-th
// (ray, triangle) pair, its ray by shuffles; a hit goes to the warp's 32
// entries of `found`, and the ray's lane takes its hits in the order of its
// triangles, the strictly closest first, as one lane alone would.
// True where an any-hit ray met a triangle.  All lanes of the warp.
template <int MODE>
__device__ __forceinline__ bool warp_triangles(const DevScene& S, TraceLane& r, uint32_t tm, int tb, float4* found,
                                               TraceStats& st) {
  if (!__any_sync(0xffffffffu, tm != 0)) return false;
  const bool any = MODE == TRACE_ANY || (MODE == TRACE_EITHER && r.any);
  const int lane = threadIdx.x & 31, cnt = __popc(tm);
  int incl = cnt;  // pairs of lanes 0..lane
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, off);
    if (lane >= off) incl += v;
  }
  const int total = __shfl_sync(0xffffffffu, incl, 31), excl = incl - cnt;
  bool met = false;
  for (int base = 0; base < total; base += 32) {
    const int j = base + lane;
    int own = 0;  // the lane of pair j: the number of lanes with incl <= j
#pragma unroll
    for (int s = 16; s; s >>= 1)
      if (__shfl_sync(0xffffffffu, incl, own + s - 1) <= j) own += s;
    int k = j - __shfl_sync(0xffffffffu, excl, own);
    uint32_t m = __shfl_sync(0xffffffffu, tm, own);
    int slot = __shfl_sync(0xffffffffu, tb, own);
    const float3 o = f3(__shfl_sync(0xffffffffu, r.ray.o.x, own), __shfl_sync(0xffffffffu, r.ray.o.y, own),
                        __shfl_sync(0xffffffffu, r.ray.o.z, own));
    const float3 d = f3(__shfl_sync(0xffffffffu, r.ray.d.x, own), __shfl_sync(0xffffffffu, r.ray.d.y, own),
                        __shfl_sync(0xffffffffu, r.ray.d.z, own));
    const float tmax = __shfl_sync(0xffffffffu, r.tmax, own);
    bool hit = false;
    if (j < total) {
      for (; k > 0; k--) m &= m - 1u;
      slot += __ffs(m) - 1;
      float t, u, v;
      hit = fast_tri(S.rtris + 3 * (size_t)slot, o, d, tmax, t, u, v);
      if (hit) found[lane] = make_float4(t, u, v, __int_as_float(slot));
    }
    const uint32_t hits = __ballot_sync(0xffffffffu, hit);
    __syncwarp();  // a vote orders no memory: the lanes' found[] before the reads of other lanes
    const int lo = max(excl - base, 0), hi = min(incl - base, 32);
    if (hits && hi > lo && !met) {
      uint32_t mine = hits & (0xffffffffu >> (32 - (hi - lo))) << lo;
      while (mine) {
        const int q = __ffs(mine) - 1;
        mine &= mine - 1u;
        const float4 f = found[q];
        if (!(f.x < r.tmax)) continue;
        r.h.ent = r.ent;
        r.h.slot = __float_as_int(f.w);
        if (any) {
          met = true;
          st.tris += base + q - excl + 1;
          break;
        }
        r.tmax = f.x;
        r.h.t = f.x;
        r.h.u = f.y;
        r.h.v = f.z;
      }
    }
    __syncwarp();  // all reads before the next pairs' hits
  }
  if (!met) st.tris += cnt;
  return met;
}

// leaves a mesh whose nodes are all visited; true past the last entity
__device__ __forceinline__ bool trace_next(const DevScene& S, TraceLane& r) {
  if ((r.g.bits & 0xFFu) == 0 && r.sp == 0) {
    r.in_mesh = false;  // this mesh is done
    r.ent++;
    return r.ent >= S.n_ents;
  }
  return false;
}

// One step of all lanes of a warp; true for a lane whose ray is answered.
template <int MODE>
__device__ __forceinline__ bool trace_step(const DevScene& S, bool busy, TraceLane& r, WGroup* stack, float4* found,
                                           TraceStats& st, uint32_t* err) {
  uint32_t tm = 0;
  int tb = 0;
  bool done = busy && trace_visit<MODE>(S, r, stack, st, err, tm, tb);
  const bool met = warp_triangles<MODE>(S, r, tm, tb, found, st);
  if (busy && !done) done = met || trace_next(S, r);
  return done;
}

// closest hit over the entity list (strict '<' in list order)
__device__ __forceinline__ bool fast_closest(const DevScene& S, float3 o, float3 d, FastHit& h, TraceStats& st,
                                             uint32_t* err) {
  h.t = 3.0e38f;
  h.ent = -1;
  h.slot = -1;
  h.u = h.v = 0.0f;
  const WRay r = make_wray(o, d);
  for (int i = 0; i < S.n_ents;) {
    const GEntF& e = S.entf[i];
    if (e.type == PR_ENT_SPHERE) {
      sphere_run_closest(S, i, o, d, h);
      continue;
    }
    float t = h.t, bu = 0.0f, bv = 0.0f;
    int slot = -1;
    bool got = false;
    if (e.type == PR_ENT_UVPLANE) got = fast_uvplane(e, o, d, h.t, t);
    else if (e.type == PR_ENT_CIRCLE) got = fast_circle(e, o, d, h.t, t);
    else if (e.type == PR_ENT_POLYGON && mesh_bounds_hit(e, r, h.t)) got = fast_qbvh<false>(S, e, r, t, slot, bu, bv, st, err);
    if (got && t < h.t) {
      h.t = t;
      h.ent = i;
      h.slot = slot;
      h.u = bu;
      h.v = bv;
    }
    i++;
  }
  return h.ent >= 0;
}

// any hit with t < tmax
__device__ __forceinline__ bool fast_occluded(const DevScene& S, float3 o, float3 d, float tmax, TraceStats& st,
                                              uint32_t* err) {
  const WRay r = make_wray(o, d);
  for (int i = 0; i < S.n_ents;) {
    const GEntF& e = S.entf[i];
    if (e.type == PR_ENT_SPHERE) {
      if (sphere_run_any(S, i, o, d, tmax) >= 0) return true;
      continue;
    }
    float t = tmax, bu, bv;
    int slot;
    bool got = false;
    if (e.type == PR_ENT_UVPLANE) got = fast_uvplane(e, o, d, tmax, t);
    else if (e.type == PR_ENT_CIRCLE) got = fast_circle(e, o, d, tmax, t);
    else if (e.type == PR_ENT_POLYGON && mesh_bounds_hit(e, r, tmax)) got = fast_qbvh<true>(S, e, r, t, slot, bu, bv, st, err);
    if (got) return true;
    i++;
  }
  return false;
}

}  // namespace pr
