// sphere_run_closest and sphere_run_any (trace_fast.cuh) against the FP64 test
// of every sphere in list order, decisions and distances exactly: walls of
// radius 1e5, shells and needle's-eye gaps, hemispheres, radii over six
// decades; origins on, just off, inside and outside of the surfaces; any-hit
// limits at the closest distance, one float to either side of it, near it and
// anywhere; directions of length 1 or the given one.
#include "host_cuda.h"

#include <cstdio>
#include <cstdlib>
#include <random>

#include "../../prender_gb300/csrc/sphere_bounds.h"
#include "../../prender_gb300/csrc/trace_fast.cuh"

using namespace pr;

static std::mt19937_64 rng(5);
static double uni(double a, double b) { return std::uniform_real_distribution<double>(a, b)(rng); }
static void unit(double* v) {
  double l;
  do {
    for (int k = 0; k < 3; k++) v[k] = uni(-1, 1);
    l = sqrt(v[0] * v[0] + v[1] * v[1] + v[2] * v[2]);
  } while (l < 0.1 || l > 1.0);
  for (int k = 0; k < 3; k++) v[k] /= l;
}

static std::vector<GEntity> scene(const char* name) {
  std::vector<GEntity> s;
  auto add = [&](double x, double y, double z, double r, int hemi = 0) {
    GEntity e;
    memset(&e, 0, sizeof(e));
    e.type = PR_ENT_SPHERE;
    e.p[0] = x;
    e.p[1] = y;
    e.p[2] = z;
    e.radius = r;
    e.hemisphere = hemi;
    s.push_back(e);
  };
  if (!strcmp(name, "walls")) {
    add(1e5 + 1, 40.8, 81.6, 1e5);
    add(-1e5 + 99, 40.8, 81.6, 1e5);
    add(50, 40.8, 1e5, 1e5);
    add(50, 40.8, -1e5 + 250, 1e5);
    add(50, 1e5, 81.6, 1e5);
    add(50, -1e5 + 81.6, 81.6, 1e5);
    add(65, 20, 20, 20);
    add(27, 16.5, 47, 16.5);
    add(77, 16.5, 78, 16.5);
    add(50, 90, 81.6, 15);
  } else if (!strcmp(name, "nested")) {
    for (double r : {1e-3, 0.5, 0.500001, 7.0, 300.0, 4.0e4}) add(1, 2, 3, r);
    add(1, 1e6 + 60, 3, 1e6);
  } else if (!strcmp(name, "hemispheres")) {
    for (int k = 0; k < 6; k++) add(uni(-5, 5), uni(-5, 5), uni(-5, 5), uni(0.5, 4), k % 2);
    add(0, -2e4, 0, 2e4, 1);
  } else {
    for (int k = 0; k < kMaxEntities; k++) add(uni(-50, 50), uni(-50, 50), uni(-50, 50), pow(10, uni(-3, 3)));
  }
  return s;
}

int main(int argc, char** argv) {
  const double len = atof(argv[2]);
  std::vector<GEntity> ents = scene(argv[1]);
  static DevScene S;
  S.ents = ents.data();
  S.n_ents = (int)ents.size();
  double mid[3] = {0, 0, 0};
  int n_small = 0;
  for (int i = 0; i < S.n_ents; i++) {
    S.entf[i].type = ents[i].type;
    if (ents[i].radius <= 1e3) {
      n_small++;
      for (int k = 0; k < 3; k++) mid[k] += ents[i].p[k];
    }
  }
  sphere_bounds(ents.data(), S.n_ents, S.entf);
  long wrong = 0, hits = 0, shadow = 0, any = 0;
  const int n = 200000;
  for (int ray = 0; ray < n; ray++) {
    const GEntity& e = ents[rng() % ents.size()];
    double u[3], d[3];
    unit(u);
    unit(d);
    if (e.radius > 1e3) {  // the side of a large sphere that faces the others
      double l = 0;
      for (int k = 0; k < 3; k++) {
        u[k] = mid[k] / n_small - e.p[k] + uni(-30, 30);
        l += u[k] * u[k];
      }
      for (int k = 0; k < 3; k++) u[k] /= sqrt(l);
    }
    const double offs[5] = {0, 1e-5, -1e-5, 1e-3, -1e-3}, off = offs[rng() % 5];
    double o[3];
    for (int k = 0; k < 3; k++)
      o[k] = ray % 4 == 0 ? uni(-60, 110) : e.p[k] + u[k] * (e.radius * (e.radius > 1e3 ? 1.0 : 1.0 + off) + off);
    if (ray % 7 == 0)  // along the surface
      for (int k = 0; k < 3; k++) d[k] = d[k] - u[k] * (d[0] * u[0] + d[1] * u[1] + d[2] * u[2]);
    const float3 of = f3((float)o[0], (float)o[1], (float)o[2]);
    const float3 df = f3((float)(len * d[0]), (float)(len * d[1]), (float)(len * d[2]));
    FastHit ref, got;
    ref.t = got.t = ray % 3 ? 3.0e38f : (float)uni(1e-4, 200);
    ref.ent = got.ent = -1;
    ref.u = got.u = 0;
    for (int i = 0; i < S.n_ents; i++) {
      float t, rest;
      if (fast_sphere(ents[i], of, df, ref.t, t, rest) && t < ref.t) {
        ref.t = t;
        ref.ent = i;
        ref.u = rest;
      }
    }
    int i = 0;
    sphere_run_closest(S, i, of, df, got);
    hits += ref.ent >= 0;
    wrong += i != S.n_ents || got.ent != ref.ent || got.t != ref.t || (ref.ent >= 0 && got.u != ref.u);
    const float t = ref.ent >= 0 ? ref.t : 10.0f;
    const float limit[7] = {t, nextafterf(t, 0.0f), nextafterf(t, 3e38f), 0.999f * t, 1.001f * t, t + 1e-3f,
                            (float)uni(1e-4, 200)};
    for (float tmax : limit) {
      bool hit = false;
      for (int k = 0; k < S.n_ents && !hit; k++) {
        float tt, rest;
        hit = fast_sphere(ents[k], of, df, tmax, tt, rest);
      }
      int j = 0;
      const int r = sphere_run_any(S, j, of, df, tmax);
      float tt, rest;
      any++;
      shadow += hit;
      wrong += (r >= 0) != hit || (r >= 0 && !fast_sphere(ents[r], of, df, tmax, tt, rest));
    }
  }
  printf("wrong %ld hits %ld of %d, occluded %ld of %ld\n", wrong, hits, n, shadow, any);
  return wrong || hits < n / 10 || shadow < any / 10;
}
