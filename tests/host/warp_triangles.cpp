// warp_triangles (trace_fast.cuh) on 32 host lanes against each lane's own
// triangles one after another, closest and any-hit rays mixed; built with the
// thread sanitizer, which reports accesses of `found` that no fence orders.
#include "host_cuda.h"

#include <cstdio>
#include <random>

#include "../../prender_gb300/csrc/trace_fast.cuh"

using namespace pr;

int main() {
  std::mt19937 rng(7);
  std::uniform_real_distribution<float> u(-1.0f, 1.0f);
  const int kTris = 96, kRounds = 24;
  std::vector<float4> tris(3 * kTris);
  for (auto& v : tris) v = make_float4(2.0f * u(rng), 2.0f * u(rng), u(rng), 0.0f);
  static DevScene S;
  S.rtris = tris.data();
  struct Task {
    TraceLane r;
    uint32_t tm;
    int tb;
  };
  std::vector<Task> in(kRounds * 32), out;
  for (size_t k = 0; k < in.size(); k++) {
    Task& t = in[k];
    const int round = (int)(k / 32);
    lane_start(t.r, f3(u(rng), u(rng), -3.0f), f3(0.2f * u(rng), 0.2f * u(rng), 1.0f), 3.0e38f);
    t.r.any = rng() % 3 == 0;
    t.r.ent = 5;
    // rounds without a triangle, with one each, with 24 on some lanes, with 24 on all
    const uint32_t bits = rng() & 0xFFFFFFu;
    t.tm = round == 0 ? 0 : round == 1 ? 1u << (rng() % 24) : round == 2 ? 0xFFFFFFu : rng() % 4 ? 0u : bits;
    t.tb = (int)(rng() % (kTris - 24));
  }
  out = in;
  std::vector<uint32_t> tests(32, 0), met(in.size(), 0);
  static float4 found[32];
  host::run_warp(32, [&](int l) {
    TraceStats st{0, 0};
    for (int r = 0; r < kRounds; r++) {
      Task& t = out[r * 32 + l];
      met[r * 32 + l] = warp_triangles<TRACE_EITHER>(S, t.r, t.tm, t.tb, found, st);
    }
    tests[l] = st.tris;
  });
  int bad = 0, hits = 0;
  for (int l = 0; l < 32; l++) {
    uint32_t n = 0;
    for (int r = 0; r < kRounds; r++) {
      Task t = in[r * 32 + l];
      bool m = false;
      for (int k = 0; k < 24 && !m; k++) {
        if (!((t.tm >> k) & 1)) continue;
        n++;
        float tt, uu, vv;
        if (!fast_tri(S.rtris + 3 * (size_t)(t.tb + k), t.r.ray.o, t.r.ray.d, t.r.tmax, tt, uu, vv)) continue;
        t.r.h.ent = t.r.ent;
        t.r.h.slot = t.tb + k;
        hits++;
        if (t.r.any) {
          m = true;
        } else {
          t.r.tmax = t.r.h.t = tt;
          t.r.h.u = uu;
          t.r.h.v = vv;
        }
      }
      const Task& o = out[r * 32 + l];
      bad += m != (met[r * 32 + l] != 0) || t.r.h.ent != o.r.h.ent || t.r.h.slot != o.r.h.slot || t.r.tmax != o.r.tmax ||
             t.r.h.t != o.r.h.t || t.r.h.u != o.r.h.u || t.r.h.v != o.r.h.v;
    }
    bad += n != tests[l];
  }
  printf("bad %d hits %d\n", bad, hits);
  return bad || hits < 50;
}
