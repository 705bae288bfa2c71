// segment_draws (geodesic_math.cuh) against the exact segment test that it
// stands in for: where it says that the test need not run, the exact test
// finds nothing within the segment, and the accretion disk's alpha test makes
// as many draws as it says.  Random scenes of every entity kind over six
// decades, origins on, near and off them, directions of the given length.
#include "host_cuda.h"

#include <cstdio>
#include <cstdlib>
#include <random>

#include "../../prender_gb300/csrc/kerr_math.cuh"

using namespace pr;

static std::mt19937_64 rng;
static double uni(double a, double b) { return std::uniform_real_distribution<double>(a, b)(rng); }
static int pick(int n) { return (int)(rng() % n); }
static dv3 unit() {
  for (;;) {
    const dv3 v = {uni(-1, 1), uni(-1, 1), uni(-1, 1)};
    const double l = sqrt(v.x * v.x + v.y * v.y + v.z * v.z);
    if (l > 0.1 && l < 1.0) return {v.x / l, v.y / l, v.z / l};
  }
}
static dv3 cross_(dv3 a, dv3 b) { return {a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x}; }
static dv3 along(dv3 o, dv3 d, double t) { return {o.x + t * d.x, o.y + t * d.y, o.z + t * d.z}; }
static void set(double* p, dv3 v) { p[0] = v.x; p[1] = v.y; p[2] = v.z; }
static void perp(dv3 n, dv3& u, dv3& v) {
  do u = cross_(n, unit());
  while (u.x * u.x + u.y * u.y + u.z * u.z < 0.01);
  const double l = sqrt(u.x * u.x + u.y * u.y + u.z * u.z);
  u = {u.x / l, u.y / l, u.z / l};
  v = cross_(n, u);
}

int main(int argc, char** argv) {
  const double len = atof(argv[1]);
  const bool unit_len = fabs(len - 1.0) < 1.0e-6;
  rng.seed(11);
  const int w = 64, h = 48;
  std::vector<uchar4> tex(w * h);
  for (auto& t : tex) {
    t = make_uchar4(pick(256), pick(256), pick(256), pick(4) ? 255 : pick(256));
    if (pick(4) == 0) t.w = 0;
    if (pick(8) == 0) t.x = t.y = t.z = 0;
  }
  long skipped = 0, wrong = 0, drawn = 0, hits = 0, total = 0;
  for (int scene = 0; scene < 400; scene++) {
    static DevScene S;
    static GEntity ents[kMaxEntities];
    static GNode node[kMaxEntities];
    static float4 tris[kMaxEntities * 3];
    memset(&S, 0, sizeof(S));
    memset(ents, 0, sizeof(ents));
    GKerr K;
    memset(&K, 0, sizeof(K));
    K.a = scene % 4 ? uni(0.0, 0.999) : 0.0;
    K.a2 = K.a * K.a;
    K.M = 1.0;
    K.Rhor = 1.0 + sqrt(1.0 - K.a2);
    K.Rmstable = K.Rhor + uni(0.05, 4.0);
    K.disk_tex = tex.data();
    K.disk_w = w;
    K.disk_h = h;
    K.use_temp = scene % 5 == 4;
    K.doppler_effect = 0.3;
    K.rms_f = (float)K.Rmstable;
    K.a2_f = (float)K.a2;
    const double world = scene % 7 == 6 ? 3.0e6 : scene % 7 == 5 ? 1000.0 : 0.0;  // the wormhole's far mouth
    if (world < 1.0) set(K.pos, {uni(-1, 1) * (scene % 2), 0, 0});
    for (int k = 0; k < 3; k++) K.pos_f[k] = (float)K.pos[k];
    S.n_ents = 1 + pick(6);
    for (int i = 0; i < S.n_ents; i++) {
      GEntity& e = ents[i];
      GEntF& f = S.entf[i];
      const dv3 c = {uni(-12, 12), uni(-12, 12), uni(-12, 12) + world}, n = unit();
      dv3 u, v;
      perp(n, u, v);
      const int kind = pick(world > 1.0 ? 4 : 5);
      set(e.p, c);
      set(e.normal, n);
      e.normal_inverse = 1;
      if (kind == 0) {
        e.type = PR_ENT_SPHERE;
        e.radius = pow(10.0, uni(-3, 5));
        if (e.radius > 20.0) set(e.p, along(c, n, e.radius));  // its surface passes by
        e.hemisphere = pick(4) == 0;
      } else if (kind == 1) {
        e.type = PR_ENT_UVPLANE;
        set(e.u_axis, u);
        set(e.v_axis, v);
        e.u_length = uni(0.5, 10);
        e.v_length = uni(0.5, 10);
      } else if (kind == 2 || kind == 4) {
        e.type = PR_ENT_CIRCLE;
        e.radius = uni(1.0, 15.0);
        e.radius_inner = pick(2) ? uni(0.0, 0.9) * e.radius : 0.0;
        if (kind == 4) {  // the accretion disk, about the hole
          e.kerr_disk = 1;
          if (pick(3)) {
            set(e.normal, {0, 0, 1});
            perp({0, 0, 1}, u, v);
          }
          set(e.p, {K.pos[0], K.pos[1], K.pos[2]});
          e.radius = uni(7.0, 15.0);
          set(e.disk_em, {2, 2, 2});
        }
        e.du_len = uni(0.5, 30);
        e.dv_len = uni(0.5, 30);
        set(e.du_axis, u);
        set(e.dv_axis, v);
        e.u_length = e.radius;
        e.v_length = e.radius_inner;
      } else {
        e.type = PR_ENT_POLYGON;
        e.node_base = i;
        GNode& g = node[i];
        memset(&g, 0, sizeof(g));
        float lo[3] = {3e38f, 3e38f, 3e38f}, hi[3] = {-3e38f, -3e38f, -3e38f};
        for (int k = 0; k < 3; k++) {
          const dv3 q = along(c, unit(), uni(0.1, 3.0));
          tris[3 * i + k] = make_float4((float)q.x, (float)q.y, (float)q.z, __int_as_float(0));
          const float x[3] = {(float)q.x, (float)q.y, (float)q.z};
          for (int a = 0; a < 3; a++) {
            lo[a] = fminf(lo[a], x[a]);
            hi[a] = fmaxf(hi[a], x[a]);
          }
        }
        for (int k = 0; k < 4; k++) {
          g.bmin_x[k] = lo[0]; g.bmin_y[k] = lo[1]; g.bmin_z[k] = lo[2];
          g.bmax_x[k] = hi[0]; g.bmax_y[k] = hi[1]; g.bmax_z[k] = hi[2];
          g.child[k] = k ? kChildInvalid : (int32_t)(kLeafBit | (uint32_t)i);
        }
        g.count[0] = 1;
        for (int a = 0; a < 3; a++) {
          f.u[a] = lo[a];
          f.v[a] = hi[a];
        }
      }
      f.type = e.type;
      f.normal_inverse = e.normal_inverse;
      for (int k = 0; k < 3; k++) {
        f.p[k] = (float)e.p[k];
        f.n[k] = (float)e.normal[k];
        if (e.type == PR_ENT_CIRCLE) {
          f.u[k] = (float)(e.du_axis[k] / e.du_len);
          f.v[k] = (float)(e.dv_axis[k] / e.dv_len);
        }
      }
      if (e.type == PR_ENT_CIRCLE) {
        f.u_length = (float)e.radius;
        f.v_length = (float)e.radius_inner;
        f.node_base = e.kerr_disk;
      }
      f.radius_eps = (float)(e.radius + 1.0e-6);
    }
    S.ents = ents;
    S.nodes = node;
    S.tris = tris;
    for (int ray = 0; ray < 1500; ray++) {
      const double within = world > 1.0 ? 0.5 : kSegment;
      const GEntity& e = ents[pick(S.n_ents)];
      dv3 o = {uni(-15, 15), uni(-15, 15), uni(-15, 15) + world}, d = unit();
      const int how = pick(5);
      if (how == 1 && e.type == PR_ENT_SPHERE)  // a segment's length off its surface
        o = along({e.p[0], e.p[1], e.p[2]}, unit(), e.radius + (pick(2) ? 1 : -1) * within * uni(0.0, 1.2));
      if (how == 2 && e.type != PR_ENT_SPHERE) o = along({e.p[0], e.p[1], e.p[2]}, unit(), uni(0, 2.2 * within));
      if (how == 3) {  // towards a point of the entity, about a segment away
        const dv3 q = along({e.p[0], e.p[1], e.p[2]}, unit(), e.type == PR_ENT_SPHERE ? e.radius : uni(0, 12));
        o = along(q, d, -within * len * uni(0.9, 1.1));
      }
      if (how == 4 && e.type == PR_ENT_SPHERE)  // at its centre, from just beyond a segment's length
        o = along({e.p[0], e.p[1], e.p[2]}, d, -e.radius - within * (1.0 + uni(0.0, 3.0e-3)));
      d = {d.x * len, d.y * len, d.z * len};
      const int draws = segment_draws(S, o, d, within, disk_alpha(K));
      total++;
      Rng r;
      r.init(1, (uint64_t)ray, 0);
      KerrDiskShading hs{&K, &r};
      uint32_t err = 0;
      uint64_t nodes = 0, nt = 0;
      double t;
      int ent, prim;
      const bool hit = exact_closest_hs(S, o, d, t, ent, prim, &err, nodes, nt, hs) && t < within;
      const int made = (int)r.ctr.z * 4 - (4 - r.idx);
      hits += hit;
      if (draws < 0) continue;
      skipped++;
      drawn += draws;
      if (hit || made != draws) {
        if (wrong++ < 5) printf("scene %d ray %d: hit %d at %g, draws %d of %d\n", scene, ray, hit, t, draws, made);
      }
    }
  }
  printf("wrong %ld skipped %ld drawn %ld hits %ld of %ld\n", wrong, skipped, drawn, hits, total);
  // most segments have nothing near them
  return wrong || hits < total / 100 || (unit_len && (skipped < total / 3 || drawn < 1000));
}
