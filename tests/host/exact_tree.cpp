// exact_closest (device_common.cuh) on malformed trees: a node that is its own
// only child (the visits' cap), a node that is all its four children (the
// stack), and for comparison a tree of one leaf.  Each call has to end.
#include "host_cuda.h"

#include <cstdio>
#include <cstdlib>

#include "../../prender_gb300/csrc/device_common.cuh"

using namespace pr;

int main(int argc, char** argv) {
  const int kind = atoi(argv[1]);  // 0: one leaf, 1: cycle, 2: cycle that fills the stack
  GNode n;
  memset(&n, 0, sizeof(n));
  for (int c = 0; c < 4; c++) {
    n.bmin_x[c] = n.bmin_y[c] = n.bmin_z[c] = -10.0f;
    n.bmax_x[c] = n.bmax_y[c] = n.bmax_z[c] = 10.0f;
    n.child[c] = kind == 2 || (kind == 1 && c == 0) ? 0 : kChildInvalid;
  }
  if (kind == 0) {
    n.child[0] = (int32_t)kLeafBit;
    n.count[0] = 1;
  }
  const float4 tri[3] = {make_float4(-1, -1, 0, __int_as_float(3)), make_float4(1, -1, 0, 0), make_float4(0, 1, 0, 0)};
  GEntity e;
  memset(&e, 0, sizeof(e));
  e.type = PR_ENT_POLYGON;
  static DevScene S;
  S.ents = &e;
  S.nodes = &n;
  S.tris = tri;
  S.n_ents = 1;
  uint32_t err = 0;
  uint64_t nodes = 0, tris = 0;
  double t;
  int ent, prim;
  const bool hit = exact_closest(S, {0, 0, -5}, {0, 0, 1}, t, ent, prim, &err, nodes, tris);
  printf("%d %d %u %llu %llu\n", hit, hit ? prim : -1, err, (unsigned long long)nodes, (unsigned long long)tris);
}
