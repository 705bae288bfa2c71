// Host side of the FP32 sphere bounds.
#pragma once
#include <algorithm>
#include <cmath>

#include "pr_internal.h"

namespace pr {

// The constants of the FP32 sphere bounds (trace_fast.cuh).  A sphere more
// than four times larger than the rest of the scene (walls of radius 1e5) is
// anchored at the point of its surface nearest to the rest, else at its centre.
inline void sphere_bounds(const GEntity* ents, int n, GEntF* entf) {
  double lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300};
  double small = 1e300;
  for (int i = 0; i < n; i++)
    if (ents[i].type == PR_ENT_SPHERE) small = std::min(small, ents[i].radius);
  for (int i = 0; i < n; i++) {
    const GEntity& e = ents[i];
    if (e.type == PR_ENT_SPHERE && e.radius > 100.0 * small) continue;
    double a[3], b[3];
    for (int k = 0; k < 3; k++) {
      a[k] = b[k] = e.p[k];
      if (e.type == PR_ENT_SPHERE || e.type == PR_ENT_CIRCLE) {
        a[k] -= e.radius;
        b[k] += e.radius;
      } else if (e.type == PR_ENT_POLYGON) {
        a[k] = e.bmin[k];
        b[k] = e.bmax[k];
      }
      lo[k] = std::min(lo[k], a[k]);
      hi[k] = std::max(hi[k], b[k]);
    }
  }
  double mid[3], extent = 0.0;
  for (int k = 0; k < 3; k++) {
    mid[k] = 0.5 * (lo[k] + hi[k]);
    extent = std::max(extent, hi[k] - lo[k]);
  }
  for (int i = 0; i < n; i++) {
    const GEntity& e = ents[i];
    if (e.type != PR_ENT_SPHERE) continue;
    GEntF& f = entf[i];
    double w[3], len = 0.0;
    for (int k = 0; k < 3; k++) {
      w[k] = mid[k] - e.p[k];
      len += w[k] * w[k];
    }
    len = std::sqrt(len);
    const bool far = e.radius > 4.0 * extent && len > 0.0;
    double c0 = 0.0;
    for (int k = 0; k < 3; k++) {
      f.u[k] = (float)(far ? e.p[k] + e.radius / len * w[k] : e.p[k]);
      const double q = (double)f.u[k] - e.p[k];
      f.v[k] = (float)q;
      f.n[k] = (float)(q - (double)f.v[k]);
      c0 += q * q;
    }
    c0 -= e.radius * e.radius;
    f.u_length = (float)c0;
    f.v_length = (float)(c0 - (double)f.u_length);
    f.node_base = e.hemisphere;
  }
}

}  // namespace pr
