// Sensor recording of one point (record_sensor_data!, first_order_steps.jl:728-811).
#pragma once
#include "kwb_internal.h"

namespace kwb {

// Record step t of point j of group g: pressure pv, velocity component d from u(d).
template <class U>
__device__ __forceinline__ void record_point(const SimDev &S, const GroupDev &g, long long t, long long j, float pv,
                                             U &&u) {
  const unsigned m = g.mask;
  const bool last = (t == S.Nt - 1);
  if (m & (1u << 0)) g.ser_p[t * g.n + j] = pv;
  if (m & (1u << 1)) g.pmax[j] = fmaxf(g.pmax[j], pv);
  if (m & (1u << 2)) g.pmin[j] = fminf(g.pmin[j], pv);
  if (m & (1u << 3)) g.prms[j] += (double)g.cnt_prms * ((double)pv * (double)pv);
  if ((m & (1u << 4)) && last) g.pfinal[j] = pv;
  const unsigned umask = (7u << 5) | (63u << 8);
  if (m & umask) {
    float uv[3] = {0.f, 0.f, 0.f};
    for (int d = 0; d < S.ndim; ++d) uv[d] = u(d);
    for (int d = 0; d < S.ndim; ++d)
      if (m & (1u << (5 + d))) g.ser_u[d][t * g.n + j] = uv[d];
    double mag2 = 0.0, i2 = 0.0;
    for (int d = 0; d < S.ndim; ++d) {
      mag2 += (double)uv[d] * (double)uv[d];
      const double pu = (double)pv * (double)uv[d];
      i2 += pu * pu;
    }
    const double mag = sqrt(mag2);
    if (m & (1u << 8)) g.umax[j] = fmax(g.umax[j], mag);
    if (m & (1u << 9)) g.urms[j] += (double)g.cnt_urms * mag2;
    if ((m & (1u << 10)) && last) g.ufinal[j] = mag;
    if (m & ((1u << 11) | (1u << 12))) {
      const double I = sqrt(i2);
      if (m & (1u << 11)) g.iavg[j] += (double)g.cnt_iavg * (I / (double)S.Nt);
      if (m & (1u << 12)) g.imax[j] = fmax(g.imax[j], I);
    }
  }
}

}  // namespace kwb
