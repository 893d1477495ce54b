// foot2d.cuh -- footprint of one pixel in a 2D B-spline projector in the
// reference's FP64 operand order (plugin/trtt_2D_projectors.c:186-383,
// plugin/trtt_2D_projectors_cubic.c:209-398).
#pragma once

#include "kernels2d.h"
#include "trtt_device.cuh"

namespace trtt {

struct Foot2D {
  int lo, n;
  double start, inc;
  double rho0;
};

// Footprint of pixel (i,j) for view V.  Returns -1 if the pixel lies on the
// source line (fan beam, wk == 0), 0 otherwise (n may be 0).
__device__ __forceinline__ int foot2d(const Params2D &P, const View2D &V, int i, int j,
                                      Foot2D &f)
{
  const double di = (double)i, dj = (double)j;
  double vc, h, scl, hs;
  if (P.fan) {
    // plugin/trtt_2D_projectors.c:330-352
    double wk = dadd(dadd(dmul(V.o2, dj), V.o4), dmul(V.o1, di));
    double num = dadd(dadd(dmul(V.b1o6, dj), V.b1o8), dmul(V.b1o5, di));
    double den = dadd(dadd(dmul(V.d_y, dj), V.d_c), dmul(V.d_x, di));
    vc = dadd(dmul(ddiv(V.a4m, den), num), V.b3);
    if (wk == 0.0) {
      f.n = 0;
      return -1;
    }
    double magn = ddiv(V.a4m, wk);
    double vca8 = dmul(dsub(vc, V.a8), P.v_scl);
    double delta_v = dsqrt(dadd(1.0, ddiv(dmul(vca8, vca8), V.a4sqr)));
    f.rho0 = dmul(dmul(P.rho0_init, magn), delta_v);
    h = dmul(dmul(P.h_init, magn), delta_v);
    scl = __drcp_rn(P.table ? dmul(h, P.step) : h);
    hs = dmul(P.hs0, h);
  } else {
    // plugin/trtt_2D_projectors.c:222-226
    vc = dadd(dadd(dmul(V.b1o6, dj), V.b1o8b3), dmul(V.b1o5, di));
    f.rho0 = V.p_rho0;
    h = V.p_h;
    scl = V.p_scl;
    hs = V.p_hs;
  }
  if (!isfinite(vc)) {
    f.n = 0;
    return 0;
  }
  const int lo = clamp_left_cell(dsub(vc, hs), P.nv);
  const int hi = clamp_right_cell(dadd(vc, hs), P.table ? P.nv - 1 : P.nv - 2);
  f.lo = lo;
  f.n = hi - lo;
  if (P.table) {
    // (vl - (vc + coord0*h)) * scl   (plugin/trtt_2D_projectors.c:94-97)
    f.start = dmul(dsub((double)lo, dadd(vc, dmul(P.coord0, h))), scl);
  } else {
    // (vl - vc) * scl   (plugin/trtt_2D_projectors_cubic.c:119)
    f.start = dmul(dsub((double)lo, vc), scl);
  }
  f.inc = scl;
  return 0;
}

// Primitive at edge l of a 2D footprint (exact FP64, reference order).
__device__ __forceinline__ double edge2d(const Params2D &P, const Foot2D &f, int l)
{
  const double x = (l == 0) ? f.start : dadd(f.start, dmul((double)l, f.inc));
  if (P.table) return __ldg(P.cum + table_slot(x, P.last));
  return cubic_prim_d(x);
}

}  // namespace trtt
