// host3d.h -- host-side derivation of the 3D projector parameters shared by
// the C ABI translation units (plan, drop-in and allocation-free entry
// points).
#pragma once

#include <cmath>
#include <cstring>
#include <vector>

#include "kernels.h"
#include "trtt_b200.h"

namespace trtt {

// Per-view constants of the 3D projectors, derived in FP64 with the operand
// order of the reference so that the device sees the reference's values
// (cone beam plugin/trtt_3D_projectors.c:1186-1230, parallel beam
// plugin/trtt_3D_projectors.c:963-1004; identical in the _cubic file).
inline void make_view3d(const Params3D &P, const double *xos, const double *xsd, View3D &V)
{
  std::memset(&V, 0, sizeof(V));
  const double a1 = xsd[0], a2 = xsd[1], a3 = xsd[2], a4 = xsd[3];
  const double a5 = xsd[4], a6 = xsd[5], a7 = xsd[6], a8 = xsd[7];
  const double a9 = xsd[8], a10 = xsd[9], a11 = xsd[10], a12 = xsd[11];
  const double o1 = xos[0], o2 = xos[1], o3 = xos[2], o4 = xos[3];
  const double o5 = xos[4], o6 = xos[5], o7 = xos[6], o8 = xos[7];
  const double o9 = xos[8], o10 = xos[9], o11 = xos[10], o12 = xos[11];
  const double a1inv = -1.0 * (1.0 / a1);
  const double b1 = a6 + a1inv * a5 * a2, c1 = a10 + a1inv * a9 * a2;
  const double b2 = a7 + a1inv * a5 * a3, c2 = a11 + a1inv * a9 * a3;
  const double b3 = a8 + a1inv * a5 * a4, c3 = a12 + a1inv * a9 * a4;
  V.o1 = o1; V.o2 = o2; V.o3 = o3; V.o4 = o4;
  V.nv_x = b1 * o5 + b2 * o9;  V.nu_x = c1 * o5 + c2 * o9;
  V.nv_y = b1 * o6 + b2 * o10; V.nu_y = c1 * o6 + c2 * o10;
  V.nv_z = b1 * o7 + b2 * o11; V.nu_z = c1 * o7 + c2 * o11;
  V.nv_c = b1 * o8 + b2 * o12; V.nu_c = c1 * o8 + c2 * o12;
  V.d_x = a1 * o1 + a2 * o5 + a3 * o9;
  V.d_y = a1 * o2 + a2 * o6 + a3 * o10;
  V.d_z = a1 * o3 + a2 * o7 + a3 * o11;
  V.d_c = a1 * o4 + a2 * o8 + a3 * o12;
  V.a4sqr = a4 * a4;
  V.a4m = -1.0 * a4;
  V.a8 = a8;
  V.a12 = a12;
  V.b3 = b3;
  V.c3 = c3;
  // parallel beam
  V.v_x = b1 * o5 + b2 * o9;  V.u_x = c1 * o5 + c2 * o9;
  V.v_y = b1 * o6 + b2 * o10; V.u_y = c1 * o6 + c2 * o10;
  V.v_z = b1 * o7 + b2 * o11; V.u_z = c1 * o7 + c2 * o11;
  V.v_c = b1 * o8 + b2 * o12 + b3; V.u_c = c1 * o8 + c2 * o12 + c3;
  const double a1sqr = a1 * a1;
  const double a5sqr = P.v_scl * P.v_scl * a5 * a5;
  const double a9sqr = P.u_scl * P.u_scl * a9 * a9;
  const double delta_u = std::sqrt(1.0 + (a9sqr / (a1sqr + a5sqr)));
  const double delta_v = std::sqrt(1.0 + (a5sqr / a1sqr));
  V.p_rho0 = P.s_scl * P.s_scl * P.s_scl * delta_u * delta_v;
  V.p_h_u = P.s_scl / P.u_scl;
  V.p_h_v = P.s_scl / P.v_scl;
  V.p_scl_u = 1.0 / V.p_h_u;
  V.p_scl_v = 1.0 / V.p_h_v;
  V.p_hs_u = P.hs0 * V.p_h_u;
  V.p_hs_v = P.hs0 * V.p_h_v;
  V.p_sclt_u = V.p_scl_u / P.step;
  V.p_sclt_v = V.p_scl_v / P.step;
  V.g0 = 0;
  V.g1 = 0;
  V.w0 = 1.0f;
  V.w1 = 0.0f;
  if (P.geom == GEOM_CONE)
    V.factorized = (V.o3 == 0.0 && V.d_z == 0.0 && V.nv_z == 0.0) ? 1 : 0;
  else
    V.factorized = (V.v_z == 0.0) ? 1 : 0;
}

inline Params3D make_params(int geom, long nx, long ny, long nz, double s_scl, int s_deg,
                     const double *cum_dev, long size, double step,
                     double coord0, long nu, long nv, double u_scl, double v_scl)
{
  Params3D P;
  std::memset(&P, 0, sizeof(P));
  P.geom = geom;
  P.model = cum_dev ? MODEL_TABLE : MODEL_CUBIC;
  P.nx = (int)nx; P.ny = (int)ny; P.nz = (int)nz;
  P.nu = (int)nu; P.nv = (int)nv;
  P.nt = 1;
  P.s_scl = s_scl;
  P.u_scl = u_scl;
  P.v_scl = v_scl;
  P.rho0_init = s_scl * s_scl * s_scl;
  P.h_u0 = s_scl / u_scl;
  P.h_v0 = s_scl / v_scl;
  P.hs0 = 0.5 * (s_deg + 1);
  P.cum = cum_dev;
  P.size = (int)size;
  P.last = (double)(size - 1);
  P.step = cum_dev ? step : 1.0;
  P.coord0 = coord0;
  return P;
}

// Range of slots outside which the table is constant.
inline void table_range(Params3D &P, const double *cum, long size)
{
  long a = 0, b = size - 1;
  while (a + 1 < size && cum[a + 1] == cum[0]) ++a;
  while (b > 0 && cum[b - 1] == cum[size - 1]) --b;
  P.tab0 = (int)(a <= b ? a : 0);
  P.tab1 = (int)(a <= b ? b : 0);
}

// Size limits shared by every 3D entry point that takes device arrays:
// dimensions in [1, 2^30) (int indices in the kernels), one volume slice
// below 2^31 voxels and the whole volume below 2^40.  Returns nullptr when
// the sizes are accepted, else the reason.
inline const char *check_sizes3d(long nx, long ny, long nz, long nu, long nv, long nviews)
{
  auto ok = [](long n) { return n >= 1 && n < (1L << 30); };
  if (!ok(nx) || !ok(ny) || !ok(nz) || !ok(nu) || !ok(nv) || !ok(nviews))
    return "sizes must be in [1, 2^30)";
  if (nx * ny >= (1L << 31) || nx * ny * nz >= (1L << 40)) return "volume too large";
  return nullptr;
}

// ---------------------------------------------------------------------------
// Orbit symmetry of a scan's views.  R(i, j) = (n-1-j, i) is the quarter turn
// of a square grid about the z axis, R^2(i, j) = (nx-1-i, ny-1-j) the half
// turn of any grid.  View b is the m-turn image of view a when it sees voxel
// (i, j, k) where view a sees voxel (R^m(i, j), k): its xos rows (p, q, r, s)
// acting as p i + q j + r k + s equal those of view a with the substitution
// applied, and its xsd equals view a's.  The footprints of view b's voxel
// column c are then view a's footprints of column R^m(c), so a group of
// views needs the footprint arithmetic of its first view only.
// ---------------------------------------------------------------------------
inline void turn_xos(const double *x, int m, long nx, long ny, double *out)
{
  for (int r = 0; r < 3; ++r) {
    const double a = x[4 * r], b = x[4 * r + 1], c = x[4 * r + 2], d = x[4 * r + 3];
    double *o = out + 4 * r;
    o[2] = c;
    if (m == 1) {
      o[0] = b; o[1] = -a; o[3] = d + a * (double)(nx - 1);
    } else if (m == 2) {
      o[0] = -a; o[1] = -b; o[3] = d + a * (double)(nx - 1) + b * (double)(ny - 1);
    } else if (m == 3) {
      o[0] = -b; o[1] = a; o[3] = d + b * (double)(ny - 1);
    } else {
      o[0] = a; o[1] = b; o[3] = d;
    }
  }
}

// Rows of two 3x4 matrices equal within tol relative to the row's magnitude.
inline bool coefs_match(const double *p, const double *q, double tol)
{
  for (int r = 0; r < 3; ++r) {
    double s = 0.0;
    for (int c = 0; c < 4; ++c) s = std::fmax(s, std::fmax(std::fabs(p[4 * r + c]), std::fabs(q[4 * r + c])));
    for (int c = 0; c < 4; ++c)
      if (!(std::fabs(p[4 * r + c] - q[4 * r + c]) <= tol * s)) return false;
  }
  return true;
}

// Greedy grouping in view order: {a, b1, b2, b3} (quarter turns, square grid
// of even side), else {a, b2} (half turn, nx or ny even), else {a}.  Each
// group is written as four view indices (unused slots -1) into the list of
// its size: groups[0] singles, groups[1] pairs, groups[2] quads.
inline void find_view_groups(long nx, long ny, long nviews, const double *xos, const double *xsd,
                             std::vector<int> groups[3], double tol = 1e-10)
{
  std::vector<char> used(nviews, 0);
  const bool quad_ok = nx == ny && nx % 2 == 0;
  const bool pair_ok = nx % 2 == 0 || ny % 2 == 0;
  auto find = [&](const double *coefs, const double *xd) -> long {
    for (long b = 0; b < nviews; ++b)
      if (!used[b] && coefs_match(xos + 12 * b, coefs, tol) && coefs_match(xsd + 12 * b, xd, tol))
        return b;
    return -1;
  };
  double t[12];
  for (long a = 0; a < nviews; ++a) {
    if (used[a]) continue;
    used[a] = 1;
    long mem[4] = {a, -1, -1, -1};
    int n = 1;
    if (quad_ok) {
      long b[3];
      for (int m = 1; m <= 3; ++m) {
        turn_xos(xos + 12 * a, m, nx, ny, t);
        b[m - 1] = find(t, xsd + 12 * a);
      }
      if (b[0] >= 0 && b[1] >= 0 && b[2] >= 0 && b[0] != b[1] && b[0] != b[2] && b[1] != b[2]) {
        mem[1] = b[0]; mem[2] = b[1]; mem[3] = b[2];
        n = 4;
      }
    }
    if (n == 1 && pair_ok) {
      turn_xos(xos + 12 * a, 2, nx, ny, t);
      const long b2 = find(t, xsd + 12 * a);
      if (b2 >= 0) {
        mem[1] = b2;
        n = 2;
      }
    }
    for (int m = 1; m < n; ++m) used[mem[m]] = 1;
    std::vector<int> &dst = groups[n == 4 ? 2 : n - 1];
    for (int m = 0; m < 4; ++m) dst.push_back((int)mem[m]);
  }
}

// Band shape of the direct kernel for a detector nu cells wide.
inline void choose_band(int nu, int nv, int &band_rows, int &warps)
{
  const long budget = 200 * 1024;
  warps = 16;
  while (warps > 2 && (long)warps * nu * 4 > budget / 3) warps /= 2;
  const long rest = budget - (long)warps * nu * 4;
  long rows = rest / ((long)nu * 4 + (long)warps * 4);
  if (rows > 32) rows = 32;  // two CTAs (2 x 16 warps) per SM at nu = 512
  if (rows > nv) rows = nv;
  band_rows = rows >= 2 ? (int)rows : 0;
}

// Bounds for the sweep and gather kernels over the factorised views of a plan:
// the detector rows of one voxel column's v footprint, and the part of the
// detector that any footprint can reach (a volume's shadow seldom fills the
// detector; the tiles cover no more than it).  Positions are quotients of affine
// functions of the voxel, so the grid's corners bound them as long as neither
// denominator changes sign over the grid.  rows = 0 where the kernels do
// not apply: a closed-form footprint that is not the cubic's 4 voxels wide (a
// walk starts at a zero of the primitive), a source within the volume, a tilted
// detector whose plane through the source crosses the volume.
inline SweepBounds sweep_bounds(const Params3D &P, const View3D *views, long nviews)
{
  SweepBounds b;
  if (P.model == MODEL_CUBIC && P.hs0 != 2.0) return b;
  double hmin = HUGE_VAL;
  double hsv = 0.0, hsu = 0.0, u0 = HUGE_VAL, u1 = -HUGE_VAL, v0 = HUGE_VAL, v1 = -HUGE_VAL;
  for (long n = 0; n < nviews; ++n) {
    const View3D &V = views[n];
    double wmin = HUGE_VAL, wmax = -HUGE_VAL, dv2 = 0.0, du2 = 0.0, dmin = HUGE_VAL, uabs = 0.0;
    int dneg = 0;  // corners behind the plane where u and v diverge
    for (int c = 0; c < 8; ++c) {
      const double i = (c & 1) ? P.nx - 1 : 0, j = (c & 2) ? P.ny - 1 : 0, k = (c & 4) ? P.nz - 1 : 0;
      double u, v;
      if (P.geom == GEOM_CONE) {
        const double w = V.o1 * i + V.o2 * j + V.o4, d = V.d_x * i + V.d_y * j + V.d_c, q = V.a4m / d;
        v = q * (V.nv_x * i + V.nv_y * j + V.nv_c) + V.b3;
        u = q * (V.nu_x * i + V.nu_y * j + V.nu_z * k + V.nu_c) + V.c3;
        wmin = std::fmin(wmin, w);
        wmax = std::fmax(wmax, w);
        dmin = std::fmin(dmin, std::fabs(d));
        dneg += d < 0.0;
        uabs = std::fmax(uabs, std::fabs(u - V.c3));
        const double va = (v - V.a8) * P.v_scl, ua = (u - V.a12) * P.u_scl;
        dv2 = std::fmax(dv2, va * va / V.a4sqr);
        du2 = std::fmax(du2, ua * ua / V.a4sqr);
      } else {
        v = V.v_x * i + V.v_y * j + V.v_c;
        u = V.u_x * i + V.u_y * j + V.u_z * k + V.u_c;
      }
      u0 = std::fmin(u0, u);
      u1 = std::fmax(u1, u);
      v0 = std::fmin(v0, v);
      v1 = std::fmax(v1, v);
    }
    if (P.geom == GEOM_CONE) {
      // a pole of u and v inside the grid: the corners bound nothing
      if (!(wmin * wmax > 0.0) || dneg % 8 != 0) return b;
      // nearest corner: largest magnification; outermost: largest obliquity
      const double magn = std::fabs(V.a4m) / std::fmin(std::fabs(wmin), std::fabs(wmax));
      hsv = std::fmax(hsv, P.hs0 * P.h_v0 * magn * std::sqrt(1.0 + dv2));
      hsu = std::fmax(hsu, P.hs0 * P.h_u0 * magn * std::sqrt(1.0 + du2));
      hmin = std::fmin(hmin, P.h_u0 * std::fabs(V.a4m) / std::fmax(std::fabs(wmin), std::fabs(wmax)));
      const double q = std::fabs(V.a4m) / dmin;
      b.du = std::fmax(b.du, q * std::fabs(V.nu_z));
      b.dcol = std::fmax(b.dcol, q * std::fabs(V.nu_x) + uabs * std::fabs(V.d_x) / dmin);
    } else {
      hmin = std::fmin(hmin, V.p_h_u);
      hsv = std::fmax(hsv, V.p_hs_v);
      hsu = std::fmax(hsu, V.p_hs_u);
      b.du = std::fmax(b.du, std::fabs(V.u_z));
      b.dcol = std::fmax(b.dcol, std::fabs(V.u_x));
    }
  }
  b.hsu = hsu;
  // table: slots along a footprint are 32-bit integers
  if (P.model == MODEL_TABLE && !(hmin > 0.0 && (2.0 * hsu + 20.0 + std::fabs(P.coord0)) / (hmin * P.step) < 1e9 &&
                                  (2.0 * P.hs0 + std::fabs(P.coord0)) / P.step < 1e9))
    return b;
  if (!(hsv > 0.0 && hsv < 1e4 && hsu < 1e4 && b.du < 1e6 && b.dcol < 1e6)) return b;
  if (!(u0 > -1e8 && u1 < 1e8 && v0 > -1e8 && v1 < 1e8)) return b;
  b.rows = (int)std::floor(2.0 * hsv * 1.0001) + 2;
  b.u0 = (int)std::fmin(std::fmax(std::floor(u0 - hsu * 1.0001) - 1.0, 0.0), P.nu);
  b.u1 = (int)std::fmin(std::fmax(std::ceil(u1 + hsu * 1.0001) + 2.0, 0.0), P.nu);
  b.v0 = (int)std::fmin(std::fmax(std::floor(v0 - hsv * 1.0001) - 1.0, 0.0), P.nv);
  b.v1 = (int)std::fmin(std::fmax(std::ceil(v1 + hsv * 1.0001) + 2.0, 0.0), P.nv);
  return b;
}

inline int geom_code(int geometry)
{
  if (geometry == TRTT_B200_PARALLEL_BEAM) return GEOM_PARALLEL;
  if (geometry == TRTT_B200_CONE_BEAM || geometry == TRTT_B200_FAN_BEAM) return GEOM_CONE;
  return -1;
}

}  // namespace trtt
