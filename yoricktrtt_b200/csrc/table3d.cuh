// table3d.cuh -- tabulated footprint: what the sweep and gather kernels
// (sweep3d.cuh, proj3d_gather.cu) do per column and voxel.
//
// Every position is the reference's own FP64 value (plugin/trtt_3D_projectors.c:
// 1253-1307), in its order of operations without contraction, so that every
// table slot is the reference's; what does not depend on the voxel is computed
// once per column.  Quotients by a column's or a launch's constant are taken
// with its correctly rounded reciprocal and two corrections of the remainder
// (Markstein, IBM J. Res. Dev. 34, 1990), which gives the correctly rounded
// quotient without the divide's branches.  The table (the range outside which it
// is constant) lies in shared memory: its slots are scattered, 32 lanes take
// about 5 passes there and about 10 in L1.
//
// Measured, 128^3 -> 256^2, 90 cone views, 10001 entries, before (the band and
// column kernels of proj3d_fast.cu) -> after: direct 7.62 -> 3.09 ms, transpose
// (dense data) 4.64 -> 3.35 ms.  Bounds: direct the latency of the FP64 chains
// with 16 warps (49% of the issue slots, 61% for a dense volume; the band and the table leave no room
// for more, 24 warps of 2 columns 2.97 ms); transpose shared-memory wavefronts
// (61%, over half of them table slots) and issue (62%).
#pragma once

#include "fast3d_items.cuh"

namespace trtt {

struct TableCol {
  double q, nyj, nxi;         // uc = q (kc + nyj + nxi) + c3 (cone), kc + nyj + nxi (parallel)
  double hm, rm, dv;          // h = hm delta_u, rho = rm delta_u dv
  double den, rden;           // delta_u = sqrt(1 + t^2 / den), and 1 / den
  double vstart, vinc;        // v axis
  int lo, n;                  // detector rows [lo, lo + n)
  int k0, k1;                 // voxels that may meet the tile
  int q_lanes;                // sweep: voxels between neighbouring lanes; 0: any, with atomics
  int c0, c1;                 // gather: cells that the k range may touch
  int col, view;              // sweep: index along the line; gather: view or -1
};

// The table in shared memory: slots [t0, t1], edge value of slot s at
// tab[min(max(s, t0), t1)] (tab points at slot 0).
struct TableSh {
  const double *tab;
  int t0, t1;
  double rstep;               // 1 / P.step
};

__host__ __device__ __forceinline__ int table_slots(const Params3D &P) { return P.tab1 - P.tab0 + 1; }
// its room, a multiple of 16 bytes
__host__ __device__ __forceinline__ size_t table_bytes(const Params3D &P)
{
  return P.model == MODEL_TABLE ? sizeof(double) * (size_t)((table_slots(P) + 1) & ~1) : 0;
}
// Largest table range the kernels take.  90 cone views of a dense 128^3: 8001 slots
// (a table of 16001 entries) 5.6 + 3.4 ms, 8501 in the general kernels 8.9 + 4.2.
constexpr int kTableSlots = 8192;

// All threads of the CTA; the caller synchronises.
__device__ __forceinline__ void table_load(const Params3D &P, double *sh, TableSh &T)
{
  for (int t = threadIdx.x; t < table_slots(P); t += blockDim.x) sh[t] = __ldg(P.cum + P.tab0 + t);
  T.tab = sh - P.tab0;
  T.t0 = P.tab0;
  T.t1 = P.tab1;
  T.rstep = __drcp_rn(P.step);
}

// a / b, r = 1 / b correctly rounded, quotient and remainder normal or a = 0.
__device__ __forceinline__ double div_by(double a, double b, double r)
{
  double q = __dmul_rn(a, r);
  q = fma(fma(-q, b, a), r, q);
  return fma(fma(-q, b, a), r, q);
}

// floor(x) for |x| < 2^31 and int -> double for non-negative values: 1.5 2^52
// puts an integer in the low word.
constexpr double kMagic52 = 6755399441055744.0;
__device__ __forceinline__ int floor52(double x) { return __double2loint(__dadd_rd(x, kMagic52)); }
__device__ __forceinline__ double int52(int i) { return __hiloint2double(0x43380000, i) - kMagic52; }

__device__ __forceinline__ double table_at(const TableSh &T, double x)
{
  return T.tab[max(min(floor52(x), T.t1), T.t0)];
}

// Weight of cell l of the v axis.
__device__ __forceinline__ float table_weight_v(const TableSh &T, const TableCol &c, int l)
{
  return (float)(table_at(T, dadd(c.vstart, dmul((double)(l + 1), c.vinc))) -
                 table_at(T, dadd(c.vstart, dmul((double)l, c.vinc))));
}

// Column (i, j) into `c`; false when it misses the detector rows.  hsm, sp:
// bound of its half support along u, least distance of neighbouring voxels'
// first cells; A, B: uc(k) = A + B k.
template <int GEOM>
__device__ __forceinline__ bool table_column(const Params3D &P, const View3D &V, int i, int j, TableCol &c, double &A,
                                             double &B, double &hsm, double &sp, int *__restrict__ err)
{
  ColGeo<MODEL_TABLE> g;
  column_geo<GEOM, MODEL_TABLE>(P, V, i, j, 0, g);
  if (g.bad) atomicOr(err, TRTT_ERR_SOURCE_PLANE);
  if (g.bad || g.vax.n <= 0) return false;
  A = g.A;
  B = g.B;
  sp = fabs(B);
  c.nyj = g.nyj;
  c.nxi = g.nxi;
  if constexpr (GEOM == GEOM_CONE) {
    c.q = g.q;
    c.hm = dmul(P.h_u0, g.magn);
    c.rm = dmul(P.rho0_init, dmul(g.magn, g.magn));
    c.dv = g.delta_v;
    c.den = dadd(V.a4sqr, g.vca8sqr);
    c.rden = __drcp_rn(c.den);
    const double ua = A - V.a12, ub = fma(B, (double)(P.nz - 1), A) - V.a12;
    const double um = fmax(fabs(ua), fabs(ub)) * P.u_scl;
    hsm = P.hs0 * fabs(c.hm) * sqrt(1.0 + um * um * c.rden) * 1.0001;
    sp -= P.hs0 * fabs(c.hm) * sp * um * P.u_scl * c.rden;
  } else {
    hsm = V.p_hs_u;
  }
  c.vstart = g.vax.start;
  c.vinc = g.vax.inc;
  c.lo = g.vax.lo;
  c.n = g.vax.n;
  return true;
}

// A voxel's footprint: first cell f (not clamped to the detector), cells
// [f + s, f + s + n) within [u0, u1), edge l of cell f + l at
// start + (l - l0) inc.
struct TableVox {
  double start, inc;
  float rho;
  int f, l0, s, n;
};

// kc: the view's constant plus k times its step, the first sum of uc.
template <int GEOM>
__device__ __forceinline__ double table_kc(const View3D &V, int k)
{
  return GEOM == GEOM_CONE ? dadd(dmul(V.nu_z, (double)k), V.nu_c) : dadd(dmul(V.u_z, (double)k), V.u_c);
}
template <int GEOM>
__device__ __forceinline__ void table_voxel(const Params3D &P, const View3D &V, const TableSh &T, const TableCol &c,
                                            double kc, int u0, int u1, TableVox &x)
{
  double uc = dadd(dadd(kc, c.nyj), c.nxi), h, hs;
  if constexpr (GEOM == GEOM_CONE) {
    uc = dadd(dmul(c.q, uc), V.c3);
    const double t = dmul(dsub(uc, V.a12), P.u_scl);
    const double du = dsqrt(dadd(1.0, div_by(dmul(t, t), c.den, c.rden)));
    x.rho = (float)dmul(dmul(c.rm, du), c.dv);
    h = dmul(c.hm, du);
    hs = dmul(P.hs0, h);
    x.inc = div_by(__drcp_rn(h), P.step, T.rstep);
  } else {
    x.rho = (float)V.p_rho0;
    h = V.p_h_u;
    hs = V.p_hs_u;
    x.inc = V.p_sclt_u;
  }
  x.f = floor52(dsub(uc, hs));
  const int e = floor52(dadd(uc, hs)) + 1;
  const int lo = min(max(x.f, 0), P.nu - 1), hi = min(max(e, 0), P.nu);
  x.l0 = lo - x.f;
  x.start = dmul(dsub(dsub(int52(lo), uc), dmul(h, P.coord0)), x.inc);
  const int a = max(lo, u0);
  x.s = a - x.f;
  x.n = max(min(hi, u1) - a, 0);
}

}  // namespace trtt
