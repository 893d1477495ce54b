// sweep3d.cuh -- direct projection of column-factorised views (closed-form
// footprint; tabulated footprint with the walks of table3d.cuh): the band of
// detector cells [v0, v1) x [u0, u1) of G views related by turns of the grid
// (find_view_groups, host3d.h; G = 1: one view), accumulated in shared memory,
// the members' values of a cell side by side.  The footprints are those of the
// first view; member m sees there the columns turned back by its turn.
//
// A warp sweeps an image line of voxel columns (along i or j, the axis on which
// neighbouring columns project further apart), NC = 32 / H consecutive columns
// at a time:
//   * their u-profiles P_g[u] are built in warp-private shared rows, H lanes per
//     column: a lane takes a pair of adjacent voxels, 2 |B| cells from the next
//     lane's, and walks the union of their footprints two cells at a time with
//     plain loads and stores; where neighbouring pairs would be less than two
//     cells apart the lanes take every q-th pair, so no step needs an atomic;
//   * the band rows that the columns cover together (about four per column
//     instead of seven or eight) then get sum_g w_g(v) P_g[u] in one update
//     each, four rows (and a strip of cells) under one lock.
//
// Positions along a column are 32.32 fixed point (uc = A + B k exact to 2^-32
// cell): the cell is the high word and the fraction the low one, so no FP64
// arithmetic or conversion is left in the voxel loop.
#pragma once

#include "fast3d_items.cuh"
#include "table3d.cuh"

namespace trtt {

struct SweepCol {
  long long A, B;             // 32.32 position of voxel 0 and step per voxel
  float h, rho, inv_den;      // ColGeo (cone beam)
  float vstart, vinc;         // ColGeo v axis
  int lo, n;                  // detector rows [lo, lo + n)
  int p0, p1;                 // voxel pairs that may meet the tile
  int q;                      // pairs between neighbouring lanes; 0: FP64 path
  int steps;                  // double cells walked per pair
  int col;                    // index along the line
};

// What a warp keeps per view: line axis, position of a column's v footprint
// along a line, half-support bound.
struct SweepView {
  int axis, ranged;           // ranged: the depth keeps its sign, lines can be cut to the band
  double hsv;
};

template <int GEOM>
__device__ __forceinline__ void sweep_view(const Params3D &P, const View3D &V, SweepView &S)
{
  const double nx1 = P.nx - 1, ny1 = P.ny - 1;
  if constexpr (GEOM == GEOM_CONE) {
    double dmin = 1e300, dmax = -1e300, wmin = 1e300, wmax = -1e300, tmax = 0.0;
    for (int c = 0; c < 4; ++c) {
      const double i = (c & 1) ? nx1 : 0.0, j = (c & 2) ? ny1 : 0.0;
      const double d = V.d_x * i + V.d_y * j + V.d_c, w = V.o1 * i + V.o2 * j + V.o4;
      const double t = fabs((V.a4m * (V.nv_x * i + V.nv_y * j + V.nv_c) / d + V.b3 - V.a8) * P.v_scl);
      dmin = fmin(dmin, d); dmax = fmax(dmax, d);
      wmin = fmin(wmin, w); wmax = fmax(wmax, w);
      tmax = fmax(tmax, t);
    }
    const double wn = fmin(fabs(wmin), fabs(wmax));
    S.ranged = dmin * dmax > 0.0 && wmin * wmax > 0.0 && wn > 1e-6 * fmax(fabs(wmin), fabs(wmax)) &&
               fmin(fabs(dmin), fabs(dmax)) > 1e-6 * fmax(fabs(dmin), fabs(dmax)) && tmax < 1e9;
    // the magnification is largest at the nearest corner, the obliquity at the outermost
    S.hsv = P.hs0 * P.h_v0 * fabs(V.a4m / wn) * sqrt(1.0 + tmax * tmax / V.a4sqr) * 1.0001 + 1.0;
    const double ci = 0.5 * nx1, cj = 0.5 * ny1;
    const double D = V.d_x * ci + V.d_y * cj + V.d_c, N = V.nv_x * ci + V.nv_y * cj + V.nv_c;
    S.axis = fabs(V.nv_y * D - N * V.d_y) > fabs(V.nv_x * D - N * V.d_x) ? 1 : 0;
  } else {
    S.ranged = 1;
    S.hsv = V.p_hs_v + 1.0;
    S.axis = fabs(V.v_y) > fabs(V.v_x) ? 1 : 0;
  }
}

// Columns [a0, a1) of line `ln` whose v footprints may meet rows [v0, v1).
template <int GEOM>
__device__ __forceinline__ void sweep_range(const Params3D &P, const View3D &V, const SweepView &S, int ln, int n,
                                            int v0, int v1, int &a0, int &a1)
{
  const double l = (double)ln, last = (double)(n - 1);
  double N0, N1, D0 = 1.0, D1 = 0.0, c = 0.0;
  if constexpr (GEOM == GEOM_CONE) {
    N0 = V.a4m * ((S.axis ? V.nv_x : V.nv_y) * l + V.nv_c);
    N1 = V.a4m * (S.axis ? V.nv_y : V.nv_x);
    D0 = (S.axis ? V.d_x : V.d_y) * l + V.d_c;
    D1 = S.axis ? V.d_y : V.d_x;
    c = V.b3;
  } else {
    N0 = (S.axis ? V.v_x : V.v_y) * l + V.v_c;
    N1 = S.axis ? V.v_y : V.v_x;
  }
  a0 = 0;
  a1 = n;
  if (!S.ranged) return;
  const double pa = N0 / D0, pb = (N0 + N1 * last) / (D0 + D1 * last);
  const double lo = (double)v0 - c - S.hsv, hi = (double)v1 - c + S.hsv;
  const double mn = fmin(pa, pb), mx = fmax(pa, pb);
  if (!(mx >= lo && mn <= hi)) {
    a1 = 0;
    return;
  }
  double kl = pa < pb ? 0.0 : last, kh = pa < pb ? last : 0.0;
  if (lo > mn) kl = (N0 - lo * D0) / (lo * D1 - N1);
  if (hi < mx) kh = (N0 - hi * D0) / (hi * D1 - N1);
  a0 = max(__double2int_rd(fmin(kl, kh)) - 1, 0);
  a1 = min(__double2int_ru(fmax(kl, kh)) + 2, n);
}

// Cells between the profile rows of a warp: walks that leave the tile end
// here, in values that nothing reads.
constexpr int kSweepGuard = 16;
// Band rows under one lock, and groups of them that one weight table covers.
constexpr int kSweepRows = 4, kSweepGroups = 8;

// 1 / sqrt(x) and 1 / x of normal numbers (2^-22 relative), without the
// denormal handling of the library forms.
__device__ __forceinline__ float rsqrt_ftz(float x)
{
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float rcp_ftz(float x)
{
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// Odd part of the primitive: P(x) - 1/2 = sign(x) (1/2 - ((2-t)_+^4 - 4
// (1-t)_+^4) / 24), t = |x|; differences of it are the weights.  Saturating
// arithmetic gives (1 - t/2)_+ and (1 - t)_+ (nine scalar operations; packing
// two powers saves two of them and costs more in register moves).
__device__ __forceinline__ float cubic_odd(float x)
{
  const float a = __saturatef(fmaf(fabsf(x), -0.5f, 1.0f)), b = __saturatef(1.0f - fabsf(x));
  const float a2 = a * a, b2 = b * b;
  return copysignf(fmaf(a2 * a2, -0.6666666666666667f, fmaf(b2 * b2, 0.1666666666666667f, 0.5f)), x);
}

// A band or profile row holds 64 Q floats: 64 Q / G cells of G values, Q pairs
// per lane, worked on in strips of SP pairs.
template <int Q, int H> struct SweepStrip {
  static constexpr int NC = 32 / H;
  static constexpr int SP = Q <= 3 ? Q : (NC >= 4 ? 2 : 4);  // registers: SP (NC + 4) pairs
  static constexpr int NS = Q / SP;
  static_assert(Q % SP == 0, "whole strips");
};

// Shared memory of one CTA: the band (rows rounded up to whole lock groups),
// one lock per group and strip, and per warp the records of a batch of columns, a
// table of row weights and NC profile rows with guards around them.
template <int MODEL> struct SweepRec {
  using T = SweepCol;
  static constexpr int batch = 32;  // columns whose records are built together
};
template <> struct SweepRec<MODEL_TABLE> {
  using T = TableCol;
  static constexpr int batch = 16;
};
template <int G, int Q, int H, int MODEL> __host__ __device__ constexpr size_t sweep_warp_bytes()
{
  constexpr int NC = 32 / H;
  return SweepRec<MODEL>::batch * sizeof(typename SweepRec<MODEL>::T) +
         sizeof(float2) * kSweepRows * kSweepGroups * NC +
         sizeof(float) * (size_t)(NC * (64 * Q + G * kSweepGuard) + G * kSweepGuard);
}
__host__ __device__ constexpr int sweep_groups(int R) { return (R + kSweepRows - 1) / kSweepRows; }
template <int G, int Q, int H, int MODEL> __host__ __device__ constexpr size_t sweep_smem(int R, int warps)
{
  return sizeof(float) * (size_t)sweep_groups(R) * kSweepRows * 64 * Q + warps * sweep_warp_bytes<G, Q, H, MODEL>() +
         sizeof(int) * (size_t)sweep_groups(R) * SweepStrip<Q, H>::NS;
}

// Turn of member m of a group of G views, and the index of column R^t(i, j),
// R(i, j) = (n-1-j, i).
template <int G> __host__ __device__ constexpr int sweep_turn(int m) { return G == 4 ? m : (G == 2 ? 2 * m : 0); }
__device__ __forceinline__ long turned_col(int i, int j, int t, int nx, int ny)
{
  t &= 3;
  const int oi = t == 0 ? i : (t == 1 ? nx - 1 - j : (t == 2 ? nx - 1 - i : j));
  const int oj = t == 0 ? j : (t == 1 ? i : (t == 2 ? ny - 1 - j : ny - 1 - i));
  return (long)oj * nx + oi;
}

// The G values of a cell: v[m] += wa xa[m] + wc xc[m].
template <int G> struct SweepVec;
template <> struct SweepVec<1> { using T = float; };
template <> struct SweepVec<2> { using T = float2; };
template <> struct SweepVec<4> { using T = float4; };
__device__ __forceinline__ void sweep_fma(float &v, float wa, float wc, const float (&xa)[1], const float (&xc)[1])
{
  v = fmaf(wc, xc[0], fmaf(wa, xa[0], v));
}
__device__ __forceinline__ void sweep_fma(float2 &v, float wa, float wc, const float (&xa)[2], const float (&xc)[2])
{
  v.x = fmaf(wc, xc[0], fmaf(wa, xa[0], v.x));
  v.y = fmaf(wc, xc[1], fmaf(wa, xa[1], v.y));
}
__device__ __forceinline__ void sweep_fma(float4 &v, float wa, float wc, const float (&xa)[4], const float (&xc)[4])
{
  v.x = fmaf(wc, xc[0], fmaf(wa, xa[0], v.x));
  v.y = fmaf(wc, xc[1], fmaf(wa, xa[1], v.y));
  v.z = fmaf(wc, xc[2], fmaf(wa, xa[2], v.z));
  v.w = fmaf(wc, xc[3], fmaf(wa, xa[3], v.w));
}

// Voxels [k0, k1) of a column uc = A + B k whose footprints (half support hsm)
// may meet cells [u0, u1).
__device__ __forceinline__ void tile_voxels(double A, double B, double hsm, int nz, int u0, int u1, int &k0, int &k1)
{
  const double lo_u = (double)u0 - 1.0 - hsm, hi_u = (double)u1 + 1.0 + hsm;
  k0 = 0;
  k1 = nz;
  if (fabs(B) > 1e-300) {
    const double ka = (lo_u - A) / B, kb = (hi_u - A) / B;
    k0 = (int)fmin(fmax(floor(fmin(ka, kb)), 0.0), (double)nz);
    k1 = (int)fmin(fmax(ceil(fmax(ka, kb)) + 1.0, 0.0), (double)nz);
  } else if (!(A > lo_u && A < hi_u)) {
    k1 = 0;
  }
}

// Record of column `a` of line `ln` into `r`; false: it misses the band or the tile.
template <int GEOM>
__device__ __forceinline__ bool sweep_record(const Params3D &P, const View3D &V, int i, int j, int v0, int v1, int u0,
                                             int u1, SweepCol &r, int *__restrict__ err)
{
  const int nz = P.nz;
  ColGeo<MODEL_CUBIC> c;
  column_geo<GEOM, MODEL_CUBIC>(P, V, i, j, 0, c);
  if (c.bad) atomicOr(err, TRTT_ERR_SOURCE_PLANE);
  if (c.bad || c.vax.n <= 0 || c.vax.lo + c.vax.n <= v0 || c.vax.lo >= v1) return false;
  // bound of the half support along the column; least distance of the first
  // cells of neighbouring voxels
  double hsm, sp = fabs(c.B);
  if constexpr (GEOM == GEOM_CONE) {
    const double ua = c.A - V.a12, ub = fma(c.B, (double)(nz - 1), c.A) - V.a12;
    const double um = fmax(fabs(ua), fabs(ub)) * P.u_scl;
    hsm = P.hs0 * (double)c.h_u0m * sqrt(1.0 + um * um * (double)c.inv_den) * 1.0001;
    sp -= P.hs0 * (double)c.h_u0m * sp * um * P.u_scl * (double)c.inv_den;
  } else {
    hsm = V.p_hs_u;
  }
  int k0, k1;
  tile_voxels(c.A, c.B, hsm, nz, u0, u1, k0, k1);
  if (k0 >= k1) return false;
  const double ue = fma(c.B, (double)nz, c.A);
  const bool fixed = fabs(c.A) < 1e9 && fabs(ue) < 1e9 && hsm < 1e6 && sp > 0.03;
  // + 2^8: the 23-bit fraction taken from the low word is then rounded
  r.A = fixed ? __double2ll_rn(c.A * 4294967296.0) + 256 : 0;
  r.B = fixed ? __double2ll_rn(c.B * 4294967296.0) : 0;
  // pairs of neighbouring lanes two cells apart (the pair steps of a parallel
  // beam are exact in fixed point; else 0.2% for the rounding of the cells)
  int q = 0;
  if (fixed) {
    const long long two = 2LL << 32, step = 2 * (r.B < 0 ? -r.B : r.B);
    q = GEOM == GEOM_CONE ? (int)ceil(2.004 / (2.0 * sp)) : (int)((two + step - 1) / step);
  }
  r.q = q;
  r.h = c.h_u0m;
  r.rho = c.rho0c;
  r.inv_den = c.inv_den;
  r.vstart = c.vax.start;
  r.vinc = c.vax.inc;
  r.lo = c.vax.lo;
  r.n = c.vax.n;
  r.p0 = k0 >> 1;
  r.p1 = (k1 + 1) >> 1;
  r.steps = fixed ? ((int)(2.0 * hsm + fabs(c.B)) + 3) >> 1 : 0;
  return true;
}

__device__ __forceinline__ bool is_finite(float x) { return fabsf(x) < __int_as_float(0x7f800000); }

// A lane's walk: `steps` double cells from cell `rel` of the row, voxels a and
// c with abscissae ax and cx at the second edge and steps da, dc per cell.  CHECK:
// cells outside [0, ncell) are left alone (some lane's walk leaves the row's
// guards).  All lanes of the warp take it.
template <int G, bool CHECK>
__device__ __forceinline__ void sweep_walk(typename SweepVec<G>::T *row, int rel, int ncell, int steps, float ax,
                                           float cx, float da, float dc, const float (&xa)[G], const float (&xc)[G])
{
  using VecG = typename SweepVec<G>::T;
  VecG *cell = row + rel;
  float pa = -0.5f, pc = -0.5f;  // both primitives are at -1/2 at the first edge
#pragma unroll 1
  for (int l = 0; l < steps; ++l) {
    bool in0 = true, in1 = true;
    if (CHECK) {
      in0 = (unsigned)rel < (unsigned)ncell;
      in1 = (unsigned)(rel + 1) < (unsigned)ncell;
    }
    VecG c0 = VecG{}, c1 = VecG{};
    if (in0) c0 = cell[0];
    if (in1) c1 = cell[1];
    const float ay = ax + da, cy = cx + dc;
    const float a1 = cubic_odd(ax), q1 = cubic_odd(cx), a2 = cubic_odd(ay), q2 = cubic_odd(cy);
    sweep_fma(c0, a1 - pa, q1 - pc, xa, xc);
    sweep_fma(c1, a2 - a1, q2 - q1, xa, xc);
    if (in0) cell[0] = c0;
    if (in1) cell[1] = c1;
    __syncwarp();
    pa = a2;
    pc = q2;
    ax = ay + da;
    cx = cy + dc;
    cell += 2;
    if (CHECK) rel += 2;
  }
}

// One column's profile by the whole warp in FP64 positions and shared-memory
// atomics: columns outside the fixed-point range or whose voxels nearly
// coincide on the detector.
template <int GEOM, int G>
__device__ __noinline__ void sweep_profile_any(const Params3D &P, const View3D &V, const float *__restrict__ vol,
                                               long gate_stride, int ci, int cj, int p0, int p1, int u0, int ncell,
                                               float *prof, int *odd)
{
  const int lane = threadIdx.x & 31;
  ColGeo<MODEL_CUBIC> c;
  column_geo<GEOM, MODEL_CUBIC>(P, V, ci, cj, 0, c);
  for (int k = 2 * p0 + lane; k < 2 * p1 && k < P.nz; k += 32) {
    UPair up;
    voxel_u_pair<GEOM>(P, V, c, k, k, up);
    const float F0 = first_edge_prim2(up).x;
    for (int m = 0; m < G; ++m) {
      const float x = vox_val(vol, gate_stride, V, turned_col(ci, cj, 4 - sweep_turn<G>(m), P.nx, P.ny) * P.nz + k);
      if (x == 0.f) continue;
      if (!is_finite(x)) {
        *odd = 1;
        continue;
      }
      float Fp = F0;
      for (int l = 0; l < up.n0; ++l) {
        const float F = cubic_prim2(f2(fmaf((float)(l + 1), up.inc.x, up.start.x))).x;
        const int cell = up.lo0 + l - u0;
        if ((unsigned)cell < (unsigned)ncell) atomicAdd(prof + cell * G + m, (F - Fp) * up.rho.x * x);
        Fp = F;
      }
    }
  }
}

// The same of the tabulated footprint.
template <int GEOM>
__device__ __forceinline__ bool sweep_record(const Params3D &P, const View3D &V, int i, int j, int v0, int v1, int u0,
                                             int u1, TableCol &r, int *__restrict__ err)
{
  double A, B, hsm, sp;
  if (!table_column<GEOM>(P, V, i, j, r, A, B, hsm, sp, err)) return false;
  if (r.lo + r.n <= v0 || r.lo >= v1) return false;
  tile_voxels(A, B, hsm, P.nz, u0, u1, r.k0, r.k1);
  // neighbouring lanes at least two cells apart (0.2% for the rounding of the cells)
  r.q_lanes = sp > 0.03 ? (int)ceil(2.004 / sp) : 0;
  return r.k0 < r.k1;
}

// Voxel k of column `col` of a (gated) view.
__device__ __forceinline__ float gate_value(const View3D &V, const float *colp, long dgate, bool gated, int k)
{
  float x = __ldg(colp + k);
  if (gated) x = V.w1 != 0.f ? fmaf(V.w0, x, V.w1 * __ldg(colp + dgate + k)) : V.w0 * x;
  return x;
}

// Profiles of a warp's columns, tabulated footprint: H lanes per column, each
// one voxel per pass, neighbouring lanes at least two cells apart, so that a
// step of two cells writes distinct cells.  row: the column's profile row; *odd is
// set where a voxel is not finite (left out).  Returns the lanes that had voxels to
// add.
template <int GEOM, int H>
__device__ __forceinline__ unsigned table_profiles(const Params3D &P, const View3D &V, const TableSh &T,
                                                   const TableCol &r, bool mine, int q, const float *colp, long dgate,
                                                   bool gated, int u0, int u1, float *row, int *odd)
{
  const int lig = threadIdx.x & (H - 1);
  const int k0 = r.k0, k1 = mine ? r.k1 : k0, nk = __reduce_max_sync(FULLM, k1 - k0);
  unsigned touched = 0;
#pragma unroll 1
  for (int pp = 0, sub = 0; pp < nk;) {
    const int k = k0 + pp + sub + q * lig;
    if (++sub == q) {
      sub = 0;
      pp += H * q;
    }
    float x = k < k1 ? gate_value(V, colp, dgate, gated, k) : 0.f;
    const unsigned some = __ballot_sync(FULLM, x != 0.f);
    if (!some) continue;
    if (!is_finite(x)) {
      *odd = 1;
      x = 0.f;
    }
    touched |= some;
    TableVox v;
    table_voxel<GEOM>(P, V, T, r, table_kc<GEOM>(V, k), u0, u1, v);
    if (x == 0.f) v.n = 0;
    const float xr = x * v.rho;
    const int steps = __reduce_max_sync(FULLM, v.n > 0 ? v.s + v.n : 0);
    float *cell = row + (v.f - u0);
    double l = (double)(-v.l0), e0 = table_at(T, dadd(v.start, dmul(l, v.inc)));
#pragma unroll 1
    for (int t = 0; t < steps; t += 2) {
      const double e1 = table_at(T, dadd(v.start, dmul(l + 1.0, v.inc)));
      l += 2.0;
      const double e2 = table_at(T, dadd(v.start, dmul(l, v.inc)));
      const bool in0 = (unsigned)(t - v.s) < (unsigned)v.n, in1 = (unsigned)(t + 1 - v.s) < (unsigned)v.n;
      float y0 = 0.f, y1 = 0.f;
      if (in0) y0 = cell[0];
      if (in1) y1 = cell[1];
      y0 = fmaf((float)(e1 - e0), xr, y0);
      y1 = fmaf((float)(e2 - e1), xr, y1);
      if (in0) cell[0] = y0;
      if (in1) cell[1] = y1;
      __syncwarp();
      e0 = e2;
      cell += 2;
    }
  }
  return touched;
}

// One column's by the whole warp with atomics: columns whose voxels nearly
// coincide on the detector.
template <int GEOM>
__device__ __noinline__ void table_profile_any(const Params3D &P, const View3D &V, const TableSh &T, const TableCol &r,
                                               const float *colp, long dgate, bool gated, int u0, int u1, float *row,
                                               int *odd)
{
  for (int k = r.k0 + (threadIdx.x & 31); k < r.k1; k += 32) {
    const float x = gate_value(V, colp, dgate, gated, k);
    if (x == 0.f) continue;
    if (!is_finite(x)) {
      *odd = 1;
      continue;
    }
    TableVox v;
    table_voxel<GEOM>(P, V, T, r, table_kc<GEOM>(V, k), u0, u1, v);
    for (int t = v.s; t < v.s + v.n; ++t) {
      const double l = (double)(t - v.l0);
      const float w = (float)(table_at(T, dadd(v.start, dmul(l + 1.0, v.inc))) -
                              table_at(T, dadd(v.start, dmul(l, v.inc))));
      atomicAdd(row + (v.f - u0) + t, w * (x * v.rho));
    }
  }
}

// All threads of the CTA call it; band, prof (this warp's profile rows) and
// locks are zero on entry, prof zero on exit; no final barrier.  `next`: the
// CTA's line counter (0 on entry); the CTA takes lines rank, rank + split, ...
// The tile has u1 - u0 <= 64 Q / G cells.  *odd (0 on entry) is set where a voxel
// is not finite; such voxels are left out, for sweep_odd.
template <int GEOM, int G, int Q, int H, int MODEL>
__device__ __forceinline__ void sweep_item(const Params3D &P, const View3D &V, const float *__restrict__ vol,
                                           long gate_stride, int v0, int v1, int u0, int u1, float *band, float *prof,
                                           typename SweepRec<MODEL>::T *recs, float2 *wtab, int *locks, int *next,
                                           int rank, int split, const TableSh &T, int *odd, int *__restrict__ err)
{
  using Rec = typename SweepRec<MODEL>::T;
  constexpr int RB = SweepRec<MODEL>::batch;
  using VecG = typename SweepVec<G>::T;
  using Strip = SweepStrip<Q, H>;
  constexpr int NC = Strip::NC, SP = Strip::SP, NS = Strip::NS;
  constexpr int PS = 64 * Q / G + kSweepGuard;  // cells of a profile row
  const int lane = threadIdx.x & 31, grp = lane / H, lig = lane & (H - 1);
  const int nx = P.nx, ny = P.ny, nz = P.nz, ncell = u1 - u0;
  SweepView S;
  sweep_view<GEOM>(P, V, S);
  const int n = S.axis ? ny : nx, nl = S.axis ? nx : ny;
  const bool gated = G == 1 && (V.w1 != 0.0f || V.w0 != 1.0f);
  const float *volg = G == 1 ? vol + (long)V.g0 * gate_stride : vol;
  const long dgate = ((long)V.g1 - V.g0) * gate_stride;
  // units of work: lines, halved where a warp has fewer than 4
  const int nseg = (4 * (int)(blockDim.x >> 5) * split) > nl ? 2 : 1;
  for (;;) {
    int un = 0;
    if (lane == 0) un = atomicAdd(next, 1);
    un = __shfl_sync(FULLM, un, 0);
    const int ln = (un / nseg) * split + rank, seg = un % nseg;
    if (ln >= nl) break;
    int a0, a1;
    sweep_range<GEOM>(P, V, S, ln, n, v0, v1, a0, a1);
    if (nseg > 1) {
      const int len = (a1 - a0 + nseg - 1) / nseg;
      a0 += seg * len;
      a1 = min(a1, a0 + len);
    }
    for (int ab = a0; ab < a1; ab += RB) {
      // ---- records of up to RB columns, without gaps ---------------------
      const int a = ab + lane;
      Rec rec;
      const bool hit = a < a1 && (RB == 32 || lane < RB) &&
                       sweep_record<GEOM>(P, V, S.axis ? ln : a, S.axis ? a : ln, v0, v1, u0, u1, rec, err);
      rec.col = a;
      const unsigned mask = __ballot_sync(FULLM, hit);
      const int cnt = __popc(mask);
      __syncwarp();
      if (hit) recs[__popc(mask & ((1u << lane) - 1u))] = rec;
      __syncwarp();
      for (int b = 0; b < cnt; b += NC) {
        // ---- profiles of columns b .. b + NC - 1 -------------------------
        const bool mine = b + grp < cnt;
        const Rec &r = recs[mine ? b + grp : b];
        unsigned touched = 0;
        if constexpr (MODEL == MODEL_TABLE) {
          if (!__any_sync(FULLM, r.q_lanes == 0)) {
            const float *colp = volg + turned_col(S.axis ? ln : r.col, S.axis ? r.col : ln, 0, nx, ny) * nz;
            touched = table_profiles<GEOM, H>(P, V, T, r, mine, __reduce_max_sync(FULLM, r.q_lanes), colp, dgate,
                                              gated, u0, u1, prof + kSweepGuard + grp * PS, odd);
          } else {
            for (int g = 0; g < NC && b + g < cnt; ++g) {
              const Rec &o = recs[b + g];
              const float *colp = volg + turned_col(S.axis ? ln : o.col, S.axis ? o.col : ln, 0, nx, ny) * nz;
              table_profile_any<GEOM>(P, V, T, o, colp, dgate, gated, u0, u1, prof + kSweepGuard + g * PS, odd);
            }
            touched = FULLM;
            __syncwarp();
          }
        } else if (!__any_sync(FULLM, r.q == 0)) {
          const int p0 = r.p0, p1 = mine ? r.p1 : p0;
          const int q = __reduce_max_sync(FULLM, r.q);
          const int steps = __reduce_max_sync(FULLM, r.steps), np = __reduce_max_sync(FULLM, p1 - p0);
          const int ci = S.axis ? ln : r.col, cj = S.axis ? r.col : ln;
          const float *colp[G];
#pragma unroll
          for (int m = 0; m < G; ++m) colp[m] = volg + turned_col(ci, cj, 4 - sweep_turn<G>(m), nx, ny) * nz;
          const long long A = r.A, B = r.B;
          const bool up = B >= 0;
          float h_c, rho_c, inv_den = 0.f;
          if constexpr (GEOM == GEOM_CONE) {
            h_c = r.h;
            rho_c = r.rho;
            inv_den = r.inv_den;
          } else {
            h_c = (float)V.p_hs_u;
            rho_c = (float)V.p_rho0;
          }
          VecG *row = reinterpret_cast<VecG *>(prof) + kSweepGuard + grp * PS;
          // pass: pairs pp + sub + q lane, sub < q; ue: position of a pair's first voxel
          const long long B2 = 2 * B, hop = B2 * (H * q - q + 1);
          long long ue = A + B2 * (p0 + q * lig);
#pragma unroll 1
          for (int pp = 0, sub = 0; pp < np;) {
            const int p = p0 + pp + sub + q * lig;
            const long long ue0 = ue;
            if (++sub < q) {
              ue += B2;
            } else {
              ue += hop;
              sub = 0;
              pp += H * q;
            }
            // a: the voxel whose footprint starts lower, c: the other
            const int ke = 2 * p, ko = ke + 1;
            const bool ine = p < p1 && ke < nz, ino = p < p1 && ko < nz;
            float xe[G], xo[G];
            float mag = 0.f;  // of the values together: 0 only if all are, infinite or NaN if one is
#pragma unroll
            for (int m = 0; m < G; ++m) {
              xe[m] = ine ? __ldg(colp[m] + ke) : 0.f;
              xo[m] = ino ? __ldg(colp[m] + ko) : 0.f;
              if (G == 1 && gated) {  // interpolation between two gates, as vox_val
                if (V.w1 != 0.f) {
                  if (ine) xe[m] = fmaf(V.w0, xe[m], V.w1 * __ldg(colp[m] + dgate + ke));
                  if (ino) xo[m] = fmaf(V.w0, xo[m], V.w1 * __ldg(colp[m] + dgate + ko));
                } else {
                  xe[m] *= V.w0;
                  xo[m] *= V.w0;
                }
              }
              mag += fabsf(xe[m]) + fabsf(xo[m]);
            }
            const unsigned some = __ballot_sync(FULLM, mag != 0.f);
            if (!some) continue;
            if (__any_sync(FULLM, !is_finite(mag))) {  // left to sweep_odd
              *odd = 1;
#pragma unroll
              for (int m = 0; m < G; ++m) {
                if (!is_finite(xe[m])) xe[m] = 0.f;
                if (!is_finite(xo[m])) xo[m] = 0.f;
              }
            }
            touched |= some;
            const long long uo = ue0 + B, ua = up ? ue0 : uo, uc = up ? uo : ue0;
            const int Ia = (int)(ua >> 32), Ic = (int)(uc >> 32);
            const float2 ph = make_float2(__uint_as_float(((unsigned)ua >> 9) | 0x3f800000u) - 1.0f,
                                          __uint_as_float(((unsigned)uc >> 9) | 0x3f800000u) - 1.0f);
            float2 scl, rho;
            float hs;
            if constexpr (GEOM == GEOM_CONE) {
              const float2 uca = mul2(add2(make_float2((float)Ia, (float)Ic), add2(ph, f2(-(float)V.a12))),
                                      f2((float)P.u_scl));
              const float2 du2 = fma2(mul2(uca, uca), f2(inv_den), f2(1.0f));
              const float2 dlt = mul2(du2, make_float2(rsqrt_ftz(du2.x), rsqrt_ftz(du2.y)));
              const float2 h = mul2(dlt, f2(h_c));
              scl = make_float2(rcp_ftz(h.x), rcp_ftz(h.y));
              rho = mul2(dlt, f2(rho_c));
              hs = (float)P.hs0 * h.x;
            } else {
              scl = f2((float)V.p_scl_u);
              rho = f2(rho_c);
              hs = h_c;
            }
            // first cell of a: Ia + floor(phi - hs); adding 1.5 2^23 with
            // rounding toward -inf leaves the floor in the low bits
            const float fm = __fadd_rd(ph.x - hs, 12582912.0f);
            const int f = Ia + (__float_as_int(fm) - 0x4B400000);
            // abscissae of the second edge, (f + 1 - uc) scl
            const float2 x1 = mul2(add2(make_float2(fm - 12582911.0f, (float)(f + 1 - Ic)),
                                        make_float2(-ph.x, -ph.y)), scl);
            float xa[G], xc[G];
#pragma unroll
            for (int m = 0; m < G; ++m) {
              xa[m] = (up ? xe[m] : xo[m]) * rho.x;
              xc[m] = (up ? xo[m] : xe[m]) * rho.y;
            }
            // lanes past the column's pairs (zeros) walk in the guard
            const int rel = p < p1 ? f - u0 : -kSweepGuard;
            if (__all_sync(FULLM, rel >= -kSweepGuard && rel + 2 * steps <= PS && 2 * steps <= kSweepGuard))
              sweep_walk<G, false>(row, rel, ncell, steps, x1.x, x1.y, scl.x, scl.y, xa, xc);
            else
              sweep_walk<G, true>(row, p < p1 ? rel : ncell, ncell, steps, x1.x, x1.y, scl.x, scl.y, xa, xc);
          }
        } else {
          for (int g = 0; g < NC && b + g < cnt; ++g) {
            const Rec &o = recs[b + g];
            sweep_profile_any<GEOM, G>(P, V, vol, gate_stride, S.axis ? ln : o.col, S.axis ? o.col : ln, o.p0, o.p1,
                                       u0, ncell, prof + G * (kSweepGuard + g * PS), odd);
          }
          touched = FULLM;
          __syncwarp();
        }
        // ---- weighted sums of the profiles into the band ------------------
        const bool on = mine && ((touched >> (grp * H)) & (H == 32 ? FULLM : (1u << (H & 31)) - 1u));
        const int r0 = __reduce_min_sync(FULLM, on ? max(r.lo, v0) : INT_MAX);
        const int r1 = __reduce_max_sync(FULLM, on ? min(r.lo + r.n, v1) : INT_MIN);
        if (r0 >= r1) continue;
        const unsigned live = __ballot_sync(FULLM, on);
        const int gend = sweep_groups(r1 - v0);
#pragma unroll 1
        for (int gb = (r0 - v0) / kSweepRows; gb < gend; gb += kSweepGroups) {
          const int ng = min(gend - gb, kSweepGroups);
          const bool last = gb + kSweepGroups >= gend;
          // table of weights [row][column], rows of lock groups gb .. gb + ng
          for (int e = lane; e < ng * kSweepRows * NC; e += 32) {
            const int g = e % NC;
            const Rec &o = recs[min(b + g, cnt - 1)];
            const int l = v0 + gb * kSweepRows + e / NC - o.lo;
            float w = 0.f;
            if (((live >> (g * H)) & 1u) && l >= 0 && l < o.n) {
              if constexpr (MODEL == MODEL_TABLE) {
                w = table_weight_v(T, o, l);
              } else {
                AxisCubic ax;
                ax.start = o.vstart;
                ax.inc = o.vinc;
                w = edge_cubic(ax, l + 1) - edge_cubic(ax, l);
              }
            }
            wtab[e] = f2(w);
          }
          __syncwarp();
#pragma unroll 1
          for (int s = 0; s < NS; ++s) {
            float2 pv[NC][SP];
#pragma unroll
            for (int g = 0; g < NC; ++g)
#pragma unroll
              for (int t = 0; t < SP; ++t) {
                float2 *c = reinterpret_cast<float2 *>(prof + G * (kSweepGuard + g * PS)) + lane + 32 * (s * SP + t);
                pv[g][t] = *c;
                if (last) *c = f2(0.f);
              }
#pragma unroll 1
            for (int k = 0; k < ng; ++k) {
              int *lock = locks + (gb + k) * NS + s;
              if (!row_lock(lock, err)) continue;
              float2 *br =
                  reinterpret_cast<float2 *>(band) + (size_t)(gb + k) * kSweepRows * (32 * Q) + lane + 32 * s * SP;
              float2 sum[kSweepRows][SP];
#pragma unroll
              for (int rr = 0; rr < kSweepRows; ++rr)
#pragma unroll
                for (int t = 0; t < SP; ++t) sum[rr][t] = br[rr * (32 * Q) + 32 * t];
#pragma unroll
              for (int rr = 0; rr < kSweepRows; ++rr)
#pragma unroll
                for (int g = 0; g < NC; ++g) {
                  const float2 w = wtab[(k * kSweepRows + rr) * NC + g];
#pragma unroll
                  for (int t = 0; t < SP; ++t) sum[rr][t] = fma2(w, pv[g][t], sum[rr][t]);
                }
#pragma unroll
              for (int rr = 0; rr < kSweepRows; ++rr)
#pragma unroll
                for (int t = 0; t < SP; ++t) br[rr * (32 * Q) + 32 * t] = sum[rr][t];
              row_unlock(lock);
            }
          }
          __syncwarp();
        }
      }
    }
  }
}

// The voxels that are not finite, which sweep_item leaves out: each is added to the
// cells and rows where its own weights are not zero.  (The sums of sweep_item over
// several columns and voxels take products with weights of 0, harmless as long as
// every factor is finite.)  Column by column: its values' profile, a voxel per lane
// with atomics, then the cells of it that are not finite into the rows, under the
// band's locks.  A second pass over the CTA's lines, so that nothing of it is alive in
// the loops of the first (called from there it cost 4 to 7% of every projection; the
// test of the values that is left there 0 to 1.5%); no call with a finite volume
// comes here.  45 pairs of views of 128^3: 2.1 ms, with one NaN voxel 3.5 ms, all of
// them NaN 11.4 (voxel by voxel into the rows 524).  All threads of the CTA call it
// after a barrier; prof is zero on entry and exit.
template <int GEOM, int G, int Q, int H, int MODEL>
__device__ __noinline__ void sweep_odd(const Params3D &P, const View3D &V, const float *__restrict__ vol,
                                       long gate_stride, const TableSh &T, int v0, int v1, int u0, int u1, float *band,
                                       float *prof, int *locks, int rank, int split, int *__restrict__ err)
{
  using Strip = SweepStrip<Q, H>;
  constexpr int SP = Strip::SP, NS = Strip::NS;
  const int lane = threadIdx.x & 31, warps = blockDim.x >> 5, ncell = u1 - u0;
  float *row = prof + G * kSweepGuard;
  SweepView S;
  sweep_view<GEOM>(P, V, S);
  const int n = S.axis ? P.ny : P.nx, nl = S.axis ? P.nx : P.ny;
  for (int unit = threadIdx.x >> 5; (unit / n) * split + rank < nl; unit += warps) {
    const int ln = (unit / n) * split + rank, a = unit % n;  // the lines that the CTA took in the first pass
    const int ci = S.axis ? ln : a, cj = S.axis ? a : ln;
    typename SweepRec<MODEL>::T o;
    if (!sweep_record<GEOM>(P, V, ci, cj, v0, v1, u0, u1, o, err)) continue;
    ColGeo<MODEL_CUBIC> c;
    int ka, kb;
    if constexpr (MODEL == MODEL_TABLE) {
      ka = o.k0;
      kb = o.k1;
    } else {
      column_geo<GEOM, MODEL_CUBIC>(P, V, ci, cj, 0, c);
      ka = 2 * o.p0;
      kb = min(2 * o.p1, P.nz);
    }
    // ---- the column's profile ---------------------------------------------
    bool any = false;
    for (int k = ka + lane; k < kb; k += 32) {
      float x[G];
      bool bad = false;
      for (int m = 0; m < G; ++m) {
        x[m] = vox_val(vol, gate_stride, V, turned_col(ci, cj, 4 - sweep_turn<G>(m), P.nx, P.ny) * P.nz + k);
        bad = bad || !is_finite(x[m]);
      }
      if (!bad) continue;
      any = true;
      auto add = [&](int u, float w, float rho) {
        if (w == 0.f || (unsigned)(u - u0) >= (unsigned)ncell) return;
        for (int m = 0; m < G; ++m)
          if (!is_finite(x[m])) atomicAdd(row + (u - u0) * G + m, w * (x[m] * rho));
      };
      if constexpr (MODEL == MODEL_TABLE) {
        TableVox t;
        table_voxel<GEOM>(P, V, T, o, table_kc<GEOM>(V, k), u0, u1, t);
        for (int l = t.s; l < t.s + t.n; ++l) {
          const double e = (double)(l - t.l0);
          add(t.f + l, (float)(table_at(T, dadd(t.start, dmul(e + 1.0, t.inc))) -
                               table_at(T, dadd(t.start, dmul(e, t.inc)))), t.rho);
        }
      } else {
        UPair up;
        voxel_u_pair<GEOM>(P, V, c, k, k, up);
        for (int l = 0; l < up.n0; ++l) {
          const float2 e = fma2(make_float2((float)l, (float)(l + 1)), f2(up.inc.x), f2(up.start.x));
          const float2 F = cubic_prim2(e);
          add(up.lo0 + l, F.y - (l == 0 ? first_edge_prim2(up).x : F.x), up.rho.x);
        }
      }
    }
    if (!__any_sync(FULLM, any)) continue;
    __syncwarp();
    // ---- into the rows ----------------------------------------------------
    const int r0 = max(o.lo, v0), r1 = min(o.lo + o.n, v1);
    for (int s = 0; s < NS; ++s) {
      float y[2 * SP];  // the floats of the lane's pairs
      bool odd = false;
#pragma unroll
      for (int q = 0; q < 2 * SP; ++q) {
        y[q] = row[2 * (lane + 32 * (s * SP + (q >> 1))) + (q & 1)];
        odd = odd || !is_finite(y[q]);
      }
      if (!__any_sync(FULLM, odd)) continue;
      for (int gr = (r0 - v0) / kSweepRows; gr < sweep_groups(r1 - v0); ++gr) {
        int *lock = locks + gr * NS + s;
        if (!row_lock(lock, err)) continue;
        for (int r = max(r0, v0 + gr * kSweepRows); r < min(r1, v0 + (gr + 1) * kSweepRows); ++r) {
          float wv;
          if constexpr (MODEL == MODEL_TABLE) {
            wv = table_weight_v(T, o, r - o.lo);
          } else {
            AxisCubic ax;
            ax.start = o.vstart;
            ax.inc = o.vinc;
            wv = edge_cubic(ax, r - o.lo + 1) - edge_cubic(ax, r - o.lo);
          }
          if (wv == 0.f) continue;
          float *br = band + (size_t)(r - v0) * (64 * Q);
#pragma unroll
          for (int q = 0; q < 2 * SP; ++q)
            if (!is_finite(y[q])) br[2 * (lane + 32 * (s * SP + (q >> 1))) + (q & 1)] += wv * y[q];
        }
        row_unlock(lock);
      }
    }
    __syncwarp();
    for (int t = lane; t < 64 * Q; t += 32) row[t] = 0.f;
    __syncwarp();
  }
}

}  // namespace trtt
