// proj2d_orbit.cu -- 2D projector pair (B-spline closed form and table,
// Long-Fessler) over groups of views related by quarter turns of the pixel
// grid.
//
// A scan over 2 pi (or pi, parallel beam) sees a square image turned by a
// quarter turn every quarter of its views: the view at theta + m pi/2 sees
// pixel p exactly where the view at theta sees R^m(p), R(i, j) = (n-1-j, i).
// The FP64 footprint of a pixel (divisions, square roots, one primitive per
// cell edge) is what a pair spends its time on, so it is evaluated once per
// group, at the group's first view, and applied to the members' pixels.
// Only the closed form and Long-Fessler group: a table weight jumps at the
// table's slots, so it stays at the reference's own positions (one view per
// group, footprints of foot2d).
//
// Direct (k_fwd2d_orbit): one CTA per (group, tile of detector cells, share
// of the image lines).  Each of its 8 warps owns a row of the tile's cells,
// interleaved [cell][member]; it walks image lines along the axis on which
// neighbouring pixels project furthest apart, lanes `lane_stride` pixels
// apart, so that the 32 footprints of a step start at distinct cells and,
// cell by cell, update the row with plain vector loads and stores (checked
// at each step; shared-memory atomics, which are compare-and-swap loops on
// this GPU, only where the check fails).  The CTAs of a cluster add their
// rows through distributed shared memory: every detector cell has one owner
// and no global atomics are used.
//
// Transpose (k_back2d_orbit): one thread per pixel position; per group one
// footprint gathers the members' rows, and the member sums are exchanged
// inside the block (a block holds whole orbits of pixels) at the end.  FP64
// sums in a fixed order; the CTAs of a cluster share the groups.
//
// Same weights both ways (foot2), so the pair is an adjoint pair up to FP32
// rounding of the direct projection's sums.
//
// Measured (B200, 512^2 image, 720 fan-beam views of 1024 cells; the per-view
// kernels of proj2d.cu before): direct 5.67 -> 1.10 ms, transpose 4.16 -> 0.97
// ms; Long-Fessler 4.47 -> 0.99 and 5.32 -> 0.78 ms; 256^2, 180 parallel views:
// 1.12 -> 0.097 and 0.25 -> 0.072 ms.  Bounds (ncu, fan beam): the direct
// kernel's shared-memory and L1 wavefronts (76% of peak: row updates, and the
// quarter-turned members' pixels read across image rows); the transpose's FP64
// (49%) and conversion (55%) pipes at 63% of the issue slots.  The direct
// result is also closer to FP64 (5e-8 instead of 7e-7): a cell's sum is spread
// over the warps' rows and the rows are added in FP64.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <climits>
#include <cmath>

#include "foot2d.cuh"
#include "host3d.h"
#include "proj2d_orbit.cuh"

namespace cg = cooperative_groups;

namespace trtt {

namespace {

constexpr unsigned FULL = 0xffffffffu;
constexpr int kWarps = 8;      // warps per CTA, both kernels
constexpr int kBatch = 16;     // group records staged together (transpose)
constexpr int kMaxSplit = 8;   // portable cluster size

template <int CLS> struct Cls;
template <> struct Cls<C2_ONE> { static constexpr int NS = 1, OS = 1; };
template <> struct Cls<C2_HALF> { static constexpr int NS = 2, OS = 2; };
template <> struct Cls<C2_QUARTER> { static constexpr int NS = 2, OS = 4; };
template <> struct Cls<C2_QUAD> { static constexpr int NS = 4, OS = 4; };

// Quarter turns of member slot s.
template <int CLS> __host__ __device__ constexpr int slot_turn(int s) { return CLS == C2_HALF ? 2 * s : s; }

__device__ __forceinline__ void turn_pix(int i, int j, int t, int nx, int ny, int &oi, int &oj)
{
  switch (t & 3) {
    case 0: oi = i; oj = j; break;
    case 1: oi = nx - 1 - j; oj = i; break;
    case 2: oi = nx - 1 - i; oj = ny - 1 - j; break;
    default: oi = j; oj = ny - 1 - i; break;
  }
}

// max(v, 0) on the integer pipe (FP64 has no min / max instruction).
__device__ __forceinline__ double pos_part(double v)
{
  const int hi = __double2hiint(v), keep = ~(hi >> 31);
  return __hiloint2double(hi & keep, __double2loint(v) & keep);
}

// Primitive of the centred cubic B-spline in its truncated-power form: with
// t = |x| the tail beyond t is g = ((2-t)_+^4 - 4 (1-t)_+^4) / 24 and
// P(x) = 1/2 + sign(x) (1/2 - g).  10 FP64 operations without a branch; the
// branchy quartics of cubic_prim_d cost a warp all four cases (about 40).
__device__ __forceinline__ double prim2(double x)
{
  const double t = fabs(x);
  const double a = pos_part(2.0 - t), b = pos_part(1.0 - t);
  const double a2 = a * a, b2 = b * b;
  const double g = fma(a2 * a2, 1.0 / 24.0, (b2 * b2) * (-1.0 / 6.0));
  return copysign(0.5 - g, x) + 0.5;
}

// Footprint of pixel (i, j) at the group's first view: cells [f, e) before
// the clamp at 0 (f may be negative), weight amp * (edge(c + 1) - edge(c)) in
// cell c, or amp * height(c).  Closed form: edge 0 at cell f.
template <int MODEL> struct Foot2;
template <> struct Foot2<M2_FAN> { int f, e; double vc, scl, amp; };
template <> struct Foot2<M2_PAR> { int f, e; double vc, scl, amp; };
template <> struct Foot2<M2_FAN_TABLE> { int f, e; Foot2D t; double amp; };
template <> struct Foot2<M2_PAR_TABLE> { int f, e; Foot2D t; double amp; };
template <> struct Foot2<M2_LF> { int f, e; double t0, t1, t2, t3, r1, r3, amp; };

__device__ __forceinline__ void swap_up(double &a, double &b)
{
  const bool s = a > b;
  const double lo = s ? b : a, hi = s ? a : b;
  a = lo;
  b = hi;
}

template <int MODEL>
__device__ __forceinline__ void foot2(const Orbit2DLaunch &A, const Orbit2D &g, const View2D *V, int i, int j,
                                      Foot2<MODEL> &ft)
{
  const Params2D &P = A.P;
  const double di = (double)i, dj = (double)j;
  if constexpr (MODEL == M2_FAN) {
    // magn = k1 / D; k0: a8, k2: (v_scl / a4)^2, k3: 1 / (h_init k1): one
    // reciprocal and one reciprocal square root per footprint
    const double D = fma(g.dj, dj, fma(g.di, di, g.d0));
    const double N = fma(g.nj, dj, fma(g.ni, di, g.n0));
    const double inv = __drcp_rn(D);
    ft.vc = fma(N, inv, g.c);
    const double va = ft.vc - g.k0;
    const double d2 = fma(va * va, g.k2, 1.0);
    const double rd = rsqrt(d2);
    const double md = (g.k1 * inv) * (d2 * rd);  // magn * delta_v
    ft.scl = (D * g.k3) * rd;
    ft.amp = P.rho0_init * md;
    const double hs = P.hs0 * (P.h_init * md);
    ft.f = __double2int_rd(ft.vc - hs);
    ft.e = min(__double2int_rd(ft.vc + hs) + 1, P.nv - 1);  // the last cell is never reached
  } else if constexpr (MODEL == M2_PAR) {
    // k1: 1 / h, k2: rho0, k3: half support
    ft.vc = fma(g.nj, dj, fma(g.ni, di, g.n0)) + g.c;
    ft.scl = g.k1;
    ft.amp = g.k2;
    ft.f = __double2int_rd(ft.vc - g.k3);
    ft.e = min(__double2int_rd(ft.vc + g.k3) + 1, P.nv - 1);
  } else if constexpr (MODEL == M2_FAN_TABLE || MODEL == M2_PAR_TABLE) {
    // the reference's own clamped range and edge positions
    foot2d(P, *V, i, j, ft.t);
    ft.amp = ft.t.rho0;
    ft.f = ft.t.lo;
    ft.e = ft.t.lo + ft.t.n;
    if (ft.t.lo == 0) {
      // first cell without the clamp (only orders the walk of the direct
      // kernel): start = (0 - (vc + coord0 h)) / (h step)
      const double h = 1.0 / (ft.t.inc * P.step);
      const double vc = -(ft.t.start * (h * P.step)) - P.coord0 * h;
      ft.f = min(__double2int_rd(vc - P.hs0 * h), 0);
    } else if (ft.t.lo == P.nv - 1 && dadd(ft.t.start, ft.t.inc) <= 0.0) {
      ft.e = ft.f;  // past the detector: the one clamped cell has weight cum[0] - cum[0]
    }
  } else {
    // Long-Fessler: lateral N (in cells times depth) and depth D of the
    // pixel's corners; k0 + i k2, k1 + j k2: the pixel seen from the source
    const double N = fma(g.nj, dj, fma(g.ni, di, g.n0)), D = fma(g.dj, dj, fma(g.di, di, g.d0));
    const double np = 0.5 * (g.ni + g.nj), nm = 0.5 * (g.ni - g.nj);
    const double dp = 0.5 * (g.di + g.dj), dm = 0.5 * (g.di - g.dj);
    const double d0 = D - dp, d1 = D + dp, d2 = D - dm, d3 = D + dm;
    const double qx = fma(di, g.k2, g.k0), qy = fma(dj, g.k2, g.k1);
    const double q2 = fma(qx, qx, qy * qy);
    const double ax = fabs(qx), ay = fabs(qy), qm = ay > ax ? ay : ax;
    // one reciprocal for the four depths and the larger component of q
    const double a = d0 * d1, b = d2 * d3, ab = a * b;
    const double r = __drcp_rn(ab * qm), rq = r * qm;
    const double ra = rq * b, rb = rq * a;
    ft.amp = g.k3 * ((q2 * rsqrt(q2)) * (r * ab));  // obliquity times the pixel's measure
    double t0 = fma(N - np, ra * d1, g.c), t1 = fma(N + np, ra * d0, g.c);
    double t2 = fma(N - nm, rb * d3, g.c), t3 = fma(N + nm, rb * d2, g.c);
    swap_up(t0, t1);
    swap_up(t2, t3);
    swap_up(t0, t2);
    swap_up(t1, t3);
    swap_up(t1, t2);
    // 1 / (2 (t1 - t0)) and 1 / (2 (t3 - t2)), 0 for a vertical flank
    const double w1 = t1 - t0, w3 = t3 - t2;
    const double c1 = w1 > 0.0 ? w1 : 1.0, c3 = w3 > 0.0 ? w3 : 1.0;
    const double rw = 0.5 * __drcp_rn(c1 * c3);
    ft.r1 = w1 > 0.0 ? rw * c3 : 0.0;
    ft.r3 = w3 > 0.0 ? rw * c1 : 0.0;
    ft.t0 = t0; ft.t1 = t1; ft.t2 = t2; ft.t3 = t3;
    const double hc = 0.5 * P.hs0;  // half a cell (pixelSize / pixelStep)
    ft.f = __double2int_rd(t0 - hc) + 1;
    ft.e = min(__double2int_ru(t3 + hc), P.nv);
  }
}

// Area of the Long-Fessler trapezoid left of p.
__device__ __forceinline__ double lf_area(const Foot2<M2_LF> &ft, double p)
{
  const double y = pos_part((p < ft.t1 ? p : ft.t1) - ft.t0);
  const double m = pos_part((p < ft.t2 ? p : ft.t2) - ft.t1);
  const double z = pos_part((p < ft.t3 ? p : ft.t3) - ft.t2);
  return fma(ft.r1 * y, y, m) + z * fma(-ft.r3, z, 1.0);
}

// Walk over the cells of a footprint: start(c) at the first one, then
// weight(c), weight(c + 1), ... (without amp).
template <int MODEL> struct Walk2 {
  double prev;

  __device__ __forceinline__ double edge(const Orbit2DLaunch &A, const Foot2<MODEL> &ft, int c) const
  {
    if constexpr (MODEL == M2_FAN || MODEL == M2_PAR) {
      return prim2(((double)c - ft.vc) * ft.scl);
    } else if constexpr (MODEL == M2_LF) {
      return lf_area(ft, (double)c - 0.5 * A.P.hs0);
    } else {
      return edge2d(A.P, ft.t, max(c - ft.t.lo, 0));
    }
  }
  __device__ __forceinline__ void start(const Orbit2DLaunch &A, const Foot2<MODEL> &ft, int c)
  {
    if constexpr (MODEL == M2_FAN || MODEL == M2_PAR) {
      prev = c == ft.f ? 0.0 : edge(A, ft, c);  // cell f starts left of the support
    } else if constexpr (MODEL == M2_LF) {
      prev = c == ft.f && A.P.hs0 == 1.0 ? 0.0 : edge(A, ft, c);
    } else {
      prev = edge(A, ft, c);
    }
  }
  __device__ __forceinline__ double weight(const Orbit2DLaunch &A, const Foot2<MODEL> &ft, int c)
  {
    if constexpr (MODEL == M2_LF) {
      if (A.line) {  // height of the trapezoid at the cell's centre
        const double p = (double)c;
        if (p >= ft.t0 && p < ft.t1) return 2.0 * ft.r1 * (p - ft.t0);
        if (p >= ft.t1 && p < ft.t2) return 1.0;
        if (p >= ft.t2 && p < ft.t3) return 2.0 * ft.r3 * (ft.t3 - p);
        return 0.0;
      }
      if (A.P.hs0 != 1.0) return lf_area(ft, (double)c + 0.5 * A.P.hs0) - edge(A, ft, c);
    }
    const double p1 = edge(A, ft, c + 1);
    const double w = p1 - prev;
    prev = p1;
    return w;
  }
};

template <int NS> struct Vec;
template <> struct Vec<1> { using T = float; };
template <> struct Vec<2> { using T = float2; };
template <> struct Vec<4> { using T = float4; };
__device__ __forceinline__ void vfma(float &v, float w, const float (&x)[1]) { v = fmaf(w, x[0], v); }
__device__ __forceinline__ void vfma(float2 &v, float w, const float (&x)[2])
{
  v.x = fmaf(w, x[0], v.x);
  v.y = fmaf(w, x[1], v.y);
}
__device__ __forceinline__ void vfma(float4 &v, float w, const float (&x)[4])
{
  v.x = fmaf(w, x[0], v.x);
  v.y = fmaf(w, x[1], v.y);
  v.z = fmaf(w, x[2], v.z);
  v.w = fmaf(w, x[3], v.w);
}

// Pixels [klo, khi) of an image line whose footprints may meet cells
// [u0, u1): the position along the line is monotone (the depth keeps its
// sign over the grid), so its inverse at the tile's ends bounds them.
__device__ __forceinline__ void line_range(const Orbit2D &g, int ln, int n, int u0, int u1, int &klo, int &khi)
{
  const double l = (double)ln;
  const double N0 = g.axis ? fma(g.ni, l, g.n0) : fma(g.nj, l, g.n0), N1 = g.axis ? g.nj : g.ni;
  const double D0 = g.axis ? fma(g.di, l, g.d0) : fma(g.dj, l, g.d0), D1 = g.axis ? g.dj : g.di;
  const double last = (double)(n - 1);
  const double pa = N0 / D0 + g.c, pb = fma(N1, last, N0) / fma(D1, last, D0) + g.c;
  const double lo = (double)u0 - 1.0 - g.hsm - g.c, hi = (double)u1 + 1.0 + g.hsm - g.c;
  const double a = pa - g.c, b = pb - g.c;
  const double mn = a < b ? a : b, mx = a < b ? b : a;
  klo = 0;
  khi = 0;
  if (!(mx >= lo && mn <= hi)) return;
  // k(v) solves N0 + N1 k = v (D0 + D1 k)
  double kl = a < b ? 0.0 : last, kh = a < b ? last : 0.0;  // positions of mn, mx
  if (lo > mn) kl = (N0 - lo * D0) / (lo * D1 - N1);
  if (hi < mx) kh = (N0 - hi * D0) / (hi * D1 - N1);
  const double k0 = kl < kh ? kl : kh, k1 = kl < kh ? kh : kl;
  klo = max(__double2int_rd(k0) - 1, 0);
  khi = min(__double2int_ru(k1) + 2, n);
}

template <int MODEL, int CLS>
__global__ void __launch_bounds__(32 * kWarps, 3) k_fwd2d_orbit(const Orbit2DLaunch A)
{
  constexpr int NS = Cls<CLS>::NS;
  using V = typename Vec<NS>::T;
  extern __shared__ __align__(16) float sm[];
  __shared__ Orbit2D g;
  __shared__ View2D sV;
  const int U = A.utile, S = A.split;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tile = blockIdx.x / S, rank = blockIdx.x - tile * S;
  const int nx = A.P.nx, ny = A.P.ny, nv = A.P.nv;
  const int u0 = tile * U, u1 = min(u0 + U, nv);
  V *rows = reinterpret_cast<V *>(sm);
  V *row = rows + warp * U;
  if (threadIdx.x < (int)(sizeof(Orbit2D) / 8))
    reinterpret_cast<double *>(&g)[threadIdx.x] =
        reinterpret_cast<const double *>(A.groups + blockIdx.y)[threadIdx.x];
  if constexpr (MODEL == M2_FAN_TABLE || MODEL == M2_PAR_TABLE) {
    if (threadIdx.x < (int)(sizeof(View2D) / 8))
      reinterpret_cast<double *>(&sV)[threadIdx.x] =
          reinterpret_cast<const double *>(A.views + A.groups[blockIdx.y].view[0])[threadIdx.x];
  }
  for (int t = lane; t < U; t += 32) row[t] = V{};
  __syncthreads();
  const int axis = g.axis, q = g.lane_stride;
  const int n = axis ? ny : nx, nl = axis ? nx : ny;
  const int W = kWarps * S, me = rank * kWarps + warp;
  for (int lb = 0; lb * W < nl; lb += 32) {
    // lane: image line (lb + lane) W + me of this warp
    const int myln = (lb + lane) * W + me;
    int klo = 0, khi = 0;
    if (myln < nl) line_range(g, myln, n, u0, u1, klo, khi);
    unsigned mask = __ballot_sync(FULL, klo < khi);
    while (mask) {
      const int src = __ffs(mask) - 1;
      mask &= mask - 1;
      const int ln = (lb + src) * W + me;
      const int k0 = __shfl_sync(FULL, klo, src), k1 = __shfl_sync(FULL, khi, src);
      // member slot s reads pixel R^-t(i, j) along the line
      const float *base[NS];
      long step[NS];
#pragma unroll
      for (int s = 0; s < NS; ++s) {
        int ai, aj, bi, bj;
        const int t = 4 - slot_turn<CLS>(s);
        turn_pix(axis ? ln : 0, axis ? 0 : ln, t, nx, ny, ai, aj);
        turn_pix(axis ? ln : 1, axis ? 1 : ln, t, nx, ny, bi, bj);
        base[s] = A.in + ((long)aj * nx + ai);
        step[s] = ((long)bj * nx + bi) - ((long)aj * nx + ai);
      }
      for (int kb = k0; kb < k1; kb += 32 * q) {
        for (int sub = 0; sub < q; ++sub) {
          const int k = kb + sub + q * lane;
          const bool in = k < k1;
          float x[NS];
          bool any = false;
#pragma unroll
          for (int s = 0; s < NS; ++s) {
            x[s] = in ? __ldg(base[s] + k * step[s]) : 0.0f;
            any = any || x[s] != 0.0f;
          }
          if (!__any_sync(FULL, any)) continue;
          const int kc = in ? k : k1 - 1;
          Foot2<MODEL> ft;
          foot2<MODEL>(A, g, &sV, axis ? ln : kc, axis ? kc : ln, ft);
          const int e = min(ft.e, u1);
          const int L = any ? max(e - ft.f, 0) : 0;
          const int Lw = __reduce_max_sync(FULL, L);
          // distinct first cells (monotone over the lanes in the range)
          const int fn = __shfl_down_sync(FULL, ft.f, 1), f0 = __shfl_sync(FULL, ft.f, 0),
                    f1 = __shfl_sync(FULL, ft.f, 1);
          const bool use = in && ft.e > ft.f;
          const bool un = __shfl_down_sync(FULL, use ? 1 : 0, 1) != 0;
          const bool ok = lane == 31 || !use || !un || (f1 > f0 ? fn > ft.f : fn < ft.f);
          const bool distinct = __all_sync(FULL, ok);
          Walk2<MODEL> wk;
          wk.start(A, ft, ft.f);
          if (distinct) {
            for (int l = 0; l < Lw; ++l) {
              const int c = ft.f + l;
              const double wd = wk.weight(A, ft, c);
              const float w = (float)(wd * ft.amp);
              // (the ends of a Long-Fessler range may have weight 0: no cells of the
              // footprint, for values that are not finite)
              if (l < L && c >= u0 && (MODEL != M2_LF || wd != 0.0)) {
                V v = row[c - u0];
                vfma(v, w, x);
                row[c - u0] = v;
              }
              __syncwarp();
            }
          } else {
            for (int l = 0; l < L; ++l) {
              const int c = ft.f + l;
              const double wd = wk.weight(A, ft, c);
              const float w = (float)(wd * ft.amp);
              if (c >= u0 && (MODEL != M2_LF || wd != 0.0)) {
#pragma unroll
                for (int s = 0; s < NS; ++s)
                  atomicAdd(reinterpret_cast<float *>(row + (c - u0)) + s, w * x[s]);
              }
            }
            __syncwarp();
          }
        }
      }
    }
  }
  __syncthreads();
  // sum of the CTA's rows, then of the cluster's CTAs
  const int nval = (u1 - u0) * NS;
  const float *flat = sm;
  double *red = reinterpret_cast<double *>(sm + kWarps * U * NS);
  if (S == 1) {
    for (int t = threadIdx.x; t < nval; t += blockDim.x) {
      double v = 0.0;
#pragma unroll
      for (int w = 0; w < kWarps; ++w) v += (double)flat[w * U * NS + t];
      float *o = A.out + (long)g.view[t % NS] * nv + u0 + t / NS;
      *o += (float)v;
    }
    return;
  }
  for (int t = threadIdx.x; t < nval; t += blockDim.x) {
    double v = 0.0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) v += (double)flat[w * U * NS + t];
    red[t] = v;
  }
  cg::cluster_group cl = cg::this_cluster();
  cl.sync();
  for (int t = rank * blockDim.x + threadIdx.x; t < nval; t += S * blockDim.x) {
    double v = 0.0;
    for (int r = 0; r < S; ++r) v += cl.map_shared_rank(red, r)[t];
    float *o = A.out + (long)g.view[t % NS] * nv + u0 + t / NS;
    *o += (float)v;
  }
  cl.sync();  // no CTA leaves while another reads its sums
}

template <int MODEL, int CLS>
__global__ void __launch_bounds__(32 * kWarps, 3) k_back2d_orbit(const Orbit2DLaunch A)
{
  constexpr int NS = Cls<CLS>::NS, OS = Cls<CLS>::OS, NO = 32 * kWarps / OS;
  constexpr bool TABLE = MODEL == M2_FAN_TABLE || MODEL == M2_PAR_TABLE;
  __shared__ Orbit2D recs[kBatch];
  __shared__ View2D vrec[TABLE ? kBatch : 1];
  __shared__ double ex[NS][32 * kWarps];
  __shared__ double part[32 * kWarps];
  const int S = A.split;
  const int blk = blockIdx.x / S, rank = blockIdx.x - blk * S;
  const int nx = A.P.nx, ny = A.P.ny, nv = A.P.nv;
  // fundamental domain of the orbits
  const int dx = OS == 1 ? nx : (OS == 2 ? ((ny & 1) ? nx / 2 : nx) : nx / 2);
  const int dy = OS == 1 ? ny : (OS == 2 ? ((ny & 1) ? ny : ny / 2) : ny / 2);
  const int rot = threadIdx.x / NO, o = threadIdx.x - rot * NO;
  // a warp covers 8 x 4 pixels, the block's orbits 16 x (NO / 16)
  const int tx = (dx + 15) / 16;
  const int bx = blk % tx, by = blk / tx;
  const int i0 = bx * 16 + ((o >> 5) & 1) * 8 + (o & 7);
  const int j0 = by * (NO / 16) + (o >> 6) * 4 + ((o >> 3) & 3);
  const bool valid = i0 < dx && j0 < dy;
  int pi, pj;
  turn_pix(min(i0, dx - 1), min(j0, dy - 1), OS == 2 ? 2 * rot : rot, nx, ny, pi, pj);
  double acc[NS];
#pragma unroll
  for (int s = 0; s < NS; ++s) acc[s] = 0.0;
  for (int gb = rank; gb < A.ngroups; gb += kBatch * S) {
    const int cnt = min(kBatch, (A.ngroups - gb + S - 1) / S);
    __syncthreads();
    for (int t = threadIdx.x; t < cnt * (int)(sizeof(Orbit2D) / 8); t += blockDim.x) {
      const int r = t / (int)(sizeof(Orbit2D) / 8), w = t - r * (int)(sizeof(Orbit2D) / 8);
      reinterpret_cast<double *>(recs + r)[w] = reinterpret_cast<const double *>(A.groups + gb + r * S)[w];
    }
    if constexpr (TABLE) {
      for (int t = threadIdx.x; t < cnt * (int)(sizeof(View2D) / 8); t += blockDim.x) {
        const int r = t / (int)(sizeof(View2D) / 8), w = t - r * (int)(sizeof(View2D) / 8);
        reinterpret_cast<double *>(vrec + r)[w] =
            reinterpret_cast<const double *>(A.views + A.groups[gb + r * S].view[0])[w];
      }
    }
    __syncthreads();
    for (int r = 0; r < cnt; ++r) {
      const Orbit2D &g = recs[r];
      Foot2<MODEL> ft;
      foot2<MODEL>(A, g, vrec + (TABLE ? r : 0), pi, pj, ft);
      int c = max(ft.f, 0);
      if constexpr (TABLE) c = ft.t.lo;
      if (c >= ft.e) continue;
      const float *rowp[NS];
#pragma unroll
      for (int s = 0; s < NS; ++s) rowp[s] = A.in + (long)g.view[s] * nv;
      double sum[NS];
#pragma unroll
      for (int s = 0; s < NS; ++s) sum[s] = 0.0;
      Walk2<MODEL> wk;
      wk.start(A, ft, c);
      for (; c < ft.e; ++c) {
        float y[NS];
#pragma unroll
        for (int s = 0; s < NS; ++s) y[s] = __ldg(rowp[s] + c);
        const double w = wk.weight(A, ft, c);
#pragma unroll
        for (int s = 0; s < NS; ++s) sum[s] = fma(w, (double)y[s], sum[s]);
      }
#pragma unroll
      for (int s = 0; s < NS; ++s) acc[s] = fma(ft.amp, sum[s], acc[s]);
    }
  }
  // member slot s's sum at position p belongs to pixel R^-t(p)
#pragma unroll
  for (int s = 0; s < NS; ++s) ex[s][threadIdx.x] = acc[s];
  __syncthreads();
  double tot = 0.0;
#pragma unroll
  for (int s = 0; s < NS; ++s) {
    const int sh = OS == 1 ? 0 : (OS == 2 ? s : slot_turn<CLS>(s));
    tot += ex[s][((rot + sh) % OS) * NO + o];
  }
  float *dst = A.out + ((long)pj * nx + pi);
  if (S == 1) {
    if (valid) *dst += (float)tot;
    return;
  }
  part[threadIdx.x] = tot;
  cg::cluster_group cl = cg::this_cluster();
  cl.sync();
  if (rank == 0) {
    for (int r = 1; r < S; ++r) tot += cl.map_shared_rank(part, r)[threadIdx.x];
    if (valid) *dst += (float)tot;
  }
  cl.sync();
}

template <class K>
cudaError_t launch_split(K kern, dim3 grid, size_t smem, int split, const Orbit2DLaunch &L, cudaStream_t st)
{
  if (smem > 48 * 1024) {
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(32 * kWarps);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)split;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = split > 1 ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kern, L);
}

int slots(int cls) { return cls == C2_QUAD ? 4 : (cls == C2_ONE ? 1 : 2); }
int orbit_size(int cls) { return cls == C2_ONE ? 1 : (cls == C2_HALF ? 2 : 4); }

}  // namespace

cudaError_t launch_fwd2d_orbit(Orbit2DLaunch L, cudaStream_t st)
{
  const int NS = slots(L.cls);
  // tiles of at most 256 (quads) or 512 cells (8 rows of 4 KB per CTA, three
  // CTAs per SM), narrower while even 8 CTAs per tile leave SMs without one;
  // then a cluster shares a tile's lines until there are 8 CTAs per SM
  int tiles = (L.P.nv + (NS == 4 ? 255 : 511)) / (NS == 4 ? 256 : 512);
  while (tiles * L.ngroups * kMaxSplit < 2 * 148 && L.P.nv / (2 * tiles) >= 64) tiles *= 2;
  L.utile = ((L.P.nv + tiles - 1) / tiles + 3) & ~3;
  L.usplit = (L.P.nv + L.utile - 1) / L.utile;
  const int lines = L.P.nx < L.P.ny ? L.P.nx : L.P.ny;
  L.split = 1;
  while (L.split < kMaxSplit && (long)L.usplit * L.ngroups * L.split < 148 * 8 && lines >= 2 * kWarps * L.split)
    L.split *= 2;
  const size_t smem = sizeof(float) * kWarps * (size_t)L.utile * NS +
                      (L.split > 1 ? sizeof(double) * (size_t)L.utile * NS : 0);
  const dim3 grid((unsigned)(L.usplit * L.split), (unsigned)L.ngroups);
#define TRTT_CASE(M, C) \
  if (L.model == M && L.cls == C) return launch_split(k_fwd2d_orbit<M, C>, grid, smem, L.split, L, st);
#define TRTT_MODEL(M) TRTT_CASE(M, C2_ONE) TRTT_CASE(M, C2_HALF) TRTT_CASE(M, C2_QUARTER) TRTT_CASE(M, C2_QUAD)
  TRTT_MODEL(M2_PAR)
  TRTT_MODEL(M2_FAN)
  TRTT_MODEL(M2_LF)
  TRTT_CASE(M2_PAR_TABLE, C2_ONE)
  TRTT_CASE(M2_FAN_TABLE, C2_ONE)
#undef TRTT_MODEL
#undef TRTT_CASE
  return cudaErrorInvalidValue;
}

cudaError_t launch_back2d_orbit(Orbit2DLaunch L, cudaStream_t st)
{
  const int OS = orbit_size(L.cls), NO = 32 * kWarps / OS;
  const int nx = L.P.nx, ny = L.P.ny;
  const int dx = OS == 1 ? nx : (OS == 2 ? ((ny & 1) ? nx / 2 : nx) : nx / 2);
  const int dy = OS == 1 ? ny : (OS == 2 ? ((ny & 1) ? ny : ny / 2) : ny / 2);
  const long blocks = (long)((dx + 15) / 16) * ((dy + NO / 16 - 1) / (NO / 16));
  // few pixels (fewer than 6 CTAs per SM): the CTAs of a cluster share the
  // groups, at least 4 each
  L.split = 1;
  while (L.split < kMaxSplit && blocks * L.split < 148 * 6 && L.ngroups >= 8 * L.split) L.split *= 2;
  const dim3 grid((unsigned)(blocks * L.split));
#define TRTT_CASE(M, C) \
  if (L.model == M && L.cls == C) return launch_split(k_back2d_orbit<M, C>, grid, 0, L.split, L, st);
#define TRTT_MODEL(M) TRTT_CASE(M, C2_ONE) TRTT_CASE(M, C2_HALF) TRTT_CASE(M, C2_QUARTER) TRTT_CASE(M, C2_QUAD)
  TRTT_MODEL(M2_PAR)
  TRTT_MODEL(M2_FAN)
  TRTT_MODEL(M2_LF)
  TRTT_CASE(M2_PAR_TABLE, C2_ONE)
  TRTT_CASE(M2_FAN_TABLE, C2_ONE)
#undef TRTT_MODEL
#undef TRTT_CASE
  return cudaErrorInvalidValue;
}

// ---------------------------------------------------------------------------
// Host: records, eligibility and groups
// ---------------------------------------------------------------------------
namespace {

// Depth of one sign and of usable magnitude at the corners of the pixel grid
// (`pad` pixels beyond its centres), hence over the whole grid.
bool depth_ok(const Orbit2D &g, double nx, double ny, double pad)
{
  double lo = HUGE_VAL, hi = -HUGE_VAL;
  for (int c = 0; c < 4; ++c) {
    const double i = (c & 1) ? nx - 1 + pad : -pad, j = (c & 2) ? ny - 1 + pad : -pad;
    const double d = g.d0 + g.di * i + g.dj * j;
    if (!(std::fabs(d) > 1e-60 && std::fabs(d) < 1e60)) return false;
    lo = std::fmin(lo, d);
    hi = std::fmax(hi, d);
  }
  // the nearest pixel at least a thousandth of the farthest one's depth away
  return lo * hi > 0.0 && std::fmin(std::fabs(lo), std::fabs(hi)) > 1e-3 * std::fmax(std::fabs(lo), std::fabs(hi));
}

double pos_at(const Orbit2D &g, double i, double j)
{
  return (g.n0 + g.ni * i + g.nj * j) / (g.d0 + g.di * i + g.dj * j) + g.c;
}

// Line axis and lane stride: the axis on which neighbouring pixels project
// further apart, lanes at least 1.02 cells apart at the grid's corners (the
// kernel checks every step).
void set_lines(Orbit2D &g, int nx, int ny)
{
  double sp[2] = {HUGE_VAL, HUGE_VAL};
  for (int c = 0; c < 4; ++c) {
    const double i = (c & 1) ? nx - 1 : 0, j = (c & 2) ? ny - 1 : 0;
    const double D = g.d0 + g.di * i + g.dj * j, p = pos_at(g, i, j) - g.c;
    sp[0] = std::fmin(sp[0], std::fabs((g.ni - p * g.di) / D));
    sp[1] = std::fmin(sp[1], std::fabs((g.nj - p * g.dj) / D));
  }
  g.axis = sp[1] > sp[0] ? 1 : 0;
  const double s = sp[g.axis];
  const double q = s > 0.02 ? std::ceil(1.02 / s) : 64.0;
  g.lane_stride = (int)std::fmin(std::fmax(q, 1.0), 64.0);
}

// All views in groups of one class, or false.
bool group_class(int cls, long nx, long ny, long nviews, const double *x12, const double *s12,
                 std::vector<int> &mem)
{
  const int NS = slots(cls);
  if (nviews % NS) return false;
  if (cls == C2_HALF ? (nx % 2 && ny % 2) : (nx != ny || nx % 2)) return false;
  std::vector<char> used(nviews, 0);
  const double tol = 1e-10;
  auto find = [&](const double *coefs, const double *xd, long self, long hint) -> long {
    auto fits = [&](long b) {
      return !used[b] && coefs_match(x12 + 12 * b, coefs, tol) && coefs_match(s12 + 12 * b, xd, tol);
    };
    // the m-turn image lies m / 4 of the scan ahead or behind
    if (fits(hint % nviews)) return hint % nviews;
    const long back = ((nviews - hint % nviews) + 2 * self) % nviews;
    if (fits(back)) return back;
    for (long b = 0; b < nviews; ++b)
      if (fits(b)) return b;
    return -1;
  };
  mem.clear();
  for (long a = 0; a < nviews; ++a) {
    if (used[a]) continue;
    used[a] = 1;
    int m[4] = {(int)a, -1, -1, -1};
    for (int s = 1; s < NS; ++s) {
      double t[12];
      const int turn = cls == C2_HALF ? 2 * s : s;
      turn_xos(x12 + 12 * a, turn, nx, ny, t);
      long b = find(t, s12 + 12 * a, a, a + s * (nviews / NS));
      if (b < 0 && cls == C2_QUARTER) {  // a is the quarter-turn image of b
        turn_xos(x12 + 12 * a, 3, nx, ny, t);
        b = find(t, s12 + 12 * a, a, a + nviews / NS);
        if (b >= 0) m[0] = (int)b;
      }
      if (b < 0) return false;
      used[b] = 1;
      m[s] = m[0] == b ? (int)a : (int)b;
    }
    mem.insert(mem.end(), m, m + 4);
  }
  return true;
}

void finish(Orbit2DScan &out, std::vector<Orbit2D> &recs, long nx, long ny, const double *x12, const double *s12,
            bool group)
{
  const long nviews = (long)recs.size();
  std::vector<int> mem;
  out.cls = C2_ONE;
  if (group && nviews > 1)
    for (int cls : {C2_QUAD, C2_HALF, C2_QUARTER})
      if (group_class(cls, nx, ny, nviews, x12, s12, mem)) {
        out.cls = cls;
        break;
      }
  out.groups.clear();
  if (out.cls == C2_ONE) {
    for (long v = 0; v < nviews; ++v) {
      Orbit2D g = recs[v];
      g.view[0] = (int)v;
      out.groups.push_back(g);
    }
    return;
  }
  for (size_t q = 0; q < mem.size(); q += 4) {
    Orbit2D g = recs[mem[q]];
    for (int s = 0; s < 4; ++s) g.view[s] = mem[q + s];
    out.groups.push_back(g);
  }
}

}  // namespace

bool orbit2d_bspline(const Params2D &P, const View2D *views, long nviews, const double *xos,
                     const double *xsd, Orbit2DScan &out)
{
  if (nviews < 1 || nviews > 65535) return false;
  // the closed form starts each footprint at a zero of the primitive
  if (!P.table && P.hs0 < 2.0) return false;
  if (!(P.hs0 > 0.0 && P.h_init > 0.0)) return false;
  std::vector<Orbit2D> recs(nviews);
  for (long v = 0; v < nviews; ++v) {
    const View2D &V = views[v];
    Orbit2D g;
    std::memset(&g, 0, sizeof(g));
    double hmax;
    if (P.fan) {
      // depth of the source distance wk and of the frame's denominator agree
      // up to the frame's scale (a detector frame that is not turned)
      const double a1 = xsd[12 * v];
      const double s = std::fabs(V.d_x) + std::fabs(V.d_y) + std::fabs(V.d_c);
      if (!(a1 > 0.0) || !(std::fabs(V.d_x - a1 * V.o1) <= 1e-15 * s) ||
          !(std::fabs(V.d_y - a1 * V.o2) <= 1e-15 * s) || !(std::fabs(V.d_c - a1 * V.o4) <= 1e-15 * s))
        return false;
      g.n0 = V.a4m * V.b1o8; g.ni = V.a4m * V.b1o5; g.nj = V.a4m * V.b1o6;
      g.d0 = V.d_c; g.di = V.d_x; g.dj = V.d_y;
      g.c = V.b3;
      if (!depth_ok(g, P.nx, P.ny, 0.0) || !(V.a4m * g.d0 > 0.0) ||
          !(V.a4m * (g.d0 + g.di * (P.nx - 1) + g.dj * (P.ny - 1)) > 0.0))
        return false;
      g.k0 = V.a8;
      g.k1 = a1 * V.a4m;
      g.k2 = P.v_scl * P.v_scl / V.a4sqr;
      g.k3 = 1.0 / (P.h_init * g.k1);
      hmax = 0.0;
      double md = 0.0, dd = 0.0;
      for (int c = 0; c < 4; ++c) {
        const double i = (c & 1) ? P.nx - 1 : 0, j = (c & 2) ? P.ny - 1 : 0;
        const double va = pos_at(g, i, j) - g.k0;
        md = std::fmax(md, std::fabs(g.k1 / (g.d0 + g.di * i + g.dj * j)));
        dd = std::fmax(dd, 1.0 + va * va * g.k2);
      }
      hmax = P.h_init * md * std::sqrt(dd);
    } else {
      g.n0 = V.b1o8b3; g.ni = V.b1o5; g.nj = V.b1o6;
      g.d0 = 1.0;
      g.k1 = P.table ? 0.0 : V.p_scl;
      g.k2 = V.p_rho0;
      g.k3 = V.p_hs;
      hmax = V.p_h;
    }
    g.hsm = P.hs0 * hmax * 1.0001;
    const double probe = g.n0 + g.ni + g.nj + g.d0 + g.di + g.dj + g.c + g.k0 + g.k1 + g.k2 + g.k3;
    if (!std::isfinite(probe) || !(g.hsm < 1e6) || !(hmax > 0.0)) return false;
    for (int c = 0; c < 4; ++c)
      if (!(std::fabs(pos_at(g, (c & 1) ? P.nx - 1 : 0, (c & 2) ? P.ny - 1 : 0)) < 1e9)) return false;
    set_lines(g, P.nx, P.ny);
    recs[v] = g;
  }
  out.model = P.fan ? (P.table ? M2_FAN_TABLE : M2_FAN) : (P.table ? M2_PAR_TABLE : M2_PAR);
  out.line = 0;
  finish(out, recs, P.nx, P.ny, xos, xsd, !P.table);
  return true;
}

bool orbit2d_lf(const LFView *views, long nviews, int line, Orbit2DScan &out)
{
  if (nviews < 1 || nviews > 65535) return false;
  std::vector<Orbit2D> recs(nviews);
  std::vector<double> x12(12 * nviews, 0.0), s12(12 * nviews, 0.0);
  for (long v = 0; v < nviews; ++v) {
    const LFView &L = views[v];
    Orbit2D g;
    std::memset(&g, 0, sizeof(g));
    g.n0 = L.scale * (L.y0 * L.sb + L.x0 * L.cb);
    g.ni = L.scale * L.cb * L.vs;
    g.nj = L.scale * L.sb * L.vs;
    g.d0 = L.sd - (L.y0 * L.cb - L.x0 * L.sb);
    g.di = L.sb * L.vs;
    g.dj = -L.cb * L.vs;
    g.c = L.off;
    g.k0 = L.x0 + L.sd * L.sb;
    g.k1 = L.y0 - L.sd * L.cb;
    g.k2 = L.vs;
    g.k3 = line ? L.vs : L.vs * L.ps;
    if (!(L.vs > 0.0 && L.size > 0.0 && L.size < 1e3) || !depth_ok(g, L.n1, L.n2, 0.5) || !(g.d0 > 0.0)) return false;
    // half width of a pixel's shadow: half its diagonal times the largest
    // slope of the position, plus half a cell
    double dmin = HUGE_VAL, tmax = 0.0;
    for (int c = 0; c < 4; ++c) {
      const double i = (c & 1) ? L.n1 - 0.5 : -0.5, j = (c & 2) ? L.n2 - 0.5 : -0.5;
      const double d = g.d0 + g.di * i + g.dj * j;
      dmin = std::fmin(dmin, d);
      tmax = std::fmax(tmax, std::fabs((g.n0 + g.ni * i + g.nj * j) / d));
    }
    g.hsm = 0.7072 * L.vs * (std::fabs(L.scale) + tmax) / dmin + 0.5 * L.size;
    const double probe = g.n0 + g.ni + g.nj + g.d0 + g.di + g.dj + g.c + g.k0 + g.k1 + g.k3;
    if (!std::isfinite(probe) || !(g.hsm < 1e6) || !(tmax < 1e9) || !(std::fabs(g.c) < 1e9)) return false;
    set_lines(g, L.n1, L.n2);
    recs[v] = g;
    double *x = &x12[12 * v], *s = &s12[12 * v];
    x[0] = g.ni; x[1] = g.nj; x[3] = g.n0;
    x[4] = g.di; x[5] = g.dj; x[7] = g.d0;
    s[0] = g.c;
    s[4] = L.size;
    s[8] = g.k3;
  }
  out.model = M2_LF;
  out.line = line;
  finish(out, recs, views[0].n1, views[0].n2, x12.data(), s12.data(), true);
  return true;
}

}  // namespace trtt
