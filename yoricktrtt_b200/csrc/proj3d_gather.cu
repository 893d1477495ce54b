// proj3d_gather.cu -- transpose 3D projection of column-factorised views
// (closed-form footprint; tabulated footprint with table3d.cuh), view by view:
// one warp gathers four neighbouring voxel columns (a k range of each) over all
// views.
//
// Per view the warp
//   * builds the four columns' v-collapsed detector profiles Q_g[u] = sum_v
//     w_g(v) y[v][u]: a detector row is loaded once for the four columns, whose
//     row ranges nearly coincide (about 10 rows instead of 4 x 7);
//   * gathers sum_u w(u) Q_g[u] for the voxels, 8 lanes per column: a lane takes
//     pairs of adjacent voxels and walks the union of their footprints two cells
//     at a time, each cell loaded once for both (the walk of the direct kernel,
//     sweep3d.cuh, with the same positions and weights: the pair is an adjoint
//     pair up to FP32 rounding).
// Views accumulate per voxel in registers with Kahan compensation.  Where the
// volume has too few columns for the SMs, the warps of a CTA share the views
// of a column group and add up in shared memory.  Gated scans: the views come
// sorted by gates, and the sums of the current two gates are in registers.
//
// Bound by instruction issue: 76 % of the slots for 90 cone views of 128^3,
// ALU 32 %, FMA 50 %; the detector images stay in L2.  One walk for two voxels
// halves the shared memory loads and a row load serves four columns, against
// one warp per column that walked each voxel for itself.  Measured, before ->
// after: cone 100 x 92 x 75 voxels x 61 views 1.07 -> 0.360 ms, parallel 97^2
// x 83 x 75 views 1.04 -> 0.66 ms, one cone view of 128^3 87 -> 51 us, 128^2
// x 64 x 10 gates x 400 views 9.04 -> 5.10 ms.  View groups keep
// k_back3d_group, whose footprint serves two or four views: at 128^3 x 90
// views 1.35 ms against 1.74 here, and 1.58 with grouped columns in this form;
// at 256^3 x 360 views 35.6 ms against 56.6 with grouped columns in this form.
#include <cuda_runtime.h>

#include <algorithm>

#include "sweep3d.cuh"

namespace trtt {

namespace {

constexpr int kH = 8, kNC = 4;    // lanes per column, columns per warp
constexpr int kTabRows = 32;      // detector rows per weight table

struct GatherCol {
  long long A, B;             // 32.32 position of voxel 0 and step per voxel
  float h, rho, inv_den;
  float vstart, vinc;
  int lo, n;                  // detector rows
  int c0, c1;                 // cells that the k range may touch, within the detector
  int steps;
  int view;                   // -1: nothing to gather
  int pad_;
};

// Shared memory of one warp: records, weight table, four profile rows of
// `cap` cells with zeros before and after them, a GatherRest.
__host__ __device__ constexpr size_t gather_row(int cap) { return (size_t)((cap + 2 * kSweepGuard + 3) & ~3); }
template <int MODEL> struct GatherRec {
  using T = GatherCol;
  static constexpr int warps = 8;          // per CTA
  static constexpr int batch = 32 / kNC;   // views whose column records are built together
};
template <> struct GatherRec<MODEL_TABLE> {
  using T = TableCol;
  static constexpr int warps = 24;
  static constexpr int batch = 16 / kNC;
};
template <int MODEL> __host__ __device__ constexpr size_t gather_warp_bytes(int cap)
{
  return GatherRec<MODEL>::batch * kNC * sizeof(typename GatherRec<MODEL>::T) + sizeof(float2) * kTabRows * kNC +
         sizeof(float) * kNC * gather_row(cap) + 32;
}

template <int GEOM>
__device__ __forceinline__ void gather_record(const Params3D &P, const View3D &V, int i, int j, int k0, int k1,
                                              GatherCol &r, int *__restrict__ err)
{
  r.view = -1;
  r.lo = 0;
  r.n = 0;
  r.c0 = INT_MAX;
  r.c1 = INT_MIN;
  r.steps = 0;
  ColGeo<MODEL_CUBIC> c;
  column_geo<GEOM, MODEL_CUBIC>(P, V, i, j, 0, c);
  if (c.bad) atomicOr(err, TRTT_ERR_SOURCE_PLANE);
  if (c.bad || c.vax.n <= 0) return;
  const double ua = fma(c.B, (double)k0, c.A), ub = fma(c.B, (double)(k1 - 1), c.A);
  double hsm;
  if constexpr (GEOM == GEOM_CONE) {
    const double um = fmax(fabs(ua - V.a12), fabs(ub - V.a12)) * P.u_scl;
    hsm = P.hs0 * (double)c.h_u0m * sqrt(1.0 + um * um * (double)c.inv_den) * 1.0001;
  } else {
    hsm = V.p_hs_u;
  }
  const double lo = fmin(ua, ub) - hsm - 1.0, hi = fmax(ua, ub) + hsm + 2.0;
  if (!(hi > 0.0 && lo < (double)P.nu)) return;
  r.c0 = (int)fmax(lo, 0.0);
  r.c1 = (int)fmin(hi, (double)P.nu);
  if (r.c0 >= r.c1) {
    r.c0 = INT_MAX;
    r.c1 = INT_MIN;
    return;
  }
  // + 2^8: the 23-bit fraction taken from the low word is then rounded
  r.A = __double2ll_rn(c.A * 4294967296.0) + 256;
  r.B = __double2ll_rn(c.B * 4294967296.0);
  r.h = c.h_u0m;
  r.rho = c.rho0c;
  r.inv_den = c.inv_den;
  r.vstart = c.vax.start;
  r.vinc = c.vax.inc;
  r.lo = c.vax.lo;
  r.n = c.vax.n;
  r.steps = ((int)(2.0 * hsm + fabs(c.B)) + 3) >> 1;
  r.view = 0;
}

// The same of the tabulated footprint.
template <int GEOM>
__device__ __forceinline__ void gather_record(const Params3D &P, const View3D &V, int i, int j, int k0, int k1,
                                              TableCol &r, int *__restrict__ err)
{
  double A, B, hsm, sp;
  if (!table_column<GEOM>(P, V, i, j, r, A, B, hsm, sp, err)) {
    r.n = 0;
    return;
  }
  const double ua = fma(B, (double)k0, A), ub = fma(B, (double)(k1 - 1), A);
  const double lo = fmin(ua, ub) - hsm - 1.0, hi = fmax(ua, ub) + hsm + 2.0;
  if (!(hi > 0.0 && lo < (double)P.nu)) return;
  const int c0 = (int)fmax(lo, 0.0), c1 = (int)fmin(hi, (double)P.nu);
  if (c0 >= c1) return;
  r.c0 = c0;
  r.c1 = c1;
  r.view = 0;
}

// acc += term, compensated.
__device__ __forceinline__ void kahan(float &acc, float &cmp, float term)
{
  const float y = term - cmp, t = acc + y;
  cmp = (t - acc) - y;
  acc = t;
}

// What a warp with a sum that is not finite has left: the sums of the gates g[0]
// and g[1] from the views start[0] and start[1] (in the order taken) on, and all
// from view `next` on.
struct GatherRest {
  int start[2], g[2], next;
};

// The terms that a warp has left, each over its voxel's own rows and cells alone,
// into the volume.  (A column's profile takes its neighbours' rows with weights of
// 0, and a walk the cells of the voxel beside its own: one detector cell there that
// is not finite spoils a voxel's sum.)  Voxel by voxel and view by view in FP64
// sums, far slower than the kernel (61 irregular views with one NaN cell each, which
// most warps meet, 0.43 -> 5.8 ms; with all cells NaN 6.1), after the kernel's loops,
// so that nothing of it is alive in them (marked and mended view by view it cost 3 to
// 4% of every transpose, here 0 to 2.6%); no call with finite data comes here.
template <int GEOM, int PP, bool GATED, int MODEL>
__device__ __noinline__ void gather_rest(const GatherLaunch &A, const GatherRest &R, int i, int j, int pb, int first,
                                         int step)
{
  const Params3D &P = A.P;
  const int lig = threadIdx.x & (kH - 1), nview = A.order ? A.norder : A.view_hi - A.view_lo;
  if (i >= P.nx) return;
  for (int e = 0; e < 2 * PP; ++e) {
    const int k = 2 * pb + (MODEL == MODEL_TABLE ? lig + kH * e : 2 * (lig + kH * (e >> 1)) + (e & 1));
    if (k >= P.nz) continue;
    float *dst = A.vol + ((long)j * P.nx + i) * P.nz + k;
    double sum[2] = {0.0, 0.0};
    int g[2] = {GATED ? -1 : 0, -1};
    for (int n = first; n < nview; ++n) {
      if ((n - first) % step >= GatherRec<MODEL>::batch) continue;  // another warp's batch
      const int view = A.order ? A.order[n] : A.view_lo + n;
      if (view < A.view_lo || view >= A.view_hi) continue;
      const View3D &V = A.views[view];
      ColGeo<MODEL> c;
      typename AxisOf<MODEL>::type ax;
      float rho, s = 0.f;
      column_geo<GEOM, MODEL>(P, V, i, j, 0, c);
      if (c.bad || c.vax.n <= 0 || !voxel_u<GEOM, MODEL>(P, V, c, k, ax, rho)) continue;
      const float *img = A.sino + (long)(view - A.view_lo) * A.sino_view_stride + (long)c.vax.lo * P.nu + ax.lo;
      for (int l = 0; l < ax.n; ++l) {
        const float w = axis_weight<MODEL>(ax, l, P);
        if (w == 0.f) continue;
        float q = 0.f;
        for (int m = 0; m < c.vax.n; ++m) {
          const float wv = axis_weight<MODEL>(c.vax, m, P);
          if (wv != 0.f) q = fmaf(wv, __ldg(img + (long)m * P.nu + l), q);
        }
        s = fmaf(w, q, s);
      }
      if (!GATED) {
        sum[0] += (double)(rho * s);
        continue;
      }
      const GatePair gp = A.pairs[view];
      for (int h = 0; h < 2; ++h) {
        const int to = h ? gp.g1 : gp.g0;
        if (to < 0) continue;
        if (n < R.next && !(to == R.g[0] && n >= R.start[0]) && !(to == R.g[1] && n >= R.start[1])) continue;
        const int a = to == g[0] ? 0 : (to == g[1] ? 1 : h);
        if (to != g[a]) {
          if (g[a] >= 0) dst[(long)g[a] * A.gate_stride] += (float)sum[a];
          g[a] = to;
          sum[a] = 0.0;
        }
        sum[a] += (double)((h ? gp.w1 : gp.w0) * (rho * s));
      }
    }
    for (int a = 0; a < 2; ++a)  // (ungated: other warps may add to the voxel)
      if (g[a] >= 0) atomicAdd(dst + (long)g[a] * A.gate_stride, (float)sum[a]);
  }
}

template <int GEOM, int PP, bool GATED, int MODEL>
__global__ void __launch_bounds__(32 * GatherRec<MODEL>::warps, MODEL == MODEL_TABLE ? 1 : (GATED || PP > 3 ? 2 : 3))
k_back3d_gather(const __grid_constant__ GatherLaunch A)
{
  extern __shared__ __align__(16) unsigned char smem_all[];
  using Rec = typename GatherRec<MODEL>::T;
  constexpr int kWarps = GatherRec<MODEL>::warps, kBatch = GatherRec<MODEL>::batch;
  TableSh T{};
  unsigned char *smem = smem_all;
  if constexpr (MODEL == MODEL_TABLE) {
    table_load(A.P, reinterpret_cast<double *>(smem_all), T);
    smem += table_bytes(A.P);
    __syncthreads();
  }
  constexpr int NA = GATED ? 2 : 1;  // sums per voxel: the current gates
  const Params3D &P = A.P;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, grp = lane / kH, lig = lane & (kH - 1);
  const int nx = P.nx, ny = P.ny, nz = P.nz, nu = P.nu;
  const int vs = warp % A.vsplit, cgi = blockIdx.x * (kWarps / A.vsplit) + warp / A.vsplit;
  const int ngx = (nx + kNC - 1) / kNC;
  const bool active = cgi < ngx * ny;
  const int i0 = (cgi % ngx) * kNC, j = min(cgi / ngx, ny - 1);
  const int col_i = i0 + grp;
  const int pb = blockIdx.y * (kH * PP);
  const int k0 = 2 * pb, k1 = min(k0 + 2 * kH * PP, nz);
  const size_t wb = gather_warp_bytes<MODEL>(A.cap);
  const int qrow = (int)gather_row(A.cap);
  Rec *recs = reinterpret_cast<Rec *>(smem + warp * wb);
  float2 *wtab = reinterpret_cast<float2 *>(recs + kBatch * kNC);
  float *Q = reinterpret_cast<float *>(wtab + kTabRows * kNC);
  GatherRest &rest = *reinterpret_cast<GatherRest *>(Q + kNC * qrow);
  for (int t = lane; t < kNC * qrow; t += 32) Q[t] = 0.f;
  __syncwarp();
  float acc[NA][PP][2], cmp[NA][PP][2];
#pragma unroll
  for (int a = 0; a < NA; ++a)
#pragma unroll
    for (int i = 0; i < PP; ++i)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        acc[a][i][e] = 0.f;
        cmp[a][i][e] = 0.f;
      }
  int ga = -1, gb = -1;  // gates of the sums
  // sum `a` into gate `g`, cleared
  auto flush = [&](int a, int g) {
    if (g >= 0 && active && col_i < nx) {
      float *dst = A.vol + (long)g * A.gate_stride + ((long)j * nx + col_i) * nz;
#pragma unroll
      for (int i = 0; i < PP; ++i) {
        // the lane's voxels: pairs of neighbours, or (table) every kH-th
        const int k = MODEL == MODEL_TABLE ? k0 + lig + 2 * kH * i : 2 * (pb + lig + kH * i);
        const int k2 = MODEL == MODEL_TABLE ? k + kH : k + 1;
        if (k < nz) dst[k] += acc[a][i][0] - cmp[a][i][0];
        if (k2 < nz) dst[k2] += acc[a][i][1] - cmp[a][i][1];
      }
    }
#pragma unroll
    for (int i = 0; i < PP; ++i)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        acc[a][i][e] = 0.f;
        cmp[a][i][e] = 0.f;
      }
  };
  // some sum of the warp is not finite
  auto spoiled = [&]() {
    float m = 0.f;
#pragma unroll
    for (int a = 0; a < NA; ++a)
#pragma unroll
      for (int i = 0; i < PP; ++i) m += fabsf(acc[a][i][0]) + fabsf(acc[a][i][1]);
    return __any_sync(FULLM, !is_finite(m));
  };
  bool left = false;
  if (GATED && lane == 0) rest = GatherRest{{0, 0}, {-1, -1}, INT_MAX};  // (lane 0 alone writes it)
  const int nview = active ? (A.order ? A.norder : A.view_hi - A.view_lo) : 0;
  const int vstep = kBatch * A.vsplit;
  for (int vb = vs * kBatch; vb < nview && !left; vb += vstep) {
    // ---- records of kBatch views x kNC columns ---------------------------
    {
      const int n = vb + lane / kNC, ci = i0 + lane % kNC;
      Rec r;
      r.view = -1;
      r.n = 0;
      r.c0 = INT_MAX;
      r.c1 = INT_MIN;
      r.lo = 0;
      if constexpr (MODEL == MODEL_CUBIC) r.steps = 0;
      if (n < nview && ci < nx && lane < kBatch * kNC) {
        const int v = A.order ? A.order[n] : A.view_lo + n;
        if (v >= A.view_lo && v < A.view_hi) {
          gather_record<GEOM>(P, A.views[v], ci, j, k0, k1, r, A.err);
          if (r.view >= 0) r.view = v;
        }
      }
      __syncwarp();
      if (lane < kBatch * kNC) recs[lane] = r;
      __syncwarp();
    }
    const int cnt = min(kBatch, nview - vb);
#pragma unroll 1
    for (int b = 0; b < cnt; ++b) {
      const Rec &r = recs[b * kNC + grp];
      const bool on = r.view >= 0;
      const int view = __reduce_max_sync(FULLM, r.view);
      if (view < 0) continue;
      const int r0 = __reduce_min_sync(FULLM, on ? r.lo : INT_MAX);
      const int r1 = __reduce_max_sync(FULLM, on ? r.lo + r.n : INT_MIN);
      int c0 = __reduce_min_sync(FULLM, r.c0) & ~3, c1 = __reduce_max_sync(FULLM, r.c1);
      if (A.vec4) c1 = (c1 + 3) & ~3;
      if (c1 - c0 > A.cap) {  // more cells than the launcher's bound: never in a correct run
        if (lane == 0) atomicOr(A.err, TRTT_ERR_BAD_INDEX);
        c1 = c0 + A.cap;
      }
      float wa = 1.f, wbv = 0.f;
      bool two = false;
      if (GATED) {
        const GatePair gp = A.pairs[view];
        wa = gp.w0;
        wbv = gp.w1;
        two = gp.g1 >= 0;
        if (gp.g0 != ga || (gp.g1 >= 0 && gp.g1 != gb)) {
          if (spoiled()) {
            left = true;
            if (lane == 0) rest.next = vb + b;
            break;
          }
          if (gp.g0 == gb) {  // the second gate becomes the first
            flush(0, ga);
#pragma unroll
            for (int i = 0; i < PP; ++i)
#pragma unroll
              for (int e = 0; e < 2; ++e) {
                acc[0][i][e] = acc[NA - 1][i][e];
                cmp[0][i][e] = cmp[NA - 1][i][e];
                acc[NA - 1][i][e] = 0.f;
                cmp[NA - 1][i][e] = 0.f;
              }
          } else {
            if (gp.g0 != ga) flush(0, ga);
            flush(NA - 1, gb);
          }
          // (slot 1 starts anew in every case; a gate that moves to slot 0 keeps its start)
          if (lane == 0) {
            if (gp.g0 != ga) rest.start[0] = gp.g0 == gb ? rest.start[1] : vb + b;
            rest.start[1] = vb + b;
            rest.g[0] = gp.g0;
            rest.g[1] = gp.g1;
          }
          ga = gp.g0;
          gb = gp.g1;
        }
      }
      // ---- v-collapsed profiles of the four columns ------------------------
      const float *img = A.sino + (long)(view - A.view_lo) * A.sino_view_stride;
      for (int rb = r0; rb < r1; rb += kTabRows) {
        const int nr = min(kTabRows, r1 - rb);
        for (int e = lane; e < nr * kNC; e += 32) {
          const Rec &o = recs[b * kNC + e % kNC];
          const int l = rb + e / kNC - o.lo;
          float w = 0.f;
          if (o.view >= 0 && l >= 0 && l < o.n) {
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
        for (int ub = c0; ub < c1; ub += 128) {
          float2 q[kNC][2];
#pragma unroll
          for (int g = 0; g < kNC; ++g) q[g][0] = q[g][1] = f2(0.f);
          if (A.vec4) {
            const int u = ub + 4 * lane;
            if (rb > r0 && u < c1) {
#pragma unroll
              for (int g = 0; g < kNC; ++g) {
                const float4 o = *reinterpret_cast<const float4 *>(Q + g * qrow + kSweepGuard + (u - c0));
                q[g][0] = make_float2(o.x, o.y);
                q[g][1] = make_float2(o.z, o.w);
              }
            }
            const float *src = img + (long)rb * nu + u;
#pragma unroll 4
            for (int m = 0; m < nr; ++m) {
              const float4 y = u < c1 ? __ldg(reinterpret_cast<const float4 *>(src + (long)m * nu))
                                      : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
              for (int g = 0; g < kNC; ++g) {
                const float2 w = wtab[m * kNC + g];
                q[g][0] = fma2(w, make_float2(y.x, y.y), q[g][0]);
                q[g][1] = fma2(w, make_float2(y.z, y.w), q[g][1]);
              }
            }
            if (u < c1) {
#pragma unroll
              for (int g = 0; g < kNC; ++g)
                *reinterpret_cast<float4 *>(Q + g * qrow + kSweepGuard + (u - c0)) =
                    make_float4(q[g][0].x, q[g][0].y, q[g][1].x, q[g][1].y);
            }
          } else {
            const int u = ub + lane;
            const bool o0 = u < c1, o1 = u + 32 < c1, o2 = u + 64 < c1, o3 = u + 96 < c1;
            if (rb > r0) {
#pragma unroll
              for (int g = 0; g < kNC; ++g) {
                const float *o = Q + g * qrow + kSweepGuard + (u - c0);
                q[g][0] = make_float2(o0 ? o[0] : 0.f, o1 ? o[32] : 0.f);
                q[g][1] = make_float2(o2 ? o[64] : 0.f, o3 ? o[96] : 0.f);
              }
            }
            const float *src = img + (long)rb * nu + u;
#pragma unroll 4
            for (int m = 0; m < nr; ++m) {
              const float *s = src + (long)m * nu;
              const float2 y0 = make_float2(o0 ? __ldg(s) : 0.f, o1 ? __ldg(s + 32) : 0.f);
              const float2 y1 = make_float2(o2 ? __ldg(s + 64) : 0.f, o3 ? __ldg(s + 96) : 0.f);
#pragma unroll
              for (int g = 0; g < kNC; ++g) {
                const float2 w = wtab[m * kNC + g];
                q[g][0] = fma2(w, y0, q[g][0]);
                q[g][1] = fma2(w, y1, q[g][1]);
              }
            }
#pragma unroll
            for (int g = 0; g < kNC; ++g) {
              float *o = Q + g * qrow + kSweepGuard + (u - c0);
              if (o0) o[0] = q[g][0].x;
              if (o1) o[32] = q[g][0].y;
              if (o2) o[64] = q[g][1].x;
              if (o3) o[96] = q[g][1].y;
            }
          }
        }
        __syncwarp();
      }
      // zeros behind the last cell (a walk may run past it)
      if (lane < kSweepGuard) {
#pragma unroll
        for (int g = 0; g < kNC; ++g) Q[g * qrow + kSweepGuard + (c1 - c0) + lane] = 0.f;
      }
      __syncwarp();
      // ---- gather ----------------------------------------------------------
      auto add = [&](int i, float te, float to) {
        if (GATED) {
          kahan(acc[0][i][0], cmp[0][i][0], wa * te);
          kahan(acc[0][i][1], cmp[0][i][1], wa * to);
          kahan(acc[NA - 1][i][0], cmp[NA - 1][i][0], two ? wbv * te : 0.f);
          kahan(acc[NA - 1][i][1], cmp[NA - 1][i][1], two ? wbv * to : 0.f);
        } else {
          kahan(acc[0][i][0], cmp[0][i][0], te);
          kahan(acc[0][i][1], cmp[0][i][1], to);
        }
      };
      if constexpr (MODEL == MODEL_TABLE) {
        const float *row = Q + grp * qrow + kSweepGuard;
        const View3D &V = A.views[view];
#pragma unroll
        for (int i = 0; i < PP; ++i) {
          // two voxels at a time: their chains of FP64 operations overlap
          TableVox v, w;
          table_voxel<GEOM>(P, V, T, r, table_kc<GEOM>(V, k0 + lig + kH * 2 * i), c0, c1, v);
          table_voxel<GEOM>(P, V, T, r, table_kc<GEOM>(V, k0 + lig + kH * (2 * i + 1)), c0, c1, w);
          if (!on) v.n = w.n = 0;
          const int steps = (__reduce_max_sync(FULLM, max(v.n > 0 ? v.s + v.n : 0, w.n > 0 ? w.s + w.n : 0)) + 1) & ~1;
          // walks that touch no cell go over the zeros in front; walks that would
          // leave the guards (none where a footprint fits them) only load their cells
          int rv = v.n > 0 ? v.f - c0 : -kSweepGuard, rw = w.n > 0 ? w.f - c0 : -kSweepGuard;
          const int rmax = c1 - c0 + kSweepGuard - steps;
          const bool safe = __all_sync(FULLM, min(rv, rw) >= -kSweepGuard && max(rv, rw) <= rmax);
          double lv = (double)(-v.l0), ev = table_at(T, dadd(v.start, dmul(lv, v.inc)));
          double lw = (double)(-w.l0), ew = table_at(T, dadd(w.start, dmul(lw, w.inc)));
          float sv = 0.f, sw = 0.f;
          const float *cv = row + rv, *cw = row + rw;
          if (safe) {
            int tv = -v.s, tw = -w.s;
#pragma unroll 1
            for (int t = 0; t < steps; t += 2) {
              const double v1 = table_at(T, dadd(v.start, dmul(lv + 1.0, v.inc)));
              const double w1 = table_at(T, dadd(w.start, dmul(lw + 1.0, w.inc)));
              lv += 2.0;
              lw += 2.0;
              const double v2 = table_at(T, dadd(v.start, dmul(lv, v.inc)));
              const double w2 = table_at(T, dadd(w.start, dmul(lw, w.inc)));
              const float y0 = cv[0], z0 = cw[0], y1 = cv[1], z1 = cw[1];
              if ((unsigned)tv < (unsigned)v.n) sv = fmaf((float)(v1 - ev), y0, sv);
              if ((unsigned)tw < (unsigned)w.n) sw = fmaf((float)(w1 - ew), z0, sw);
              if ((unsigned)(tv + 1) < (unsigned)v.n) sv = fmaf((float)(v2 - v1), y1, sv);
              if ((unsigned)(tw + 1) < (unsigned)w.n) sw = fmaf((float)(w2 - w1), z1, sw);
              ev = v2;
              ew = w2;
              cv += 2;
              cw += 2;
              tv += 2;
              tw += 2;
            }
          } else {
#pragma unroll 1
            for (int t = 0; t < steps; ++t) {
              lv += 1.0;
              lw += 1.0;
              const double v1 = table_at(T, dadd(v.start, dmul(lv, v.inc)));
              const double w1 = table_at(T, dadd(w.start, dmul(lw, w.inc)));
              if ((unsigned)(t - v.s) < (unsigned)v.n) sv = fmaf((float)(v1 - ev), cv[t], sv);
              if ((unsigned)(t - w.s) < (unsigned)w.n) sw = fmaf((float)(w1 - ew), cw[t], sw);
              ev = v1;
              ew = w1;
            }
          }
          add(i, v.n > 0 ? sv * v.rho : 0.f, w.n > 0 ? sw * w.rho : 0.f);
        }
      } else {
        const int steps = __reduce_max_sync(FULLM, r.steps);
        const long long B = r.B, B2 = 2 * B;
        const bool up = B >= 0;
        float h_c = 0.f, rho_c = 0.f, inv_den = 0.f;
        if constexpr (GEOM == GEOM_CONE) {
          h_c = r.h;
          rho_c = on ? r.rho : 0.f;
          inv_den = r.inv_den;
        } else {
          h_c = (float)A.views[view].p_hs_u;
          rho_c = on ? (float)A.views[view].p_rho0 : 0.f;
        }
        const float a12 = (float)A.views[view].a12, pscl = GEOM == GEOM_CONE ? 0.f : (float)A.views[view].p_scl_u;
        long long ue = r.A + B2 * (pb + lig);
        const float *row = Q + grp * qrow + kSweepGuard;
        const int rmax = c1 - c0 + kSweepGuard - 2 * steps;  // last start of a walk
  #pragma unroll
        for (int i = 0; i < PP; ++i) {
          const long long uo = ue + B, ua = up ? ue : uo, uc = up ? uo : ue;
          ue += B2 * kH;
          const int Ia = (int)(ua >> 32), Ic = (int)(uc >> 32);
          const float2 ph = make_float2(__uint_as_float(((unsigned)ua >> 9) | 0x3f800000u) - 1.0f,
                                        __uint_as_float(((unsigned)uc >> 9) | 0x3f800000u) - 1.0f);
          float2 scl, rho;
          float hs;
          if constexpr (GEOM == GEOM_CONE) {
            const float2 uca = mul2(add2(make_float2((float)Ia, (float)Ic), add2(ph, f2(-a12))), f2((float)P.u_scl));
            const float2 du2 = fma2(mul2(uca, uca), f2(inv_den), f2(1.0f));
            const float2 dlt = mul2(du2, make_float2(rsqrt_ftz(du2.x), rsqrt_ftz(du2.y)));
            const float2 h = mul2(dlt, f2(h_c));
            scl = make_float2(rcp_ftz(h.x), rcp_ftz(h.y));
            rho = mul2(dlt, f2(rho_c));
            hs = (float)P.hs0 * h.x;
          } else {
            scl = f2(pscl);
            rho = f2(rho_c);
            hs = h_c;
          }
          const float fm = __fadd_rd(ph.x - hs, 12582912.0f);
          const int f = Ia + (__float_as_int(fm) - 0x4B400000);
          const float2 x1 = mul2(add2(make_float2(fm - 12582911.0f, (float)(f + 1 - Ic)),
                                      make_float2(-ph.x, -ph.y)), scl);
          // a walk that would start before the guard or end behind it touches no
          // cell of the detector: it is moved into the zeros in front
          int rel = f - c0;
          const bool in = on && rel >= -kSweepGuard && rel <= rmax;
          rel = in ? rel : -kSweepGuard;
          const int st = in ? steps : 0;
          const float *cell = row + rel;
          float ax = x1.x, cx = x1.y, pa = -0.5f, pc = -0.5f, sa = 0.f, sc = 0.f;
  #pragma unroll 1
          for (int l = 0; l < st; ++l) {
            const float y0 = cell[0], y1 = cell[1];
            const float ay = ax + scl.x, cy = cx + scl.y;
            const float a1 = cubic_odd(ax), q1 = cubic_odd(cx), a2 = cubic_odd(ay), q2 = cubic_odd(cy);
            sa = fmaf(a2 - a1, y1, fmaf(a1 - pa, y0, sa));
            sc = fmaf(q2 - q1, y1, fmaf(q1 - pc, y0, sc));
            pa = a2;
            pc = q2;
            ax = ay + scl.x;
            cx = cy + scl.y;
            cell += 2;
          }
          const float ta = in ? sa * rho.x : 0.f, tc = in ? sc * rho.y : 0.f;
          const float te = up ? ta : tc, to = up ? tc : ta;
          add(i, te, to);
        }
      }
      __syncwarp();
    }
  }
  left = left || spoiled();
  __syncwarp();
  if (GATED) {
    if (!left) {
      flush(0, ga);
      flush(NA - 1, gb);
    }
  } else if (A.vsplit == 1) {
    if (!left) flush(0, 0);
  } else {
    // the warps of a column group add up: sums and compensations to shared memory
    __syncthreads();
    float2 *part = reinterpret_cast<float2 *>(smem);
#pragma unroll
    for (int i = 0; i < PP; ++i)
#pragma unroll
      for (int e = 0; e < 2; ++e)
        part[(2 * i + e) * (32 * kWarps) + threadIdx.x] =
            left ? f2(0.f) : make_float2(acc[0][i][e], cmp[0][i][e]);
    __syncthreads();
    if (vs == 0) {
#pragma unroll
      for (int i = 0; i < PP; ++i)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          double s = 0.0;
          for (int w = 0; w < A.vsplit; ++w) {
            const float2 p = part[(2 * i + e) * (32 * kWarps) + threadIdx.x + 32 * w];
            s += (double)p.x - (double)p.y;
          }
          acc[0][i][e] = (float)s;
          cmp[0][i][e] = 0.f;
        }
      flush(0, 0);
    }
    __syncthreads();
  }
  if (left && active) gather_rest<GEOM, PP, GATED, MODEL>(A, rest, col_i, j, pb, vs * kBatch, vstep);
}

template <int GEOM, int PP, int MODEL>
cudaError_t launch(GatherLaunch L, cudaStream_t st)
{
  constexpr int kWarps = GatherRec<MODEL>::warps, kBatch = GatherRec<MODEL>::batch;
  const int pairs = (L.P.nz + 1) / 2, chunks = (pairs + kH * PP - 1) / (kH * PP);
  const long groups = (long)((L.P.nx + kNC - 1) / kNC) * L.P.ny;
  // warps that share the views of a column group, each with at least a batch
  L.vsplit = 1;
  if (!L.pairs) {
    const long slots = 148 * (MODEL == MODEL_TABLE ? 1 : (PP > 3 ? 2 : 3));
    double best = 1e300;
    for (int s = 1; s <= 8 && (s == 1 || L.view_hi - L.view_lo >= kBatch * s); s *= 2) {
      // waves of CTAs (and a part for the uneven ends) times the work of each
      const long ctas = (groups * s + kWarps - 1) / kWarps * chunks;
      const double cost = ((double)((ctas + slots - 1) / slots) + 0.3) * (1.0 / s + 0.04);
      if (cost < 0.97 * best) {
        best = cost;
        L.vsplit = s;
      }
    }
  }
  // cells of a k range: its voxels' positions in four neighbouring columns and
  // their half supports
  const double len = L.b.du * 2 * kH * PP + L.b.dcol * (kNC - 1) + 2.0 * L.b.hsu + 16.0;
  L.cap = len < (double)L.P.nu ? (int)len : (L.P.nu + 3) & ~3;
  const size_t smem = table_bytes(L.P) +
                      std::max(kWarps * gather_warp_bytes<MODEL>(L.cap), sizeof(float2) * 2 * PP * 32 * kWarps);
  if (smem > 227 * 1024) return cudaErrorInvalidConfiguration;
  const dim3 grid((unsigned)((groups * L.vsplit + kWarps - 1) / kWarps), (unsigned)chunks);
  auto go = [&](auto kern) {
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    kern<<<grid, 32 * kWarps, smem, st>>>(L);
    return cudaGetLastError();
  };
  return L.pairs ? go(k_back3d_gather<GEOM, PP, true, MODEL>) : go(k_back3d_gather<GEOM, PP, false, MODEL>);
}

// Voxel pairs per lane (at most `most`): the fewest passes over the column's
// pairs; each range of k also builds its own profiles, about a pass's work.
int pairs_per_lane(int nz, int most)
{
  const int pairs = (nz + 1) / 2;
  int best = 1, cost = INT_MAX;
  for (int pp = most; pp >= 1; --pp) {
    const int s = (pairs + kH * pp - 1) / (kH * pp) * (pp + 1);
    if (s < cost) {
      cost = s;
      best = pp;
    }
  }
  return best;
}

template <int GEOM, int MODEL>
cudaError_t launch_geom(const GatherLaunch &L, cudaStream_t st)
{
  // (gated sums of the tabulated footprint: beyond 2 pairs the registers spill)
  switch (pairs_per_lane(L.P.nz, MODEL == MODEL_TABLE && L.pairs ? 2 : 5)) {
    case 1: return launch<GEOM, 1, MODEL>(L, st);
    case 2: return launch<GEOM, 2, MODEL>(L, st);
    case 3: return launch<GEOM, 3, MODEL>(L, st);
    case 4: return launch<GEOM, 4, MODEL>(L, st);
    default: return launch<GEOM, 5, MODEL>(L, st);
  }
}

}  // namespace

bool gather_fits(const Params3D &P, const SweepBounds &b)
{
  const double len = b.du * 2 * kH * pairs_per_lane(P.nz, 5) + b.dcol * (kNC - 1) + 2.0 * b.hsu + 16.0;
  const int cap = len < (double)P.nu ? (int)len : (P.nu + 3) & ~3;
  if (P.model == MODEL_TABLE)
    return b.rows > 0 && table_slots(P) <= kTableSlots && (P.nz + 1) / 2 / kH < 65535 &&
           table_bytes(P) + GatherRec<MODEL_TABLE>::warps * gather_warp_bytes<MODEL_TABLE>(cap) <= 227 * 1024;
  // (the last test: a walk over two voxels' cells fits the zeros beside a profile,
  // voxels of up to about 2.4 cells on the detector; 60 views of 64^3, voxels of 2.33
  // cells 0.45 ms, of 2.47 cells 0.61 in the column kernel)
  return b.rows > 0 && GatherRec<MODEL_CUBIC>::warps * gather_warp_bytes<MODEL_CUBIC>(cap) <= 113 * 1024 &&
         (P.nz + 1) / 2 / kH < 65535 && 2.0 * b.hsu + b.du + 4.0 < 2.0 * kSweepGuard - 16.0;
}

cudaError_t launch_back3d_gather(const GatherLaunch &L, cudaStream_t st)
{
  if (L.view_hi <= L.view_lo) return cudaSuccess;
  if (L.P.model == MODEL_TABLE)
    return L.P.geom == GEOM_CONE ? launch_geom<GEOM_CONE, MODEL_TABLE>(L, st)
                                 : launch_geom<GEOM_PARALLEL, MODEL_TABLE>(L, st);
  return L.P.geom == GEOM_CONE ? launch_geom<GEOM_CONE, MODEL_CUBIC>(L, st)
                               : launch_geom<GEOM_PARALLEL, MODEL_CUBIC>(L, st);
}

}  // namespace trtt
