// proj3d_sweep.cu -- direct 3D projection of column-factorised views: launches
// of the sweep item (sweep3d.cuh) over (view or view group, band of detector
// rows, u tile), the image lines of a tile shared by a cluster of CTAs where
// there are too few tiles for the SMs.
//
// Measured (B200; the band kernel of proj3d_fast.cu, for groups the kernel of
// proj3d_group.cu before):
//   61 irregular cone views, 100 x 92 x 75 -> 151 x 133      1.60 -> 0.50 ms
//   75 parallel views, dense 97 x 97 x 83 -> 129 x 141       2.14 -> 0.81 ms
//   one cone view, 128^3 -> 256^2 (8 CTAs before)            1.48 -> 0.08 ms
//   347 gated cone views, 128 x 128 x 64 -> 256^2 (phantom)  8.0 -> 4.1 ms
//   45 half-turn pairs of views, dense 128^3 -> 256^2        3.03 -> 2.11 ms
//   90 quads of views, 256^3 -> 512^2 (51% zero voxels)      35.8 -> 31.8 ms
// Bounds (ncu): pairs and quads shared-memory wavefronts (66% of peak for the
// pairs: half of them the band rows, the rest the walks, a quarter of those
// bank conflicts) at 60% of the issue slots; single views of 128^3 issue (76% of
// the slots), of smaller volumes the latencies of their walks and of the row locks
// (the 61 irregular views 55%).
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "sweep3d.cuh"

namespace cg = cooperative_groups;

namespace trtt {

namespace {

constexpr int kMaxSplit = 8;    // portable cluster size

template <int GEOM, int G, int Q, int H, int WARPS, int MINB, int MODEL>
__global__ void __launch_bounds__(32 * WARPS, MINB) k_fwd3d_sweep(const __grid_constant__ SweepLaunch A)
{
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ View3D sV;
  __shared__ int s_next, s_odd;
  const Params3D &P = A.P;
  constexpr int US = 64 * Q;  // floats of a band row
  constexpr size_t WB = sweep_warp_bytes<G, Q, H, MODEL>();
  const int warp = threadIdx.x >> 5;
  const int R = A.band_rows, U = A.utile, S = A.split;
  const int tile = blockIdx.x / S, rank = blockIdx.x - tile * S;
  const int bnd = tile / A.usplit, ut = tile - bnd * A.usplit;
  const int v0 = A.b.v0 + bnd * R, v1 = min(v0 + R, A.b.v1), u0 = A.b.u0 + ut * U, u1 = min(u0 + U, A.b.u1);
  constexpr int NC = 32 / H;
  const int rows = sweep_groups(R) * kSweepRows;
  using Rec = typename SweepRec<MODEL>::T;
  TableSh T{};
  unsigned char *base = smem;
  if constexpr (MODEL == MODEL_TABLE) {
    table_load(P, reinterpret_cast<double *>(smem), T);
    base += table_bytes(P);
  }
  float *band = reinterpret_cast<float *>(base);
  unsigned char *mine = base + sizeof(float) * (size_t)rows * US + warp * WB;
  Rec *recs = reinterpret_cast<Rec *>(mine);
  float2 *wtab = reinterpret_cast<float2 *>(mine + SweepRec<MODEL>::batch * sizeof(Rec));
  float *prof = reinterpret_cast<float *>(wtab + kSweepRows * kSweepGroups * NC);
  int *locks = reinterpret_cast<int *>(base + sizeof(float) * (size_t)rows * US + WARPS * WB);
  if (threadIdx.x < (int)(sizeof(View3D) / 8))
    reinterpret_cast<double *>(&sV)[threadIdx.x] =
        reinterpret_cast<const double *>(
            A.views + (A.groups ? A.groups[4 * blockIdx.y] : (int)blockIdx.y))[threadIdx.x];
  if (threadIdx.x == 0) {
    s_next = 0;
    s_odd = 0;
  }
  for (int t = threadIdx.x; t < rows * US; t += blockDim.x) band[t] = 0.f;
  for (int t = threadIdx.x; t < sweep_groups(R) * SweepStrip<Q, H>::NS; t += blockDim.x) locks[t] = 0;
  for (int t = threadIdx.x & 31; t < NC * (US + G * kSweepGuard) + G * kSweepGuard; t += 32) prof[t] = 0.f;
  __syncthreads();
  sweep_item<GEOM, G, Q, H, MODEL>(P, sV, A.vol, A.gate_stride, v0, v1, u0, u1, band, prof, recs, wtab, locks, &s_next,
                                   rank, S, T, &s_odd, A.err);
  __syncthreads();
  if (s_odd) {
    sweep_odd<GEOM, G, Q, H, MODEL>(P, sV, A.vol, A.gate_stride, T, v0, v1, u0, u1, band, prof, locks, rank, S,
                                    A.err);
    __syncthreads();
  }
  const int nrow = v1 - v0, ncell = u1 - u0;
  cg::cluster_group cl = cg::this_cluster();
  if (S > 1) cl.sync();
  // the cluster's bands, added in rank order; each CTA writes its share
#pragma unroll
  for (int m = 0; m < G; ++m) {
    float *out = A.sino + (long)(A.groups ? A.groups[4 * blockIdx.y + m] : (int)blockIdx.y) * A.sino_view_stride;
    for (int t = rank * blockDim.x + threadIdx.x; t < nrow * ncell; t += S * blockDim.x) {
      const int r = t / ncell, u = t - r * ncell, at = r * US + u * G + m;
      float v = 0.f;
      if (S == 1)
        v = band[at];
      else
        for (int k = 0; k < S; ++k) v += cl.map_shared_rank(band, k)[at];
      out[(long)(v0 + r) * P.nu + u0 + u] += v;
    }
  }
  if (S > 1) cl.sync();  // no CTA leaves while another reads its band
}

template <int GEOM, int G, int Q, int H, int WARPS, int MINB, int MODEL = MODEL_CUBIC>
cudaError_t launch(SweepLaunch L, cudaStream_t st)
{
  const long slots = MINB * 148;
  const int nu = L.b.u1 - L.b.u0, nv = L.b.v1 - L.b.v0;
  L.usplit = (nu + 64 * Q / G - 1) / (64 * Q / G);
  L.utile = (nu + L.usplit - 1) / L.usplit;
  // rows per band: what the CTAs of an SM have room for; bands of one height
  const size_t tab = table_bytes(L.P), room = (227 * 1024) / MINB - 1024 - tab;
  int nb = 1, R = nv;
  while (R > 96 || sweep_smem<G, Q, H, MODEL>(R, WARPS) > room) {
    ++nb;
    R = (nv + nb - 1) / nb;
  }
  // few views: lower bands, down to 16 rows, until clusters of 8 CTAs per tile
  // fill the SMs
  while ((long)L.usplit * nb * L.count * kMaxSplit < slots && R >= 32) {
    nb *= 2;
    R = (nv + nb - 1) / nb;
  }
  nb = (nv + R - 1) / R;
  L.band_rows = R;
  // CTAs per tile: the number of waves, rounded up, times the work per CTA
  // (0.02: clearing and adding up the bands)
  const int lines = L.P.nx < L.P.ny ? L.P.nx : L.P.ny;
  const long tiles = (long)L.usplit * nb * L.count;
  double best = 1e300;
  L.split = 1;
  for (int s = 1; s <= kMaxSplit; ++s) {
    if (s > 1 && lines < WARPS * s) break;
    const double cost = (double)((tiles * s + slots - 1) / slots) * (1.0 / s + 0.02);
    if (cost < best * 0.97) {
      best = cost;
      L.split = s;
    }
  }
  const size_t smem = tab + sweep_smem<G, Q, H, MODEL>(R, WARPS);
  auto kern = k_fwd3d_sweep<GEOM, G, Q, H, WARPS, MINB, MODEL>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(L.usplit * nb * L.split), (unsigned)L.count);
  cfg.blockDim = dim3(32 * WARPS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)L.split;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = L.split > 1 ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kern, L);
}

// Shapes <G, pairs of floats per lane and row, lanes per column, warps per CTA,
// CTAs per SM>: the fastest of those measured, by the cells of the tile.  8
// lanes per column keep short columns' lanes busy (75 voxels are 38 pairs: 95%
// of 5 x 8 lanes, 59% of 2 x 32), 16 where the wider rows' profiles would
// leave the SM too few warps.
template <int GEOM>
cudaError_t launch_geom(const SweepLaunch &L, int G, cudaStream_t st)
{
  const int nu = L.b.u1 - L.b.u0, nv = L.b.v1 - L.b.v0;
  if (G == 4) return launch<GEOM, 4, 8, 16, 16, 1>(L, st);
  if (G == 2) return launch<GEOM, 2, 8, 16, 8, 2>(L, st);
  // single views: as few tiles as 256 cells each allow (a column's set-up costs
  // as much as 30 of its voxels), narrower ones for few views
  const int tiles = (nu + 255) / 256;
  int q = ((nu + tiles - 1) / tiles + 63) / 64;
  while (q > 1 && (long)((nu + 64 * q - 1) / (64 * q)) * ((nv + 63) / 64) * L.count * kMaxSplit < 2 * 148) --q;
  if (L.P.model == MODEL_TABLE) {
    // one CTA per SM: each holds the table (40 KB for the cubic's 10001 entries)
    switch (q) {
      case 1: return launch<GEOM, 1, 1, 8, 16, 1, MODEL_TABLE>(L, st);
      case 2: return launch<GEOM, 1, 2, 8, 16, 1, MODEL_TABLE>(L, st);
      case 3: return launch<GEOM, 1, 3, 8, 16, 1, MODEL_TABLE>(L, st);
      default: return launch<GEOM, 1, 4, 8, 16, 1, MODEL_TABLE>(L, st);
    }
  }
  switch (q) {
    case 1: return launch<GEOM, 1, 1, 8, 8, 4>(L, st);
    case 2: return launch<GEOM, 1, 2, 8, 8, 3>(L, st);
    case 3: return launch<GEOM, 1, 3, 8, 12, 2>(L, st);
    default: return launch<GEOM, 1, 4, 16, 12, 2>(L, st);
  }
}

}  // namespace

cudaError_t launch_fwd3d_sweep(const SweepLaunch &L, int G, cudaStream_t st)
{
  if (L.count <= 0 || L.b.u1 <= L.b.u0 || L.b.v1 <= L.b.v0) return cudaSuccess;
  return L.P.geom == GEOM_CONE ? launch_geom<GEOM_CONE>(L, G, st) : launch_geom<GEOM_PARALLEL>(L, G, st);
}

}  // namespace trtt
