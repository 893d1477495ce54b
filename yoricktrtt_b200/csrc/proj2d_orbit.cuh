// proj2d_orbit.cuh -- host side of the 2D projector pair over view groups
// (proj2d_orbit.cu): the per-group records, the launch descriptions and the
// test of whether a scan may take that path.
#pragma once

#include <vector>

#include "kernels2d.h"

namespace trtt {

// Footprint models of the group kernels.
enum { M2_PAR = 0, M2_FAN = 1, M2_PAR_TABLE = 2, M2_FAN_TABLE = 3, M2_LF = 4 };

// View groups: every group of a scan has the same members, the views that see
// the grid of the group's first view turned by
//   C2_ONE: -       C2_HALF: 2 quarter turns       C2_QUARTER: 1       C2_QUAD: 1, 2, 3
enum { C2_ONE = 0, C2_HALF = 1, C2_QUARTER = 2, C2_QUAD = 3 };

// One group.  Positions are affine or linear-fractional in the pixel indices:
// p(i, j) = (n0 + ni i + nj j) / (d0 + di i + dj j) + c detector cells.
struct Orbit2D {
  double n0, ni, nj, d0, di, dj, c;
  double k0, k1, k2, k3;  // model constants (proj2d_orbit.cu, foot2)
  double hsm;             // bound of the half support of a footprint, in cells
  int view[4];            // member views by slot
  int axis;               // image lines run along i (0) or j (1)
  int lane_stride;        // pixels between neighbouring lanes of the direct kernel
};

struct Orbit2DScan {
  int model = 0, cls = 0, line = 0;
  std::vector<Orbit2D> groups;
};

// Groups of a B-spline scan (views made by make_view2d from xos, xsd) or a
// Long-Fessler scan.  False: the scan keeps the per-view kernels (a pixel on
// or near the source line, a detector frame that is not a translation).
bool orbit2d_bspline(const Params2D &P, const View2D *views, long nviews, const double *xos,
                     const double *xsd, Orbit2DScan &out);
bool orbit2d_lf(const LFView *views, long nviews, int line, Orbit2DScan &out);

struct Orbit2DLaunch {
  Params2D P;             // nx, ny, nv and the B-spline model (Long-Fessler: sizes only)
  const View2D *views;    // table models: exact footprints (foot2d)
  const Orbit2D *groups;
  int ngroups, model, cls, line;
  int utile, usplit, split;  // direct: cells per tile, tiles; CTAs sharing one tile or pixel block
  const float *in;
  float *out;
};

cudaError_t launch_fwd2d_orbit(Orbit2DLaunch L, cudaStream_t st);
cudaError_t launch_back2d_orbit(Orbit2DLaunch L, cudaStream_t st);

}  // namespace trtt
