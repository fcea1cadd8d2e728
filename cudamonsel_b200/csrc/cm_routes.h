// cm_routes.h -- what the host derives from a scene so that the kernels can take a short route: the inside
// of each shape (FastRegion), the child grids (ChildGrid) and the search guides of the table axes (AxisGuide).  Plain C++ over the
// scene's structs, so that a CPU test can compare the routes with the general searches.
#pragma once
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "cm_device.cuh"

namespace cm {

// The half-spaces and cylinders whose common part lies strictly (by kFastMarginNm or more) inside a shape,
// appended to fp and fc; false when the shape has no such description.  A step with both ends in there
// crosses nothing as the boundary search sees it: its plane solves find u outside (0, 1] by a margin far
// above rounding, and an intersection or a union of shapes (one part of it holding the step) reports none.
// The margin grows with what the searches round: by 1e-14 of the distance of the point a plane or cylinder
// is given by (their dot products round to a few 1e-16 of it), and in a cylinder so that the squared
// distance from the wall, 2 rad m, stays above 1e-14 len^2 (the search takes it as the difference of squares
// of the length, rounded to at most 7e-15 len^2).
static bool inside_of(const std::vector<Shape>& shapes, const std::vector<Plane>& planes, int id,
                      std::vector<FastPlane>& fp, std::vector<FastCyl>& fc) {
  const Shape& sh = shapes[id];
  auto rounding = [](const double* p) { return 1e-14 * (fabs(p[0]) + fabs(p[1]) + fabs(p[2])); };
  // n . p < d, given by a point at
  auto half_space = [&](const double* n, double d, const double* at) {
    const double len = sqrt(n[0] * n[0] + n[1] * n[1] + n[2] * n[2]);
    if (!(len > 0) || !std::isfinite(len) || !std::isfinite(d)) return false;
    fp.push_back(FastPlane{{n[0] / len, n[1] / len, n[2] / len}, d / len - kFastMarginNm - rounding(at)});
    return true;
  };
  switch (sh.kind) {
    case SHAPE_PLANES:
      for (int i = 0; i < sh.np; ++i) {
        const Plane& p = planes[sh.plane0 + i];
        if (!half_space(p.n, p.n[0] * p.p[0] + p.n[1] * p.p[1] + p.n[2] * p.p[2], p.p)) return false;
      }
      return true;
    case SHAPE_INTERSECTION:
      return inside_of(shapes, planes, sh.a, fp, fc) && inside_of(shapes, planes, sh.b, fp, fc);
    case SHAPE_UNION: {
      const size_t np = fp.size(), nc = fc.size();
      if (inside_of(shapes, planes, sh.a, fp, fc) && fc.size() == nc) return true;
      fp.resize(np);
      fc.resize(nc);
      if (inside_of(shapes, planes, sh.b, fp, fc)) return true;
      fp.resize(np);
      fc.resize(nc);
      return false;
    }
    case SHAPE_CYLINDER: {
      // only a cylinder whose axis is normalised is ever struck (see cm_shape_cylinder)
      const double u = sh.nax[0] * sh.nax[0] + sh.nax[1] * sh.nax[1] + sh.nax[2] * sh.nax[2];
      const double rad = sqrt(sh.rad2), m = 1e-3 + 1e-9 * sh.len + 1e-14 * sh.len2 / rad + rounding(sh.e0);
      if (!(fabs(u - 1.0) < 1e-9) || !(rad > 2 * m) || !(sh.len > 4 * m)) return false;
      const double back[3] = {-sh.nax[0], -sh.nax[1], -sh.nax[2]};
      const double a0 = sh.nax[0] * sh.e0[0] + sh.nax[1] * sh.e0[1] + sh.nax[2] * sh.e0[2];
      if (!half_space(sh.nax, a0 + sh.len - m, sh.e0) || !half_space(back, -a0 - m, sh.e0)) return false;
      fc.push_back(FastCyl{{sh.e0[0], sh.e0[1], sh.e0[2]}, {sh.nax[0], sh.nax[1], sh.nax[2]}, (rad - m) * (rad - m)});
      return true;
    }
    default:
      return false;  // spheres: the full form
  }
}

// Whether the steps of a region may take the fast flight: it has no children and its model has mechanisms,
// at most the four the fast flight picks among.  In a region without mechanisms (vacuum) every step ends at
// a boundary, so a fast flight would only hand it on to the next iteration's full flight.
template <typename R> static bool fast_model(const Region& r, const Msm<R>& m) {
  return r.nchild == 0 && m.nmech > 0 && m.nmech <= 4;
}

// The x-y grid over the children of region r, its cells and items appended; false when r has too few children
// with bounded boxes.
static bool child_grid(const std::vector<Region>& regions, const std::vector<int>& children, const Region& r, ChildGrid& g,
                       std::vector<int>& cell_start, std::vector<int>& grid_items) {
  if (r.nchild < kGridMinChildren) return false;
  std::vector<int> bounded, unbounded;
  double lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
  for (int i = 0; i < r.nchild; ++i) {
    const double* bb = regions[children[r.child0 + i]].bb;
    if (std::isinf(bb[0]) || std::isinf(bb[1]) || std::isinf(bb[3]) || std::isinf(bb[4]) || bb[0] > bb[3] ||
        bb[1] > bb[4]) {
      unbounded.push_back(i);
      continue;
    }
    bounded.push_back(i);
    for (int a = 0; a < 3; ++a) {
      lo[a] = std::min(lo[a], bb[a]);
      hi[a] = std::max(hi[a], bb[3 + a]);
    }
  }
  if ((int)bounded.size() < kGridMinChildren) return false;
  const double wx = std::max(hi[0] - lo[0], 1e-3), wy = std::max(hi[1] - lo[1], 1e-3);
  const double cells = std::min(65536.0, std::max(16.0, 2.0 * bounded.size()));
  g.nx = std::max(1, std::min(4096, (int)ceil(sqrt(cells * wx / wy))));
  g.ny = std::max(1, std::min(4096, (int)ceil(cells / g.nx)));
  g.x0 = lo[0];
  g.y0 = lo[1];
  g.dx = wx / g.nx;
  g.dy = wy / g.ny;
  g.z0 = lo[2];
  g.z1 = hi[2];
  std::vector<std::vector<int>> lists((size_t)g.nx * g.ny);
  for (int i : bounded) {  // ascending positions, so every cell list is ascending
    const double* bb = regions[children[r.child0 + i]].bb;
    const int ix0 = std::max(0, (int)floor((bb[0] - g.x0) / g.dx)), ix1 = std::min(g.nx - 1, (int)floor((bb[3] - g.x0) / g.dx));
    const int iy0 = std::max(0, (int)floor((bb[1] - g.y0) / g.dy)), iy1 = std::min(g.ny - 1, (int)floor((bb[4] - g.y0) / g.dy));
    for (int iy = iy0; iy <= iy1; ++iy)
      for (int ix = ix0; ix <= ix1; ++ix) lists[(size_t)iy * g.nx + ix].push_back(i);
  }
  g.cell0 = (int)cell_start.size();
  for (auto& l : lists) {
    cell_start.push_back((int)grid_items.size());
    grid_items.insert(grid_items.end(), l.begin(), l.end());
  }
  cell_start.push_back((int)grid_items.size());
  g.unb0 = (int)grid_items.size();
  g.nunb = (int)unbounded.size();
  grid_items.insert(grid_items.end(), unbounded.begin(), unbounded.end());
  return true;
}

// The search guide of an ascending axis: linear buckets or the leading bits of the argument, whichever
// leaves at most one node in every bucket of at most 4096; kind 0 (bisection) when neither does.
static AxisGuide make_guide(const double* x, int n, std::vector<GuideEntry>& out) {
  AxisGuide g;
  memset(&g, 0, sizeof(g));
  if (n < 4 || n > 60000) return g;
  for (int i = 0; i < n; ++i)
    if (!std::isfinite(x[i]) || (i > 0 && !(x[i] > x[i - 1]))) return g;
  auto bucket = [&](double v) -> int {  // as guide_below does
    if (g.kind == 1) {
      const double t = (v - g.x0) * g.scale;
      return t > 0.0 ? (t < (double)(g.n - 1) ? (int)t : g.n - 1) : 0;
    }
    long long bits;
    memcpy(&bits, &v, 8);
    const int b = ((int)(bits >> 32) >> g.shift) - g.base;
    return b < 0 ? 0 : b > g.n - 1 ? g.n - 1 : b;
  };
  auto fits = [&]() {
    for (int i = 1; i < n; ++i)
      if (bucket(x[i]) == bucket(x[i - 1])) return false;
    return true;
  };
  bool ok = false;
  g.kind = 1;
  g.x0 = x[0];
  for (int per = 1; per <= 8 && !ok; per *= 2) {
    g.n = (n - 1) * per + 1;
    if (g.n > 4096) break;
    g.scale = (double)(g.n - 1) / (x[n - 1] - x[0]);
    ok = std::isfinite(g.scale) && fits();
  }
  if (!ok && x[0] > 0) {
    g.kind = 2;
    for (g.shift = 20; g.shift >= 10 && !ok; --g.shift) {
      long long b0, b1;
      memcpy(&b0, &x[0], 8);
      memcpy(&b1, &x[n - 1], 8);
      g.base = (int)(b0 >> 32) >> g.shift;
      const long long cells = (((long long)(int)(b1 >> 32)) >> g.shift) - g.base + 1;
      if (cells > 4096) break;
      g.n = (int)cells;
      if ((ok = fits())) break;
    }
  }
  if (!ok) {
    memset(&g, 0, sizeof(g));
    return g;
  }
  // the order-3 window of an argument with k nodes below it, from the reference's own search
  auto first3 = [&](int k) {
    const double v = k == n ? INFINITY : x[k];  // has exactly k nodes below it
    int first, nearest;
    nu_locate<double>(v, x, n, 3, first, nearest);
    return (unsigned short)first;
  };
  g.off = (int)out.size();
  int k = 0;
  for (int b = 0; b < g.n; ++b) {
    while (k < n && bucket(x[k]) < b) ++k;
    out.push_back(GuideEntry{(unsigned short)k, first3(k), first3(std::min(k + 1, n)), 0});
  }
  return g;
}

}  // namespace cm
