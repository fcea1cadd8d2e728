// The short routes against the general searches at the ends of their ranges, on the CPU: the device functions
// compiled as plain C++.  Run with the name of one group of checks.
#define __host__
#define __device__
#define __global__
#define __shared__
#define __forceinline__ inline
#define __noinline__
#define __align__(n) __attribute__((aligned(n)))
#include <cstdio>
#include <cstdlib>
#include <limits>
#include <random>
#include <string>

#include "cm_routes.h"

using namespace cm;

static int failures = 0;
static long checks = 0;
#define CHECK(c, ...) \
  do {                \
    ++checks;         \
    if (!(c) && ++failures <= 10) { printf("line %d: ", __LINE__); printf(__VA_ARGS__); printf("\n"); } \
  } while (0)

// ---- table windows of arguments beyond both ends of an axis, the axis on either side of zero or across it
static void check_axis_ends() {
  const double inf = std::numeric_limits<double>::infinity();
  for (int n : {4, 5, 40})
    for (double end : {-1e300, -1e6, -20.0, -1.0, -0.5, 0.0, 0.5, 20.0, 1e6, std::numeric_limits<double>::max()})
      for (int form = 0; form < 3; ++form) {
        std::vector<double> x(n);
        x[n - 1] = end;
        const double size = fabs(end) > 1 ? fabs(end) : 1.0;
        for (int i = n - 2; i >= 0; --i) {
          const double below = n - 1 - i;
          x[i] = end - size * (form == 0 ? below / 64 : form == 1 ? 1 - pow(1.03, -below) : below * below / 4096);
        }
        std::vector<GuideEntry> e(2);  // entries of another axis before this one's
        const AxisGuide g = make_guide(x.data(), n, e);
        for (double v : {std::nextafter(end, inf), end + 0.01 * size, end + size, end + 100 * size, 0.0, 1.0, inf, end,
                         std::nextafter(x[0], -inf), x[0] - size, -inf}) {
          int first, nearest;
          nu_locate<double>(v, x.data(), n, 3, first, nearest);
          const int got = nu_first3(g, e.data(), v, x.data(), n);
          CHECK(got == first, "%d nodes %.17g..%.17g (guide kind %d): window at %.17g is %d, the search's %d", n, x[0], end,
                g.kind, v, got, first);
        }
      }
}

// ---- the inside of shapes far larger than they are wide, or given by points far away: a step with both ends
// strictly inside is one the boundary search finds no boundary for
struct OneShape {
  std::vector<Shape> shapes;
  std::vector<Plane> planes;
};

static OneShape cylinder(const double* e0, const double* ax, double rad) {
  Shape s;
  memset(&s, 0, sizeof(s));
  s.kind = SHAPE_CYLINDER;
  s.len2 = ax[0] * ax[0] + ax[1] * ax[1] + ax[2] * ax[2];
  s.len = sqrt(s.len2);
  for (int k = 0; k < 3; ++k) {
    s.e0[k] = e0[k];
    s.ax[k] = ax[k];
    s.nax[k] = ax[k] / s.len;
  }
  s.rad2 = rad * rad;
  return OneShape{{s}, {}};
}

// steps from at(a point) to at(another), kept when both ends are strictly inside
template <typename F> static void check_inside(const char* name, const OneShape& sh, F at) {
  std::vector<FastPlane> fp;
  std::vector<FastCyl> fc;
  if (!inside_of(sh.shapes, sh.planes, 0, fp, fc)) return;  // not described: the full flight
  SceneView<double> v;
  memset(&v, 0, sizeof(v));
  v.shapes = sh.shapes.data();
  v.planes = sh.planes.data();
  v.fast_planes = fp.data();
  v.fast_cyls = fc.data();
  const FastRegion f{0, 0, 0, (int)fp.size(), fc.empty() ? -1 : 0, {0, 0, 0}};
  for (int k = 0; k < 200000; ++k) {
    double p0[3], p1[3];
    at(k, p0, p1);
    if (!point_inside(v, f, p0) || !point_inside(v, f, p1)) continue;
    CHECK((shape_contains<double, 0>(v, 0, p0)), "%s: start not contained", name);
    const NV nv = shape_first_normal<double, 0>(v, 0, p0, p1);
    CHECK(!(nv.u <= 1.0), "%s: boundary at u = %.17g", name, nv.u);
  }
}

static void check_far_shapes() {
  std::mt19937_64 r(11);
  std::uniform_real_distribution<double> u(-1.0, 1.0);
  const double dir[2][3] = {{0, 1, 0}, {0.48, 0.6, 0.64}};
  for (double len : {1e3, 1e5, 1e6, 1e7, 1e8, 2e8})
    for (double rad : {0.5, 2.0, 5.0, 100.0, 1e4, 1e6})
      for (const double* n : dir) {
        double e0[3], ax[3], side[2][3];
        for (int a = 0; a < 3; ++a) {
          ax[a] = len * n[a];
          e0[a] = -0.5 * ax[a];
          side[0][a] = a == 0 ? (n[0] > 0 ? 0.8 : 1.0) : a == 1 && n[0] > 0 ? -0.64 : 0.0;
        }
        const double m = sqrt(side[0][0] * side[0][0] + side[0][1] * side[0][1]), dot = side[0][0] * n[0] + side[0][1] * n[1];
        for (int a = 0; a < 3; ++a) side[0][a] = (side[0][a] - dot * n[a]) / m;
        for (int a = 0; a < 3; ++a)
          side[1][a] = n[(a + 1) % 3] * side[0][(a + 2) % 3] - n[(a + 2) % 3] * side[0][(a + 1) % 3];
        const double margin = 1e-3 + 1e-9 * len;
        char name[64];
        snprintf(name, sizeof(name), "cylinder %g x %g", len, rad);
        check_inside(name, cylinder(e0, ax, rad), [&](int k, double* p0, double* p1) {
          const double w0 = 0.5 * len * u(r), w1 = k % 2 ? w0 + 3 * rad * u(r) : 0.5 * len * u(r);
          for (int e = 0; e < 2; ++e) {
            // from the axis to within a few margins of the wall
            const double rr = k % 3 ? rad - margin * (1 + 3 * fabs(u(r))) : rad * fabs(u(r)), th = 3.14159265358979 * u(r);
            for (int a = 0; a < 3; ++a)
              (e ? p1 : p0)[a] = n[a] * (e ? w1 : w0) + rr * (cos(th) * side[0][a] + sin(th) * side[1][a]);
          }
        });
      }
  // a slab whose planes are given by points far from it
  for (double far : {0.0, 1e8, 1e9, 1e10, 1e12, 1e14})
    for (int tilted = 0; tilted < 2; ++tilted) {
      const double n[3] = {tilted ? 0.48 : 0.0, tilted ? 0.6 : 0.0, tilted ? 0.64 : 1.0};
      const double t[3] = {tilted ? 0.8 : 1.0, 0.0, tilted ? -0.6 : 0.0};  // along the slab
      OneShape s;
      Shape sh;
      memset(&sh, 0, sizeof(sh));
      sh.kind = SHAPE_PLANES;
      sh.np = 2;
      s.shapes.push_back(sh);
      for (int sg = -1; sg <= 1; sg += 2) {
        Plane P;
        for (int a = 0; a < 3; ++a) {
          P.n[a] = sg * n[a];
          P.p[a] = sg * 10 * n[a] + far * t[a];
        }
        s.planes.push_back(P);
      }
      char name[64];
      snprintf(name, sizeof(name), "slab through points %g away", far);
      check_inside(name, s, [&](int k, double* p0, double* p1) {
        for (int e = 0; e < 2; ++e) {
          const double h = k % 3 ? (10 - 3 * kFastMarginNm * fabs(u(r))) * (u(r) > 0 ? 1 : -1) : 10 * u(r);
          const double x = 1e3 * u(r), off = far * (n[0] * t[0] + n[1] * t[1] + n[2] * t[2]);
          for (int a = 0; a < 3; ++a) (e ? p1 : p0)[a] = n[a] * (h + off) + t[a] * x;
        }
      });
    }
}

// ---- which regions take the fast flight: childless ones whose model has one to four mechanisms
static void check_fast_models() {
  for (int nmech = 0; nmech <= kMaxMech; ++nmech)
    for (int nchild = 0; nchild < 3; ++nchild) {
      Region r;
      Msm<float> m;
      memset(&r, 0, sizeof(r));
      memset(&m, 0, sizeof(m));
      r.nchild = nchild;
      m.nmech = nmech;
      CHECK(fast_model(r, m) == (nchild == 0 && nmech >= 1 && nmech <= 4), "%d mechanisms, %d children", nmech, nchild);
    }
}

// ---- the walk through a child grid
struct GridScene {
  std::vector<Shape> shapes;
  std::vector<Plane> planes;
  std::vector<Region> regions;
  std::vector<int> children, cell_start, grid_items;
  std::vector<ChildGrid> grids;
  SceneView<double> v;

  int region(int parent, const Shape& sh, const double* lo, const double* hi) {
    Region r;
    memset(&r, 0, sizeof(r));
    r.parent = parent;
    r.shape = (int)shapes.size();
    r.grid = -1;
    for (int a = 0; a < 3; ++a) {
      r.bb[a] = lo[a] - 1e-3;
      r.bb[3 + a] = hi[a] + 1e-3;
    }
    shapes.push_back(sh);
    regions.push_back(r);
    return (int)regions.size() - 1;
  }
  GridScene() {  // the chamber
    Shape s;
    memset(&s, 0, sizeof(s));
    s.kind = SHAPE_SPHERE;
    s.r = 1e8;
    const double lo[3] = {-1e8, -1e8, -1e8}, hi[3] = {1e8, 1e8, 1e8};
    region(-1, s, lo, hi);
  }
  void box(const double* lo, const double* hi) {
    Shape s;
    memset(&s, 0, sizeof(s));
    s.kind = SHAPE_PLANES;
    s.plane0 = (int)planes.size();
    s.np = 6;
    for (int a = 0; a < 3; ++a)
      for (int k = 0; k < 2; ++k) {
        Plane P{{0, 0, 0}, {0, 0, 0}};
        P.n[a] = k ? 1 : -1;
        P.p[a] = k ? hi[a] : lo[a];
        planes.push_back(P);
      }
    children.push_back(region(0, s, lo, hi));
  }
  // the chamber's grid; its cells list the children by their boxes
  ChildGrid& finish() {
    regions[0].nchild = (int)children.size();
    ChildGrid g;
    CHECK(child_grid(regions, children, regions[0], g, cell_start, grid_items), "no grid over %zu children", children.size());
    grids.push_back(g);
    regions[0].grid = 0;
    memset(&v, 0, sizeof(v));
    v.shapes = shapes.data();
    v.planes = planes.data();
    v.regions = regions.data();
    v.children = children.data();
    v.grids = grids.data();
    v.cell_start = cell_start.data();
    v.grid_items = grid_items.data();
    return grids[0];
  }
};

static void check_grid_walk() {
  std::mt19937_64 r(29);
  std::uniform_real_distribution<double> u(-1.0, 1.0);
  GridScene s;
  for (int k = 0; k < 90; ++k) {  // boxes of unlike sizes, some of them overlapping, in a layer of 300 nm
    double lo[3], hi[3];
    for (int a = 0; a < 3; ++a) {
      const double c = (a == 2 ? 100 : 500) * u(r), w = (a == 2 ? 50 : 40) * fabs(u(r)) + 0.5;
      lo[a] = c - w;
      hi[a] = c + w;
    }
    s.box(lo, hi);
  }
  const ChildGrid g = s.finish();
  long hits = 0, down = 0;
  for (int k = 0; k < 400000; ++k) {
    double p0[3], d[3];
    for (int a = 0; a < 3; ++a) {
      p0[a] = (a == 2 ? 300 : 600) * u(r);
      d[a] = u(r);
    }
    const double len = k % 4 == 0 ? 2e8 : k % 4 == 1 ? 1000 * fabs(u(r)) : k % 4 == 2 ? 5 * fabs(u(r)) : 300;
    if (k % 5 < 3) d[k % 5] = 0;              // within a plane across an axis
    if (k % 7 < 3) d[(k + 1) % 3] = d[(k + 2) % 3] = 0;  // along an axis
    if (k % 11 == 0) p0[0] = g.x0 + g.dx * (int)(g.nx * fabs(u(r)));  // on a cell's border
    if (k % 13 == 0) p0[2] = k % 2 ? g.z0 : g.z1;             // on the layer's
    double a1[3], b1[3], an[3], bn[3];
    bool ac = false, bc = false;
    for (int a = 0; a < 3; ++a) a1[a] = b1[a] = p0[a] + len * d[a];
    down += d[0] == 0 && d[1] == 0 && d[2] != 0;
    s.regions[0].grid = 0;
    const int ra = find_end_of_step<double, 0>(s.v, 0, p0, a1, an, &ac);
    s.regions[0].grid = -1;
    const int rb = find_end_of_step<double, 0>(s.v, 0, p0, b1, bn, &bc);
    hits += rb > 0;
    CHECK(ra == rb && ac == bc && !memcmp(a1, b1, sizeof(a1)) && (!ac || !memcmp(an, bn, sizeof(an))),
          "step %d from %g %g %g: region %d through the grid, %d by the scan", k, p0[0], p0[1], p0[2], ra, rb);
  }
  CHECK(hits > 10000 && down > 10000, "only %ld hits, %ld steps straight down", hits, down);
}

// a step that stays out of the children's layer visits no cell: a child put outside the layer that the grid
// states is struck only by steps that do visit its cell
static void check_grid_layer() {
  GridScene s;
  for (int iy = 0; iy < 6; ++iy)
    for (int ix = 0; ix < 6; ++ix) {
      const double lo[3] = {20.0 * ix, 20.0 * iy, 20}, hi[3] = {20.0 * ix + 15, 20.0 * iy + 15, 30};
      s.box(lo, hi);
    }
  ChildGrid& g = s.finish();
  g.z0 = 0;
  g.z1 = 10;
  for (double ex : {0.0, 1e-3, 2.0})
    for (double ey : {0.0, 1e-3, 2.0})
      for (int layer = 0; layer < 2; ++layer) {
        const double p0[3] = {42, 42, layer ? 5.0 : 15.0};
        double p1[3] = {p0[0] + ex, p0[1] + ey, 28}, n[3];
        const int reg = find_end_of_step<double, 0>(s.v, 0, p0, p1, n);
        CHECK((reg > 0) == (layer == 1), "ex %g ey %g from z %g: region %d", ex, ey, p0[2], reg);
      }
}

int main(int argc, char** argv) {
  const std::string what = argc > 1 ? argv[1] : "";
  if (what == "axis_ends") check_axis_ends();
  else if (what == "far_shapes") check_far_shapes();
  else if (what == "fast_models") check_fast_models();
  else if (what == "grid_walk") check_grid_walk();
  else if (what == "grid_layer") check_grid_layer();
  else return 2;
  printf("%s: %ld checks, %d failures\n", what.c_str(), checks, failures);
  return failures ? 1 : 0;
}
