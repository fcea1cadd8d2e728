// The short routes against the general searches, on the CPU: the device functions compiled as plain C++.
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

#include "cm_routes.h"

using namespace cm;

static int failures = 0;
static long checks = 0;
#define CHECK(c, ...) \
  do {                \
    ++checks;         \
    if (!(c) && ++failures <= 10) { printf("line %d: ", __LINE__); printf(__VA_ARGS__); printf("\n"); } \
  } while (0)

// ---- table windows
static void check_axis(const char* name, const std::vector<double>& x, int want_kind) {
  const int n = (int)x.size();
  std::vector<GuideEntry> e(3);  // entries of other axes before this one's
  const AxisGuide g = make_guide(x.data(), n, e);
  CHECK(want_kind < 0 || g.kind == want_kind, "%s: guide kind %d, expected %d", name, g.kind, want_kind);
  std::vector<double> at;
  const double inf = std::numeric_limits<double>::infinity();
  for (int i = 0; i < n; ++i) {
    for (double v : {x[i], std::nextafter(x[i], -inf), std::nextafter(x[i], inf)}) at.push_back(v);
    if (i) at.push_back(0.5 * (x[i] + x[i - 1]));
  }
  std::mt19937_64 r(n);
  std::uniform_real_distribution<double> u(0.0, 1.0);
  const double lo = std::min(x[0], x[n - 1]), hi = std::max(x[0], x[n - 1]);
  for (int k = 0; k < 20000; ++k) at.push_back(lo + (hi - lo) * (1.2 * u(r) - 0.1));
  for (double v : {-inf, inf, 0.0, -0.0, 1e-310, -1e300, 1e300}) at.push_back(v);
  std::vector<double> f(n);
  for (double& v : f) v = u(r);
  const AxisGuide none{};
  for (double v : at) {
    int first, nearest;
    nu_locate<double>(v, x.data(), n, 3, first, nearest);
    if (n > 3) CHECK(nu_first3(g, e.data(), v, x.data(), n) == first, "%s: window at %.17g", name, v);
    if (std::isfinite(v)) {
      const double a = nu_d1_order1<double>(g, e.data(), f.data(), x.data(), x.data(), n, v);
      const double b = nu_d1_order1<double>(none, e.data(), f.data(), x.data(), x.data(), n, v);
      CHECK(a == b || (a != a && b != b), "%s: order 1 at %.17g: %.17g %.17g", name, v, a, b);
    }
  }
}

// ---- shapes
struct Shapes {
  std::vector<Shape> shapes;
  std::vector<Plane> planes;
  int add(Shape s) {
    shapes.push_back(s);
    return (int)shapes.size() - 1;
  }
  int planes_of(const std::vector<Plane>& p) {
    Shape s;
    memset(&s, 0, sizeof(s));
    s.kind = SHAPE_PLANES;
    s.plane0 = (int)planes.size();
    s.np = (int)p.size();
    planes.insert(planes.end(), p.begin(), p.end());
    return add(s);
  }
  int pair(int kind, int a, int b) {
    Shape s;
    memset(&s, 0, sizeof(s));
    s.kind = kind;
    s.a = a;
    s.b = b;
    s.anyunion = kind == SHAPE_UNION || shapes[a].anyunion || shapes[b].anyunion;
    return add(s);
  }
  int cylinder(const double* e0, const double* ax, double rad, bool normalised) {
    Shape s;
    memset(&s, 0, sizeof(s));
    s.kind = SHAPE_CYLINDER;
    s.len2 = ax[0] * ax[0] + ax[1] * ax[1] + ax[2] * ax[2];
    s.len = sqrt(s.len2);
    for (int k = 0; k < 3; ++k) {
      s.e0[k] = e0[k];
      s.ax[k] = ax[k];
      s.nax[k] = normalised ? ax[k] / s.len : ax[k] / 0.0;
    }
    s.rad2 = rad * rad;
    return add(s);
  }
};

// a step with both ends strictly inside must be one the general search finds no boundary for
static void check_shape(const char* name, const Shapes& sh, int id, double size, bool described) {
  std::vector<FastPlane> fp;
  std::vector<FastCyl> fc;
  const bool ok = inside_of(sh.shapes, sh.planes, id, fp, fc) && fc.size() <= 1;
  CHECK(ok == described, "%s: described %d", name, ok);
  if (!ok) return;
  SceneView<double> v;
  memset(&v, 0, sizeof(v));
  v.shapes = sh.shapes.data();
  v.planes = sh.planes.data();
  v.fast_planes = fp.data();
  v.fast_cyls = fc.data();
  FastRegion f{0, 0, 0, (int)fp.size(), fc.empty() ? -1 : 0, {0, 0, 0}};
  std::mt19937_64 r(17);
  std::uniform_real_distribution<double> u(-1.0, 1.0);
  long inside = 0;
  for (int k = 0; k < 400000; ++k) {
    double p0[3], p1[3];
    const double len = size * pow(10.0, -6.0 * fabs(u(r)));  // from across the shape to grazing lengths
    for (int a = 0; a < 3; ++a) {
      p0[a] = size * u(r);
      p1[a] = p0[a] + len * u(r);
    }
    if (k % 4 == 0)  // ends within a few margins of a plane
      for (const FastPlane& P : fp) {
        const double d = P.d - (P.n[0] * p1[0] + P.n[1] * p1[1] + P.n[2] * p1[2]) - kFastMarginNm * u(r);
        if (fabs(d) < size * 0.2) {
          for (int a = 0; a < 3; ++a) p1[a] += d * P.n[a];
          break;
        }
      }
    if (!point_inside(v, f, p0) || !point_inside(v, f, p1)) continue;
    ++inside;
    CHECK((shape_contains<double, 4>(v, id, p0)), "%s: start not contained", name);
    const NV nv = shape_first_normal<double, 4>(v, id, p0, p1);
    CHECK(!(nv.u <= 1.0), "%s: boundary at u = %.17g", name, nv.u);
  }
  CHECK(inside > 1000, "%s: only %ld steps inside", name, inside);
}

// the box test never leaves out a plane box that the step strikes
static void check_boxes() {
  std::mt19937_64 r(5);
  std::uniform_real_distribution<double> u(-1.0, 1.0);
  for (int k = 0; k < 300000; ++k) {
    double lo[3], hi[3], bb[6], p0[3], p1[3], rd[3];
    std::vector<Plane> pl;
    for (int a = 0; a < 3; ++a) {
      const double c = 50 * u(r), w = 20 * fabs(u(r)) + 0.01;
      lo[a] = c - w;
      hi[a] = c + w;
      bb[a] = lo[a] - 1e-3;
      bb[3 + a] = hi[a] + 1e-3;
      for (int s = 0; s < 2; ++s) {
        Plane P{{0, 0, 0}, {0, 0, 0}};
        P.n[a] = s ? 1 : -1;
        P.p[a] = s ? hi[a] : lo[a];
        pl.push_back(P);
      }
      p0[a] = 80 * u(r);
    }
    const double len = k % 3 == 0 ? 2e8 : 60;
    for (int a = 0; a < 3; ++a) {
      p1[a] = k % 5 == a ? p0[a] : p0[a] + len * u(r);
      if (k % 7 == 0) p1[a] = (lo[a] + hi[a]) / 2 + (hi[a] - lo[a]) / 2 * (u(r) > 0 ? 1 : -1);  // through corners
      rd[a] = 1.0 / (p1[a] - p0[a]);
    }
    const NV nv = planes_first_normal(pl.data(), 6, p0, p1);
    if (nv.u <= 1.0) CHECK(segment_meets_box(bb, p0, p1, rd), "struck box left out (u %.17g)", nv.u);
  }
}

// NormalMultiPlaneShape::getFirstNormal with every quotient formed
static NV first_normal_plain(const std::vector<Plane>& pl, const double* p0, const double* p1) {
  double umin = -INFINITY, umax = INFINITY;
  int lo = -1, hi = -1;
  for (int i = 0; i < (int)pl.size(); ++i) {
    double num = 0, den = 0;
    for (int a = 0; a < 3; ++a) {
      num += (p0[a] - pl[i].p[a]) * pl[i].n[a];
      den += (p1[a] - p0[a]) * pl[i].n[a];
    }
    if (den == 0) {
      if (num < 0 || (num == 0 && tie_break(pl[i].n))) continue;
      return nv_none();
    }
    const double u = -num / den;
    if (den > 0) {
      if (u < umax) {
        if (u < 0 || u <= umin) return nv_none();
        umax = u;
        hi = i;
      }
    } else if (u > umin) {
      if (u > 1 || u >= umax) return nv_none();
      umin = u;
      lo = i;
    }
  }
  NV r = nv_none();
  const int k = umin > 0 ? lo : umax <= 1 && umax > 0 ? hi : -1;
  if (k < 0) return r;
  r.u = umin > 0 ? umin : umax;
  for (int a = 0; a < 3; ++a) r.n[a] = pl[k].n[a];
  return r;
}

static void check_planes() {
  std::mt19937_64 r(23);
  std::uniform_real_distribution<double> u(-1.0, 1.0);
  long hits = 0;
  for (int k = 0; k < 400000; ++k) {
    const int np = 1 + k % 8;
    std::vector<Plane> pl;
    double p0[3], p1[3];
    const double len = pow(10.0, 4 * u(r));
    for (int a = 0; a < 3; ++a) {
      p0[a] = 30 * u(r);
      p1[a] = p0[a] + len * u(r);
    }
    for (int i = 0; i < np; ++i) {
      Plane P;
      double m = 0;
      for (int a = 0; a < 3; ++a) {
        P.n[a] = k % 3 == 0 ? (double)(int)(2.5 * u(r)) : u(r);
        P.p[a] = k % 3 == 0 ? (double)(int)(30 * u(r)) : 30 * u(r);
        m += P.n[a] * P.n[a];
      }
      if (m == 0) P.n[2] = 1;
      if (k % 5 == 0)  // a plane through an end of the step
        for (int a = 0; a < 3; ++a) P.p[a] = i % 2 ? p0[a] : p1[a];
      pl.push_back(P);
    }
    const NV a = planes_first_normal(pl.data(), np, p0, p1), b = first_normal_plain(pl, p0, p1);
    hits += b.u <= 1;
    CHECK(a.u == b.u && (a.u > 1 || (a.n[0] == b.n[0] && a.n[1] == b.n[1] && a.n[2] == b.n[2])), "planes: u %.17g %.17g", a.u, b.u);
  }
  CHECK(hits > 10000, "planes: only %ld crossings", hits);
}

int main() {
  auto axis = [](int n, auto f) {
    std::vector<double> x;
    for (int i = 0; i < n; ++i) x.push_back(f(i));
    return x;
  };
  check_axis("unit 33", axis(33, [](int i) { return i / 32.0; }), 1);
  check_axis("unit 65", axis(65, [](int i) { return i / 64.0; }), 1);
  check_axis("tenths", axis(11, [](int i) { return 0.1 * i; }), 1);
  check_axis("negative to positive", axis(40, [](int i) { return -3.0 + 0.37 * i; }), 1);
  check_axis("factor 1.05", axis(150, [](int i) { return 16.0 * pow(1.049, i); }), 2);
  check_axis("factor 1.2", axis(40, [](int i) { return 16.0 * pow(1.2, i); }), 2);
  check_axis("factor 1.0005", axis(300, [](int i) { return 1e-3 * pow(1.0005, i); }), -1);
  check_axis("quadratic", axis(50, [](int i) { return 1.0 + 0.01 * i * i; }), -1);
  check_axis("clusters", {0.0, 1e-9, 2e-9, 1.0, 1.0 + 1e-9, 5.0, 1e6}, 0);
  check_axis("four nodes", {1.0, 2.0, 3.0, 4.0}, 1);
  check_axis("descending", axis(20, [](int i) { return 20.0 - i; }), 0);
  check_axis("three nodes", {1.0, 2.0, 4.0}, 0);

  Shapes s;
  auto box = [&](double cx, double cy, double cz, double hw, double scale) {
    std::vector<Plane> p;
    const double c[3] = {cx, cy, cz};
    for (int a = 0; a < 3; ++a)
      for (int sg = -1; sg <= 1; sg += 2) {
        Plane P{{0, 0, 0}, {cx, cy, cz}};
        P.n[a] = scale * sg;
        P.p[a] = c[a] + sg * hw;
        p.push_back(P);
      }
    return p;
  };
  const double th = 0.05;
  const std::vector<Plane> walls = {{{cos(th), 0, sin(th)}, {20, 0, 0}}, {{-cos(th), 0, sin(th)}, {-20, 0, 0}}};
  const int b0 = s.planes_of(box(0, 0, 0, 50, 1.0)), b1 = s.planes_of(box(5, 0, 0, 40, 3.0));
  const int half = s.planes_of({{{0, 0, -1}, {0, 0, 0}}}), wedge = s.planes_of(walls);
  const double e0[3] = {0, -60, 0}, ax[3] = {0, 120, 0};
  const int cyl = s.cylinder(e0, ax, 30, true), ghost = s.cylinder(e0, ax, 30, false);
  const int line = s.pair(SHAPE_INTERSECTION, wedge, b0), both = s.pair(SHAPE_INTERSECTION, b0, b1);
  const int uni = s.pair(SHAPE_UNION, b1, cyl), uni2 = s.pair(SHAPE_UNION, cyl, b1);
  const int deep = s.pair(SHAPE_INTERSECTION, s.pair(SHAPE_UNION, wedge, cyl), b0);
  const int cut = s.pair(SHAPE_INTERSECTION, cyl, b1), two = s.pair(SHAPE_INTERSECTION, cyl, cyl);
  const int ghosts = s.pair(SHAPE_UNION, ghost, b1);
  Shape ball;
  memset(&ball, 0, sizeof(ball));
  ball.kind = SHAPE_SPHERE;
  ball.r = 10;
  const int sphere = s.add(ball);
  check_shape("box", s, b0, 60, true);
  check_shape("scaled normals", s, b1, 60, true);
  check_shape("half space", s, half, 60, true);
  check_shape("half space, far", s, half, 1e8, true);
  check_shape("line", s, line, 60, true);
  check_shape("boxes", s, both, 60, true);
  check_shape("cylinder", s, cyl, 60, true);
  check_shape("union, planes first", s, uni, 60, true);
  check_shape("union, cylinder first", s, uni2, 60, true);
  check_shape("intersection of a union", s, deep, 60, true);
  check_shape("cut cylinder", s, cut, 60, true);
  check_shape("two cylinders", s, two, 60, false);
  check_shape("unnormalised cylinder", s, ghost, 60, false);
  check_shape("union with an unnormalised cylinder", s, ghosts, 60, true);
  check_shape("sphere", s, sphere, 60, false);
  check_boxes();
  check_planes();
  printf("%ld checks, %d failures\n", checks, failures);
  return failures ? 1 : 0;
}
