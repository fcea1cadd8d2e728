// The fast flight against the full one, on the CPU, in the build that records steps: the same electron gets
// the same step and leaves the same record.
#define __host__
#define __device__
#define __global__
#define __shared__
#define __forceinline__ inline
#define __noinline__
#define __align__(n) __attribute__((aligned(n)))
#define CM_TRACE
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>

#include "../../include/cudamonsel_b200.h"
#include "cm_routes.h"
#include "cm_wave.cuh"

using namespace cm;

static int failures = 0;
static long checks = 0;
#define CHECK(c, ...) \
  do {                \
    ++checks;         \
    if (!(c) && ++failures <= 10) { printf("line %d: ", __LINE__); printf(__VA_ARGS__); printf("\n"); } \
  } while (0)

struct HostSink {
  int append(int* c) { return (*c)++; }
  void count(uint32_t* h) { ++*h; }
  unsigned long long ticket(unsigned long long* c) { return (*c)++; }
};

template <typename R> static void check(const char* name) {
  // a box of 40 nm of a model with a phonon mechanism (and, for the second model, a polaron trap)
  std::vector<Shape> shapes(1);
  std::vector<Plane> planes;
  memset(shapes.data(), 0, sizeof(Shape));
  shapes[0].kind = SHAPE_PLANES;
  shapes[0].np = 6;
  for (int a = 0; a < 3; ++a)
    for (int sg = -1; sg <= 1; sg += 2) {
      Plane P{{0, 0, 0}, {0, 0, 0}};
      P.n[a] = sg;
      P.p[a] = 20 * sg;
      planes.push_back(P);
    }
  std::vector<FastPlane> fp;
  std::vector<FastCyl> fc;
  CHECK(inside_of(shapes, planes, 0, fp, fc), "%s: box not described", name);
  for (int nmech = 1; nmech <= 2; ++nmech) {
    Region reg;
    memset(&reg, 0, sizeof(reg));
    reg.parent = -1;
    reg.grid = -1;
    Mech<R> mech[2];
    memset(mech, 0, sizeof(mech));
    mech[0].kind = MECH_PHONON;
    mech[0].phononE = 0.063;
    mech[0].prefactor64 = 2.0;
    mech[0].prefactor = 2;
    mech[1].kind = MECH_POLARON;
    mech[1].prefactor = R(0.05);
    mech[1].extinction = R(0.25);
    mech[1].cutoff = 10;
    Msm<R> msm;
    memset(&msm, 0, sizeof(msm));
    msm.nmech = nmech;
    msm.kinds = MECH_PHONON | MECH_POLARON << 4;
    msm.minE = 1;
    const FastRegion fast{0, 0, 0, (int)fp.size(), -1, {0, 0, 0}};
    RunView<R> v;
    memset(&v, 0, sizeof(v));
    std::vector<TraceRec> rec(4);
    int n = 0;
    v.trace = rec.data();
    v.ntrace = &n;
    v.tracecap = 4;
    v.s.shapes = shapes.data();
    v.s.planes = planes.data();
    v.s.regions = &reg;
    v.s.msms = &msm;
    v.s.mechs = mech;
    v.s.fast = &fast;
    v.s.fast_planes = fp.data();
    std::mt19937_64 r(5);
    std::uniform_real_distribution<double> u(-1.0, 1.0);
    HostSink sink;
    long same = 0, slow = 0, ended = 0;
    for (int k = 0; k < 20000; ++k) {
      El<R> a;
      memset(&a, 0, sizeof(a));
      double m = 0, d[3];
      for (int j = 0; j < 3; ++j) {
        a.p[j] = 19.99 * u(r);
        d[j] = u(r);
        m += d[j] * d[j];
      }
      for (int j = 0; j < 3; ++j) a.d[j] = (R)(d[j] / sqrt(m));
      a.E = (R)(1.5 + 12 * fabs(u(r)));
      a.key = r();
      a.step = (uint32_t)(k % 50);
      El<R> b = a;
      StepCounts sa, sb;
      n = 0;
      memset(rec.data(), 0, sizeof(TraceRec) * rec.size());
      const int qa = flight_fast(v, a, sink, sa, [](El<R>&) {});
      const int na = n;
      if (qa == Q_SLOW) {
        ++slow;
        CHECK(na == 0 && sa.steps == 0, "%s: a step handed on was recorded", name);
        continue;
      }
      const int qb = flight_apply<R, 0>(v, b, sink, sb);
      CHECK(qa == qb && sa.steps == sb.steps && sa.scat == sb.scat, "%s: queue %d, %d", name, qa, qb);
      CHECK(n == 2 * na && na == (qa >= 0 ? 1 : 0), "%s: queue %d, %d records of the fast flight, %d of the full", name, qa, na, n - na);
      if (qa < 0) {
        ++ended;
        continue;
      }
      ++same;
      CHECK(a.E == b.E && a.Ep == b.Ep && a.step == b.step && !memcmp(a.p, b.p, sizeof(a.p)) && aux_kind(a.aux) == aux_kind(b.aux) &&
                aux_val(a.aux) == aux_val(b.aux), "%s: different steps", name);
      if (n == 2) CHECK(!memcmp(&rec[0], &rec[1], sizeof(TraceRec)), "%s: different records", name);
    }
    CHECK(same > 1000 && slow > 1000 && (nmech == 1 || ended > 100), "%s: %ld fast, %ld handed on, %ld ended", name, same, slow, ended);
  }
}

int main() {
  check<double>("fp64");
  check<float>("fp32");
  printf("trace: %ld checks, %d failures\n", checks, failures);
  return failures ? 1 : 0;
}
