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

int main(int argc, char** argv) {
  const std::string what = argc > 1 ? argv[1] : "";
  if (what == "axis_ends") check_axis_ends();
  else return 2;
  printf("%s: %ld checks, %d failures\n", what.c_str(), checks, failures);
  return failures ? 1 : 0;
}
