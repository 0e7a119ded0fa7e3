// The FP64 step's estimate of "no bailout, no rebase" (no_event_by_estimate) and
// the eps it leaves out (absorbed), pixel_fp64.cuh, against the FP64 operations
// they stand for, on the host build of the same header.
//
//   fp64_estimate count seed
//
// Prints "checks decided absorbed mismatches".
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>

#include "../../newman_gb300/csrc/pixel_fp64.cuh"

using namespace nmg;

int main(int argc, char** argv) {
  const long n = std::atol(argv[1]);
  std::mt19937_64 g(std::strtoull(argv[2], nullptr, 10));
  std::uniform_real_distribution<double> u(-1.0, 1.0);
  auto mag = [&](double lo, double hi) { return std::exp2(lo + (hi - lo) * 0.5 * (u(g) + 1.0)); };
  long decided = 0, skipped = 0, bad = 0;
  for (long k = 0; k < n; k++) {
    const int kind = (int)(g() % 6);
    // sizes of Z and delta: as the loop meets them, out to the bailout, small,
    // vanishing or beyond the estimates' range; a third of them near a tie
    // |Y| = |delta| or near |Y| = 1024
    const double zs = kind == 0 ? mag(-2, 2) : kind == 1 ? mag(8, 12) : kind == 2 ? mag(-70, -10)
                    : kind == 3 ? mag(-3, 11) : kind == 4 ? mag(-1000, 1000) : 0.0;
    Dbl2 z{zs * u(g), zs * u(g)};
    const double ds = kind == 4 ? mag(-1000, 1000) : zs == 0.0 ? mag(-80, 80) : zs * mag(-24, 4);
    double dr = ds * u(g), di = ds * u(g);
    if (g() % 3 == 0) {
      // delta = Y - Z with |Y| a little off |delta| or 1024
      const double t = g() % 2 ? 1.0 + u(g) * std::exp2(-(double)(g() % 30)) : 1.0;
      if (g() % 2) {
        // |Z + d| = t |d|: d along Z's bisector, scaled
        const double a = -0.5 * t;
        const double h = std::sqrt(std::fabs(1.0 - a * a)) * (g() % 2 ? 1 : -1);
        dr = z.x * a - z.y * h;
        di = z.y * a + z.x * h;
      } else {
        const double ph = 3.2 * u(g);
        dr = 1024.0 * t * std::cos(ph) - z.x;
        di = 1024.0 * t * std::sin(ph) - z.y;
      }
    }
    if (g() % 16 == 0) (g() % 2 ? z.x : dr) = 0.0;
    const double yr = z.x + dr, yi = z.y + di;
    const double r2 = yr * yr + yi * yi, d2 = dr * dr + di * di;
    const bool event = r2 > 1048576.0 || r2 < d2;
    if (no_event_by_estimate(z, dr, di)) {
      decided++;
      if (event) bad++;
    }
    const double e = dr * std::exp2((double)(int)(g() % 120) - 100.0) * (g() % 2 ? 1.0 : u(g));
    if (exp_field(z.x) >= 1 && exp_field(z.x) < 2047 && absorbed(z.x, e)) {
      skipped++;
      if (z.x + e != z.x || z.x - e != z.x) bad++;
    }
    // the boundary: a power of two less just under a quarter of its ulp
    const double p = std::ldexp(1.0, (int)(g() % 600) - 300);
    const double q = p * (0x1p-53 * mag(-3, 2));
    if (absorbed(p, q) && (p + q != p || p - q != p)) bad++;
  }
  std::printf("%ld checks %ld decided %ld absorbed %ld mismatches\n", n, decided, skipped, bad);
  return bad ? 1 : 0;
}
