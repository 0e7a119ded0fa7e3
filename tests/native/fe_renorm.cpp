// The FP32 path's scaled steps (newman_gb300/csrc/fe_core.cuh, compiled for the host):
// the state after a number of steps is the same bits in whatever pieces they are made.
//
//   fe_renorm re im step nr nc N samples steps seed
//
// Prints "samples mismatches renormalisations".
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>

// what the header takes from the device compiler
using std::max;
using std::min;
static inline float __int_as_float(int i) {
  float f;
  std::memcpy(&f, &i, 4);
  return f;
}
static inline float __fsub_rd(float a, float b) {
  const float f = a - b;
  return (double)f > (double)a - (double)b ? std::nextafter(f, -INFINITY) : f;
}
static inline int __clz(int x) { return x ? __builtin_clz((unsigned)x) : 32; }
static inline int __popc(unsigned x) { return __builtin_popcount(x); }
static inline unsigned __ballot_sync(unsigned, bool p) { return p ? 1u : 0u; }

#include "../../newman_gb300/csrc/fe_core.cuh"
#include "../../newman_gb300/csrc/mpview.hpp"

using namespace nmg;

int main(int argc, char** argv) {
  if (argc != 10) return 2;
  MPView v(std::atoi(argv[4]), std::atoi(argv[5]));
  if (v.set_view(argv[1], argv[2], argv[3], argv[3], std::atoi(argv[6]), 1e-10, 0)) return 3;
  OrbitData od;
  if (v.precompute(4, od, REFERENCE_CENTER, false, nullptr, nullptr)) return 4;
  std::vector<RFE> er, ei;
  v.eps_tables_fe(er, ei);
  std::vector<Flt4> zf(od.z.size());
  for (size_t k = 0; k < zf.size(); k++) {
    const FF x = ff_from_double(od.z[k].x), y = ff_from_double(od.z[k].y);
    zf[k] = {x.h, y.h, x.l, y.l};
  }
  DeviceView view{};
  view.N = std::atoi(argv[6]);
  view.zf = zf.data();
  view.zlen = (int)zf.size();
  view.sa_fe = 1;
  std::mt19937_64 g(std::strtoull(argv[9], nullptr, 10));
  const int samples = std::atoi(argv[7]), steps = std::atoi(argv[8]);
  long bad = 0, renorms = 0;
  for (int s = 0; s < samples; s++) {
    const RFE a = er[g() % er.size()], b = ei[g() % ei.size()];
    FeState start{};
    start.E = std::max(a.e, b.e);
    start.dr = start.er = ff_from_double(std::scalbn(a.m, a.e - start.E));
    start.di = start.ei = ff_from_double(std::scalbn(b.m, b.e - start.E));
    start.err = up_mul(kFeU, up_add(fabsf(start.dr.h), fabsf(start.di.h)));
    start.j = start.i = 1;
    start.certified = 1;
    const int renorm = 1 + (int)(g() % 100);
    FeState whole = start, parts = start;
    FeResult res;
    unsigned long long n = 0, r = 0;
    int e = whole.E;
    while (whole.i < 1 + steps && whole.E != 0) {
      if (fe_advance(view, whole, min(renorm, 1 + steps - whole.i), renorm, res, n, r)) break;
      renorms += whole.E != e;
      e = whole.E;
    }
    // in pieces of 16 steps, cut short here and there, as a warp's rounds make them
    while (parts.i < whole.i && parts.E != 0)
      if (fe_advance(view, parts, min((int)(g() % 4 ? 16 : 1 + g() % 16), whole.i - parts.i), renorm,
                     res, n, r))
        break;
    if (std::memcmp(&whole, &parts, sizeof whole)) bad++;
  }
  std::printf("%d %ld %ld\n", samples, bad, renorms);
  return bad ? 1 : 0;
}
