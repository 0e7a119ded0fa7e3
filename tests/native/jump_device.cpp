// The FP32 path's jumps as the device makes them (newman_gb300/csrc/fe_jump.cuh,
// its host build) against the records' polynomials in long double.
//
//   jump_device what re im step nr nc N probes|center samples seed
//
// what = slope: the factor by which a chain jump multiplies a start's bound is at
// least the derivative of the whole polynomial, orders of eps included, at the
// start: samples stand at a chain's first index with delta on the edge of a
// record's ball and eps a corner of the grid, and jump with two bounds.
// what = range: eps at a corner of the grid jumps, eps beyond it in one component
// does not (a preview's last row can lie outside the grid of the view whose tables it
// shares).  "violations": jumps beyond; "worst": the part of those inside that jump.
//
// what = start: a sample whose eps lies in a start record's ball, on one of the
// axes or off them, jumps, to within the bound of the polynomial.
// what = precision: against the exact iteration, jumps are off by no more than the
// float-float steps they stand for, root mean square and at most, from random samples
// of the grid at the series stop and from the balls at the chains' starts.
// "violations": of those four; "worst": the largest ratio.
//
// what = sizes: prints for grids of 2^17 - 1, 2^17, 499,999 and 500,000 samples whether
// they have tables (1) or none (0), as one number.
//
// what = tie: a rebase test near its tie counts as tied at every size of delta that
// the unscaled steps meet, as long as the bound is below 2^-23 |delta|.
//
// what = side: near a tie, what fe_tie_side decides is what the FP64 path's sums give
// for both paths' deltas; "worst": the part decided where |Z| > 2^-26 |delta|.
//
// Prints "jumps violations worst", worst the largest ratio.
#include <cmath>
#include <complex>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include <string>

#include "../../newman_gb300/csrc/fe_jump.cuh"
#include "../../newman_gb300/csrc/jump.hpp"

using namespace nmg;
typedef long double LD;
typedef std::complex<LD> CL;

static JumpTables tables;
static std::vector<JumpRec> records;
static std::vector<RFE> er, ei;
static DeviceView view;
static EpsRange range;

static CL eps_at(size_t c, size_t r) { return CL(ldexpl(er[c].m, er[c].e), ldexpl(ei[r].m, ei[r].e)); }

static FF ff(LD x) {
  const float h = (float)x;
  return FF{h, (float)(x - (LD)h)};
}

// A sample at the first index of `chain` with delta d, eps and bound e.
static FeState state(int chain, CL d, CL eps, float e) {
  FeState st{};
  st.dr = ff(d.real());
  st.di = ff(d.imag());
  st.er = ff(eps.real());
  st.ei = ff(eps.imag());
  st.err = e;
  st.j = view.jump_from[chain];
  st.i = st.j;
  st.certified = 1;
  return st;
}

// The derivative at x = y 2^p of the record's polynomial, all orders of eps.
static CL slope(const JumpRec& r, CL y, CL eps) {
  CL g = 0;
  for (int k = kJumpDegree; k >= 1; k--) {
    const CL c = k <= kJumpExact ? CL((LD)r.b[k - 1].x + r.b[k - 1].y, (LD)r.b[k - 1].z + r.b[k - 1].w)
                                 : CL(r.c[k - kJumpExact - 1].x, r.c[k - kJumpExact - 1].y);
    g = g * y + (LD)k * c;
  }
  const Flt2* tab[4] = {r.q1, r.q2, r.q3, r.q4};
  const int len[4] = {kJumpEps1, kJumpEps2, kJumpEps3, kJumpEps4};
  CL e = 1;
  for (int b = 0; b < 4; b++) {
    e *= 0x1p32L * eps;
    CL t = 0;
    for (int k = len[b] - 1; k >= 1; k--) {
      CL c(tab[b][k].x, tab[b][k].y);
      if (b == 0 && k < kEpsExact) c += CL(r.q1l[k].x, r.q1l[k].y);
      t = t * y + (LD)k * c;
    }
    g += t * e;
  }
  return g;
}

// The record of `chain` that a sample jumped by, from its new index.
static const JumpRec* taken(int chain, const FeState& a, const FeState& b) {
  for (int i = 0; i < kChainClasses; i++) {
    const JumpRec& r = tables.chain[(size_t)chain * kChainClasses + i];
    if (r.rho2 > 0 && r.n - r.fire == b.j - a.j && (float)r.scale != 0.0f) return &r;
  }
  return nullptr;
}

static int check_slope(int samples, std::mt19937_64& g) {
  std::uniform_real_distribution<double> U(0.0, 1.0);
  long jumps = 0, bad = 0;
  LD worst = 0;
  for (int s = 0; s < samples; s++) {
    const int chain = (int)(g() % kChains), i = (int)(g() % kChainClasses);
    const JumpRec& r = tables.chain[(size_t)chain * kChainClasses + i];
    if (tables.start_index[chain] < 0 || !(r.rho2 > 0)) continue;
    const CL eps = eps_at(g() % 2 ? 0 : er.size() - 1, g() % 2 ? 0 : ei.size() - 1);
    // x on the ball's edge, delta = x - Gamma eps
    const LD a = ldexpl(sqrtl(r.rho2) * (0.9L + 0.09L * U(g)), r.p), ph = 6.2831853L * U(g);
    const CL gamma((LD)r.gamma.x + r.gamma.y, (LD)r.gamma.z + r.gamma.w);
    const CL x = CL(a * cosl(ph), a * sinl(ph)), d = x - gamma * eps;
    const float e = (float)(0x1p-27L * a);
    FeState st1 = state(chain, d, eps, e), st2 = state(chain, d, eps, 4.0f * e), st0 = st1;
    fe_chain_jump(view, st1);
    fe_chain_jump(view, st2);
    const JumpRec* t = taken(chain, st0, st1);
    if (st1.j == st0.j || st2.j != st1.j || t != &r) continue;  // by another class's record
    jumps++;
    const LD got = ((LD)st2.err - st1.err) / (3 * (LD)e) / r.scale * ldexpl(1, r.p);
    const LD want = std::abs(slope(r, CL(ldexpl(x.real(), -r.p), ldexpl(x.imag(), -r.p)), eps));
    // (the bounds' own rounding: 2^-23 of themselves)
    worst = std::max(worst, want / got);
    if (want > got * (1 + 0x1p-20L)) bad++;
  }
  std::printf("%ld %ld %.7f\n", jumps, bad, (double)worst);
  return bad ? 1 : 0;
}

static int check_range(int samples, std::mt19937_64& g) {
  std::uniform_real_distribution<double> U(0.0, 1.0);
  long inside = 0, jumped = 0, bad = 0;
  for (int s = 0; s < samples; s++) {
    const int chain = (int)(g() % kChains), i = (int)(g() % kChainClasses);
    const JumpRec& r = tables.chain[(size_t)chain * kChainClasses + i];
    if (tables.start_index[chain] < 0 || !(r.rho2 > 0)) continue;
    CL eps = eps_at(g() % 2 ? 0 : er.size() - 1, g() % 2 ? 0 : ei.size() - 1);
    // the corners that are the farthest in both components
    if (fabsl(eps.real()) != ldexpl(range.re, range.e) || fabsl(eps.imag()) != ldexpl(range.im, range.e))
      continue;
    const LD a = ldexpl(0.7L * sqrtl(r.rho2), r.p), ph = 6.2831853L * U(g);
    const CL gamma((LD)r.gamma.x + r.gamma.y, (LD)r.gamma.z + r.gamma.w);
    const LD f = 1.0L + std::exp2(-20.0 + 20.0 * U(g));
    for (int beyond = 0; beyond < 3; beyond++) {
      const CL e(beyond == 1 ? f * eps.real() : eps.real(), beyond == 2 ? f * eps.imag() : eps.imag());
      const CL d = CL(a * cosl(ph), a * sinl(ph)) - gamma * e;
      FeState st = state(chain, d, e, (float)(0x1p-27L * a));
      const int j = st.j;
      fe_chain_jump(view, st);
      if (beyond == 0) {
        inside++;
        jumped += st.j != j;
      } else {
        bad += st.j != j;
      }
    }
  }
  std::printf("%ld %ld %.7f\n", jumped, bad, (double)jumped / std::max(1L, inside));
  return bad ? 1 : 0;
}

static FFE ffe(LD x) {
  if (x == 0) return FFE{0.0f, 0.0f, 0, 0};
  const int k = ilogbl(x);
  const FF m = ff(ldexpl(x, -k));
  return FFE{m.h, m.l, k, 0};
}

static int check_start(int samples, std::mt19937_64& g) {
  std::uniform_real_distribution<double> U(0.0, 1.0);
  long jumps = 0, bad = 0;
  LD worst = 0;
  for (int s = 0; s < samples; s++) {
    const JumpRec& r = tables.start[g() % tables.start.size()];
    if (!(r.rho2 > 0)) continue;
    const LD a = ldexpl(sqrtl(r.rho2) * (0.5L + 0.49L * U(g)), r.p), ph = 6.2831853L * U(g);
    const int axis = (int)(g() % 3);
    const FFE fr = ffe(axis == 0 ? 0 : axis == 1 ? a : a * cosl(ph));
    const FFE fi = ffe(axis == 0 ? -a : axis == 1 ? 0 : a * sinl(ph));
    CFF d;
    float bound = 0.0f;
    int found = -1;
    if (!fe_jump(view, r.fire, fr, fi, d, bound, found)) {
      bad++;
      continue;
    }
    jumps++;
    // the record it took: the smallest radius that holds it
    const JumpRec* use = nullptr;
    for (const JumpRec& q : tables.start)
      if (q.fire == r.fire && q.rho2 > 0 && q.n == found && q.err == bound && q.s == d.e) use = &q;
    if (!use) {
      bad++;
      continue;
    }
    const CL y(ldexpl((LD)fr.h + fr.l, fr.e - use->p), ldexpl((LD)fi.h + fi.l, fi.e - use->p));
    CL p = 0;
    for (int k = kJumpDegree; k >= 1; k--) {
      const CL c = k <= kJumpExact
                       ? CL((LD)use->b[k - 1].x + use->b[k - 1].y, (LD)use->b[k - 1].z + use->b[k - 1].w)
                       : CL(use->c[k - kJumpExact - 1].x, use->c[k - kJumpExact - 1].y);
      p = (p + c) * y;
    }
    const LD e = std::abs(p - CL((LD)d.re.h + d.re.l, (LD)d.im.h + d.im.l)) / bound;
    worst = std::max(worst, e);
    if (!(e <= 1)) bad++;
  }
  std::printf("%ld %ld %.7f\n", jumps, bad, (double)worst);
  return bad ? 1 : 0;
}

// Steps from orbit index j to k (of z) in float-float, and exactly.
static void step_to(const OrbitData& od, int j, int k, FF er_, FF ei_, FF& dr, FF& di, CL& exact) {
  const CL eps((LD)er_.h + er_.l, (LD)ei_.h + ei_.l);
  for (; j < k; j++) {
    const FF zr = ff_from_double(od.z[j].x), zi = ff_from_double(od.z[j].y);
    const FF tr = ff_add_twice_raw(zr.h, zr.l, dr), ti = ff_add_twice_raw(zi.h, zi.l, di);
    FF nr, ni;
    ff_cmul_add(tr, ti, dr, di, er_, ei_, nr, ni);
    dr = nr;
    di = ni;
    // X[j - 1] is z[j]
    const CL X((LD)od.xhi[j - 1].x + od.xlo[j - 1].x, (LD)od.xhi[j - 1].y + od.xlo[j - 1].y);
    exact = (X + X + exact) * exact + eps;
  }
}

struct Errors {
  long n = 0;
  LD sum = 0, most = 0;
  void add(CL got, CL exact) {
    const LD e = std::abs(got - exact) / std::abs(exact);
    n++;
    sum += e * e;
    most = std::max(most, e);
  }
  LD rms() const { return sqrtl(sum / std::max(1L, n)); }
};

static int check_precision(const OrbitData& od, int samples, std::mt19937_64& g) {
  std::uniform_real_distribution<double> U(0.0, 1.0);
  Errors jump[2], steps[2];
  for (int s = 0; s < samples; s++) {
    const int chain = (int)(g() % kChains), i = (int)(g() % kChainClasses);
    const JumpRec& r = tables.chain[(size_t)chain * kChainClasses + i];
    if (tables.start_index[chain] < 0 || !(r.rho2 > 0)) continue;
    const CL eps = eps_at(g() % er.size(), g() % ei.size());
    const LD a = ldexpl(sqrtl(r.rho2) * (0.5L + 0.49L * U(g)), r.p), ph = 6.2831853L * U(g);
    const CL gamma((LD)r.gamma.x + r.gamma.y, (LD)r.gamma.z + r.gamma.w);
    FeState st = state(chain, CL(a * cosl(ph), a * sinl(ph)) - gamma * eps, eps, 0.0f);
    FF dr = st.dr, di = st.di;
    CL exact((LD)dr.h + dr.l, (LD)di.h + di.l);
    const int j = st.j;
    fe_chain_jump(view, st);
    if (st.j == j) continue;
    step_to(od, j, st.j, st.er, st.ei, dr, di, exact);
    jump[0].add(CL((LD)st.dr.h + st.dr.l, (LD)st.di.h + st.di.l), exact);
    steps[0].add(CL((LD)dr.h + dr.l, (LD)di.h + di.l), exact);
  }
  auto co = [](const CFE& x) { return CL(ldexpl(x.re, x.e), ldexpl(x.im, x.e)); };
  for (int s = 0; s < samples; s++) {
    const CL eps = eps_at(g() % er.size(), g() % ei.size());
    const LD u = std::norm(eps);
    int fire = 1, hi = od.xlen;
    while (fire < hi) {
      const int mid = (fire + hi) / 2;
      const RFE& t = od.sa_min_fe[mid];
      if (!std::isinf(t.m) && ldexpl(t.m, t.e) < u) hi = mid; else fire = mid + 1;
    }
    CFF d;
    float bound = 0.0f;
    int found = -1;
    if (!fe_jump(view, fire, ffe(eps.real()), ffe(eps.imag()), d, bound, found)) continue;
    const int f = std::max(1, fire - 3) - 1;
    CL exact = (co(od.a_fe[f]) + (co(od.b_fe[f]) + co(od.c_fe[f]) * eps) * eps) * eps;
    FF dr = ff(exact.real()), di = ff(exact.imag());
    step_to(od, f + 1, found + 1, ff(eps.real()), ff(eps.imag()), dr, di, exact);
    jump[1].add(CL(ldexpl((LD)d.re.h + d.re.l, d.e), ldexpl((LD)d.im.h + d.im.l, d.e)), exact);
    steps[1].add(CL((LD)dr.h + dr.l, (LD)di.h + di.l), exact);
  }
  int bad = 0;
  LD worst = 0;
  for (int k = 0; k < 2; k++) {
    const LD ratio[2] = {jump[k].rms() / steps[k].rms(), jump[k].most / steps[k].most};
    for (LD q : ratio) {
      worst = std::max(worst, q);
      if (!(q <= 1)) bad++;
    }
  }
  std::printf("%ld %d %.4f\n", std::min(jump[0].n, jump[1].n), bad, (double)worst);
  return bad ? 1 : 0;
}

static int check_tie(int samples, std::mt19937_64& g) {
  std::uniform_real_distribution<double> U(0.0, 1.0);
  long bad = 0;
  for (int s = 0; s < samples; s++) {
    const double d = std::exp2(-59.0 * U(g)), near = (2.0 * U(g) - 1.0) * 0x1p-20;
    const float d2 = (float)(d * d), r2 = (float)(d * d * (1.0 + near));
    const double e = std::exp2(-40.0 * U(g));  // bound / |delta|
    if (e > 0x1p-24 && e < 0x1p-22) continue;
    if (fe_tied(r2, d2, (float)(e * d)) != (e < 0x1p-23)) bad++;
    if (fe_tied((float)(d * d * (1.0 - 0x1p-17)), d2, (float)(e * d))) bad++;
  }
  std::printf("%d %ld 0\n", samples, bad);
  return bad ? 1 : 0;
}

static int check_side(int samples, std::mt19937_64& g) {
  std::uniform_real_distribution<double> U(-1.0, 1.0);
  long bad = 0, n = 0, decided = 0;
  for (int s = 0; s < samples; s++) {
    // delta of any size, Z from as large down to far below its rounding
    const double d = std::exp2(29.5 * (U(g) - 1.0)), q = std::exp2(25.0 * (U(g) - 1.0));
    const double p1 = 3.15 * U(g);
    double dx = d * std::cos(p1), dy = d * std::sin(p1);
    // Z at an angle of delta with |Z + delta| near |delta|: cos = -q / 2, moved
    const double c = -0.5 * q + (g() % 2 ? U(g) : U(g) * std::exp2(-24.0 * std::fabs(U(g))));
    if (std::fabs(c) > 1.0) continue;
    const double h = std::sqrt(1.0 - c * c) * (g() % 2 ? 1.0 : -1.0);
    const double zx = q * (dx * c - dy * h), zy = q * (dy * c + dx * h);
    const float fx = (float)dx, fy = (float)dy, wx = (float)zx, wy = (float)zy;
    const float yx = wx + fx, yy = wy + fy;
    const float r2 = fmaf(yx, yx, yy * yy), d2 = fmaf(fx, fx, fy * fy);
    if (!(r2 < d2 * (1.0f + kFeTie)) || !fe_tied(r2, d2, 0.0f)) continue;
    n++;
    const int side = fe_tie_side(wx, wy, fx, fy, d2);
    if (q > 0x1p-26) decided += side >= 0;
    else n--;
    if (side < 0) continue;
    // the FP64 path's delta, up to 2^-23 off
    for (int k = 0; k < 4; k++) {
      const double t = k ? 0x1p-23 * d : 0.0, p2 = 3.15 * U(g);
      const double ex = dx + t * std::cos(p2), ey = dy + t * std::sin(p2);
      const double vx = zx + ex, vy = zy + ey;
      const bool rebase = vx * vx + vy * vy < ex * ex + ey * ey;
      if (rebase != (side == 1)) bad++;
    }
  }
  std::printf("%ld %ld %.4f\n", n, bad, (double)decided / std::max(1L, n));
  return bad ? 1 : 0;
}

int main(int argc, char** argv) {
  if (argc != 11) return 2;
  const char* what = argv[1];
  std::mt19937_64 g(std::strtoull(argv[10], nullptr, 10));
  const int samples = std::atoi(argv[9]);
  if (!std::strcmp(what, "tie")) return check_tie(samples, g);
  if (!std::strcmp(what, "side")) return check_side(samples, g);
  MPView v(std::atoi(argv[5]), std::atoi(argv[6]));
  if (v.set_view(argv[2], argv[3], argv[4], argv[4], std::atoi(argv[7]), 1e-10, 0)) return 3;
  OrbitData od;
  const bool center = !std::strcmp(argv[8], "center");
  if (v.precompute(4, od, center ? REFERENCE_CENTER : REFERENCE_PROBES, false, nullptr, nullptr))
    return 4;
  v.eps_tables_fe(er, ei);
  range = eps_range(er, ei);
  if (!std::strcmp(what, "sizes")) {
    for (long long n : {(1ll << 17) - 1, 1ll << 17, 499999ll, 500000ll}) {
      JumpTables t;
      build_jumps(od, range.norm(), range.e, 4, t, n);
      bool any = t.start[0].fire >= 0;
      for (int k = 0; k < kChains; k++) any |= t.start_index[k] >= 0;
      for (const JumpRec& r : t.chain) any |= r.rho2 > 0;
      std::printf("%d", any);
    }
    std::printf(" 0 0\n");
    return 0;
  }
  build_jumps(od, range.norm(), range.e, 4, tables);
  records = tables.start;
  records.insert(records.end(), tables.chain.begin(), tables.chain.end());
  view.N = 1 << 30;
  view.jump = records.data();
  view.jump_x2 = 0x1p-16f;
  view.jump_er = range.re_limit();
  view.jump_ei = range.im_limit();
  for (int k = 0; k < kChains; k++)
    view.jump_from[k] = tables.start_index[k] < 0 ? -1 : tables.start_index[k] + 1;
  if (!std::strcmp(what, "slope")) return check_slope(samples, g);
  if (!std::strcmp(what, "range")) return check_range(samples, g);
  if (!std::strcmp(what, "precision")) return check_precision(od, samples, g);
  if (!std::strcmp(what, "start")) return check_start(samples, g);
  return 2;
}
