// Checks the FP32 path's jumps (newman_gb300/csrc/jump.hpp) against the
// iteration they stand for, on the host: from the reference's series at the
// stop index, every sample is iterated to the jump's index in long double
// against the exact orbit and in double against its FP64 copy (the plain FP64
// path's operations), and both must lie within the record's bound of the
// polynomial, with neither a bailout nor a rebase on the way.
//
//   jump_check re im step nr nc N probes|center samples seed
//
// Prints "samples jumped violations mean-steps worst-ratio".
#include <cmath>
#include <complex>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include <string>

#include "../../newman_gb300/csrc/jump.hpp"

using namespace nmg;
typedef long double LD;
typedef std::complex<LD> CL;

int main(int argc, char** argv) {
  if (argc != 10) return 2;
  const int nr = std::atoi(argv[4]), nc = std::atoi(argv[5]);
  MPView v(nr, nc);
  if (v.set_view(argv[1], argv[2], argv[3], argv[3], std::atoi(argv[6]), 1e-10, 0)) return 3;
  OrbitData od;
  const bool center = !std::strcmp(argv[7], "center");
  if (v.precompute(4, od, center ? REFERENCE_CENTER : REFERENCE_PROBES, false, nullptr, nullptr))
    return 4;
  std::vector<RFE> er, ei;
  v.eps_tables_fe(er, ei);
  LD mx = 0, my = 0;
  for (const RFE& x : er) mx = std::max(mx, fabsl(ldexpl(x.m, x.e)));
  for (const RFE& y : ei) my = std::max(my, fabsl(ldexpl(y.m, y.e)));
  const LD m = sqrtl(mx * mx + my * my);
  const int e = ilogbl(m);
  JumpTables tables;
  build_jumps(od, (double)ldexpl(m, -e) * (1.0 + 0x1p-40), e, 4, tables);
  const std::vector<JumpRec>& recs = tables.start;
  // to 53 bits: the FP64 path's rounding, with its unbounded exponent
  auto r53 = [](LD x) {
    if (x == 0) return x;
    const int k = ilogbl(x) - 52;
    return ldexpl(rintl(ldexpl(x, -k)), k);
  };
  std::mt19937_64 g(std::strtoull(argv[9], nullptr, 10));
  const int samples = std::atoi(argv[8]);
  long jumped = 0, bad = 0;
  LD worst = 0, steps = 0;
  for (int s = 0; s < samples; s++) {
    const RFE& a = er[g() % er.size()];
    const RFE& b = ei[g() % ei.size()];
    const CL eps(ldexpl(a.m, a.e), ldexpl(b.m, b.e));
    const LD u = std::norm(eps);
    int lo = 1, hi = od.xlen;
    while (lo < hi) {
      const int mid = (lo + hi) / 2;
      const RFE& t = od.sa_min_fe[mid];
      if (!std::isinf(t.m) && ldexpl(t.m, t.e) < u) hi = mid; else lo = mid + 1;
    }
    const int fire = lo, f = std::max(1, fire - 3) - 1;
    const JumpRec* use = nullptr;
    for (int c = 0; c < kJumpClasses; c++)
      for (int k = 0; k < kJumpSubs; k++) {
        const JumpRec& r = recs[(size_t)c * kJumpSubs + k];
        if (r.fire == fire && r.rho2 > 0 && ldexpl(u, -2 * r.p) <= r.rho2) use = &r;
      }
    if (!use) continue;
    jumped++;
    auto co = [](const CFE& x) { return CL(ldexpl(x.re, x.e), ldexpl(x.im, x.e)); };
    CL d = (co(od.a_fe[f]) + (co(od.b_fe[f]) + co(od.c_fe[f]) * eps) * eps) * eps;
    LD dr = r53(d.real()), di = r53(d.imag());
    const LD e_r = eps.real(), e_i = eps.imag();
    bool event = false;
    for (int n = f; n < use->n; n++) {
      const CL X = CL((LD)od.xhi[n].x + od.xlo[n].x, (LD)od.xhi[n].y + od.xlo[n].y);
      d = (X + X + d) * d + eps;
      const LD zr = od.xhi[n].x, zi = od.xhi[n].y;
      const LD tr = r53(2 * zr + dr), ti = r53(2 * zi + di);
      const LD nre = r53(r53(r53(tr * dr) - r53(ti * di)) + e_r);
      const LD nim = r53(r53(r53(tr * di) + r53(ti * dr)) + e_i);
      dr = nre;
      di = nim;
      const LD yr = r53(od.xhi[n + 1].x + dr), yi = r53(od.xhi[n + 1].y + di);
      const LD r2 = yr * yr + yi * yi, d2 = dr * dr + di * di;
      if (r2 > 1048576.0L || r2 <= d2) event = true;
    }
    steps += use->n - f;
    const CL x(ldexpl(eps.real(), -use->p), ldexpl(eps.imag(), -use->p));
    CL p = 0;
    for (int k = kJumpDegree - kJumpExact - 1; k >= 0; k--) p = p * x + CL(use->c[k].x, use->c[k].y);
    for (int k = kJumpExact - 1; k >= 0; k--)
      p = p * x + CL((LD)use->b[k].x + use->b[k].y, (LD)use->b[k].z + use->b[k].w);
    p *= x;
    const LD bound = (LD)use->err;
    const LD e1 = std::abs(p - CL(ldexpl(d.real(), -use->s), ldexpl(d.imag(), -use->s)));
    const LD e2 = std::abs(p - CL(ldexpl(dr, -use->s), ldexpl(di, -use->s)));
    worst = std::max(worst, std::max(e1, e2) / bound);
    if (event || !(e1 <= bound) || !(e2 <= bound)) bad++;
  }
  // chain jumps: delta on a circle of the ball's size at each chain's start
  long rj = 0, rbad = 0;
  LD rworst = 0, rsteps = 0;
  std::uniform_real_distribution<double> U(0.0, 1.0);
  auto X = [&](int n) { return CL((LD)od.xhi[n].x + od.xlo[n].x, (LD)od.xhi[n].y + od.xlo[n].y); };
  for (int s = 0; s < samples; s++) {
    const int chain = s % kChains, from = tables.start_index[chain];
    if (from < 0) continue;
    const JumpRec* rb = &tables.chain[(size_t)chain * kChainClasses];
    const RFE& a = er[g() % er.size()];
    const RFE& b = ei[g() % ei.size()];
    const CL eps(ldexpl(a.m, a.e), ldexpl(b.m, b.e));
    const LD dm = exp2l(-0.5L * (kChainTop + 2 * kChainClasses * U(g))), ph = 6.2831853L * U(g);
    const CL d0(r53(dm * cosl(ph)), r53(dm * sinl(ph)));
    int i = (-(ilogbl(std::norm(d0)) + 1) - kChainTop) >> 1;
    const JumpRec* use = nullptr;
    CL x = 0;
    for (int t = 0; t < 3 && !use; t++, i--) {
      if (i < 0 || i >= kChainClasses || !(rb[i].rho2 > 0)) continue;
      const Flt4 g = rb[i].gamma;
      x = d0 + CL((LD)g.x + g.y, (LD)g.z + g.w) * eps;
      if (ldexpl(std::norm(x), -2 * rb[i].p) <= rb[i].rho2) use = &rb[i];
    }
    if (!use) continue;
    rj++;
    const int n = use->n;
    if (use->fire != from) rbad++;
    rsteps += n - from;
    // the polynomial
    const CL y(ldexpl(x.real(), -use->p), ldexpl(x.imag(), -use->p));
    CL p = 0, q = 0;
    for (int k = kJumpDegree - kJumpExact - 1; k >= 0; k--) p = p * y + CL(use->c[k].x, use->c[k].y);
    for (int k = kJumpExact - 1; k >= 0; k--)
      p = p * y + CL((LD)use->b[k].x + use->b[k].y, (LD)use->b[k].z + use->b[k].w);
    const Flt2* tab[4] = {use->q4, use->q3, use->q2, use->q1};
    const int len[4] = {kJumpEps4, kJumpEps3, kJumpEps2, kJumpEps1};
    for (int o = 0; o < 4; o++) {
      CL t = 0;
      for (int k = len[o] - 1; k >= 0; k--) {
        t = t * y + CL(tab[o][k].x, tab[o][k].y);
        if (o == 3 && k < kEpsExact) t += CL(use->q1l[k].x, use->q1l[k].y);
      }
      q = (q + t) * 0x1p32L * eps;
    }
    p = p * y + q;
    // the exact orbit, and the FP64 path's steps
    CL d = d0;
    LD dr = d0.real(), di = d0.imag();
    bool event = false;
    for (int k = from; k < n; k++) {
      d = (X(k) + X(k) + d) * d + eps;
      const LD tr = r53(2 * (LD)od.xhi[k].x + dr), ti = r53(2 * (LD)od.xhi[k].y + di);
      const LD nre = r53(r53(r53(tr * dr) - r53(ti * di)) + eps.real());
      const LD nim = r53(r53(r53(tr * di) + r53(ti * dr)) + eps.imag());
      dr = nre;
      di = nim;
      const LD yr = od.xhi[k + 1].x + dr, yi = od.xhi[k + 1].y + di;
      if (yr * yr + yi * yi <= dr * dr + di * di || yr * yr + yi * yi > 1048576.0L) event = true;
    }
    const LD e1 = std::abs(p - CL(ldexpl(d.real(), -use->s), ldexpl(d.imag(), -use->s)));
    const LD e2 = std::abs(p - CL(ldexpl(dr, -use->s), ldexpl(di, -use->s)));
    rworst = std::max(rworst, std::max(e1, e2) / use->err);
    if (event || !(e1 <= use->err) || !(e2 <= use->err)) rbad++;
  }
  std::printf("%ld %ld %.1f %.4f\n", rj, rbad, (double)(rsteps / std::max(1L, rj)), (double)rworst);
  if (std::getenv("JUMP_RECORDS"))
    for (size_t i = 0; i < tables.chain.size(); i++) {
      const JumpRec& r = tables.chain[i];
      if (r.rho2 > 0)
        std::printf("chain %d class %zu n %d p %d s %d err 2^%.1f q0 %.2g rho %.2f\n", r.fire,
                    i % kChainClasses, r.n, r.p, r.s, std::log2(r.err), r.q1[0].x,
                    std::sqrt(r.rho2));
    }
  if (rbad) bad += rbad;
  std::printf("%d %ld %ld %.1f %.4f\n", samples, jumped, bad, (double)(steps / std::max(1L, jumped)),
              (double)worst);
  if (std::getenv("JUMP_RECORDS"))
    for (const JumpRec& r : recs)
      if (r.fire >= 0)
        std::printf("fire %d n %d rho %.3f p %d s %d |b1| %.3f err %.3g (2^%.1f of the linear term)\n",
                    r.fire, r.n, std::sqrt(std::max(0.0f, r.rho2)), r.p, r.s,
                    std::hypot(r.b[0].x, r.b[0].z), r.err,
                    std::log2(r.err / (std::hypot(r.b[0].x, r.b[0].z) * std::sqrt(r.rho2))));
  return bad ? 1 : 0;
}
