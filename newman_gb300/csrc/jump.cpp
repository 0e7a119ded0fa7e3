// The polynomials of jump.hpp, on the host in double.
#if defined(__GNUC__)
#pragma GCC optimize("O3", "no-math-errno")  // (square roots in vectors)
#endif
#include "jump.hpp"

#include <algorithm>
#include <atomic>
#include <cmath>
#include <thread>

namespace nmg {

namespace {

constexpr int D = kJumpDegree;
// Orders of eps (chain jumps) and the terms x^0 .. of each: order 0 has x^1 ..
// x^D, the others what FP32 holds of them (JumpRec).
constexpr int B = kJumpOrders;
constexpr int kTerms[B] = {D + 1, kJumpEps1, kJumpEps2, kJumpEps3, kJumpEps4};
// R stays below 2^-46 of the linear term: half the FP32 path's rounding of one
// step, and since R grows by 2^D an octave of delta, a tighter or looser limit
// moves the target by a few steps only.
constexpr double kTail = 0x1p-46;
// A record is worth its evaluation (four steps' work and a lane's wait for
// its warp) from here on.
constexpr int kMinSteps = 16;

// A chain's jumps go at most this far.
constexpr int kChainReach = 4096;

double norm(double re, double im) { return std::sqrt(re * re + im * im); }

// 2^e as a double, 0 below the range.
double pow2(int e) { return e < -1022 ? 0.0 : std::ldexp(1.0, std::min(e, 1023)); }

// The same for n radii at once.
void sums_pow(const double* a, int lo, int hi, const double* rho, int n, double* out) {
  for (int i = 0; i < n; i++) out[i] = 0.0;
  for (int k = hi; k >= lo; k--)
    for (int i = 0; i < n; i++) out[i] = out[i] * rho[i] + a[k];
  for (int k = 0; k < lo; k++)
    for (int i = 0; i < n; i++) out[i] *= rho[i];
}

// Coefficients of eps^b x^k, times 2^s, for orders b < NB.
template <int NB>
struct Poly {
  double re[NB][D + 1], im[NB][D + 1];
  int s;
};

// sum_k a[k] rho^k over [lo, hi].
double sum_pow(const double* a, int lo, int hi, double rho) {
  double s = 0.0;
  for (int k = hi; k >= lo; k--) s = s * rho + a[k];
  for (int k = 0; k < lo; k++) s *= rho;
  return s;
}

// The record of polynomial u (index n) for |x| <= rho 2^p, its bound q on
// everything but the device's evaluation; eps: the largest |eps|.
template <int NB>
bool make_record(const Poly<NB>& u, int fire, int n, int p, double rho, double q, double eps,
                 JumpRec& r) {
  // x in units of 2^pr with rho in (1/2, 1], the linear coefficient in [1, 2)
  int sh = std::ilogb(rho) + 1;
  if (std::ldexp(rho, -sh) == 0.5) sh--;
  const double rr = std::ldexp(rho, -sh);
  const int k0 = std::ilogb(norm(u.re[0][1], u.im[0][1])) + sh;
  double mag[D + 1] = {}, err = 0.0, lip = 0.0, lip_eps = 0.0, lip2 = 0.0, rk = 1.0;
  JumpRec o{};
  for (int k = 1; k <= D; k++) {
    const double re = std::ldexp(u.re[0][k], sh * k - k0);
    const double im = std::ldexp(u.im[0][k], sh * k - k0);
    const double m = norm(re, im);
    lip += k * m * rk;
    o.d[k - 1] = {(float)(k * re), (float)(k * im)};
    if (k > 1) lip2 += 0.5 * k * (k - 1) * m * rk / rr;
    rk *= rr;
    if (!(m < 0x1p100)) return false;
    if (m < 0x1p-100) {  // far below the bound's own terms
      err += m * rk;
      continue;
    }
    mag[k] = m;
    if (k <= kJumpExact) {
      Flt4& b = o.b[k - 1];
      b.x = (float)re;
      b.y = (float)(re - (double)b.x);
      b.z = (float)im;
      b.w = (float)(im - (double)b.z);
    } else {
      o.c[k - kJumpExact - 1] = {(float)re, (float)im};
    }
    // plain FP32: the coefficient, x^k, and at most 3 of 2^-24 a Horner step on
    // the partial sums it is part of
    if (k > kJumpExact) err += (8.0 + 4.0 * k) * 0x1p-24 * m * rk;
  }
  // the orders of eps in plain FP32, coefficients times 2^-32b for (2^32 eps)^b
  Flt2* const tab[B] = {nullptr, o.q1, o.q2, o.q3, o.q4};
  for (int b = 1; b < NB; b++) {
    rk = std::pow(std::ldexp(eps, 32), b);
    for (int k = 0; k < kTerms[b]; k++) {
      const int e = sh * k - k0 - 32 * b;
      const double re = std::ldexp(u.re[b][k], e), im = std::ldexp(u.im[b][k], e);
      const double m = norm(re, im);
      if (!(m < 0x1p100)) return false;
      tab[b][k] = {(float)re, (float)im};
      const bool ff = b == 1 && k < kEpsExact;
      if (ff) o.q1l[k] = {(float)(re - (double)(float)re), (float)(im - (double)(float)im)};
      // rounded: the coefficient, y^k, at most 3 of 2^-24 a Horner step on the
      // partial sums it is part of, and the product and sum with the next order
      err += ((8.0 + 4.0 * (k + 2.0 * b)) * (ff ? 0x1p-43 : 0x1p-24) * m + 0x1p-100) * rk;
      // d / dx of it, at most, which the device does not evaluate, and half d2 / dx2
      if (k > 0) lip_eps += k * m * rk / rr;
      if (k > 1) lip2 += 0.5 * k * (k - 1) * m * rk / (rr * rr);
      rk *= rr;
    }
  }
  // Horner in float-float: p_k = p_{k+1} x + b_k rounds by at most
  // u (|p_{k+1}|_1 |x|_1 + |b_k|_1) <= 2 u m_k with m_k = |b_k| + rho m_{k+1}
  // (u = 1.125 * 2^-43, fe_core.cuh), then is multiplied by x k times; x (its
  // last operation included) and b_k are float-float to 2^-45 of themselves
  const double uu = 0x1.2p-43;
  double m = 0.0;
  for (int k = D; k >= 1; k--) {
    m = mag[k] + rr * m;
    rk = std::pow(rr, k);
    if (k <= kJumpExact) err += 2.0 * uu * m * rk;
    err += 0x1p-44 * k * mag[k] * rk;
  }
  err += 2.0 * uu * m * rr;
  err = 1.01 * (err + std::ldexp(q, -k0));
  // (a bound above a thousand FP32 steps' rounding is not worth the jump)
  if (!(err < 0x1p-31)) return false;
  o.fire = fire;
  o.n = n;
  o.p = p + sh;
  o.s = u.s + k0;
  o.unit = (float)pow2(-o.p);
  o.scale = (float)pow2(o.s);
  o.rho2 = (float)(rr * rr * (1.0 - 0x1p-20));
  o.err = std::nextafter((float)err, INFINITY);
  // the device's FP32 derivative of order 0 (of its terms' sum, at most 2^-18 in
  // the Horner steps and 2^-21 in the norm) and the orders of eps
  o.slack = (float)(1.01 * (0x1p-17 * lip + lip_eps));
  o.lip2 = (float)(2.0 * lip2);
  r = o;
  return true;
}

// Adds order c times order b - c of u to order b of its square, the terms kept.
template <int b, int c, int NB>
inline void add_product(const Poly<NB>& u, double* sr, double* si) {
  constexpr int m = kTerms[c], n = kTerms[b - c], keep = kTerms[b];
  constexpr bool square = 2 * c == b;
  const double *yr = u.re[b - c], *yi = u.im[b - c];
  for (int i = 0; i < m; i++) {
    // a square's pairs once: j >= i
    const int lo = square ? i : 0, mid = std::min(n, std::max(lo, keep - i));
    const double xr = 2.0 * u.re[c][i], xi = 2.0 * u.im[c][i];
    for (int j = lo; j < mid; j++) {
      sr[i + j] += xr * yr[j] - xi * yi[j];
      si[i + j] += xr * yi[j] + xi * yr[j];
    }
    if (square && 2 * i < keep) {  // and the diagonal half
      sr[2 * i] -= 0.5 * (xr * yr[i] - xi * yi[i]);
      si[2 * i] -= 0.5 * (xr * yi[i] + xi * yr[i]);
    }
  }
  if constexpr (2 * (c + 1) <= b) add_product<b, c + 1>(u, sr, si);
}

// One step, u' = 2 X u + F (u^2) + eps (eps_x: of order 0's x, as start jumps
// have it; else of order 1's constant), over orders [0, nb).
template <int b, int NB>
inline void step_order(const Poly<NB>& u, int nb, double xr, double xi, double F, Poly<NB>& o) {
  double sr[D + 1] = {}, si[D + 1] = {};
  add_product<b, 0>(u, sr, si);
  for (int k = 0; k < kTerms[b]; k++) {
    o.re[b][k] = 2.0 * (xr * u.re[b][k] - xi * u.im[b][k]) + F * sr[k];
    o.im[b][k] = 2.0 * (xr * u.im[b][k] + xi * u.re[b][k]) + F * si[k];
  }
  if constexpr (b + 1 < NB) {
    if (b + 1 < nb) step_order<b + 1>(u, nb, xr, xi, F, o);
  }
}
template <int NB>
void step_poly(Poly<NB>& u, int nb, double xr, double xi, double F, double eps_x) {
  Poly<NB> o;
  o.s = u.s;
  step_order<0>(u, nb, xr, xi, F, o);
  o.re[0][1] += eps_x;
  if constexpr (NB > 1) {
    if (nb > 1) o.re[1][0] += 1.0;
    for (int b = nb; b < NB; b++) {
      std::fill(o.re[b], o.re[b] + kTerms[b], 0.0);
      std::fill(o.im[b], o.im[b] + kTerms[b], 0.0);
    }
  }
  u = o;
}

// What a square drops at radius rho, out[b] = the sum over the pairs of order b's
// terms |u_i| |u_j| rho^(i + j) beyond its degree (a: the coefficients' magnitudes).
// At a radius t rho, t <= 1, it is at most t^kTerms[b] of that: the least power it
// has.  (The sums by degree, taken at each radius, cost as much again as the step.)
template <int NB>
void dropped_by_square(const double (*a)[D + 1], int nb, double rho, double* out) {
  double A[NB][D + 1], S[NB][D + 2];
  for (int b = 0; b < nb; b++) {
    double p = 1.0;
    for (int k = 0; k < kTerms[b]; k++) {
      A[b][k] = a[b][k] * p;
      p *= rho;
    }
    S[b][kTerms[b]] = 0.0;
    for (int k = kTerms[b] - 1; k >= 0; k--) S[b][k] = S[b][k + 1] + A[b][k];
  }
  for (int b = 0; b < nb; b++) {
    double sum = 0.0;
    for (int c = 0; c <= b; c++)
      for (int i = 0; i < kTerms[c]; i++) {
        const int j = std::max(0, kTerms[b] - i);
        if (j < kTerms[b - c]) sum += A[c][i] * S[b - c][j];
      }
    out[b] = sum;
  }
}

// x^n for the numbers of terms.
double power(double x, int n) {
  double p = 1.0;
  for (; n; n >>= 1, x *= x)
    if (n & 1) p *= x;
  return p;
}

// With x' = x + theta eps, theta = the constant of order 1 over the linear
// coefficient, order 1 loses its constant: u(x' - theta eps) re-expanded,
//   u'_b,k = sum_m (-theta)^m binom(k + m, m) u_{b-m},{k+m},
// to the terms kept.
struct Shift {
  double tr, ti, tm;       // theta, |theta|
  double d[B + 1][D + 1];  // dropped, by order (the last: beyond the orders) and degree
  double dp[D + 1];        // |u_0'|
  double kept[B][D + 1];   // the magnitudes summed in what is kept
  void recentre(Poly<B>& u, int nb) {
    const double m2 = u.re[0][1] * u.re[0][1] + u.im[0][1] * u.im[0][1];
    tr = (u.re[1][0] * u.re[0][1] + u.im[1][0] * u.im[0][1]) / m2;
    ti = (u.im[1][0] * u.re[0][1] - u.re[1][0] * u.im[0][1]) / m2;
    tm = norm(tr, ti);
    Poly<B> o{};
    o.s = u.s;
    for (int b = 0; b <= nb; b++) {
      std::fill(d[b], d[b] + D + 1, 0.0);
      for (int k = 0; k <= D; k++) {
        double cr = 1.0, ci = 0.0, cm = 1.0, sr = 0.0, si = 0.0, sm = 0.0;
        for (int m = 0; m <= b; m++) {
          if (k + m <= D && b - m < nb && k + m < kTerms[b - m]) {
            const double x = u.re[b - m][k + m], y = u.im[b - m][k + m];
            sr += cr * x - ci * y;
            si += cr * y + ci * x;
            sm += cm * norm(x, y);
          }
          const double f = (double)(k + m + 1) / (m + 1);
          const double t = -f * (cr * tr - ci * ti);
          ci = -f * (cr * ti + ci * tr);
          cr = t;
          cm *= f * tm;
        }
        if (b < nb && k < kTerms[b]) {
          o.re[b][k] = sr;
          o.im[b][k] = si;
        } else {
          // beyond the orders: a shift of at most 2^-5 of the ball (as the
          // chain takes), each further one is less than half the one before
          d[b][k] = b < nb ? sm : 2.0 * sm;
        }
        if (b < nb) kept[b][k] = k < kTerms[b] ? sm : 0.0;
      }
    }
    for (int k = 0; k < D; k++) dp[k] = (k + 1) * norm(u.re[0][k + 1], u.im[0][k + 1]);
    dp[D] = 0.0;
    o.re[1][0] = o.im[1][0] = 0.0;
    u = o;
  }
  double dropped(int nb, double rho, double eps) const {
    double s = 0.0;
    for (int b = nb; b >= 0; b--) s = s * eps + sum_pow(d[b], 0, D, rho);
    return s;
  }
  // The same for any shift, u the polynomial before it: all of the expansion,
  // sum_b eps^b |u_b|(rho + |theta| eps), less what is kept (and 2^-46 of it for
  // the difference's own rounding).
  double dropped_any(const Poly<B>& u, int nb, double rho, double eps) const {
    double all = 0.0, in = 0.0, a[D + 1];
    for (int b = nb - 1; b >= 0; b--) {
      for (int k = 0; k <= D; k++) a[k] = k < kTerms[b] ? norm(u.re[b][k], u.im[b][k]) : 0.0;
      all = all * eps + sum_pow(a, 0, D, rho + tm * eps);
      in = in * eps + sum_pow(kept[b], 0, D, rho);
    }
    return std::max(0.0, all - in) + 0x1p-46 * all;
  }
  // of the terms moved, theta eps u_0' above all
  double rounding(double rho, double eps) const {
    return 0x1p-47 * tm * eps * sum_pow(dp, 0, D, rho);
  }
};

struct Start {
  int fire;
  double hi, lo;  // |eps| of the class's samples, in units of 2^p: (lo, hi]
};

// The radii of a class's records: steps of 2^-1/4 to half, then octaves.
double sub_radius(double hi, int i) {
  for (int k = 0; k < i; k++) hi *= k < 4 ? 0.84089641525371461 : 0.5;
  return hi;
}

void build_class(const OrbitData& od, const Start& st, int p, JumpRec* out, int* stop) {
  *stop = -1;
  const int f = std::max(1, st.fire - 3) - 1;
  const int last = od.xlen - 2;
  if (f < 1 || f >= last) return;
  Poly<1> u{};
  {
    const CFE t[3] = {od.a_fe[f], od.b_fe[f], od.c_fe[f]};
    u.s = t[0].e + p;  // the linear term's exponent
    for (int k = 1; k <= 3; k++) {
      const int e = t[k - 1].e + k * p - u.s;
      if (e > 900) return;
      u.re[0][k] = e < -1000 ? 0.0 : std::ldexp(t[k - 1].re, e);
      u.im[0][k] = e < -1000 ? 0.0 : std::ldexp(t[k - 1].im, e);
    }
  }
  double a[1][D + 1] = {};
  for (int k = 1; k <= 3; k++) a[0][k] = norm(u.re[0][k], u.im[0][k]);
  if (!(a[0][1] > 0.0)) return;
  double rho[kJumpSubs], R[kJumpSubs], Q[kJumpSubs], P[kJumpSubs];
  bool alive[kJumpSubs];
  for (int i = 0; i < kJumpSubs; i++) {
    rho[i] = sub_radius(st.hi, i);
    alive[i] = rho[i] > 0.0 && (i == 0 || rho[i] > st.lo);
    R[i] = P[i] = 0.0;
    // the FP64 path's rounding of its start
    Q[i] = 0x1p-49 * sum_pow(a[0], 1, 3, rho[i]);
  }
  Poly<1> prev = u;
  double prev_q[kJumpSubs] = {}, fall[kJumpSubs] = {};  // (rho[i] / rho[top])^kTerms[0]
  int top = -1;
  for (int n = f; n <= last; n++) {
    if (u.s < -900) return;  // the products below would leave the double range
    const double xr = od.xhi[n].x, xi = od.xhi[n].y, xm = norm(xr, xi) * (1.0 + 0x1p-50);
    const double F = pow2(u.s);
    for (int k = 1; k <= D; k++) a[0][k] = norm(u.re[0][k], u.im[0][k]);
    bool any = false;
    sums_pow(a[0], 1, D, rho, kJumpSubs, P);
    for (int i = 0; i < kJumpSubs; i++) {
      if (!alive[i]) continue;
      const double dmax = (P[i] + R[i] + Q[i]) * F;
      // the FP64 path has this sample at the same orbit index: it does not
      // rebase while |delta| < |X| - |delta|, nor bail out below 1000
      const bool good = R[i] <= kTail * a[0][1] * rho[i] && Q[i] <= 0x1p-20 * a[0][1] * rho[i] &&
                        xm > 2.1 * dmax && xm + dmax < 1000.0;
      if (!good || n == last) {
        alive[i] = false;
        if (*stop < 0 && !(xm > 2.1 * dmax)) *stop = n;
        if (n - 1 - f >= kMinSteps)
          make_record(prev, st.fire, n - 1, p, rho[i], prev_q[i], 0.0, out[i]);
        continue;
      }
      any = true;
    }
    if (!any) return;
    prev = u;
    std::copy(Q, Q + kJumpSubs, prev_q);
    const double eps = pow2(p - u.s);  // eps = x 2^p
    step_poly(u, 1, xr, xi, F, eps);
    if (top < 0 || !alive[top]) {
      for (top = 0; !alive[top];) top++;
      for (int i = top; i < kJumpSubs; i++) fall[i] = power(rho[i] / rho[top], kTerms[0]);
    }
    double drop = 0.0;
    dropped_by_square<1>(a, 1, rho[top], &drop);
    for (int i = 0; i < kJumpSubs; i++) {
      if (!alive[i]) continue;
      const double h = F * drop * fall[i];
      // R: (p + R)^2 = p^2 + (2p + R) R, and p^2's terms beyond the degree
      R[i] = (2.0 * xm + F * (2.0 * P[i] + R[i])) * R[i] + h;
      // Q adds, a step: the FP64 path's rounding and its truncated orbit,
      // 2^-50 (2|X| + |d|)|d| + 2^-52 |eps|; the coefficients' rounding, 2^-50
      // of 2|X| p for the products and sums, 2^-47 of p^2 for the at most D
      // products of a convolution, and 2^-51.5 of 2|X| p for the truncated
      // orbit: 2.36 * 2^-50 of 2|X| p and 9 * 2^-50 of p^2
      Q[i] = (2.0 * xm + F * (2.0 * P[i] + Q[i])) * Q[i] + h +
             0x1p-50 * (2.5 * 2.0 * xm * P[i] + 9.5 * F * P[i] * P[i]) + 0x1p-51 * eps * rho[i];
    }
    const double big = std::fabs(u.re[0][1]) + std::fabs(u.im[0][1]);
    if (!(big < 0x1p200) || !(big > 0.0)) return;
    if (big > 0x1p30 || big < 0x1p-30) {
      const int sh = std::ilogb(big);
      for (int k = 1; k <= D; k++) {
        u.re[0][k] = std::ldexp(u.re[0][k], -sh);
        u.im[0][k] = std::ldexp(u.im[0][k], -sh);
      }
      for (int i = 0; i < kJumpSubs; i++) {
        R[i] = std::ldexp(R[i], -sh);
        Q[i] = std::ldexp(Q[i], -sh);
      }
      u.s += sh;
    }
  }
}

}  // namespace

// The stop indexes in use, from the outermost samples inward, in units of 2^p with
// |eps| <= hi0 2^p, hi0 in [1/2, 1).
static std::vector<Start> starts_of(const OrbitData& od, double eps_m, int p) {
  const double hi0 = std::ldexp(eps_m, -(std::ilogb(eps_m) + 1));
  // fire = i for T_i < |eps|^2 <= T_{i-1}, T the prefix minima of the thresholds
  auto radius = [&](int i) {  // sqrt(T_i) in units of 2^p (infinite: 4)
    const RFE& t = od.sa_min_fe[i];
    if (std::isinf(t.m)) return 4.0;
    if (!(t.m > 0.0)) return 0.0;
    const int e = t.e - 2 * p, odd = e & 1;
    const int k = (e - odd) / 2 + std::ilogb(t.m) / 2;
    if (k > 4) return 4.0;
    if (k < -200) return 0.0;
    return std::sqrt(std::ldexp(t.m, odd)) * pow2((e - odd) / 2);
  };
  std::vector<Start> starts;
  double above = std::min(hi0, radius(1));
  int i = 1;
  while ((int)starts.size() < kJumpClasses && above > 0x1p-12) {
    int lo = i, hi = od.xlen;  // the first index past i with a threshold below `above`
    while (lo < hi) {
      const int mid = (lo + hi) / 2;
      if (radius(mid) < above)
        hi = mid;
      else
        lo = mid + 1;
    }
    if (lo >= od.xlen) break;
    const double r = radius(lo);
    starts.push_back({lo, above * (1.0 + 0x1p-16), r});
    above = r;
    i = lo;
  }
  return starts;
}

// The mean of the steps that start jumps save over |eps| <= hi0 2^p.
static double mean_steps(const std::vector<Start>& starts, const std::vector<JumpRec>& recs,
                         double hi0) {
  double sum = 0.0;
  for (size_t k = 0; k < starts.size(); k++) {
    const int f = std::max(1, starts[k].fire - 3) - 1;
    double x = starts[k].hi;
    for (int i = 0; i < kJumpSubs; i++) {
      const double in = i + 1 < kJumpSubs ? sub_radius(starts[k].hi, i + 1) : starts[k].lo;
      const double y = std::max(starts[k].lo, std::min(x, in));
      if (recs[k * kJumpSubs + i].rho2 > 0.0f) sum += (x * x - y * y) * (recs[k * kJumpSubs + i].n - f);
      x = y;
    }
  }
  return sum / (hi0 * hi0);
}

// The classes in use first: the device stops at the first unused one, and
// knows a class by its first record.
static void pack_starts(const std::vector<Start>& starts, std::vector<JumpRec>& out,
                        const JumpRec& none) {
  size_t at = 0;
  for (size_t k = 0; k < starts.size(); k++) {
    JumpRec* r = &out[k * kJumpSubs];
    bool used = false;
    for (int j = 0; j < kJumpSubs; j++) used |= r[j].fire >= 0;
    if (!used) continue;
    for (int j = 0; j < kJumpSubs; j++) r[j].fire = starts[k].fire;
    if (at != k) std::copy(r, r + kJumpSubs, &out[at * kJumpSubs]);
    at++;
  }
  for (size_t k = at * kJumpSubs; k < out.size(); k++) out[k] = none;
}

namespace {

// The records of the chain that starts at orbit index s (X[s]) from delta = x,
// x the whole of it; out: kChainClasses records.  stop: where its balls ended at
// an element of the orbit near 0, most often (-1: nowhere).
void build_chain(const OrbitData& od, int s, double eps, JumpRec* out, int* stop) {
  constexpr int C = kChainClasses;
  *stop = -1;
  const int last = std::min(od.xlen - 2, s + kChainReach);
  // an order of eps weighs at most about 2^9 eps over the smallest ball's 2^-43
  // against the one before: as many as come to 2^-50 (below 2^-110 eps itself
  // is far under every bound)
  int nb = 1;
  if (eps >= 0x1p-110) {
    const double ratio = std::ldexp(eps, 52);
    nb = 2;
    for (double t = ratio * ratio; nb < B && t > 0x1p-50; t *= ratio) nb++;
  }
  Poly<B> u{};
  u.re[0][1] = 1.0;
  double rho[C], R[C], Q[C], P[C], E[C], S[C], T[C], order[B][C], epow[2 * B];
  double fall[B][C];  // (rho[i] / rho[first])^kTerms[b]
  int fall_of = -1;   // first, as those were taken
  bool alive[C], open[C];
  epow[0] = 1.0;
  for (int b = 1; b < 2 * B; b++) epow[b] = epow[b - 1] * eps;
  for (int i = 0; i < C; i++) {
    rho[i] = std::exp2(-0.5 * kChainTop - i);
    R[i] = P[i] = E[i] = 0.0;
    // the FP64 path's rounding of the step that gave x
    Q[i] = 0x1p-49 * rho[i];
    alive[i] = open[i] = true;
  }
  double most = 0.0;
  double gr = 0.0, gi = 0.0;  // Gamma: x = delta_s + Gamma eps
  Poly<B> prev = u;
  double prev_q[C] = {}, prev_rho[C] = {}, prev_g[2] = {};
  double a[B][D + 1] = {};
  Shift shift;
  int stops[C], nstops = 0;
  for (int n = s; n <= last; n++) {
    const double xr = od.xhi[n].x, xi = od.xhi[n].y, xm = norm(xr, xi) * (1.0 + 0x1p-50);
    for (int b = 0; b < nb; b++)
      for (int k = 0; k < kTerms[b]; k++) a[b][k] = norm(u.re[b][k], u.im[b][k]);
    const bool end = n == last || !(a[0][D] < 0x1p900) || !(a[0][1] > 0.0);
    // |delta|'s bounds: the polynomial's sums for the classes down to the first
    // that is nearly linear (`lin`).  From there on a smaller ball's nonlinear
    // part is at most the square of the ratio of the radii times that one's, an
    // order of eps its constant and the rest times the ratio.
    int first = 0;
    while (first < C - 1 && !alive[first]) first++;
    int lin = C - 1;
    for (int i = first; i < C; i++) {  // (a guess by the first two terms)
      if (a[0][2] * rho[i] < 0x1p-14 * a[0][1]) {
        lin = i;
        break;
      }
    }
    const int full = lin - first + 1;
    sums_pow(a[0], 1, D, rho + first, full, P + first);
    for (int i = first; i <= lin; i++) E[i] = 0.0;
    double flat = 0.0;
    for (int b = nb - 1; b > 0; b--) {
      sums_pow(a[b], 0, kTerms[b] - 1, rho + first, full, S + first);
      for (int i = first; i <= lin; i++) {
        E[i] = (E[i] + S[i]) * eps;
        order[b][i] = S[i];
      }
      flat = (flat + a[b][0]) * eps;
    }
    const double bend = P[lin] - a[0][1] * rho[lin] + 0x1p-50 * P[lin];
    const double slope = E[lin] * (1.0 + 0x1p-50) - flat;
    for (int i = lin + 1; i < C; i++) {
      const double t = rho[i] / rho[lin];
      P[i] = a[0][1] * rho[i] + bend * t * t;
      E[i] = flat + slope * t;
    }
    bool any = false;
    for (int i = 0; i < C; i++) {
      if (!open[i]) continue;
      // the FP64 path holds the sample at the same orbit index: it does not
      // rebase while |delta| < |X| - |delta|, nor bail out below 1000
      const double d = P[i] + E[i] + R[i] + Q[i];
      const bool near = n > s && !(xm > 2.1 * d);
      const bool good = alive[i] && !end && R[i] <= kTail * a[0][1] * rho[i] &&
                        Q[i] <= 0x1p-20 * a[0][1] * rho[i] && !near && xm + d < 1000.0;
      if (good) {
        any = true;
        continue;
      }
      open[i] = false;
      if (near && alive[i] && n - s > 256) stops[nstops++] = n;
      if (n - 1 - s < kMinSteps) continue;
      // the record's own Gamma, which takes the constant of order 1 out
      Poly<B> at = prev;
      double r = prev_rho[i], q = prev_q[i];
      shift.tr = shift.ti = 0.0;
      if (nb > 1) {
        shift.recentre(at, nb);
        if (shift.tm * eps < 0x1p-3 * r) {
          r -= shift.tm * eps;
          q += shift.dropped_any(prev, nb, r, eps) + shift.rounding(r, eps);
        } else {
          at = prev;
          shift.tr = shift.ti = 0.0;
        }
      }
      if (!make_record(at, s, n - 1, 0, r, q, nb > 1 ? eps : 0.0, out[i])) continue;
      const double g1 = prev_g[0] + shift.tr, g2 = prev_g[1] + shift.ti;
      Flt4& g = out[i].gamma;
      g.x = (float)g1;
      g.y = (float)(g1 - (double)g.x);
      g.z = (float)g2;
      g.w = (float)(g2 - (double)g.z);
    }
    if (!any) break;
    prev = u;
    std::copy(Q, Q + C, prev_q);
    std::copy(rho, rho + C, prev_rho);
    prev_g[0] = gr;
    prev_g[1] = gi;
    step_poly(u, nb, xr, xi, 1.0, 0.0);
    // the square's terms beyond the degrees and beyond the orders
    while (first < C && !alive[first]) first++;
    if (fall_of != first) {
      fall_of = first;
      for (int i = first; i < C; i++)
        for (int b = 0; b < nb; b++) fall[b][i] = power(rho[i] / rho[first], kTerms[b]);
    }
    double drop[B];
    dropped_by_square<B>(a, nb, rho[first], drop);
    for (int b = 1; b < nb; b++) drop[b] *= epow[b];
    const int from = std::min(first, lin);
    for (int i = from; i <= lin; i++) T[i] = nb == 1 ? eps : 0.0;
    for (int b = 1; b < nb; b++)
      for (int c = nb - b; c < nb; c++)
        for (int i = from; i <= lin; i++) T[i] += order[b][i] * order[c][i] * epow[b + c];
    for (int i = lin + 1; i < C; i++) T[i] = T[lin];
    for (int b = 0; b < nb; b++)
      for (int i = first; i < C; i++) T[i] += drop[b] * fall[b][i];
    // (the balls that have ended among them: for whole vectors)
    for (int i = first; i < C; i++) {
      const double h = T[i];
      const double d = P[i] + E[i];
      R[i] = (2.0 * xm + 2.0 * d + R[i]) * R[i] + h;
      // as build_class, with eps's own terms
      Q[i] = (2.0 * xm + 2.0 * d + Q[i]) * Q[i] + h +
             0x1p-50 * (2.5 * 2.0 * xm * d + 9.5 * d * d) + 0x1p-48 * eps;
    }
    for (int i = first; i < C; i++)
      if (!(R[i] <= 0x1p-6 * P[i])) alive[i] = false;
    if (nb == 1) continue;
    // Recentre (Shift) where the linear coefficient is the largest so far:
    // theta goes with its inverse, and after a near return of the orbit it is
    // small for a while.
    const double m = u.re[0][1] * u.re[0][1] + u.im[0][1] * u.im[0][1];
    if (!(m > most) || !(m < 1e300)) continue;
    // (a constant far below every ball stays)
    if (norm(u.re[1][0], u.im[1][0]) * eps < 0x1p-16 * rho[C - 1] * std::sqrt(m)) continue;
    most = m;
    shift.recentre(u, nb);
    gr += shift.tr;
    gi += shift.ti;
    for (int i = 0; i < C; i++) {
      if (!alive[i]) continue;
      const double r = shift.dropped(nb, rho[i], eps);
      R[i] += r;
      Q[i] += r + shift.rounding(rho[i], eps);
      rho[i] -= shift.tm * eps;
      fall_of = -1;
      // (see Shift::dropped), and half of it in all
      if (rho[i] < 0.5 * std::exp2(-0.5 * kChainTop - i) || shift.tm * eps > 0x1p-5 * rho[i])
        alive[i] = false;
    }
  }
  int count = 0;
  for (int i = 0; i < nstops; i++) {
    int c = 0;
    for (int j = 0; j < nstops; j++) c += stops[j] == stops[i];
    if (c > count) {
      count = c;
      *stop = stops[i];
    }
  }
}

}  // namespace

EpsRange eps_range(const std::vector<double>& re, const std::vector<double>& im) {
  EpsRange r{0.0, 0.0, 0};
  for (double x : re) r.re = std::max(r.re, std::fabs(x));
  for (double y : im) r.im = std::max(r.im, std::fabs(y));
  return r;
}

EpsRange eps_range(const std::vector<RFE>& re, const std::vector<RFE>& im) {
  // every component at the largest exponent
  EpsRange r{0.0, 0.0, -(1 << 30)};
  for (const auto* v : {&re, &im})
    for (const RFE& x : *v)
      if (x.m != 0.0) r.e = std::max(r.e, x.e + std::ilogb(x.m));
  for (const RFE& x : re) r.re = std::max(r.re, std::fabs(std::scalbn(x.m, x.e - r.e)));
  for (const RFE& y : im) r.im = std::max(r.im, std::fabs(std::scalbn(y.m, y.e - r.e)));
  return r;
}

// work(0) .. work(n - 1) on at most `threads` threads, the caller's included.  work
// throws nothing; a thread that cannot be had is done without.
template <class Work>
static void run_on(int threads, size_t n, const Work& work) {
  std::atomic<size_t> next{0};
  auto loop = [&] {
    for (size_t k; (k = next.fetch_add(1)) < n;) work(k);
  };
  const size_t nt = std::min(n, (size_t)std::max(1, threads));
  std::vector<std::thread> pool;
  pool.reserve(nt);
  try {
    for (size_t t = 1; t < nt; t++) pool.emplace_back(loop);
  } catch (...) {  // with those there are
  }
  loop();
  for (std::thread& t : pool) t.join();
}

// Where tables are built, by what a first render of a new view gains less the build
// (2-3 ms on 16 threads for most views; precompute and render together, without -> with,
// on nine views at widths from 1e-13 to 1e-120, and in brackets later renders):
// * grids of 500,000 samples and more: 960x540 at 1e-15 9.2 -> 9.9 ms (7.3 -> 5.4), at
//   3e-17 29.7 -> 30.4 (24.3 -> 22.0), at 2e-13 32.5 -> 32.4, at 1e-20 32.8 -> 29.0;
//   1280x720 from 13.2 -> 12.4 at 1e-15 to 39.8 -> 31.4 at 1e-20;
// * from 2^17 on where the start jumps alone save 0.42e9 steps in all: 517x333 at 1e-20
//   27.5 -> 27.0 (12.4 -> 10.4), at 1e-25 37.4 -> 37.0 (14.6 -> 11.7); at 1e-15, where
//   they do not, it was 7.6 -> 9.9 (5.9 -> 5.4).  That is known only once they are
//   built (1.3 ms in vain at 1e-15), so first the stop index, which they rarely pass,
//   has to allow it;
// * never on smaller grids: 320x240 at 1e-20 24.7 -> 26.2, at 1e-15 6.7 -> 9.4;
// * and nowhere that no sample stops the series: all end about where the reference
//   orbit does (the frames below 1e-16 of a zoom into a center of 15 digits).
constexpr long long kJumpSamples = 500000, kJumpFewSamples = 1 << 17;
constexpr double kJumpStopSteps = 0.7e9, kJumpStartSteps = 0.42e9;

void build_jumps(const OrbitData& od, double eps_m, int eps_e, int threads, JumpTables& t,
                 long long samples) {
  JumpRec none{};
  none.fire = -1;
  none.rho2 = -1.0f;
  auto clear = [&] {
    t.start.assign((size_t)kJumpClasses * kJumpSubs, none);
    t.chain.assign((size_t)kChains * kChainClasses, none);
    t.start_index.assign(kChains, -1);
  };
  clear();
  if (od.xlen < 64 || !(eps_m >= 0.0) || !std::isfinite(eps_m)) return;
  const double eps = eps_e < -1000 ? 0x1p-1000 : std::ldexp(eps_m, eps_e);
  const bool chains = eps < 0x1p-16;
  std::vector<Start> starts;
  int p = 0;
  if (eps_m > 0.0) {
    p = std::ilogb(eps_m) + 1 + eps_e;
    starts = starts_of(od, eps_m, p);
  }
  const bool few = samples < kJumpSamples;
  if (starts.empty() || samples < kJumpFewSamples ||
      (few && (double)samples * starts[0].fire < kJumpStopSteps))
    return;
  // The chain from a rebase, mostly the longest of these, the start classes, and, on
  // threads to spare, the chains that are likely to be wanted next: from past the
  // smallest element of the orbit and past the smallest within a chain's reach.
  std::vector<int> stops(starts.size(), -1);
  int stop[kChains] = {-1, -1, -1};
  std::vector<int> guess;
  if (chains && threads > 2) {
    for (const int reach : {kChainReach, od.xlen}) {
      int at = -1;
      double least = INFINITY;
      for (int n = 64; n < std::min(reach, od.xlen); n++) {
        const double m = od.xhi[n].x * od.xhi[n].x + od.xhi[n].y * od.xhi[n].y;
        if (m < least) {
          least = m;
          at = n;
        }
      }
      if (at >= 0 && std::find(guess.begin(), guess.end(), at + 1) == guess.end())
        guess.push_back(at + 1);
    }
  }
  std::vector<JumpRec> guessed(guess.size() * kChainClasses, none);
  const size_t first = chains ? 1 + guess.size() : 0;
  run_on(threads, first + starts.size(), [&](size_t k) {
    int unused;
    if (chains && k == 0)
      build_chain(od, 0, eps, &t.chain[0], &stop[0]);
    else if (k < first)
      build_chain(od, guess[k - 1], eps, &guessed[(k - 1) * kChainClasses], &unused);
    else
      build_class(od, starts[k - first], p, &t.start[(k - first) * kJumpSubs], &stops[k - first]);
  });
  t.start_steps = mean_steps(starts, t.start, std::ldexp(eps_m, -(std::ilogb(eps_m) + 1)));
  if (few && (double)samples * t.start_steps < kJumpStartSteps) {
    clear();
    return;
  }
  pack_starts(starts, t.start, none);
  if (!chains) return;
  // and the chains from past the elements near 0 at which most start jumps (outermost
  // samples first) and the rebase chain's end
  std::vector<int> from{0};
  auto add = [&](int at) {
    if (at >= 0 && at + 1 + 4 * kMinSteps < od.xlen && (int)from.size() < kChains &&
        std::find(from.begin(), from.end(), at + 1) == from.end())
      from.push_back(at + 1);
  };
  for (size_t k = 0; k < stops.size() && k < 2; k++) add(stops[k]);
  add(stop[0]);
  std::vector<size_t> rest;
  for (size_t k = 1; k < from.size(); k++) {
    const size_t g = std::find(guess.begin(), guess.end(), from[k]) - guess.begin();
    if (g < guess.size())
      std::copy_n(&guessed[g * kChainClasses], kChainClasses, &t.chain[k * kChainClasses]);
    else
      rest.push_back(k);
  }
  run_on(threads, rest.size(), [&](size_t i) {
    const size_t k = rest[i];
    build_chain(od, from[k], eps, &t.chain[k * kChainClasses], &stop[k]);
  });
  for (size_t k = 0; k < from.size(); k++) t.start_index[k] = from[k];
}

}  // namespace nmg
