// The FP32 path's jumps (jump.hpp: the records and what their bounds hold) on one
// sample: the start jump of the series front and the chain jumps between steps.
// Host and device, so that the host's tests run the device's operations.
#pragma once

#include <cmath>
#include <cstring>

#include "ff32.cuh"
#include "view_device.cuh"

namespace nmg {

constexpr float kFeU = 0x1.2p-43f;    // float-float multiply-add rounding per step (worst case)

// Arithmetic on error bounds, rounded upward.
#if defined(__CUDA_ARCH__)
NM_HD float up_add(float a, float b) { return __fadd_ru(a, b); }
NM_HD float up_mul(float a, float b) { return __fmul_ru(a, b); }
NM_HD float up_fma(float a, float b, float c) { return __fmaf_ru(a, b, c); }
#else
// (to nearest in double, then up)
inline float up_float(double x) {
  const float f = (float)x;
  return (double)f < x ? std::nextafter(f, INFINITY) : f;
}
inline float up_add(float a, float b) { return up_float((double)a + (double)b); }
inline float up_mul(float a, float b) { return up_float((double)a * (double)b); }
inline float up_fma(float a, float b, float c) { return up_float(std::fma((double)a, (double)b, (double)c)); }
#endif

NM_HD int float_bits(float x) {
#if defined(__CUDA_ARCH__)
  return __float_as_int(x);
#else
  int i;
  std::memcpy(&i, &x, 4);
  return i;
#endif
}

// sqrt(x) from the hardware reciprocal square root (relative error below
// 2^-22.9; with the product's rounding within 2^-21).  Below x = 2^-120 the
// result is 2^-60, above sqrt(x): the FE32 step only uses the estimate of |Y|
// as an upper bound (its error amplification, the bailout gap 1024 - |Y|),
// and the flush-to-zero form needs no subnormal handling.
NM_HD float approx_sqrt(float x) {
  float r;
#if defined(__CUDA_ARCH__)
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
#else
  r = 1.0f / std::sqrt(x);
#endif
  return x > 0x1p-120f ? x * r : 0x1p-60f;
}
NM_HD float approx_norm(float x, float y) {
  return approx_sqrt(fmaf(x, x, y * y));
}

// A rebase test |Y|^2 < |delta|^2 nearer to a tie than this may come out unlike in
// FP32 and FP64: the sample ends uncertified unless fe_tie_side decides, so that on the
// others both paths rebase at the same steps for as long as their bound is small.  (The estimates
// are within 2^-20; a bound of 2^-23 |delta| on each path moves the squares by
// 2^-20.)  With a larger bound a sample no longer jumps (fe_chain_jump).
constexpr float kFeTie = 0x1p-19f;
// r2 = |Y|^2 below d2 (1 + kFeTie), d2 = |delta|^2: near the tie, with a bound below
// 2^-23 |delta|.  (Compared as magnitudes: their squares leave the float range from
// |delta| = 2^-52 down.  approx_sqrt's floor only takes in more.)
NM_HD bool fe_tied(float r2, float d2, float err) {
  return r2 >= d2 * (1.0f - kFeTie) && err < 0x1p-23f * approx_sqrt(d2);
}

// The rebase test near its tie, from |Y|^2 - |delta|^2 = Z . (Z + 2 delta): 1 below,
// 0 above, -1 where the FP64 path may see it the other way.  High words alone give
// each product to 2^-22 of itself; the two paths' deltas (each within 2^-23 |delta|)
// move the sum by 2^-21 |Z||delta|; the FP64 path rounds its squares, and Y, by 2^-49
// |delta|^2 in all.  Where Z is small beside delta (past a near return of the orbit to
// 0), |Y|^2 and |delta|^2 agree to 2^-19 for whole regions of a view, and this decides
// them down to |Z| = 2^-27 |delta|: on a 960x540 part of the 1920x1080x16 view at 1e-12
// 16 % of the samples ended there.
NM_HD int fe_tie_side(float zx, float zy, float dx, float dy, float d2) {
  const float s = fmaf(zx, fmaf(2.0f, dx, zx), zy * fmaf(2.0f, dy, zy));
  const float z1 = fabsf(zx) + fabsf(zy);
  // (2^-120: the products keep their bits above it)
  const float band = fmaf(0x1p-20f * z1, fmaf(2.0f, fabsf(dx) + fabsf(dy), z1),
                          fmaf(0x1p-47f, d2, 0x1p-120f));
  return fabsf(s) <= band ? -1 : s < 0.0f ? 1 : 0;
}

struct alignas(16) FeState {
  FF dr, di;      // delta * 2^-E
  FF er, ei;      // eps * 2^-E
  float err;      // error bound of delta, in the same units
  int32_t E;      // 0: unscaled
  int32_t j, i;   // orbit index, iteration count (getIterations' i)
  int32_t certified;
  int32_t frame;  // frame of a batch
  float e64;      // double-loop views: bound on the double loop's own error
  int32_t since;  // steps since the exponent was set (while E != 0)
};

struct CFF {  // ((re) + i (im)) * 2^e, float-float mantissas
  FF re, im;
  int e;
};

NM_HD FF ffe_scaled(float h, float l, int d) {
  if (h == 0.0f || d < -140) return FF{0.0f, 0.0f};
  return ff_scale(FF{h, l}, d);
}

// The polynomial of a jump's record at x (in its units), without the eps part,
// times 2^-s: the first kJumpExact terms in float-float, the rest in FP32 (their
// rounding is in the record's bound).
NM_HD void jump_poly(const JumpRec& rec, FF xr, FF xi, FF& dr, FF& di) {
  constexpr int n = kJumpDegree - kJumpExact;
  float hr = rec.c[n - 1].x, hi = rec.c[n - 1].y;
#pragma unroll
  for (int k = n - 2; k >= 0; k--) {
    const Flt2 c = rec.c[k];
    const float t = fmaf(hr, xr.h, fmaf(-hi, xi.h, c.x));
    hi = fmaf(hr, xi.h, fmaf(hi, xr.h, c.y));
    hr = t;
  }
  FF pr{hr, 0.0f}, pi{hi, 0.0f};
#pragma unroll 1
  for (int k = kJumpExact - 1; k >= 0; k--) {
    const Flt4 b = rec.b[k];
    FF nr, ni;
    ff_cmul_add(pr, pi, xr, xi, FF{b.x, b.y}, FF{b.z, b.w}, nr, ni);
    pr = nr;
    pi = ni;
  }
  ff_cmul_add(pr, pi, xr, xi, FF{0.0f, 0.0f}, FF{0.0f, 0.0f}, dr, di);
}

// The jump (jump.hpp) of a sample that stops the series at `fire`: its delta at
// the jump's index `found`, within `dbound`; false when it has none.
// Bit-for-bit the same start in every kernel.
NM_HD bool fe_jump(const DeviceView& v, int fire, const FFE& er, const FFE& ei, CFF& d,
                   float& dbound, int& found) {
  if (!v.jump) return false;
  const JumpRec* rec = v.jump;
  int c = 0;
  for (; c < kJumpClasses; c++, rec += kJumpSubs) {
    if (rec->fire == fire) break;
    if (rec->fire < 0) return false;
  }
  if (c == kJumpClasses) return false;
  // the smallest radius that holds the sample
  const JumpRec* use = nullptr;
  FF xr{0.0f, 0.0f}, xi{0.0f, 0.0f};
  // (a component that is 0, on the row or column of the reference, has no exponent)
  const int e = er.h == 0.0f ? ei.e : ei.h == 0.0f ? er.e : er.e > ei.e ? er.e : ei.e;
  for (int k = kJumpSubs - 1; k >= 0 && !use; k--) {
    if (!(rec[k].rho2 > 0.0f) || e - rec[k].p > 20) continue;
    xr = ffe_scaled(er.h, er.l, er.e - rec[k].p);
    xi = ffe_scaled(ei.h, ei.l, ei.e - rec[k].p);
    if (fmaf(xr.h, xr.h, xi.h * xi.h) <= rec[k].rho2) use = rec + k;
  }
  // (an x whose square vanishes would lose its own low bits: 2^-40 and below
  // starts at the series stop)
  if (!use || fmaxf(fabsf(xr.h), fabsf(xi.h)) < 0x1p-40f) return false;
  jump_poly(*use, xr, xi, d.re, d.im);
  d.e = use->s;
  dbound = use->err;
  found = use->n;
  return true;
}

// The chain a sample at orbit index j with delta small may jump along, or -1.
NM_HD int fe_chain_at(const DeviceView& v, int j) {
  int k = -1;
#pragma unroll
  for (int c = 0; c < kChains; c++)
    if (j == v.jump_from[c]) k = c;
  return k;
}

// The jump (jump.hpp) of a sample at a chain's first index: its next steps at
// once, where x = delta + Gamma eps lies in the ball of a record.  The bound
// passes through the jump by the polynomial's derivative at x: e' = |d delta/dx| e
// + err, the orders of eps by the largest they reach in the ball.  A bound above 2^-24 |x| keeps the sample from jumping: below it
// every rebase so far was decided alike in both paths (kFeTie).
NM_HD void fe_chain_jump(const DeviceView& v, FeState& st) {
  const int c = fe_chain_at(v, st.j);
  if (c < 0) return;
  const float x2 = fmaf(st.dr.h, st.dr.h, st.di.h * st.di.h);
  if (!(x2 < v.jump_x2) || fabsf(st.er.h) > v.jump_er || fabsf(st.ei.h) > v.jump_ei) return;
  // class i: |x|^2 < 2^-(kChainTop + 2 i), i from the exponent of |delta|^2
  int i = (126 - kChainTop - (float_bits(x2) >> 23)) >> 1;
  const JumpRec* base = v.jump + kJumpClasses * kJumpSubs + c * kChainClasses;
  const FF zero{0.0f, 0.0f};
  const JumpRec* use = nullptr;
  FF sr = zero, si = zero;
  const bool with_eps = fabsf(st.er.h) + fabsf(st.ei.h) > 0x1p-110f;
  // its own class, or up to two larger ones (below the smallest class its bound
  // would be far above delta's own scale)
  for (int t = 0; t < 3 && !use; t++, i--) {
    if (i < 0) return;
    if (i >= kChainClasses || !(base[i].rho2 > 0.0f)) continue;
    // x = delta + Gamma eps, in the record's units
    FF xr = st.dr, xi = st.di;
    if (with_eps) {
      const Flt4 g = base[i].gamma;
      ff_cmul_add(st.er, st.ei, FF{g.x, g.y}, FF{g.z, g.w}, st.dr, st.di, xr, xi);
    }
    const float u = base[i].unit;
    sr = FF{xr.h * u, xr.l * u};
    si = FF{xi.h * u, xi.l * u};
    if (fmaf(sr.h, sr.h, si.h * si.h) <= base[i].rho2) use = base + i;
  }
  if (!use) return;
  const int n = use->n - use->fire;  // steps
  if (st.i + n >= v.N) return;
  // bound of x: delta's, and the product's rounding
  const float el1 = up_add(fabsf(st.er.h), fabsf(st.ei.h));
  const float gl1 = up_add(fabsf(use->gamma.x), fabsf(use->gamma.z));
  const float xl1 = up_add(fabsf(st.dr.h), fabsf(st.di.h));
  float ex = up_fma(kFeU, up_fma(up_mul(2.0f, gl1), el1, xl1), st.err);
  ex = up_add(up_mul(ex, use->unit), 0x1p-100f);
  if (!(ex * ex < 0x1p-48f * fmaf(sr.h, sr.h, si.h * si.h))) return;
  FF dr, di;
  jump_poly(*use, sr, si, dr, di);
  // the orders of eps, and |d delta / dx| at x, in FP32
  const float xh = sr.h, yh = si.h;
  auto horner = [&](const Flt2* c, int m, float& pr, float& pi) {
    pr = c[m - 1].x;
    pi = c[m - 1].y;
    for (int k = m - 2; k >= 0; k--) {
      const float t = fmaf(pr, xh, fmaf(-pi, yh, c[k].x));
      pi = fmaf(pr, yh, fmaf(pi, xh, c[k].y));
      pr = t;
    }
  };
  const float er = st.er.h * 0x1p32f, ei = st.ei.h * 0x1p32f;
  if (with_eps) {
    float qr, qi, tr, ti;
    auto times_eps = [&]() {
      const float t = fmaf(qr, er, -qi * ei);
      qi = fmaf(qr, ei, qi * er);
      qr = t;
    };
    horner(use->q4, kJumpEps4, qr, qi);
    times_eps();
    horner(use->q3, kJumpEps3, tr, ti);
    qr += tr;
    qi += ti;
    times_eps();
    horner(use->q2, kJumpEps2, tr, ti);
    qr += tr;
    qi += ti;
    times_eps();
    // order 1: its first terms in float-float (2^-17 of delta on the 1e-12 view),
    // the later ones and the orders above in FP32
    horner(use->q1 + kEpsExact, kJumpEps1 - kEpsExact, tr, ti);
    const float ur = fmaf(tr, xh, -ti * yh), ui = fmaf(tr, yh, ti * xh);
    FF or_{ur, 0.0f}, oi{ui, 0.0f};
#pragma unroll 1
    for (int k = kEpsExact - 1; k >= 0; k--) {
      const Flt2 c = use->q1[k], l = use->q1l[k];
      or_ = ff_add(or_, FF{c.x, l.x});
      oi = ff_add(oi, FF{c.y, l.y});
      if (k > 0) {
        FF nr, ni;
        ff_cmul_add(or_, oi, sr, si, zero, zero, nr, ni);
        or_ = nr;
        oi = ni;
      }
    }
    or_ = ff_add(or_, FF{qr, 0.0f});
    oi = ff_add(oi, FF{qi, 0.0f});
    const FF er2{er, st.er.l * 0x1p32f}, ei2{ei, st.ei.l * 0x1p32f};
    FF nr, ni;
    ff_cmul_add(or_, oi, er2, ei2, dr, di, nr, ni);
    dr = nr;
    di = ni;
  }
  float gr = 0.0f, gi = 0.0f;
#pragma unroll
  for (int k = kJumpDegree - 1; k >= 0; k--) {
    const Flt2 c = use->d[k];
    const float t = fmaf(gr, xh, fmaf(-gi, yh, c.x));
    gi = fmaf(gr, yh, fmaf(gi, xh, c.y));
    gr = t;
  }
  // its FP32 rounding and the derivative of the orders of eps (slack), and the
  // second derivative over the ball of radius ex
  const float amp = up_fma(use->lip2, ex, up_add(use->slack, approx_norm(gr, gi)));
  const float err = up_fma(amp, ex, use->err);
  const float sc = use->scale;
  st.dr = FF{dr.h * sc, dr.l * sc};
  st.di = FF{di.h * sc, di.l * sc};
  st.err = up_add(up_mul(err, sc), 0x1p-120f);
  st.j += n;
  st.i += n;
}

}  // namespace nmg
