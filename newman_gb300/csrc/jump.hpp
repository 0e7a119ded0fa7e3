// Jumps of the FP32 path over the steps where delta is small: there delta is a
// polynomial in what it started from to far below the path's own error bound,
// for hundreds to thousands of steps.  Two kinds, both tables of records for
// balls of start values, built on the host at precompute:
//
// * From the series stop .  A class is one series stop index
//   (`fire`, the first unstable term of mandelbrot.cpp:165-181): its samples
//   start at index f = fire - 4 from A_f eps + B_f eps^2 + C_f eps^3 -- the
//   reference's own series, whose B and C are not the Taylor coefficients of
//   the orbit, so that each stop index needs polynomials of its own, in
//   x = eps.  A few indexes cover a view (the 1920x1080x16 view at 1e-12: 8,
//   five of them 98 % of the samples).
//
// * From an orbit index (chains).  Any sample that stands at a chain's first
//   index with delta small jumps, whatever it did before: the first element of
//   the orbit, one step after a rebase with Y small, and the elements past a
//   near return of the orbit to 0 at which other jumps have to end (a sample
//   rebases there or passes with delta small again).  The eps added at each
//   later step acts almost as if Gamma eps were added at the first (Gamma =
//   sum 1 / (dX_k/dX_s) up to the record's index), so x = delta + Gamma eps, and
//   what is left are powers of eps times polynomials of low degree.
//
// The host carries the polynomial of degree kJumpDegree through
// delta' = 2 X delta + delta^2 + eps step by step, with bounds for |x| <= rho on
//   R  the terms left out (beyond the degrees),
//   Q  R, the rounding of the coefficients, the truncation of the FP64 orbit
//      and the rounding of the FP64 path's own steps,
// until R would pass 2^-46 of delta, or the FP64 path could rebase or bail out;
// a record holds the polynomial at the last index before that.
//
// The FP32 path rebases at the steps where the FP64 path does (fe_core.cuh), so
// both hold a sample against the same orbit element.  That matters beyond the
// bounds: the orbit at 64 bits of precision is one of z^2 + c only to 2^-64 a
// step, the same for both paths while they are at the same element.
#pragma once

#include <cmath>
#include <vector>

#include "mpview.hpp"
#include "view_device.cuh"

namespace nmg {

struct JumpTables {
  std::vector<JumpRec> start;    // kJumpClasses * kJumpSubs; unused: fire -1, rho2 -1
  std::vector<JumpRec> chain;    // kChains * kChainClasses (class i: |x|^2 <
                                 // 2^-(kChainTop + 2 i)); unused: rho2 -1
  std::vector<int> start_index;  // kChains: X index each starts at; -1: none
  double start_steps = 0.0;      // that start jumps save, the mean over the disk of |eps|
};

// The largest |component|s of a grid's eps: re 2^e and im 2^e.
struct EpsRange {
  double re, im;
  int e;
  double norm() const { return std::sqrt(re * re + im * im) * (1.0 + 0x1p-40); }
  // as floats, not below them
  float re_limit() const { return std::nextafter((float)std::scalbn(re, e), INFINITY); }
  float im_limit() const { return std::nextafter((float)std::scalbn(im, e), INFINITY); }
};
EpsRange eps_range(const std::vector<double>& re, const std::vector<double>& im);
EpsRange eps_range(const std::vector<RFE>& re, const std::vector<RFE>& im);

// The tables of a precomputed deep view whose `samples` samples have |eps| <= m 2^e,
// on at most `threads` threads; unused throughout where they would not pay for
// themselves in one render (kJumpSamples).
void build_jumps(const OrbitData& od, double eps_m, int eps_e, int threads, JumpTables& t,
                 long long samples = 1ll << 62);

}  // namespace nmg
