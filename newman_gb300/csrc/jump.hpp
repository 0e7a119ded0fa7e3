// Jumps of the FP32 path over the steps where delta is small: there delta is a
// polynomial in what it started from to far below the path's own error bound,
// for hundreds to thousands of steps.  Two kinds, both tables of records for
// balls of start values, built on the host at precompute:
//
// * From the series stop (build_start_jumps).  A class is one series stop index
//   (`fire`, the first unstable term of mandelbrot.cpp:165-181): its samples
//   start at index f = fire - 4 from A_f eps + B_f eps^2 + C_f eps^3 -- the
//   reference's own series, whose B and C are not the Taylor coefficients of
//   the orbit, so that each stop index needs polynomials of its own, in
//   x = eps.  A few indexes cover a view (the 1920x1080x16 view at 1e-12: 8,
//   five of them 98 % of the samples).
//
// * From a rebase (build_rebase_jumps).  A sample that rebases with Y = w small
//   restarts at Z[0] = 0, and one step later at delta = w^2 + eps: one chain
//   from the orbit's first element serves every rebase of every sample.  The
//   eps added at each later step acts almost as if Gamma eps were added at the
//   first (Gamma = sum 1 / (dX_k/dX_0) up to the record's index), so
//   x = w^2 + (1 + Gamma) eps, and what is left are powers of eps times
//   polynomials of low degree, in plain FP32.
//
// The host carries the polynomial of degree kJumpDegree through
// delta' = 2 X delta + delta^2 + eps step by step, with bounds for |x| <= rho on
//   R  the terms left out (beyond the degrees),
//   Q  R, the rounding of the coefficients, the truncation of the FP64 orbit
//      and the rounding of the FP64 path's own steps,
// until R would pass 2^-46 of delta, or the FP64 path could rebase or bail out;
// a record holds the polynomial at the last index before that.
#pragma once

#include <vector>

#include "mpview.hpp"
#include "view_device.cuh"

namespace nmg {

// The records of a precomputed deep view whose samples have |eps| <= m 2^e:
// kJumpClasses * kJumpSubs of the first kind (unused ones: fire -1, rho2 -1).
void build_start_jumps(const OrbitData& od, double eps_m, int eps_e, int threads,
                       std::vector<JumpRec>& out);

// kRebaseClasses of the second kind (class i: |x|^2 < 2^-(kRebaseTop + 2 i);
// unused ones: rho2 -1).  Empty when the orbit is too short.
void build_rebase_jumps(const OrbitData& od, double eps_m, int eps_e, std::vector<JumpRec>& out);

}  // namespace nmg
