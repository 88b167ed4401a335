/*
 * gc_root.h -- x**y, y the double nearest 1/3, for the step-size factor
 * FacSafe / Err**(ONE/ros_ELO) of the cooperative kernel's FMA build.
 *
 * gc_pow's double-double series is a chain of ~1,000 dependent operations, a
 * fifth of an attempt of a single cell.  This starts from c = cbrt(x) and adds
 * the residual of one double-double cube and the difference d between 1/3 and
 * y (x**(1/3 - d) = x**(1/3) (1 - d ln x), d = 1.850371707708594e-17).  The
 * corrections are a few ulp of c and known to their own rounding, so that the
 * one rounding that counts is the last addition: the result is gc_pow's.
 *
 * The residual is a difference of nearly equal numbers.  Its operations are
 * written with the macros of gc_pow.h, which no compiler contracts: x - q as
 * fma(-p, c, x) would already hold the rounding error of q that ql holds too
 * (up to 0.75 ulp, and 8% of the results a rounding off).
 */
#pragma once
#include "gc_pow.h"

/* 0 < x < 1e300 */
GC_HD double gc_root3(double x) {
  const double c = cbrt(x);
  const gc_dd p = gc_two_prod(c, c);
  const gc_dd q = gc_two_prod(p.hi, c);
  const double ql = GC_FMA(p.lo, c, q.lo);
  const double r = GC_SUB(GC_SUB(x, q.hi), ql);
  const double e = GC_SUB(GC_DIV(r, GC_MUL(3.0, p.hi)), GC_MUL(c, GC_MUL(1.850371707708594e-17, log(x))));
  return GC_ADD(c, e);
}
