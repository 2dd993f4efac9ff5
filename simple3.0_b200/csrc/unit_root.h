// unit_root.h -- exp(2 pi i e / n) in double precision, rounded once: the angle is reduced to an
// eighth of a turn in whole numbers, so that the quarter turns are exact, and what is left evaluated
// in extended precision (a rounded angle alone is off by up to 4e-16).  Host code only.
#pragma once

#include <cmath>

namespace pftcc {

inline void unit_root(long long e, long long n, double *c, double *s)
{
    e = ((e % n) + n) % n;
    const long long q = (8 * e + n) / (2 * n), r = 4 * e - q * n;   // e / n = q / 4 + r / (4 n), |r| <= n / 2
    const long double a = 3.141592653589793238462643383279502884L * (long double)r / (long double)(2 * n);
    const double x = (double)cosl(a), y = (double)sinl(a);
    switch (q & 3) {
    case 0: *c = x; *s = y; break;
    case 1: *c = -y; *s = x; break;
    case 2: *c = -x; *s = -y; break;
    default: *c = y; *s = -x; break;
    }
}

}  // namespace pftcc
