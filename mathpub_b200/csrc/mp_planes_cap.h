// mp_planes_cap.h -- the capacity of a tile's bucket in the residue-plane sieve (mp_planes.cu): plain host
// arithmetic, so that it can be compiled and checked on its own.
#pragma once
#include <math.h>
#include <stdint.h>

// Records that a tile of pt bits (one plane, 30 integers a bit) may get from the bucket primes, in a range that
// begins at plane bit i0.  inv_sum is the sum of 1/q over those primes, qmax the largest of them.
//   e      expected: a prime hits a block of pt bits pt / q times
//   2% and 10 sqrt(e) and 256   the spread of the counts far from 0, and small ones
//   edge   The tile's records are the q u in its pt bits with u coprime to 30, u >= 7 (the primes themselves are no
//          records).  For each u the primes are those of an interval of 30 pt / u integers at x / u, of which
//          the plane takes the eighth in one class mod 30: f(u) = 30 pt / (8 u ln(x / u)) of them.  Near 0 the
//          u are few, from t = max(7, x / qmax) on, and their sum differs from the integral that e stands for.
//          [a, b] holds at most (b - a) 4/15 + 28/15 units mod 30 (worst: 11 .. 19), and f falls with u, so the
//          sum is above the integral by at most 28/15 f(t) = 7 pt / (t ln qmax).  At the smallest t, a range from 0
//          up to 1e14, tiles hold up to 1.13 e; from x = 1000 qmax on the term is below 900 records.
static inline uint32_t plane_bucket_cap(uint32_t pt, double inv_sum, uint64_t i0, uint32_t qmax)
{
    const double e = (double)pt * inv_sum, t = fmax(7.0, 30.0 * (double)i0 / (double)qmax);
    return ((uint32_t)(e * 1.02 + 10.0 * sqrt(e + 1.0) + 256.0 + 7.0 * pt / (t * log((double)qmax))) + 3u) & ~3u;
}
