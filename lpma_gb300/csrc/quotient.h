// r / n for a whole n from the rounded reciprocal of n.
#pragma once
#include <cmath>

#ifdef __CUDACC__
#define LPMA_HD __host__ __device__ __forceinline__
#else
#define LPMA_HD inline
#endif

namespace lpma {

// The quotient r / n of a finite r, rounded as a division rounds it, from
// y = 1 / n (rounded): one correction of q = r y by its remainder (Markstein,
// "Computation of elementary functions on the IBM RISC System/6000 processor",
// 1990).  n is a whole number of at most 2^22, so r / n lies no nearer than
// 2^-23 of a last place to a rounding boundary, where the corrected value
// before its rounding is off by some 2^-52 of one.  (Below the normal range
// the last place is not promised.)
LPMA_HD double quotient(double r, double n, double y) {
    const double q = r * y;
    return fma(fma(-q, n, r), y, q);
}

}  // namespace lpma
