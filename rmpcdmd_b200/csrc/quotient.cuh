// Quotients by a divisor that is used again.
#pragma once
#include <math.h>

namespace rmpcd {

// a / b rounded to nearest, as the division gives it: with y = 1 / b rounded to
// nearest, two corrections by exact residuals give the correctly rounded
// quotient (P. Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", IBM J. Res. Dev. 34(1), 1990); operands near the ends of the
// exponent range, zeros and non-finite ones take the division itself.
struct Quotient {
    double b, y;
    bool safe;
    __host__ __device__ void set(double d)
    {
        b = d;
        y = 1.0 / d;
        safe = fabs(d) > 1e-100 && fabs(d) < 1e100;
    }
    __host__ __device__ __forceinline__ double of(double a) const
    {
        if (!(safe && fabs(a) > 1e-180 && fabs(a) < 1e180)) return a / b;
        double q = a * y;
        q = fma(fma(-b, q, a), y, q);
        return fma(fma(-b, q, a), y, q);
    }
};

}  // namespace rmpcd
