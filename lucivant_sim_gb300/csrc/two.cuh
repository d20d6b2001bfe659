// Host arithmetic on pairs of doubles, for coefficients that many amplitudes are multiplied by.
#pragma once

#include <cmath>

namespace lsg {

// A real as v + e, e what the roundings of the operations that made v left over, to first order. A
// rotation or a diagonal's entry takes some twenty operations from the matrices it comes from, and its
// error is common to all amplitudes it multiplies: coefficients formed in double precision were
// most of a program's error. Each is now rounded once. Measured, 12 seeds of 11 qubits x 20 layers
// of u3 and cx in complex128, against the gates as given (their double matrices) in 80 bits: 2.6e-15
// before, 1.4e-15 now, dense products 1.1e-15; against the gates the angles stand for: 3.3e-15 before,
// 2.9e-15 now, dense products 3.1e-15. The arithmetic on the amplitudes has 0.8e-15 of it.
// (inlined by force: as calls, g++ 13 loses parts of the pairs it holds in vector registers at -O1 and -O2
// with FMA instructions)
#define LSG_INLINE __attribute__((always_inline)) inline
struct Two {
    double v = 0.0, e = 0.0;
    Two() = default;
    Two(double x, double y = 0.0) : v(x), e(y) {}
    double value() const { return v + e; }
};
LSG_INLINE Two operator-(Two a) { return Two(-a.v, -a.e); }
LSG_INLINE Two operator+(Two a, Two b) {
    const double s = a.v + b.v, t = s - a.v;
    return Two(s, ((a.v - (s - t)) + (b.v - t)) + (a.e + b.e));
}
LSG_INLINE Two operator-(Two a, Two b) { return a + -b; }
LSG_INLINE Two operator*(Two a, Two b) {
    const double p = a.v * b.v;
    return Two(p, std::fma(a.v, b.v, -p) + (a.v * b.e + a.e * b.v));
}
LSG_INLINE Two tidy(Two a) {  // v the rounding of the sum (after a cancellation it may not be)
    const double s = a.v + a.e;
    return Two(s, a.e - (s - a.v));
}
LSG_INLINE Two operator/(Two a, Two b) {
    b = tidy(b);
    const double q = a.v / b.v;
    return Two(q, (std::fma(-q, b.v, a.v) + (a.e - q * b.e)) / b.v);
}
LSG_INLINE Two root(Two a) {
    a = tidy(a);
    if (!(a.v > 0.0)) return Two();
    const double r = std::sqrt(a.v);
    return Two(r, (std::fma(-r, r, a.v) + a.e) / (2.0 * r));
}

}  // namespace lsg
