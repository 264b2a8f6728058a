// FP64 activation of the complex RBM and the deep nets, shared by rbm64.cu and deep.cu.
#pragma once

#include <cuda_runtime.h>

namespace rbmg {

// The rational log-cosh (include/quantum_state/psi_functions.hpp:49-57) in FP64, kept open as
// f + C = A u + n / D(u): u = sign(Re z) z, n / D = (nr + i ni) inv.  FP64 instructions issue
// at 1/64 of the FP32 rate and are all that these kernels wait for, so they are counted: the
// quartic with real coefficients runs on u's trace 2p and norm |u|^2 (11 operations against
// 13 of the complex Horner scheme), the sign is folded in by integer operations, and one
// reciprocal serves both parts: the hardware's estimate (at least 19 bits) and one cubic step
// r (1 + e + e^2), e = 1 - den r, which leaves e^3 < 2^-57.  32 FP64 operations with the
// difference and its sum, against 61 with two divisions.
// All of it is 64 bits, but not the same roundings.  Against 113 bits (emulated, Re z and Im z normal
// with deviation 0.1 / 0.3 / 1 / 3 / 10) the activation's rms error is 5.4e-17 / 4.7e-17 / 6.3e-17 /
// 1.6e-16 / 4.5e-16, with Horner's scheme and divisions 4.6e-17 / 4.2e-17 / 6.9e-17 / 1.6e-16 / 4.5e-16.
// In a whole log psi the angles' sums count for more, and these have fewer roundings by groups of
// spins: 2.5e-16 against 2.4e-16 at N = 12, M = 24, 4.5e-16 / 5.0e-16 at 36, 75, 9.4e-16 / 1.4e-15 at 75, 150,
// 3.0e-15 / 5.4e-15 at 140, 400.  The distance of deep nets, a difference down to the last bits, keeps
// the other order (lc64_plain).
constexpr double kLcC = 0.598139;
constexpr double kLcA = 0.9003320053750442;

__device__ __forceinline__ double rcp64(double den) {
    // |D|^2 overflows for |z| > 1e38 only; the clamp keeps 0 rather than NaN there, as a
    // division does
    const int hi = min(__double2hiint(den), 0x7FD00000);
    den = __hiloint2double(hi, __double2loint(den));
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(den));
    const double e = fma(-den, r, 1.0);
    return fma(r, fma(e, e, e), r);
}

struct Lc64 {
    double p, q, r, n, dr, di, nr, ni, inv;   // u = p + i q, its trace and norm, D(u), numerator conj(D), 1 / |D|^2
    long long flip;                            // the sign bit of Re z where u = -z
    __device__ __forceinline__ double2 open() const { return make_double2(fma(kLcA, p, nr * inv), fma(kLcA, q, ni * inv)); }
    // d += (f + C) - g
    __device__ __forceinline__ void add_difference(double2 g, double2& d) const {
        d.x += fma(kLcA, p, fma(nr, inv, -g.x));
        d.y += fma(kLcA, q, fma(ni, inv, -g.y));
    }
    __device__ __forceinline__ double2 value() const {
        const double2 v = open();
        return make_double2(v.x - kLcC, v.y);
    }
    // my_tanh (psi_functions.hpp:97-114), sign u Q(u) / D(u)^2, from the same D and reciprocal (its
    // D has the constant 10.218021346543315 in place of 10.2180213465)
    __device__ __forceinline__ double2 tanh() const {
        const double b7 = 0.9003320053750442, b6 = fma(r, b7, 6.746450656267947);
        const double b5 = fma(r, b6, fma(-n, b7, 26.632014683761202));
        const double b4 = fma(r, b5, fma(-n, b6, 70.82878897882324));
        const double b3 = fma(r, b4, fma(-n, b5, 146.36284300074402));
        const double b2 = fma(r, b3, fma(-n, b4, 199.24474920889975));
        const double b1 = fma(r, b2, fma(-n, b3, 177.6769746361748));
        const double qr = fma(p, b1, fma(-n, b2, 83.68563506532087)), qi = q * b1;
        const double ur = fma(p, qr, -(q * qi)), ui = fma(p, qi, q * qr);
        // D with my_tanh's constant: D + (10.218021346543315 - 10.2180213465) u
        constexpr double kD = 10.218021346543315 - 10.2180213465;
        const double tr = fma(kD, p, dr), ti = fma(kD, q, di);
        const double sr = fma(tr, tr, -(ti * ti)), si = 2.0 * tr * ti;
        const double i1 = rcp64(fma(tr, tr, ti * ti)), i2 = i1 * i1;
        const double hr = fma(ur, sr, ui * si) * i2, hi = fma(ui, sr, -(ur * si)) * i2;
        return make_double2(__longlong_as_double(__double_as_longlong(hr) ^ flip),
                            __longlong_as_double(__double_as_longlong(hi) ^ flip));
    }
};

__device__ __forceinline__ Lc64 lc64(double2 z) {
    // sign = z.x > 0 ? 1 : -1 (positive doubles are positive integers; zero counts as -1)
    Lc64 f;
    f.flip = __double_as_longlong(z.x) > 0 ? 0ll : static_cast<long long>(0x8000000000000000ull);
    f.p = __longlong_as_double(__double_as_longlong(z.x) ^ f.flip);
    f.q = __longlong_as_double(__double_as_longlong(z.y) ^ f.flip);
    f.r = f.p + f.p;
    f.n = fma(f.q, f.q, f.p * f.p);
    const double b3 = f.r + 3.746646023906276;
    const double b2 = fma(f.r, b3, 7.771429504240965 - f.n);
    const double b1 = fma(f.r, b2, fma(-f.n, b3, 10.2180213465));
    const double dr = f.dr = fma(f.p, b1, fma(-f.n, b2, 9.19376335670885)), di = f.di = f.q * b1;
    const double ur = fma(-2.16564366435, f.p, 5.49914721954), ui = -2.16564366435 * f.q;
    f.nr = fma(ur, dr, ui * di);
    f.ni = fma(ui, dr, -(ur * di));
    f.inv = rcp64(fma(dr, dr, di * di));
    return f;
}

}  // namespace rbmg
