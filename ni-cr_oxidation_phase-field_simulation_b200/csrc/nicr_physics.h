// Pointwise physics of the Ni-Cr oxidation model, shared by host C++ and the
// CUDA kernels. Every expression keeps the reference's operand order and
// association, so that with FMA contraction disabled (nvcc -fmad=false, gcc on
// x86-64 without -march) device and host results are bit-identical to the
// reference's. Reference: 3S = mpi3d-slab/NiCr3D_grains.cpp,
// 2D = mpi2d/NiCr2D_grains.cpp.
#pragma once
#include <cmath>
#include <limits>

#ifdef __CUDACC__
#define NICR_HD __host__ __device__ __forceinline__
#else
#define NICR_HD inline
#endif

namespace nicr {

// struct Physics (3S:73-79). Vm = 1 divides exactly and is left out.
struct Phys {
    static constexpr double W = 1e4, ko = 1e-9, kc = 7.5e-9, kp = 1.7e-10, L = 0.2;
    static constexpr double bmo = 2.21e-16, bmc = 3.5436e-20, boo = 2.21e-18, boc = 3.5436e-21;
    static constexpr double ckO = 2e-10, ckCr = 2e-10, ksp = 1.28e-7;
    static constexpr double bulkO = 0., bulkCr = 0.1986, layerO = 0.0023, layerCr = 0.182;
    static constexpr double oxideO = 0.56300203, oxideCr = 0.35677915;
};

constexpr double PI = 3.14159265358979323846;

// h(phi) interpolation (3S:171) and its derivative (3S:87)
NICR_HD double h(double p) { return p * p * p * (10. - 15. * p + 6. * p * p); }
// the same for the reciprocal form: 10 - 15 p + 6 p^2 = 1 + (p - 1)(6 p - 9), whose
// rounding vanishes with 1 - p (by Horner's rule 6 p - 15 rounds by 8 units of
// the last place of h at p = 1, and a grain boundary's mobility multiplies 1 - h)
NICR_HD double h_fast(double p) { return (p * p) * p * fma(p - 1., fma(6., p, -9.), 1.); }
NICR_HD double hp(double p) { return 30. * p * p * (p - 1.) * (p - 1.); }
// minimum-image offset for a periodic axis (3S:172)
NICR_HD double min_image(double d, double period) { return d - period * round(d / period); }

// chemical free energies (3S:198-206)
NICR_HD double fmetal(double o, double cr) {
    return (6000000. * o * o + 583264.303945031 * cr * cr + 3200000. * o * cr
            - 298432. * o - 97045.64 * cr - 61732.2974223055);
}
NICR_HD double foxide(double o, double cr) {
    return (12000000. * o * o + 7000000. * cr * cr - 13800000. * o * cr
            - 8880000. * o + 2680000. * cr + 1860990.);
}
// chemical potentials without the gradient term (refresh, 3S:604-612)
NICR_HD double mu_o_local(double o, double cr, double hh) {
    return (1. - hh) * (12000000. * o + 3200000. * cr - 298432.) + hh * (24000000. * o - 13800000. * cr - 8880000.);
}
NICR_HD double mu_cr_local(double o, double cr, double hh) {
    return (1. - hh) * (1166528.60789006 * cr + 3200000. * o - 97045.64)
         + hh * (14000000. * cr - 13800000. * o + 2680000.);
}
// mobility(conc, p, gb) (3S:207-215); active_gb is gb when grains are on, else 0,
// gbm1 = gb_factor - 1 evaluated once per run (same value as the reference's).
NICR_HD double mobility(double conc, double hh, double active_gb, double bm, double bo, double gbm1) {
    return conc * ((1. - hh) * bm * (1. + gbm1 * active_gb) + hh * bo);
}
// std::min / std::max / std::clamp tie and NaN semantics
NICR_HD double smin(double a, double b) { return (b < a) ? b : a; }
NICR_HD double smax(double a, double b) { return (a < b) ? b : a; }
NICR_HD double sclamp(double v, double lo, double hi) { return (v < lo) ? lo : (hi < v) ? hi : v; }

// Evolving-grain energy terms (3S:104-113); W = eta_W, A = eta_A
NICR_HD double grain_deta(double e, double S, double phi, double W, double A) {
    return e * (W * (S - (1. - h(phi)) + 2. * (S - e * e)) + A * h(phi));
}
NICR_HD double grain_dphi(double S, double phi, double W, double A) {
    return 0.5 * hp(phi) * (W * (S - (1. - h(phi))) + A * S);
}
NICR_HD double grain_energy_density(double S, double P, double phi, double W, double A) {
    const double H = h(phi), d = S - (1. - H);
    return 0.25 * W * d * d + W * P + 0.5 * A * H * S;
}

// Derived eta coefficients (3S:88-103). Evaluated on the host only.
struct EtaCoef {
    double K, ell, A, scale;
};
inline double reference_gb_width(double fwhm, double dx) {
    return fwhm * dx * std::sqrt(PI) / (2. * std::sqrt(std::log(2.)));
}
inline EtaCoef eta_coef(double fwhm, double dx, double W, double kappa, double penalty) {
    EtaCoef e;
    if (kappa > 0.) e.K = kappa;
    else {
        const double ell = 3. * reference_gb_width(fwhm, dx) / 8.;
        e.K = 2. * W * ell * ell;
    }
    e.ell = std::sqrt(e.K / (2. * W));
    e.A = penalty < 0. ? W : penalty;
    e.scale = reference_gb_width(fwhm, dx) / (8. * e.ell / 3.);
    return e;
}

// Division by a run constant b, correctly rounded (bit-identical to a / b).
// The host stores y = RN(1/b) and the double-word reciprocal zh = RD(1/b),
// zl = RN(1/b - zh) >= 0 (Brisebarre, Muller, Raina, "Accelerating correctly
// rounded floating-point division when the divisor is known in advance",
// IEEE Trans. Comput. 53(8), 2004), also times 2^128 (uh, ul). For b > 0 with
// 2^-60 <= b <= 2^60 and a numerator a:
//   as = a * 2^128                  exact for |a| < 2^895, subnormals included,
//   q0 = RN(as*zh + RN(as*zl))      = RN(a*uh + RN(a*ul)), the same products:
//                                   within (1/2 + 2^-51) ulp of as/b,
//   e  = q0*b - as                  exact: q0 is within one ulp of as/b, and
//                                   as/b >= 2^-1006 keeps its bits normal,
//   qs = RN(q0 - e*y)               = RN(as/b), Markstein's correction theorem
//                                   (IBM J. Res. Dev. 34(1), 1990: q0 within one
//                                   ulp, y within half an ulp of 1/b, exact
//                                   remainder => the correctly rounded quotient),
//   q  = qs * 2^-128                exact whenever a/b is normal or zero.
// For most divisors q0 is RN(as/b) already, whatever the numerator, and
// division_in_two() proves it (the same paper): two operations instead of five.
// The scaling keeps tiny numerators (the tails of diffusing fields) exact.
// Zeros come out with the IEEE sign because zl >= 0 and e is formed as
// q0*b - as. A quotient that is subnormal (qs nonzero below 2^-894, which the
// final scaling would round a second time), infinite or NaN (infinite, NaN or
// huge numerators) is flagged, and so is any quotient of a divisor outside the
// range, whose reciprocals are NaN here. tests/division_check.c restates this
// on the host and checks it against IEEE division, near-midpoint quotients
// included. Sums and products of scaled quotients round as the unscaled ones
// do (a power of two, and sums that reach the subnormal range are exact), so
// the kernels keep quotients scaled through a sum and fold 2^-128 into the
// constant that follows it.
struct DivC {
    double b, rb;      // divisor and y = RN(1/b) (the reciprocal form multiplies by it)
    double uh, ul;     // 2^128 times RD(1/b) and RN(1/b - RD(1/b))
};
struct DivF : DivC {   // numerators in the carried scale too
    double zh, zl;     // RD(1/b) and RN(1/b - RD(1/b))
};
inline bool div_in_range(double b) {
    return std::isnormal(b) && b > 0. && b >= std::ldexp(1.0, -60) && b <= std::ldexp(1.0, 60);
}
inline DivF make_divc(double b) {
    DivF d;
    d.b = b;
    d.rb = 1.0 / b;
    double zh = d.rb;
    double rem = std::fma(-zh, b, 1.0);   // exact: zh is within one ulp of 1/b
    if (rem < 0.) {
        zh = std::nextafter(zh, 0.0);
        rem = std::fma(-zh, b, 1.0);
    }
    d.zh = zh;
    d.zl = rem / b;
    if (!div_in_range(b)) d.zh = d.zl = std::numeric_limits<double>::quiet_NaN();
    d.uh = std::ldexp(d.zh, 128);
    d.ul = std::ldexp(d.zl, 128);
    return d;
}
// Whether RN(X*zh + RN(X*zl)) = RN(X/b) for every numerator. With zl at most
// 2^-52 of zh and two roundings of relative size 2^-53 in X*zl, the sum before
// its rounding lies within 2^-103 of X/b (relative), so it can round otherwise
// only if a rounding midpoint lies that close to X/b. For significands X and Y
// (53-bit integers) midpoints are M/2^s with M odd, 2^53 < M < 2^54 and s = 53
// (X >= Y) or 54; X/Y - M/2^s = k/(2^s Y) with k = 2^s X - M Y an integer, not
// zero, and the distance bounds |k| by 16. Each k leaves few M modulo 2^s:
// those numerators are tried against IEEE division.
inline bool division_in_two(double b) {
    if (!div_in_range(b)) return false;
    int e;
    const double y = std::ldexp(std::frexp(b, &e), 53);   // Y, an integer below 2^53
    const DivF d = make_divc(y);
    const unsigned long long Y = (unsigned long long)y;
    const int t = __builtin_ctzll(Y);
    const unsigned long long Yo = Y >> t;
    unsigned long long inv = Yo;   // 1 / Yo modulo 2^64 (Newton)
    for (int i = 0; i < 6; ++i) inv *= 2 - Yo * inv;
    for (int s = 53; s <= 54; ++s) {
        const unsigned long long mod = 1ull << (s - t), most = 1ull << 54;
        for (int k = -16; k <= 16; ++k) {
            if (k == 0 || t > 4 || k % (1 << t) != 0 || (k / (1 << t)) % 2 == 0) continue;   // M odd needs k / 2^t odd
            // M Y = -k modulo 2^s
            for (unsigned long long M = (0ull - (unsigned long long)(long long)(k / (1 << t))) * inv & (mod - 1); M < most; M += mod) {
                if (M <= (most >> 1)) continue;
                const __int128 n = (__int128)M * (__int128)Y + k;
                const double X = (double)(long long)(n >> s);
                if (X < 0x1p52 || X >= 0x1p53) continue;
                if (std::fma(X, d.zh, X * d.zl) != X / y) return false;
            }
        }
    }
    return true;
}
#ifdef __CUDACC__
// IEEE division kept out of line: it is only the rare fallback, and inlining
// it at every call site would multiply the kernels' instruction footprint.
__device__ __noinline__ double ieee_div(double a, double b);
// the scaled quotient (uncertified) of an unscaled numerator
__device__ __forceinline__ double xdiv_up(double a, const DivC& d) {
    const double q0 = __fma_rn(a, d.uh, __dmul_rn(a, d.ul));
    const double e = __fma_rn(q0, d.b, -__dmul_rn(a, 0x1p128));
    return __fma_rn(-e, d.rb, q0);
}
// and of a scaled one
__device__ __forceinline__ double xdiv_scaled(double as, const DivF& d) {
    const double q0 = __fma_rn(as, d.zh, __dmul_rn(as, d.zl));
    const double e = __fma_rn(q0, d.b, -as);
    return __fma_rn(-e, d.rb, q0);
}
// The same where division_in_two(d.b)
__device__ __forceinline__ double xdiv_up2(double a, const DivC& d) { return __fma_rn(a, d.uh, __dmul_rn(a, d.ul)); }
__device__ __forceinline__ double xdiv_scaled2(double as, const DivF& d) {
    return __fma_rn(as, d.zh, __dmul_rn(as, d.zl));
}
// |qs| in (0, 2^-894): a subnormal quotient; >= 2^1024: infinite or NaN
__device__ __forceinline__ unsigned xdiv_uncertified(double qs) {
    const unsigned u = (unsigned)__double2hiint(qs) & 0x7FFFFFFFu;
    return ((u - 1u) < 0x080FFFFFu || u >= 0x7FF00000u) ? 1u : 0u;
}
// The exact quotient; a flagged one (see DivC) sets `bad` (the value returned
// for it is then not the IEEE quotient), so a caller can test once for a
// whole group of divisions and recompute the group with IEEE division.
__device__ __forceinline__ double xdiv_flag(double a, const DivC& d, unsigned& bad) {
    const double qs = xdiv_up(a, d);
    bad |= xdiv_uncertified(qs);
    return __dmul_rn(qs, 0x1p-128);
}
__device__ __forceinline__ double xdiv(double a, const DivC& d) {
    unsigned bad = 0;
    const double q = xdiv_flag(a, d, bad);
    return bad ? ieee_div(a, d.b) : q;
}
#endif

// Double-double accumulation (Knuth two-sum). Budget sums that the reference
// keeps in 80-bit long double are kept as hi+lo pairs with ~106-bit precision.
struct DD {
    double hi, lo;
};
NICR_HD DD dd_add(DD a, double b) {
    const double s = a.hi + b;
    const double bb = s - a.hi;
    const double err = (a.hi - (s - bb)) + (b - bb);
    const double lo = a.lo + err;
    const double hi = s + lo;
    return DD{hi, lo - (hi - s)};
}
NICR_HD DD dd_add(DD a, DD b) {
    DD r = dd_add(a, b.hi);
    return dd_add(r, b.lo);
}

}  // namespace nicr
