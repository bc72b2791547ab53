// FP64 division and square root without branches, for the step kernels.
//
// An IEEE division as the compiler emits it ends in a test and a branch to a
// slow path, so the divisions of one face solve run one after another: 35
// clocks each per SM sub-partition at 16 warps per SM, with or without
// independent work beside them (126 clocks of latency). The routines here
// return the same bits for operands in a wide normal range, as straight-line
// code that the compiler interleaves; operands outside the range raise a flag
// instead of branching, and the caller repeats the whole face, cell or state
// with the plain operators when the flag is up (out-of-line, practically
// never taken). Quotients with a common divisor share its reciprocal: 8
// clocks each after 14 for the reciprocal, 4 for the constants gamma and
// gamma - 1 (the FP64 pipe issues one warp instruction per 2 clocks).
//
// Division: a quotient q of a / b within half a last place and a little, from
// a reciprocal in two parts or corrected once, is corrected by its exact
// remainder, q + (a - b q) y (P. Markstein, Computation of elementary
// functions on the IBM RISC System/6000 processor, IBM J. Res. Dev. 34,
// 1990). With a, b scaled to [1, 2) the value before the last rounding is off
// by 1/2 b |y - 1/b| <= b 2^-55 (1 + 2^-50) last places, and a / b is never
// nearer to a rounding boundary than 2^-53 / b, so the result is the rounded
// quotient where b^2 < 4 (1 - 2^-50): for every b but the last four below 2,
// whose few numerators near a boundary the tests go through. The reciprocal y
// is the hardware's estimate (relative error below 2^-19) after one cubic and
// one linear correction, its error below 2^-105 before the last rounding.
//
// Square root: a cubic step on the pair g ~ sqrt(a), h ~ 1 / (2 sqrt(a)), then
// g + (a - g^2) h from the exact residual (the same paper). With g within 1.5
// last places and the relative error of h below 2^-52 the value before the
// last rounding is off by less than 10 2^-106 (a in [1, 4)); a boundary M
// 2^-53 (M odd) with a 2^106 - M^2 = D is at least |D| / 4 2^-106 away, so
// only |D| < 40 can round wrongly, a few significands as D = -1 mod 8. The
// tests go through all with |D| < 130.
//
// Constants: q = fma(x, zh, x * zl) with zh + zl the reciprocal of c to 106
// bits is correctly rounded for all but listed x (N. Brisebarre, J.-M. Muller,
// S. K. Raina, Accelerating correctly rounded floating-point division when the
// divisor is known in advance, IEEE Trans. Computers 53, 2004); for 5/3, 5/3 -
// 1 and sqrt(4 pi) as doubles the numerators near a rounding boundary (two or
// three significands each) all round correctly.
#pragma once

#include "fluid.cuh"

namespace dgpu {
namespace f64 {

// Ranges. Divisors lie in [2^-120, 2^50), numerators are zero or in [2^-920,
// 2^850): no quotient leaves the normal range and no remainder loses a bit
// that matters. Values ahead of a front fall off through every magnitude down
// to zero. A quotient that is a velocity, a field or a flux component raises
// the flag when its numerator is smaller (quots); one that is only added to
// something of normal size, which it then cannot change, passes as it is
// (quot). A numerator that is infinite, NaN or too large needs no test of its
// own there: it makes the quotient NaN or huge, and the sum, pressure, energy
// or radicand it goes into has a test.
//
// In centimetres and seconds some divisors are far above 2^50. A quotient of
// its own (div) takes divisors below 2^102: its remainders are exact down to
// quotients of 2^-1022, where the second part of a reciprocal has lost its
// bits. The others are a WideRec: a cell width, a pressure, the square of a
// speed, a density times one or two speeds.

constexpr unsigned kNumFloor = (1023u - 920u) << 20;  // 2^-920

// The flag of one face, cell or state. With LOCAL the quotients of small
// numerators are divided by the plain operator on the spot: a branch per group
// of quotients (the shear layer 8 % slower), which the gas ahead of a 3D blast
// repays (its step 7 % faster). Elsewhere a raised flag first repeats the work
// out of line with LOCAL, and with the plain operators if that raises it too.
template <bool LOCAL>
struct Flag {
    static constexpr bool kLocal = LOCAL;
    bool bad = false;
    // |x| in [2^-120, 2^MAX)
    template <unsigned MAX = 50>
    __device__ __forceinline__ void den(double x) {
        const unsigned u = (unsigned)__double2hiint(x) & 0x7fffffffu;
        bad |= u - ((1023u - 120u) << 20) >= ((MAX + 120u) << 20);
    }
    // x in [2^-120, 2^50)
    __device__ __forceinline__ void posden(double x) {
        bad |= (unsigned)__double2hiint(x) - ((1023u - 120u) << 20) >= (170u << 20);
    }
    // x in [2^-400, 2^400)
    __device__ __forceinline__ void pos(double x) {
        bad |= (unsigned)__double2hiint(x) - ((1023u - 400u) << 20) >= (800u << 20);
    }
    // |x| < 2^850 (not a NaN)
    __device__ __forceinline__ void fin(double x) {
        bad |= ((unsigned)__double2hiint(x) & 0x7fffffffu) >= ((1023u + 850u) << 20);
    }
    // x == 0 or |x| in [lo, 2^1770 lo), lo a high word (2^-920, or what num_floor gives)
    __device__ __forceinline__ void num(double x, unsigned lo = kNumFloor) {
        const unsigned u = (unsigned)__double2hiint(x) & 0x7fffffffu;
        const unsigned z = u | (unsigned)__double2loint(x);
        bad |= (u - lo >= (1770u << 20)) && z != 0u;
    }
    __device__ __forceinline__ void raise(bool c) { bad |= c; }
};
using Chk = Flag<false>;

// max(2^-920, 2^-970 |b|) as a high word, of that of |b|: the smallest numerator
// for a divisor of any size.
__device__ __forceinline__ unsigned floor_of(unsigned b) { return max(b, (1023u + 50u) << 20) - (970u << 20); }
// 0 < |x| < lo
__device__ __forceinline__ bool tiny(double x, unsigned lo) {
    const unsigned u = (unsigned)__double2hiint(x) & 0x7fffffffu;
    return u < lo && (u | (unsigned)__double2loint(x)) != 0u;
}
static __device__ __noinline__ double div_plain(double a, double b) { return a / b; }

// 1 / b, rounded. The corrections round down the one case whose exact value
// lies just above a rounding boundary, a significand of all ones: 2^k for 2^k
// (1 + 2^-52).
__device__ __forceinline__ double reciprocal(double b) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
    double e = __fma_rn(-b, y, 1.0);
    y = __fma_rn(y, __fma_rn(e, e, e), y);
    e = __fma_rn(-b, y, 1.0);
    y = __fma_rn(y, e, y);
    const bool ones = ((__double2hiint(b) | (int)0xfff00000) & __double2loint(b)) == -1;
    return __hiloint2double(__double2hiint(y), ones ? 1 : __double2loint(y));
}

// A divisor and its reciprocal in two parts, for several quotients.
struct Rec {
    double b, y, l;
};
// without a look at the range of b
__device__ __forceinline__ Rec rec_of(double b) {
    const double y = reciprocal(b);
    return Rec{b, y, __dmul_rn(y, __fma_rn(-b, y, 1.0))};
}
template <class C>
__device__ __forceinline__ Rec rec(double b, C& ck) {
    ck.den(b);
    return rec_of(b);
}
// of a divisor that is positive (anything else raises the flag)
struct PosRec : Rec {};
template <class C>
__device__ __forceinline__ PosRec posrec(double b, C& ck) {
    ck.posden(b);
    return PosRec{rec_of(b)};
}
// of a divisor in [2^-120, 2^400), whose numerators' floor goes with it: two
// integer instructions (for every divisor 0.5 to 1.8 % of a step)
struct WideRec : Rec {};
template <class C>
__device__ __forceinline__ WideRec widerec(double b, C& ck) {
    ck.template den<400>(b);
    return WideRec{rec_of(b)};
}
__device__ __forceinline__ unsigned num_floor(const Rec&) { return kNumFloor; }
__device__ __forceinline__ unsigned num_floor(const WideRec& r) {
    return floor_of((unsigned)__double2hiint(r.b) & 0x7fffffffu);
}

// The sign a zero quotient takes (the corrections lose it); others have it already.
__device__ __forceinline__ double signed_as(double q, double a, double b) {
    return __hiloint2double(__double2hiint(q) | ((__double2hiint(a) ^ __double2hiint(b)) & (int)0x80000000),
                            __double2loint(q));
}
__device__ __forceinline__ double signed_as(double q, double a, const Rec& r) { return signed_as(q, a, r.b); }
__device__ __forceinline__ double signed_as(double q, double a, const PosRec&) {
    return __hiloint2double(__double2hiint(q) | (__double2hiint(a) & (int)0x80000000), __double2loint(q));
}

// a / r.b, the numerator checked by the caller or known to be in range: the
// quotient from both parts of the reciprocal, corrected once by its remainder
// (a zero without its sign: for values that are not zero, or then added to one
// that is not).
__device__ __forceinline__ double quot(double a, const Rec& r) {
    const double q = __fma_rn(a, r.y, __dmul_rn(a, r.l));
    const double m = __fma_rn(-r.b, q, a);
    return __fma_rn(m, r.y, q);
}
// a / r.b for several values at once.
template <class Q, class C, class... D>
__device__ __forceinline__ void quots(const Q& r, C& ck, D&... a) {
    const unsigned lo = num_floor(r);
    if constexpr (C::kLocal) {
        (ck.fin(a), ...);
        const bool small = (tiny(a, lo) || ...);
        const double n[sizeof...(D)] = {a...};
        ((a = signed_as(quot(a, r), a, r)), ...);
        if (small) {
            int k = 0;
            ((a = div_plain(n[k++], r.b)), ...);
        }
    } else {
        (ck.num(a, lo), ...);
        ((a = signed_as(quot(a, r), a, r)), ...);
    }
}
// a / b, one quotient (the first correction takes the place of the second
// part of the reciprocal), without a look at the ranges or a zero's sign
__device__ __forceinline__ double div_of(double a, double b) {
    const double y = reciprocal(b);
    double q = __dmul_rn(a, y);
    q = __fma_rn(__fma_rn(-b, q, a), y, q);
    return __fma_rn(__fma_rn(-b, q, a), y, q);
}
template <class C>
__device__ __forceinline__ double div(double a, double b, C& ck) {
    ck.num(a);
    ck.template den<102>(b);
    return signed_as(div_of(a, b), a, b);
}

__device__ __forceinline__ double root_of(double a) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a));
    double g = __dmul_rn(a, y), h = __dmul_rn(0.5, y);
    const double r = __fma_rn(-g, h, 0.5);
    const double t = __fma_rn(__dmul_rn(1.5, r), r, r);
    g = __fma_rn(g, t, g);
    h = __fma_rn(h, t, h);
    return __fma_rn(__fma_rn(-g, g, a), h, g);
}
// sqrt(a), a > 0 in range
template <class C>
__device__ __forceinline__ double root(double a, C& ck) {
    ck.raise((unsigned)__double2hiint(a) - ((1023u - 900u) << 20) >= (1800u << 20));
    return root_of(a);
}
// sqrt(a), a >= 0 of a value that a root below 2^-450 cannot change (0 then)
template <class C>
__device__ __forceinline__ double root0(double a, C& ck) {
    const unsigned u = (unsigned)__double2hiint(a);
    const bool z = u < ((1023u - 900u) << 20) || (u == 0x80000000u && __double2loint(a) == 0);
    ck.raise(!z && u >= ((1023u + 900u) << 20));
    return z ? 0.0 : root_of(a);
}

// x / (gamma - 1), x / gamma for x > 0 in range.
__device__ __forceinline__ double by_gm1(double x) {
    return __fma_rn(x, 0x1.7ffffffffffffp+0, __dmul_rn(x, 0x1.0000000000001p-54));
}
__device__ __forceinline__ double by_gamma(double x) {
    return __fma_rn(x, 0x1.3333333333333p-1, __dmul_rn(x, -0x1.47ae147ae1479p-58));
}

// x / sqrt(4 pi) for x >= 0, zero or in range.
__device__ __forceinline__ double by_sq4pi(double x) {
    return __fma_rn(x, 0x1.20dd750429b6dp-2, __dmul_rn(x, 0x1.f189d3b48513cp-56));
}

// ---------------------------------------------------------------------------
// FluidElement's conversions (fluid.cuh has them with the plain operators and
// the reference's lines), the same operand order.

template <bool MHD>
__device__ __forceinline__ double energy(const Prim<double>& w) {
    double E = by_gm1(w.p) + (w.rho * 0.5) * dot3(w.vx, w.vy, w.vz, w.vx, w.vy, w.vz);
    if constexpr (MHD) E += dot3(w.Bx, w.By, w.Bz, w.Bx, w.By, w.Bz) * k1_8pi;
    return E;
}
template <bool MHD>
__device__ __forceinline__ Cons<double> to_cons(const Prim<double>& w) {
    Cons<double> u;
    u.rho = w.rho;
    u.mx = w.vx * w.rho;
    u.my = w.vy * w.rho;
    u.mz = w.vz * w.rho;
    u.E = f64::energy<MHD>(w);
    if constexpr (MHD) { u.Bx = w.Bx; u.By = w.By; u.Bz = w.Bz; }
    else { u.Bx = 0; u.By = 0; u.Bz = 0; }
    return u;
}
// a / (2 b) is half of a / b: a quotient near the smallest normal number, where
// it would not be, does not change E
template <bool MHD, class C>
__device__ __forceinline__ double pressure(const Cons<double>& u, const Rec& r, C& ck) {
    ck.pos(u.E);
    double Eth = u.E - 0.5 * quot(dot3(u.mx, u.my, u.mz, u.mx, u.my, u.mz), r);
    if constexpr (MHD) Eth -= dot3(u.Bx, u.By, u.Bz, u.Bx, u.By, u.Bz) * k1_8pi;
    return kGm1 * Eth;
}
template <bool MHD, class C>
__device__ __forceinline__ Prim<double> to_prim(const Cons<double>& u, const PosRec& r, C& ck) {
    Prim<double> w;
    w.rho = u.rho;
    w.vx = u.mx;
    w.vy = u.my;
    w.vz = u.mz;
    quots(r, ck, w.vx, w.vy, w.vz);
    w.p = f64::pressure<MHD>(u, r, ck);
    if constexpr (MHD) { w.Bx = u.Bx; w.By = u.By; w.Bz = u.Bz; }
    else { w.Bx = 0; w.By = 0; w.Bz = 0; }
    return w;
}
// The flag unless is_physical holds for a state that to_prim gave without
// one (its density is positive and its velocities are finite then).
template <bool MHD, class C>
__device__ __forceinline__ void sound_state(const Prim<double>& w, C& ck) {
    ck.pos(w.p);
    if constexpr (MHD) {
        ck.fin(w.Bx);
        ck.fin(w.By);
        ck.fin(w.Bz);
    }
}
// The plain conversions out of line: of a state whose flag is up.
template <bool MHD>
__device__ __noinline__ void corrected_plain(Prim<double>* w, const Cons<double>* d) {
    *w = dgpu::to_prim<MHD>(dgpu::c_sub<MHD>(dgpu::to_cons<MHD>(*w), *d));
}
// to_prim(to_cons(w) - d): a half state with its transverse correction.
template <bool MHD, bool LOCAL = false>
__device__ __forceinline__ Prim<double> corrected(const Prim<double>& w, const Cons<double>& d) {
    Flag<LOCAL> ck;
    ck.pos(w.p);
    const Cons<double> u = c_sub<MHD>(f64::to_cons<MHD>(w), d);
    Prim<double> r = f64::to_prim<MHD>(u, posrec(u.rho, ck), ck);
    if (ck.bad) {
        Prim<double> t = w;
        const Cons<double> e = d;
        corrected_plain<MHD>(&t, &e);
        r = t;
    }
    return r;
}

// The reciprocals of the cell widths of a 2D or 3D grid.
struct Widths {
    Rec x, y, z;
    bool three, bad;
};
__device__ __forceinline__ Widths widths(int dim, double dx, double dy, double dz) {
    Chk ck;
    Widths d;
    ck.raise(!(dx > 1e-14 && dy > 1e-14 && (dim < 3 || dz > 1e-14)));  // cfl_speed leaves these axes out
    d.three = dim > 2;
    d.x = widerec(dx, ck);  // (of numerators that are speeds: above 2^-275)
    d.y = widerec(dy, ck);
    d.z = widerec(d.three ? dz : 1.0, ck);
    d.bad = ck.bad;
    return d;
}
// cfl_speed of a cell with sound (or fast) speed a, for the sum and the
// maximum over the axes; the p-norm raises the flag.
template <class C>
__device__ __forceinline__ double cfl_speed(const Prim<double>& w, double a, int cfl, const Widths& d, C& ck) {
    ck.raise(d.bad || cfl > 1);
    ck.fin(w.vx);
    ck.fin(w.vy);
    ck.fin(w.vz);
    double s = quot(fabs(w.vx) + a, d.x);
    const double t = quot(fabs(w.vy) + a, d.y);
    s = cfl == 0 ? smax(s, t) : s + t;
    if (d.three) {
        const double t = quot(fabs(w.vz) + a, d.z);
        s = cfl == 0 ? smax(s, t) : s + t;
    }
    return s;
}

// ConservativeState::flux with the pressure given.
template <bool MHD>
__device__ __forceinline__ Cons<double> flux_of(const Cons<double>& u, double p, double vx, double vy, double vz) {
    Cons<double> F;
    F.rho = u.mx;
    F.mx = u.mx * vx;
    F.my = u.my * vx;
    F.mz = u.mz * vx;
    F.mx += p;
    F.E = (u.E + p) * vx;
    if constexpr (MHD) {
        const double pmag = dot3(u.Bx, u.By, u.Bz, u.Bx, u.By, u.Bz) * k1_8pi;
        F.mx += pmag;
        F.E += pmag * vx;
        const double tx = (u.Bx * u.Bx) * k1_4pi, ty = (u.By * u.Bx) * k1_4pi, tz = (u.Bz * u.Bx) * k1_4pi;
        F.mx -= tx;
        F.my -= ty;
        F.mz -= tz;
        F.E -= dot3(vx, vy, vz, tx, ty, tz);
        F.By = u.By * vx - vy * u.Bx;
        F.Bz = u.Bz * vx - vz * u.Bx;
        F.Bx = 0;
    } else {
        F.Bx = 0; F.By = 0; F.Bz = 0;
    }
    return F;
}

// Wave speeds (fluid.cuh), r the reciprocal of the density.
template <class C>
__device__ __forceinline__ double sound_speed(const Prim<double>& w, const Rec& r, C& ck) {
    ck.pos(w.p);
    return root(quot(kGamma * w.p, r), ck);
}
template <class C>
__device__ __forceinline__ double fast_speed(const Prim<double>& w, double Bk, const Rec& r, C& ck) {
    const double c = f64::sound_speed(w, r, ck);
    const double a = by_sq4pi(root0(quot(dot3(w.Bx, w.By, w.Bz, w.Bx, w.By, w.Bz), r), ck));
    const double c2 = c * c, a2 = a * a, ak2 = quot(Bk * Bk, r) * k1_4pi;
    const double s = c2 + a2;
    const double disc = smax(0.0, (s * s) * 0.25 - ak2 * c2);
    return root((c2 + a2) * 0.5 + root0(disc, ck), ck);
}
template <class C>
__device__ __forceinline__ double fast_speed_max(const Prim<double>& w, const Rec& r, C& ck) {
    double Bk;
    if (w.Bx * w.Bx < w.By * w.By) Bk = (w.Bx * w.Bx < w.Bz * w.Bz) ? w.Bx : w.Bz;
    else Bk = (w.By * w.By < w.Bz * w.Bz) ? w.By : w.Bz;
    return f64::fast_speed(w, Bk, r, ck);
}

// The flag unless the conservative state u is physical beyond doubt: its
// pressure test E - m^2 / (2 rho) - B^2 / (8 pi) > 0, rounded as the plain
// test rounds it, follows from the inequality without a division where it
// holds with a margin of 2^-44 E; the states between go to the plain test.
template <bool MHD, class C>
__device__ __forceinline__ void surely_physical(const Cons<double>& u, C& ck) {
    const double m2 = dot3(u.mx, u.my, u.mz, u.mx, u.my, u.mz);
    ck.pos(u.rho);
    ck.pos(u.E);
    double e = u.E * (1.0 - 0x1p-44);
    if constexpr (MHD) {
        const double b2 = dot3(u.Bx, u.By, u.Bz, u.Bx, u.By, u.Bz);
        e -= b2 * k1_8pi;
    }
    ck.raise(!(e * (2.0 * u.rho) > m2));
}

}  // namespace f64
}  // namespace dgpu
