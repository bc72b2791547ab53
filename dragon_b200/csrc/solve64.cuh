// FP64 reconstruction and Riemann solvers of the step kernels on the
// branch-free divisions of fast64.cuh: the same results as muscl() and
// face_flux() bit for bit, but for the exact solver, whose star pressure may
// differ in its last places (exact_f). Each first computes without a branch per division
// and raises a flag on anything out of the ordinary (an operand out of range,
// an unphysical or borderline state, a fallback of the solver); the face or
// cell is then repeated out of line, in the end by the plain routine.
#pragma once

#include "fast64.cuh"
#include "recon.cuh"
#include "riemann.cuh"

namespace dgpu {
namespace f64 {

// n / d for slopes of one sign (on), 0 otherwise. With n at least 2^-900 the
// divisor may lie in [2^-450, 2^120) (div_of needs no more than a normal
// quotient). WIDE: up to 2^400, with n at least 2^-950 d, for a sum of squares.
template <bool WIDE, class C>
__device__ __forceinline__ double slope_quot(double n, double d, bool on, C& ck) {
    const unsigned un = (unsigned)__double2hiint(n) & 0x7fffffffu, ud = (unsigned)__double2hiint(d) & 0x7fffffffu;
    const unsigned lo = WIDE ? floor_of(ud) + (20u << 20) : (1023u - 900u) << 20;
    const bool odd = on && (un - lo >= (1800u << 20) || ud - ((1023u - 450u) << 20) >= ((WIDE ? 850u : 570u) << 20));
    if constexpr (C::kLocal) {
        if (odd) return div_plain(n, d);
    } else {
        ck.raise(odd);
    }
    const double q = div_of(n, on ? d : 1.0);
    return on ? q : 0.0;
}
template <class C>
__device__ __forceinline__ double limit1(int lim, double a, double b, C& ck) {
    switch (lim) {
        case LIM_MC: return lim_mc(a, b);
        // the plain form divides (2 a) b by a + b unless a b <= 0
        case LIM_VANLEER: return slope_quot<false>((2.0 * a) * b, a + b, !(a * b <= 0.0), ck);
        case LIM_SUPERBEE: return lim_superbee(a, b);
        case LIM_VANALBADA: return slope_quot<true>((a * b) * (a + b), a * a + b * b, !(a * b <= 0.0), ck);
        default: return lim_minmod(a, b);
    }
}

// TVD::MUSCL with both predicted states physical (else the flag).
template <bool MHD, class C>
__device__ __forceinline__ void muscl_body(int lim, const Prim<double>& wL, Prim<double>& outL, const Prim<double>& wC,
                                           Prim<double>& outR, const Prim<double>& wR, double dt_dL, double dBx,
                                           double dBy, double dBz, C& ck) {
    Prim<double> dW, L, Rr;
    dW.rho = f64::limit1(lim, wC.rho - wL.rho, wR.rho - wC.rho, ck);
    dW.vx = f64::limit1(lim, wC.vx - wL.vx, wR.vx - wC.vx, ck);
    dW.vy = f64::limit1(lim, wC.vy - wL.vy, wR.vy - wC.vy, ck);
    dW.vz = f64::limit1(lim, wC.vz - wL.vz, wR.vz - wC.vz, ck);
    dW.p = f64::limit1(lim, wC.p - wL.p, wR.p - wC.p, ck);
    L.rho = wC.rho - 0.5 * dW.rho;
    Rr.rho = wC.rho + 0.5 * dW.rho;
    L.vx = wC.vx - dW.vx * 0.5;
    L.vy = wC.vy - dW.vy * 0.5;
    L.vz = wC.vz - dW.vz * 0.5;
    Rr.vx = wC.vx + dW.vx * 0.5;
    Rr.vy = wC.vy + dW.vy * 0.5;
    Rr.vz = wC.vz + dW.vz * 0.5;
    L.p = wC.p - 0.5 * dW.p;
    Rr.p = wC.p + 0.5 * dW.p;
    if constexpr (MHD) {
        dW.Bx = f64::limit1(lim, wC.Bx - wL.Bx, wR.Bx - wC.Bx, ck);
        dW.By = f64::limit1(lim, wC.By - wL.By, wR.By - wC.By, ck);
        dW.Bz = f64::limit1(lim, wC.Bz - wL.Bz, wR.Bz - wC.Bz, ck);
        L.Bx = wC.Bx - dW.Bx * 0.5;
        L.By = wC.By - dW.By * 0.5;
        L.Bz = wC.Bz - dW.Bz * 0.5;
        Rr.Bx = wC.Bx + dW.Bx * 0.5;
        Rr.By = wC.By + dW.By * 0.5;
        Rr.Bz = wC.Bz + dW.Bz * 0.5;
    } else {
        L.Bx = L.By = L.Bz = Rr.Bx = Rr.By = Rr.Bz = 0.0;
    }
    ck.pos(L.p);
    ck.pos(Rr.p);
    const Cons<double> UL = f64::to_cons<MHD>(L), UR = f64::to_cons<MHD>(Rr);
    const double pL = f64::pressure<MHD>(UL, posrec(UL.rho, ck), ck), pR = f64::pressure<MHD>(UR, posrec(UR.rho, ck), ck);
    Cons<double> corr = c_mul<MHD>(c_sub<MHD>(flux_of<MHD>(UR, pR, Rr.vx, Rr.vy, Rr.vz),
                                              flux_of<MHD>(UL, pL, L.vx, L.vy, L.vz)), 0.5 * dt_dL);
    if constexpr (MHD) {
        const double a_s = (Rr.Bx - L.Bx) * dt_dL;
        const double vy = 0.5 * (L.vy + Rr.vy), vz = 0.5 * (L.vz + Rr.vz);
        const double dBy_ = 0.5 * wC.vy * lim_minmod(dBx, -dBy) - 0.5 * vy * a_s;
        const double dBz_ = 0.5 * wC.vz * lim_minmod(dBx, -dBz) - 0.5 * vz * a_s;
        corr.By -= dBy_;
        corr.Bz -= dBz_;
        corr.E -= k1_4pi * (wC.By * dBy_ + wC.Bz * dBz_);
    }
    const Cons<double> oL = c_sub<MHD>(UL, corr), oR = c_sub<MHD>(UR, corr);
    outL = f64::to_prim<MHD>(oL, posrec(oL.rho, ck), ck);
    outR = f64::to_prim<MHD>(oR, posrec(oR.rho, ck), ck);
    sound_state<MHD>(outL, ck);
    sound_state<MHD>(outR, ck);
}

// Out of line, for a cell whose flag is up: with small numerators divided on
// the spot (AGAIN), else with the plain operators.
template <bool MHD, bool AGAIN>
__device__ __noinline__ bool muscl_slow(int lim, const Prim<double>* w3, Prim<double>* out2, double dt_dL, double dBx,
                                        double dBy, double dBz) {
    if constexpr (AGAIN) {
        Flag<true> ck;
        muscl_body<MHD>(lim, w3[0], out2[0], w3[1], out2[1], w3[2], dt_dL, dBx, dBy, dBz, ck);
        if (!ck.bad) return true;
        return muscl_slow<MHD, false>(lim, w3, out2, dt_dL, dBx, dBy, dBz);
    } else {
        return dgpu::muscl<MHD>(lim, w3[0], out2[0], w3[1], out2[1], w3[2], dt_dL, dBx, dBy, dBz);
    }
}

template <bool MHD, bool LOCAL = false>
__device__ __forceinline__ bool muscl(int lim, const Prim<double>& wL, Prim<double>& outL, const Prim<double>& wC,
                                      Prim<double>& outR, const Prim<double>& wR, double dt_dL, double dBx, double dBy,
                                      double dBz) {
    Flag<LOCAL> ck;
    muscl_body<MHD>(lim, wL, outL, wC, outR, wR, dt_dL, dBx, dBy, dBz, ck);
    if (!ck.bad) return true;
    const Prim<double> w3[3] = {wL, wC, wR};
    Prim<double> out2[2];
    const bool ok = muscl_slow<MHD, !LOCAL>(lim, w3, out2, dt_dL, dBx, dBy, dBz);
    outL = out2[0];
    outR = out2[1];
    return ok;
}

// ---------------------------------------------------------------------------
// Hydro solvers

struct FaceSide {
    Rec r;
    Cons<double> U;
    double a, sq, h;  // sound speed, sqrt(rho), enthalpy
};
template <class C>
__device__ __forceinline__ void face_side(const Prim<double>& w, FaceSide& s, C& ck) {
    ck.pos(w.p);
    s.r = posrec(w.rho, ck);
    s.U = f64::to_cons<false>(w);
    s.a = root(quot(kGamma * w.p, s.r), ck);
    s.sq = root(w.rho, ck);
}
// Roe-averaged normal velocity and sound speed (HLL::roeAvg)
template <class C>
__device__ __forceinline__ void roe_mean(const Prim<double>& L, const Prim<double>& Rt, const FaceSide& sL,
                                         const FaceSide& sR, double& vx, double& aM, C& ck) {
    const PosRec rs = posrec(sL.sq + sR.sq, ck);
    const double _sql = quot(sL.sq, rs), _sqr = quot(sR.sq, rs);
    const double rho = sL.sq * sR.sq;
    vx = L.vx * _sql + Rt.vx * _sqr;
    const double vy = L.vy * _sql + Rt.vy * _sqr, vz = L.vz * _sql + Rt.vz * _sqr;
    const double hL = quot(sL.U.E + L.p, sL.r), hR = quot(sR.U.E + Rt.p, sR.r);
    const double H = _sql * hL + _sqr * hR;
    const double a2 = kGm1 * (H - dot3(vx, vy, vz, vx, vy, vz) * 0.5);
    const double ar = a2 * rho;
    ck.pos(ar);
    aM = root(div(kGamma * by_gamma(ar), rho, ck), ck);
}
// x-flux of one side's state
template <class C>
__device__ __forceinline__ Cons<double> side_flux(const Prim<double>& w, const FaceSide& s, C& ck) {
    return flux_of<false>(s.U, f64::pressure<false>(s.U, s.r, ck), w.vx, w.vy, w.vz);
}

// Riemann::HLLC: one path for the supersonic and the star cases, the flux of
// the upwind side plus the star part.
template <class C>
__device__ __forceinline__ Cons<double> hllc(const Prim<double>& L, const Prim<double>& Rt, FaceSide& sL, FaceSide& sR,
                                             C& ck) {
    face_side(L, sL, ck);
    face_side(Rt, sR, ck);
    double vM, aM;
    roe_mean(L, Rt, sL, sR, vM, aM, ck);
    const double sl = smin(L.vx - sL.a, vM - aM), sr = smax(Rt.vx + sR.a, vM + aM);
    const bool out_l = sl >= 0.0, out_r = !out_l && sr <= 0.0;
    const double mr = Rt.rho * (Rt.vx - sr), ml = L.rho * (L.vx - sl);
    const double _pr = Rt.p + Rt.rho * Rt.vx * (Rt.vx - sr), _pl = L.p + L.rho * L.vx * (L.vx - sl);
    double sc = 0.0;
    const bool star = !(out_l || out_r);
    if (star) sc = div(_pr - _pl, mr - ml, ck);
    const bool left = star ? sc > 0.0 : out_l;
    const Prim<double> X = left ? L : Rt;
    const FaceSide S = left ? sL : sR;
    Cons<double> F = side_flux(X, S, ck);
    if (star) {
        const double sx = left ? sl : sr;
        const double w = sx - X.vx;
        const Rec rd = rec(sx - sc, ck);
        Cons<double> U;
        const double rw = S.U.rho * w;
        U.rho = quot(rw, rd);
        U.E = quot(S.U.E * w, rd);
        U.my = S.U.my * w;
        U.mz = S.U.mz * w;
        quots(rd, ck, U.my, U.mz);
        U.Bx = U.By = U.Bz = 0;
        U.mx = U.rho * sc;
        U.E += U.rho * (sc - X.vx) * (sc + div(X.p, rw, ck));
        F = c_add<false>(F, c_mul<false>(c_sub<false>(U, S.U), sx));
    }
    return F;
}

// Riemann::HLL(SL, SR)
template <class C>
__device__ __forceinline__ Cons<double> hll_speeds(const Prim<double>& L, const Prim<double>& Rt, const FaceSide& sL,
                                                   const FaceSide& sR, double sl, double sr, C& ck) {
    const Cons<double> FL = side_flux(L, sL, ck), FR = side_flux(Rt, sR, ck);
    if (sl >= 0.0) return FL;
    if (sr <= 0.0) return FR;
    const Cons<double> n = c_add<false>(c_sub<false>(c_mul<false>(FL, sr), c_mul<false>(FR, sl)),
                                        c_mul<false>(c_sub<false>(sR.U, sL.U), sl * sr));
    Cons<double> F = n;
    quots(rec(sr - sl, ck), ck, F.rho, F.E, F.mx, F.my, F.mz);
    return F;
}
template <class C>
__device__ __forceinline__ Cons<double> hll(const Prim<double>& L, const Prim<double>& Rt, FaceSide& sL, FaceSide& sR,
                                            C& ck) {
    face_side(L, sL, ck);
    face_side(Rt, sR, ck);
    double vM, aM;
    roe_mean(L, Rt, sL, sR, vM, aM, ck);
    return hll_speeds(L, Rt, sL, sR, smin(L.vx - sL.a, vM - aM), smax(Rt.vx + sR.a, vM + aM), ck);
}
template <class C>
__device__ __forceinline__ Cons<double> hlle(const Prim<double>& L, const Prim<double>& Rt, FaceSide& sL, FaceSide& sR,
                                             C& ck) {
    face_side(L, sL, ck);
    face_side(Rt, sR, ck);
    const double sql = sL.sq, sqr = sR.sq, aL = sL.a, aR = sR.a;
    const PosRec rs = posrec(sql + sqr, ck);
    const double _sql = quot(sql, rs), _sqr = quot(sqr, rs);
    const double _v = quot(Rt.vx - L.vx, rs);
    double d = (_sql * aL * aL + _sqr * aR * aR) + 0.5 * (sql * sqr) * _v * _v;
    d = root(d, ck);
    const double u = _sql * L.vx + _sqr * Rt.vx;
    return hll_speeds(L, Rt, sL, sR, smin(L.vx - aL, u - d), smax(Rt.vx + aR, u + d), ck);
}

// Riemann::Roe with the Harten-Hyman fix; the two entropy-fix returns raise
// the flag (transonic rarefactions are few).
template <class C>
__device__ __forceinline__ Cons<double> roe(const Prim<double>& L, const Prim<double>& Rt, FaceSide& sL, FaceSide& sR,
                                            C& ck) {
    face_side(L, sL, ck);
    face_side(Rt, sR, ck);
    const PosRec rs = posrec(sL.sq + sR.sq, ck);
    const double _sql = quot(sL.sq, rs), _sqr = quot(sR.sq, rs);
    const double _rho = sL.sq * sR.sq;
    const double vx = L.vx * _sql + Rt.vx * _sqr, vy = L.vy * _sql + Rt.vy * _sqr, vz = L.vz * _sql + Rt.vz * _sqr;
    const double _H = _sql * quot(sL.U.E + L.p, sL.r) + _sqr * quot(sR.U.E + Rt.p, sR.r);
    const double V2 = dot3(vx, vy, vz, vx, vy, vz);
    const double _a = root(kGm1 * (_H - V2 * 0.5), ck);
    const double dp = Rt.p - L.p, ra = _rho * _a, du = Rt.vx - L.vx;
    // (2 a) a is exactly twice a a, so all three quotients share 1 / (a a)
    const WideRec r2 = widerec(_a * _a, ck);
    double q0 = dp - ra * du, q1 = dp, q4 = dp + ra * du;
    quots(r2, ck, q0, q1, q4);
    const double al0 = 0.5 * q0, al1 = (Rt.rho - L.rho) - q1, al2 = _rho * (Rt.vy - L.vy), al3 = _rho * (Rt.vz - L.vz),
                 al4 = 0.5 * q4;
    const Cons<double> K0{1.0, _H - vx * _a, vx - _a, vy - 0.0, vz - 0.0, 0, 0, 0};
    const Cons<double> K4{1.0, _H + vx * _a, vx + _a, vy + 0.0, vz + 0.0, 0, 0, 0};
    {
        const Cons<double> SL = c_add<false>(sL.U, c_mul<false>(K0, al0));
        const Rec r = rec(SL.rho, ck);
        const double aSL = root(quot(kGamma * f64::pressure<false>(SL, r, ck), r), ck);
        ck.raise(L.vx - sL.a < 0.0 && quot(SL.mx, r) - aSL > 0.0);
        const Cons<double> SR = c_sub<false>(sR.U, c_mul<false>(K4, al4));
        const Rec q = rec(SR.rho, ck);
        const double aSR = root(quot(kGamma * f64::pressure<false>(SR, q, ck), q), ck);
        ck.raise(Rt.vx + sR.a > 0.0 && quot(SR.mx, q) + aSR < 0.0);
    }
    Cons<double> F = c_add<false>(side_flux(L, sL, ck), side_flux(Rt, sR, ck));
    const Cons<double> K1{1.0, V2 * 0.5, vx, vy, vz, 0, 0, 0}, K2{0.0, vy, 0.0, 1.0, 0.0, 0, 0, 0},
        K3{0.0, vz, 0.0, 0.0, 1.0, 0, 0, 0};
    F = c_sub<false>(F, c_mul<false>(K0, al0 * fabs(vx - _a)));
    F = c_sub<false>(F, c_mul<false>(K1, al1 * fabs(vx)));
    F = c_sub<false>(F, c_mul<false>(K2, al2 * fabs(vx)));
    F = c_sub<false>(F, c_mul<false>(K3, al3 * fabs(vx)));
    F = c_sub<false>(F, c_mul<false>(K4, al4 * fabs(vx + _a)));
    return c_mul<false>(F, 0.5);
}

// ---------------------------------------------------------------------------
// The exact solver (Exact.cpp) with the reference's mean guess. What bounds it
// is pow, so a power of one (a uniform or a resting gas, both sides of most
// faces ahead of a front) is not taken, and the derivative's power -(g + 1) /
// (2 g) is the function's (g - 1) / (2 g) divided by the argument (their sum
// is -1): it steers the Newton step alone, whose end the tolerance sets.

__device__ __forceinline__ double pow1(double x, double y) { return x == 1.0 ? 1.0 : pow(x, y); }

struct ExactSide {
    Rec rp;              // 1 / p
    double a, A, B, ra;  // sound speed, Riemann::f's A and B, rho a
};
template <class C>
__device__ __forceinline__ void exact_side(const Prim<double>& w, ExactSide& s, C& ck) {
    const Rec r = rec(w.rho, ck);
    ck.pos(w.rho);
    ck.pos(w.p);
    s.a = root(quot(kGamma * w.p, r), ck);
    s.A = quot(k2_Gp1, r);
    s.B = kGm1_Gp1 * w.p;
    s.ra = w.rho * s.a;
    s.rp = widerec(w.p, ck);  // (here and in exact_f of numerators above 2^-460)
}
template <bool DERIV, class C>
__device__ __forceinline__ double exact_f(double p, const Prim<double>& w, const ExactSide& s, double& df, C& ck) {
    if (p > w.p) {
        const Rec r = widerec(s.B + p, ck);
        const double q = root(quot(s.A, r), ck), d = p - w.p;
        if constexpr (DERIV) df = q * (1.0 - 0.5 * quot(d, r));
        return d * q;
    }
    ck.pos(p);
    const double x = quot(p, s.rp), y = pow1(x, kGm1_2G);
    if constexpr (DERIV) df = div(y, x * s.ra, ck);
    return k2_Gm1 * s.a * (y - 1.0);
}
template <class C>
__device__ __forceinline__ double exact_rho(double p, const Prim<double>& w, const ExactSide& s, C& ck) {
    if (p > w.p) return div(w.rho * (p + s.B), kGm1_Gp1 * p + w.p, ck);
    return w.rho * pow1(quot(p, s.rp), kGinv);
}
// the flux of the exact solution at x / t = 0; ps: its star pressure
template <class C>
__device__ __forceinline__ Cons<double> exact(const Prim<double>& L, const Prim<double>& Rt, const ExactOpts& o,
                                              FaceStats* st, double& ps, C& ck) {
    ExactSide sL, sR;
    exact_side(L, sL, ck);
    exact_side(Rt, sR, ck);
    double v, p, rhoL, rhoR, dfL = 0.0, dfR = 0.0;
    const double p_min = smin(L.p, Rt.p);
    if (exact_f<false>(p_min, L, sL, dfL, ck) + exact_f<false>(p_min, Rt, sR, dfR, ck) + Rt.vx - L.vx >= 0.0) {
        st->trrs += 1;
        const double _LR = div(pow1(quot(L.p, sR.rp), kGm1_2G) * sR.a, sL.a, ck);
        v = div(_LR * L.vx + Rt.vx + k2_Gm1 * (_LR * sL.a - sR.a), _LR + 1.0, ck);
        p = L.p * pow1(1.0 - div(kGm1_2 * (v - L.vx), sL.a, ck), k2G_Gm1);
        ck.pos(p);
        rhoL = L.rho * pow1(quot(p, sL.rp), kGinv);
        rhoR = Rt.rho * pow1(quot(p, sR.rp), kGinv);
    } else {
        p = (L.p + Rt.p) * 0.5;
        double CHA;
        int iters = o.max_iters, n = 0;
        do {
            const double fL = exact_f<true>(p, L, sL, dfL, ck), fR = exact_f<true>(p, Rt, sR, dfR, ck);
            double delta = fL + fR + Rt.vx - L.vx;
            delta = smin(div(delta, dfL + dfR, ck), 0.8 * p);
            p -= delta;
            CHA = fabs(div(delta, p + delta * 0.5, ck));
            n++;
        } while (CHA > o.tol && --iters != 0 && !ck.bad);
        st->newton_iters += n;
        st->exact_calls += 1;
        st->cap_hits += CHA > o.tol;
        const double fR = exact_f<false>(p, Rt, sR, dfR, ck);
        v = (L.vx + Rt.vx + fR - exact_f<false>(p, L, sL, dfL, ck)) * 0.5;
        rhoL = exact_rho(p, L, sL, ck);
        rhoR = exact_rho(p, Rt, sR, ck);
    }
    ck.pos(p);
    ck.num(v);
    ps = p;
    Prim<double> w;
    w.Bx = w.By = w.Bz = 0;
    if (fabs(v - 0.0) < 1e-12) {
        // on the contact: the root-density mean of both star states
        const double sql = root(rhoL, ck), sqr = root(rhoR, ck);
        const Prim<double> a{rhoL, p, v, L.vy, L.vz, 0, 0, 0}, b{rhoR, p, v, Rt.vy, Rt.vz, 0, 0, 0};
        Cons<double> u = c_add<false>(c_mul<false>(f64::to_cons<false>(a), sql), c_mul<false>(f64::to_cons<false>(b), sqr));
        quots(rec(sql + sqr, ck), ck, u.rho, u.E, u.mx, u.my, u.mz);
        w = f64::to_prim<false>(u, posrec(u.rho, ck), ck);
    } else {
        // the side the contact leaves behind, mirrored to be the right one
        const bool left = 0.0 < v;
        Prim<double> W = left ? L : Rt;
        const double a = left ? sL.a : sR.a, rho = left ? rhoL : rhoR;
        const Rec rp = left ? sL.rp : sR.rp;
        if (left) W.vx *= -1.0;
        const double sv = left ? v * -1.0 : v, x_t = left ? -0.0 : 0.0;
        w = W;
        int zone;
        if (p > W.p) {
            const double scale = root(quot(kGp1_2G * p, rp) + kGm1_2G, ck);
            zone = (x_t - W.vx > scale * a) ? 1 : 3;
        } else {
            if (x_t - W.vx > a) zone = 1;
            else if (x_t - sv > a) zone = 2;
            else zone = (x_t - sv > a * pow1(quot(p, rp), kGm1_2G)) ? 2 : 3;
        }
        if (zone == 3) {
            w.rho = rho;
            w.p = p;
            w.vx = sv;
        } else if (zone == 2) {
            const double scale = k2_Gp1 - div(kGm1_Gp1 * (W.vx - x_t), a, ck);
            w.rho *= pow1(scale, k2_Gm1);
            w.p *= pow1(scale, k2G_Gm1);
            w.vx = k2_Gp1 * (x_t - a + W.vx * kGm1_2);
        }
        if (left) w.vx *= -1.0;
    }
    ck.pos(w.rho);
    ck.pos(w.p);
    const Cons<double> U = f64::to_cons<false>(w);
    return flux_of<false>(U, f64::pressure<false>(U, rec(U.rho, ck), ck), w.vx, w.vy, w.vz);
}

// ---------------------------------------------------------------------------
// MHD solvers. The normal field is averaged into both sides first, as the
// plain routines do.

struct MhdSide {
    Rec r;        // of the density
    double E, c;  // energy, fast speed along x
};
template <class C>
__device__ __forceinline__ void mhd_side(const Prim<double>& w, MhdSide& s, C& ck) {
    s.r = posrec(w.rho, ck);
    s.c = f64::fast_speed(w, w.Bx, s.r, ck);
    s.E = f64::energy<true>(w);
}
__device__ __forceinline__ Cons<double> mhd_cons(const Prim<double>& w, const MhdSide& s) {
    return Cons<double>{w.rho, s.E, w.vx * w.rho, w.vy * w.rho, w.vz * w.rho, w.Bx, w.By, w.Bz};
}
template <class C>
__device__ __forceinline__ Cons<double> mhd_flux(const Prim<double>& w, const MhdSide& s, C& ck) {
    const Cons<double> U = mhd_cons(w, s);
    return flux_of<true>(U, f64::pressure<true>(U, s.r, ck), w.vx, w.vy, w.vz);
}
__device__ __forceinline__ double b2_of(const Prim<double>& w) { return dot3(w.Bx, w.By, w.Bz, w.Bx, w.By, w.Bz); }

// The state behind one outer wave: its velocity and field, and with FLUX its
// conservative state and flux. d: SK - SM and its reciprocal; ZERO: the branch
// without a normal field.
struct MhdStar {
    Cons<double> u, F;
    Prim<double> w;
};
template <bool ZERO, bool FLUX, class C>
__device__ __forceinline__ void mhd_star(const Prim<double>& K, const MhdSide& s, double x, double SK, double SM,
                                         const Rec& d, double rho, double pT, double Bx, MhdStar& o, C& ck) {
    Cons<double> u;
    u.rho = rho;
    double vy, vz;
    if constexpr (ZERO) {
        ck.raise(!(fabs(d.b) >= 1e-12));
        const double num = SK - K.vx;
        u.Bx = 0;
        u.By = K.By * num;
        u.Bz = K.Bz * num;
        quots(d, ck, u.By, u.Bz);
        vy = K.vy;
        vz = K.vz;
    } else {
        const double bb = (Bx * Bx) * k1_4pi;
        const double den = x * d.b - bb, num = x * (SK - K.vx) - bb, dv = SM - K.vx;
        // a density times two speeds: always below 1e-12 in the units of thin gas
        const bool degen = fabs(den) < 1e-12;
        const WideRec q = widerec(degen ? 1.0 : den, ck);
        u.Bx = Bx;
        u.By = degen ? K.By : K.By * num;
        u.Bz = degen ? K.Bz : K.Bz * num;
        double ty = degen ? 0.0 : (K.By * Bx) * dv, tz = degen ? 0.0 : (K.Bz * Bx) * dv;
        quots(q, ck, u.By, u.Bz, ty, tz);
        vy = K.vy - ty * k1_4pi;
        vz = K.vz - tz * k1_4pi;
    }
    u.mx = SM * u.rho;
    u.my = vy * u.rho;
    u.mz = vz * u.rho;
    double E = s.E * (SK - K.vx);
    E += pT * SM - (K.p + b2_of(K) * k1_8pi) * K.vx;
    if constexpr (!ZERO)
        E += Bx * (dot3(K.vx, K.vy, K.vz, K.Bx, K.By, K.Bz) - dot3(SM, vy, vz, u.Bx, u.By, u.Bz)) * k1_4pi;
    u.E = quot(E, d);
    ck.pos(u.E);
    const PosRec q = posrec(u.rho, ck);
    Prim<double> w;
    w.rho = u.rho;
    w.vx = u.mx;
    w.vy = u.my;
    w.vz = u.mz;
    quots(q, ck, w.vx, w.vy, w.vz);
    w.Bx = u.Bx;
    w.By = u.By;
    w.Bz = u.Bz;
    w.p = pT - b2_of(w) * k1_8pi;
    sound_state<true>(w, ck);
    if constexpr (!ZERO) surely_physical<true>(u, ck);
    o.w = w;
    o.u = u;
    if constexpr (FLUX) {
        o.F = c_add<true>(mhd_flux(K, s, ck), c_mul<true>(c_sub<true>(u, mhd_cons(K, s)), SK));
        o.F.Bx = 0;
    }
}

// Riemann::HLLD and HLLD_zero_B; an unphysical star state (their way to HLLE)
// raises the flag. Only the side the contact leaves behind needs its star flux
// and energy (SsL >= 0 implies SM >= 0, SsR <= 0 implies SM <= 0), so the
// other side's star state comes first and leaves its velocity and field:
// fewer values alive at a time (both sides whole spilled 700 bytes). Where an
// inner wave stands on the face (SsL or SsR zero) the other side's star state
// is not used, but an unphysical one still takes the face to HLLE.
template <class C>
__device__ __forceinline__ Cons<double> hlld(Prim<double> L, Prim<double> Rt, C& ck) {
    const double Bx = (L.Bx + Rt.Bx) * 0.5;
    L.Bx = Bx;
    Rt.Bx = Bx;
    MhdSide sL, sR;
    mhd_side(L, sL, ck);
    mhd_side(Rt, sR, ck);
    const double SL = smin(L.vx - sL.c, Rt.vx - sR.c);
    const double SR = smax(L.vx + sL.c, Rt.vx + sR.c);
    const bool outer = SL >= 0.0 || SR <= 0.0;
    double SM = SL >= 0.0 ? 1.0 : -1.0, pT = 0.0, xL = 0.0, xR = 0.0;
    if (!outer) {
        const double pTL = L.p + b2_of(L) * k1_8pi, pTR = Rt.p + b2_of(Rt) * k1_8pi;
        xL = L.rho * (SL - L.vx);
        xR = Rt.rho * (SR - Rt.vx);
        const WideRec rx = widerec(xR - xL, ck);
        SM = (xR * Rt.vx - xL * L.vx) - (pTR - pTL);
        quots(rx, ck, SM);
        pT = quot(xR * pTL - xL * pTR + xL * xR * (Rt.vx - L.vx), rx);
    }
    const bool left = SM >= 0.0;
    const Prim<double> K = left ? L : Rt;
    const MhdSide sK = left ? sL : sR;
    if (outer) return mhd_flux(K, sK, ck);
    const double cutoff = smax(b2_of(L) + b2_of(Rt), 1e-100);
    const bool zero = Bx * Bx < 1e-12 * cutoff || Bx == 0.0;
    const Prim<double> O = left ? Rt : L;
    const MhdSide sO = left ? sR : sL;
    const double SK = left ? SL : SR, SO = left ? SR : SL, xK = left ? xL : xR, xO = left ? xR : xL;
    const Rec dK = rec(SK - SM, ck), dO = rec(SO - SM, ck);
    const double rhoK = quot(xK, dK), rhoO = quot(xO, dO);
    MhdStar k, o;
    if (zero) {
        mhd_star<true, true>(K, sK, xK, SK, SM, dK, rhoK, pT, Bx, k, ck);
        if (SM != 0.0) return k.F;
        mhd_star<true, true>(O, sO, xO, SO, SM, dO, rhoO, pT, Bx, o, ck);
        const double sql = root(rhoK, ck), sqr = root(rhoO, ck);
        const Rec q = rec(sql + sqr, ck);
        return c_add<true>(c_mul<true>(k.F, quot(sql, q)), c_mul<true>(o.F, quot(sqr, q)));
    }
    const double sqK = root(rhoK, ck), sqO = root(rhoO, ck);
    const double ab = fabs(Bx), s4 = sq4pi();
    const double aK = div(ab, s4 * sqK, ck), aO = div(ab, s4 * sqO, ck);
    const double SsL = SM - (left ? aK : aO), SsR = SM + (left ? aO : aK);
    const bool inner = !(SsL >= 0.0) && !(SsR <= 0.0);
    if (!(SsL > 0.0) && !(SsR < 0.0)) mhd_star<false, false>(O, sO, xO, SO, SM, dO, rhoO, pT, Bx, o, ck);
    mhd_star<false, true>(K, sK, xK, SK, SM, dK, rhoK, pT, Bx, k, ck);
    ck.raise(SsL >= 0.0 ? !left : SsR <= 0.0 && left);
    if (!inner) return k.F;
    const double lvy = left ? k.w.vy : o.w.vy, lvz = left ? k.w.vz : o.w.vz, rvy = left ? o.w.vy : k.w.vy,
                 rvz = left ? o.w.vz : k.w.vz, lBy = left ? k.w.By : o.w.By, lBz = left ? k.w.Bz : o.w.Bz,
                 rBy = left ? o.w.By : k.w.By, rBz = left ? o.w.Bz : k.w.Bz, sqL = left ? sqK : sqO,
                 sqR = left ? sqO : sqK;
    const Rec q = rec(sqL + sqR, ck);
    const double _sqL = quot(sqL, q), _sqR = quot(sqR, q);
    const double sbx = Bx > 0.0 ? s4 : -s4;
    Prim<double> w;
    w.rho = rhoK;
    w.vx = SM;
    double tvy = (rBy - lBy) * sbx * k1_4pi, tvz = (rBz - lBz) * sbx * k1_4pi, tBy = (rvy - lvy) * sbx * sqL * sqR,
           tBz = (rvz - lvz) * sbx * sqL * sqR;
    quots(q, ck, tvy, tvz, tBy, tBz);
    w.vy = (lvy * _sqL + rvy * _sqR) + tvy;
    w.vz = (lvz * _sqL + rvz * _sqR) + tvz;
    w.Bx = Bx;
    w.By = (rBy * _sqL + lBy * _sqR) + tBy;
    w.Bz = (rBz * _sqL + lBz * _sqR) + tBz;
    const double dE = sbx * (dot3(k.w.vx, k.w.vy, k.w.vz, k.w.Bx, k.w.By, k.w.Bz) -
                             dot3(w.vx, w.vy, w.vz, w.Bx, w.By, w.Bz)) * k1_4pi * sqK;
    const Cons<double> u{rhoK, left ? k.u.E - dE : k.u.E + dE, w.vx * rhoK, w.vy * rhoK, w.vz * rhoK, w.Bx, w.By, w.Bz};
    w.p = pT - b2_of(w) * k1_8pi;
    sound_state<true>(w, ck);
    ck.fin(u.E);
    ck.fin(u.mx);
    ck.fin(u.my);
    ck.fin(u.mz);
    return c_add<true>(k.F, c_mul<true>(c_sub<true>(u, k.u), left ? SsL : SsR));
}

// Riemann::HLLE for MHD states
template <class C>
__device__ __forceinline__ Cons<double> hlle_mhd(Prim<double> L, Prim<double> Rt, C& ck) {
    const double Bx = (L.Bx + Rt.Bx) * 0.5;
    L.Bx = Bx;
    Rt.Bx = Bx;
    MhdSide sL, sR;
    mhd_side(L, sL, ck);
    mhd_side(Rt, sR, ck);
    const double sql = root(L.rho, ck), sqr = root(Rt.rho, ck), aL = sL.c, aR = sR.c;
    const PosRec rs = posrec(sql + sqr, ck);
    const double _sql = quot(sql, rs), _sqr = quot(sqr, rs);
    const double _v = quot(Rt.vx - L.vx, rs);
    const double d = root((_sql * aL * aL + _sqr * aR * aR) + 0.5 * (sql * sqr) * _v * _v, ck);
    const double u = _sql * L.vx + _sqr * Rt.vx;
    const double sl = smin(L.vx - aL, u - d), sr = smax(Rt.vx + aR, u + d);
    const Cons<double> FL = mhd_flux(L, sL, ck), FR = mhd_flux(Rt, sR, ck);
    if (sl >= 0.0) return FL;
    if (sr <= 0.0) return FR;
    const Cons<double> n = c_add<true>(c_sub<true>(c_mul<true>(FL, sr), c_mul<true>(FR, sl)),
                                       c_mul<true>(c_sub<true>(mhd_cons(Rt, sR), mhd_cons(L, sL)), sl * sr));
    Cons<double> F = n;
    quots(rec(sr - sl, ck), ck, F.rho, F.E, F.mx, F.my, F.mz, F.Bx, F.By, F.Bz);
    return F;
}

// The solver and the physicality test of its flux (verify_and_fallback,
// Flux.cpp:77-97); a test that fails or is close raises the flag.
template <bool MHD, int SOLVER, class C>
__device__ __forceinline__ void face_body(const Prim<double>& L, const Prim<double>& Rt, double dt_dL,
                                          const ExactOpts& eo, Cons<double>& F, FaceStats* st, double& ps, C& ck) {
    if constexpr (MHD) {
        if constexpr (SOLVER == RS_HLLE) F = hlle_mhd(L, Rt, ck);
        else F = hlld(L, Rt, ck);
    } else {
        FaceSide sL, sR;
        if constexpr (SOLVER == RS_HLL) F = hll(L, Rt, sL, sR, ck);
        else if constexpr (SOLVER == RS_HLLE) F = hlle(L, Rt, sL, sR, ck);
        else if constexpr (SOLVER == RS_ROE) F = roe(L, Rt, sL, sR, ck);
        else if constexpr (SOLVER == RS_EXACT) {
            F = exact(L, Rt, eo, st, ps, ck);
            sL.U = f64::to_cons<false>(L);
            sR.U = f64::to_cons<false>(Rt);
        } else F = hllc(L, Rt, sL, sR, ck);
        // (a face without the test has no other look at its flux)
        ck.raise(!(dt_dL > 0.0));
        if (dt_dL > 0.0) {
            surely_physical<false>(c_sub<false>(sL.U, c_mul<false>(F, dt_dL)), ck);
            surely_physical<false>(c_add<false>(sR.U, c_mul<false>(F, dt_dL)), ck);
        }
    }
}
// The exact solver's face while its solves are logged: false if it raises the
// flag (then nothing is logged here).
template <bool LOCAL>
__device__ __noinline__ bool exact_logged(const Prim<double>* LR, double dt_dx, const ExactOpts* eo, Cons<double>* F,
                                          FaceStats* st) {
    Flag<LOCAL> ck;
    FaceStats s = *st;
    double ps;
    face_body<false, RS_EXACT>(LR[0], LR[1], dt_dx, *eo, *F, &s, ps, ck);
    if (ck.bad) return false;
    // (without a flag both states and the pressure are positive and finite)
    if (s.exact_calls != st->exact_calls && s.cap_hits == st->cap_hits)
        newton_log_push(eo->log, LR[0].rho, LR[0].vx, LR[0].p, LR[1].rho, LR[1].vx, LR[1].p, ps,
                        s.newton_iters - st->newton_iters);
    *st = s;
    return true;
}
template <bool MHD, int SOLVER, bool AGAIN, bool LOCAL>
__device__ __noinline__ bool face_slow(const Prim<double>* LR, double dt_dx, const ExactOpts* eo, Cons<double>* F,
                                       FaceStats* st) {
    if constexpr (AGAIN) {
        Flag<true> ck;
        FaceStats s = *st;
        double ps;
        face_body<MHD, SOLVER>(LR[0], LR[1], dt_dx, *eo, *F, &s, ps, ck);
        if (!ck.bad) {
            *st = s;
            return true;
        }
        return face_slow<MHD, SOLVER, false, LOCAL>(LR, dt_dx, eo, F, st);
    } else {
        if constexpr (!MHD && SOLVER == RS_EXACT)
            if (eo->log.rows && eo->guess == GUESS_MEAN && exact_logged<LOCAL>(LR, dt_dx, eo, F, st)) return true;
        return face_flux_x<MHD, SOLVER, double>(LR[0], LR[1], dt_dx, *eo, *F, st);
    }
}

// The flux along x of the states on both sides of a face, as face_flux_x. MHD
// HLL is rare and takes the plain routine, and so does the exact solver with
// another guess than the mean. While its solves are logged they run out of line
// (a branch to the log behind every exact solve here cost 1.8 %, its star
// pressure kept to the end of the face 1.2 %: 3D blast 110 x 87 x 93).
template <bool MHD, int SOLVER, bool LOCAL = false>
__device__ __forceinline__ bool face_flux_x(const Prim<double>& L, const Prim<double>& Rt, double dt_dL,
                                            const ExactOpts& eo, Cons<double>& F, FaceStats* st) {
    if constexpr (MHD && SOLVER == RS_HLL) {
        return dgpu::face_flux_x<MHD, SOLVER>(L, Rt, dt_dL, eo, F, st);
    } else {
        constexpr bool kExact = !MHD && SOLVER == RS_EXACT;
        Flag<LOCAL> ck;
        FaceStats s = *st;
        const bool aside = kExact && (eo.guess != GUESS_MEAN || eo.log.rows);
        if (!aside) {
            double ps;
            face_body<MHD, SOLVER>(L, Rt, dt_dL, eo, F, &s, ps, ck);
            if (!ck.bad) {
                if constexpr (kExact) *st = s;
                return true;
            }
        }
        const Prim<double> LR[2] = {L, Rt};
        Cons<double> G;
        const ExactOpts e = eo;
        FaceStats t = *st;
        const bool ok = face_slow<MHD, SOLVER, !LOCAL && !kExact, LOCAL>(LR, dt_dL, &e, &G, &t);
        *st = t;
        F = G;
        return ok;
    }
}
template <bool MHD, int SOLVER, int AX, bool LOCAL = false>
__device__ __forceinline__ bool face_flux(Prim<double> L, Prim<double> Rt, double dt_dL, const ExactOpts& eo,
                                          Cons<double>& F, FaceStats* st) {
    swap_axis<AX>(L);
    swap_axis<AX>(Rt);
    const bool ok = f64::face_flux_x<MHD, SOLVER, LOCAL>(L, Rt, dt_dL, eo, F, st);
    swap_axis<AX>(F);
    return ok;
}

// ---------------------------------------------------------------------------
// The conservative update of a cell

// protect_thermal's gate 8 pi p / B^2 <= 0.1 without the division, the flag
// where the rounded quotient could fall on either side.
template <class C>
__device__ __forceinline__ bool keeps_thermal(const Prim<double>& w, int mode, C& ck) {
    if (mode == 0) return false;
    if (mode == 1) return true;
    const double B2 = b2_of(w);
    const double n = k8pi * w.p, t = 0.1 * B2;
    const bool under = n < t * (1.0 - 0x1p-48);
    ck.raise(!under && !(n > t * (1.0 + 0x1p-48)));
    return under && B2 != 0.0;
}
// computeBodyField (B_fields.cpp:70-79): the cell with its field replaced, r
// the reciprocal of its density.
template <class C>
__device__ __forceinline__ Prim<double> body_field(Prim<double> w, double bx, double by, double bz, int mode,
                                                   const PosRec& r, C& ck) {
    const bool keep = keeps_thermal(w, mode, ck);
    ck.pos(w.p);
    Cons<double> U = f64::to_cons<true>(w);
    U.Bx = bx; U.By = by; U.Bz = bz;
    const Prim<double> n = f64::to_prim<true>(U, r, ck);
    w.Bx = bx; w.By = by; w.Bz = bz;
    return keep ? w : n;
}

// A half state w plus its transverse correction d, with the normal field
// (component ax) replaced by b.
static __device__ __noinline__ void corrected_mhd_plain(Prim<double>* w, const Cons<double>* d, int ax, double b) {
    Cons<double> u = dgpu::c_add<true>(dgpu::to_cons<true>(*w), *d);
    (ax == 0 ? u.Bx : ax == 1 ? u.By : u.Bz) = b;
    *w = dgpu::to_prim<true>(u);
}
template <int AX>
__device__ __forceinline__ Prim<double> corrected_mhd(const Prim<double>& w, const Cons<double>& d, double b) {
    Chk ck;
    ck.pos(w.p);
    Cons<double> u = c_add<true>(f64::to_cons<true>(w), d);
    (AX == 0 ? u.Bx : AX == 1 ? u.By : u.Bz) = b;
    Prim<double> r = f64::to_prim<true>(u, posrec(u.rho, ck), ck);
    if (ck.bad) {
        Prim<double> t = w;
        const Cons<double> e = d;
        corrected_mhd_plain(&t, &e, AX, b);
        r = t;
    }
    return r;
}

}  // namespace f64
}  // namespace dgpu
