// The conservative update of a cell, its physicality and its CFL speed on the
// branch-free divisions of fast64.cuh (hydro cells and 1D MHD cells; the MHD
// grids' constrained transport has its own, step_mhd.cuh).
#pragma once

#include "grid.cuh"
#include "solve64.cuh"

namespace dgpu {
namespace f64 {

// The committed state of a cell, the stage of the error it raises (0: none)
// and its CFL speed.
struct Updated {
    Prim<double> w;
    int stage;
    double speed;
};
template <bool MHD>
__device__ __noinline__ void updated_plain(Updated* r, const Cons<double>* dU, int nd, const StepArgs* sa) {
    Cons<double> U = dgpu::to_cons<MHD>(r->w);
    for (int k = 0; k < nd; k++) U = c_add<MHD>(U, dU[k]);
    r->w = dgpu::to_prim<MHD>(U);
    r->stage = !is_finite<MHD>(U) ? ST_NAN : !is_physical<MHD>(r->w) ? ST_UNPHYSICAL : 0;
    r->speed = grid_cfl_speed<MHD>(r->w, nd, sa->cfl, sa->dx, sa->dy, nd > 2 ? sa->dz : 0.0);
}
// The update by the flux differences d of the grid's axes, in turn
// (applyFluxes, Unsplit.cpp:256-288).
template <bool MHD, class... D>
__device__ __forceinline__ Updated updated(const Prim<double>& w, const StepArgs& sa, const Widths& wd, const D&... d) {
    Chk ck;
    ck.pos(w.p);
    Cons<double> U = f64::to_cons<MHD>(w);
    ((U = c_add<MHD>(U, d)), ...);
    const PosRec r = posrec(U.rho, ck);
    Updated o;
    o.w = f64::to_prim<MHD>(U, r, ck);
    sound_state<MHD>(o.w, ck);
    ck.fin(U.E);
    o.stage = 0;
    double a;
    if constexpr (MHD) a = f64::fast_speed_max(o.w, r, ck);
    else a = f64::sound_speed(o.w, r, ck);
    if constexpr (sizeof...(D) == 1) o.speed = fabs(o.w.vx) + a;
    else o.speed = f64::cfl_speed(o.w, a, sa.cfl, wd, ck);
    if (ck.bad) {
        const Cons<double> all[] = {d...};
        const StepArgs s = sa;
        Updated t;
        t.w = w;
        updated_plain<MHD>(&t, all, sizeof...(D), &s);
        o = t;
    }
    return o;
}

}  // namespace f64
}  // namespace dgpu
