// FP64 fused 2D CTU hydro launchers (every hydro solver).
#include "launchers.h"
#include "step_hydro.cuh"

namespace dgpu {

// Tiles of 14 x 26 cells, 256 threads, two CTAs per SM (128 registers, 106 KB
// each): bound by FP64 issue, so one CTA's barriers, tile load and last rounds
// of a phase fall under the other's arithmetic. Step time on the 1024^2 shear
// layer, results bit-identical: 0.288 ms against 0.333 ms for one CTA of 19 x
// 22 cells on 512 threads (the better shape while the divisions branched:
// 0.471 against 0.51), 0.312 for 8 x 32, 0.296 for 12 x 30, 0.30 for 16 x 24
// and 0.33 for three CTAs of 10 x 24 cells on 160 threads; x and y items in
// one instruction sequence with a runtime direction 0.294.
constexpr int k2dTI = 14, k2dTJ = 26, k2dNT = 256;

template <int S>
static int go(const Geo& G, const double* win, double* wout, StepCtl* ctl, const StepArgs& sa, const CUtensorMap* map,
              cudaStream_t st) {
    auto kern = k_step2d_hydro<S, k2dTI, k2dTJ, k2dNT>;
    const size_t smem = sizeof(Smem2DH<k2dTI, k2dTJ>);
    static bool attr_set = false;
    if (!attr_set) {
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return 1;
        attr_set = true;
    }
    dim3 grid((G.n[1] + k2dTJ - 1) / k2dTJ, (G.n[0] + k2dTI - 1) / k2dTI);
    kern<<<grid, k2dNT, smem, st>>>(G, win, wout, ctl, sa, *map);
    return cudaGetLastError() == cudaSuccess ? 0 : 1;
}

int step2d_tile_box(int mixed, int box[3]) {
    box[0] = (mixed ? kMx2dTJ : k2dTJ) + 6;
    box[1] = (mixed ? kMx2dTI : k2dTI) + 4;
    box[2] = 5;
    return 0;
}

int launch_step2d_hydro(int solver, const Geo& G, const double* win, double* wout, StepCtl* ctl, const StepArgs& sa,
                        const CUtensorMap* map, cudaStream_t st) {
    switch (solver) {
        case RS_HLLC: return go<RS_HLLC>(G, win, wout, ctl, sa, map, st);
        case RS_HLL: return go<RS_HLL>(G, win, wout, ctl, sa, map, st);
        case RS_HLLE: return go<RS_HLLE>(G, win, wout, ctl, sa, map, st);
        case RS_ROE: return go<RS_ROE>(G, win, wout, ctl, sa, map, st);
        default: return go<RS_EXACT>(G, win, wout, ctl, sa, map, st);
    }
}

}  // namespace dgpu
