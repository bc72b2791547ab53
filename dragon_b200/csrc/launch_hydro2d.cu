// FP64 fused 2D CTU hydro launchers (every hydro solver).
#include "chain.cuh"
#include "launchers.h"
#include "step_hydro.cuh"

namespace dgpu {

// Tiles of 16 x 24 cells, 256 threads, two CTAs per SM (128 registers, 111 KB
// each): bound by FP64 issue, so one CTA's barriers, tile load and last rounds
// of a phase fall under the other's arithmetic. Step time on the 1024^2 shear
// layer, results bit-identical: 0.256 ms (14 x 26 cells 0.261, 20 x 20 0.256, 18
// x 22 0.263); one CTA of 28 x 30 cells on 512 threads 0.268, three of 10 x 24
// on 160 threads 0.302, four of 8 x 22 on 128 threads 0.315. With divisions that
// branched, one CTA of 19 x 22 cells on 512 threads was the best at 0.471.
constexpr int k2dTI = 16, k2dTJ = 24, k2dNT = 256;

// A grid whose large tiles do not fill the GPU waits for the longest CTA, not
// for its arithmetic, so smaller grids take smaller tiles: 6 x 30 cells, whose
// 256 half states are one round of the threads (faces and corrections two),
// and 6 x 14, whose every phase is one round (128 half states, 232 and 188
// faces, 208 corrections, 84 updates). Step times in us (CTAs), shear layer:
//          6 x 14        6 x 30       16 x 24
//  96^2   17.5 (112)   19.1  (64)   27.2  (24)
// 128^2   18.9 (220)   20.5 (110)   27.8  (48)
// 160^2   26.0 (324)   24.9 (162)   27.4  (70)
// 256^2   40.1 (817)   33.9 (387)   38.5 (176)
// 300^2   50.2         40.7 (500)   38.7 (247)
// 320^2   54.5         43.5 (594)   38.6 (280)
// 350^2   60.1         48.8 (708)   51.6 (330)
// 384^2   74.0         55.4 (832)   52.3 (384)
// Hence the lines: 6 x 14 while its CTAs are all resident (two per SM), 6 x 30
// up to three per SM, and up to five where the large tiles need a second wave.
enum Tile2D { kTile16x24, kTile6x30, kTile6x14 };
constexpr long long kSms = 148;  // of a B200
static Tile2D pick_tile(const Geo& G) {
    auto ctas = [&](int ti, int tj) { return (long long)((G.n[0] + ti - 1) / ti) * ((G.n[1] + tj - 1) / tj); };
    if (ctas(6, 14) <= 2 * kSms) return kTile6x14;
    const long long mid = ctas(6, 30);
    if (mid <= 3 * kSms || (mid <= 5 * kSms && ctas(k2dTI, k2dTJ) > 2 * kSms)) return kTile6x30;
    return kTile16x24;
}

template <int S, int TI, int TJ>
static int go_tile(const Geo& G, const double* win, double* wout, StepCtl* ctl, const StepArgs& sa,
                   const CUtensorMap* map, cudaStream_t st) {
    auto kern = k_step2d_hydro<S, TI, TJ, k2dNT>;
    const size_t smem = sizeof(Smem2DH<TI, TJ>);
    static bool attr_set = false;
    if (!attr_set) {
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return 1;
        attr_set = true;
    }
    dim3 grid((G.n[1] + TJ - 1) / TJ, (G.n[0] + TI - 1) / TI);
    chain(kern, grid, k2dNT, smem, st, G, win, wout, ctl, sa, *map);
    return cudaGetLastError() == cudaSuccess ? 0 : 1;
}
template <int S>
static int go(const Geo& G, const double* win, double* wout, StepCtl* ctl, const StepArgs& sa, const CUtensorMap* map,
              cudaStream_t st) {
    switch (pick_tile(G)) {
        case kTile6x14: return go_tile<S, 6, 14>(G, win, wout, ctl, sa, map, st);
        case kTile6x30: return go_tile<S, 6, 30>(G, win, wout, ctl, sa, map, st);
        default: return go_tile<S, k2dTI, k2dTJ>(G, win, wout, ctl, sa, map, st);
    }
}

int step2d_tile_box(int mixed, const Geo& G, int box[3]) {
    const Tile2D t = pick_tile(G);
    box[0] = (mixed ? kMx2dTJ : t == kTile6x14 ? 14 : t == kTile6x30 ? 30 : k2dTJ) + 6;
    box[1] = (mixed ? kMx2dTI : t == kTile16x24 ? k2dTI : 6) + 4;
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
