// bp_fp32.cuh -- the FP32 form's backprojection kernel and the choice of its
// instance, for bp_fast.cu and bp_exact.cu.
#pragma once

#include "bp_body.cuh"

namespace jfdk {
namespace {

// One CTA = one TX x (128 / TX) x ZPT voxel tile of one launch's grid.
template <int ZPT, bool FINALIZE, bool EXACT, int G, int TX, bool WV = false>
__global__ void __launch_bounds__(kBPThreads, bp_fp32_min_blocks(ZPT)) bp_kernel(BPParams p) {
    bp_block<ZPT, FINALIZE, EXACT, G, GridTile<TX>, WV>(p, GridTile<TX>{});
}

template <int ZPT, bool F, bool E, int G, int TX>
cudaError_t go(const BPParams& p, cudaStream_t s) {
    if constexpr (F) {
        if (p.wvol) {
            bp_kernel<ZPT, F, E, G, TX, true><<<bp_grid<TX>(p, ZPT), dim3(TX, kBPThreads / TX), 0, s>>>(p);
            return cudaGetLastError();
        }
    }
    bp_kernel<ZPT, F, E, G, TX><<<bp_grid<TX>(p, ZPT), dim3(TX, kBPThreads / TX), 0, s>>>(p);
    return cudaGetLastError();
}

// Tile widths 4, 8 and 32 for the tile depths the autotuner chooses between
// (4 and 8 slices); 16-slice tiles are 4 wide.
template <int ZPT, bool F, bool E, int G>
cudaError_t go_tx(const BPParams& p, int tx, cudaStream_t s) {
    if constexpr (ZPT != 16) {
        if (tx == 8) return go<ZPT, F, E, G, 8>(p, s);
        if (tx == 32) return go<ZPT, F, E, G, 32>(p, s);
    }
    return go<ZPT, F, E, G, 4>(p, s);
}

template <bool F, bool E, int G>
cudaError_t go_zpt(const BPParams& p, int zpt, int tx, cudaStream_t s) {
    switch (zpt) {
        case 16: return go_tx<16, F, E, G>(p, tx, s);
        case 8: return go_tx<8, F, E, G>(p, tx, s);
        default: return go_tx<4, F, E, G>(p, tx, s);
    }
}

// EXACT runs the loop of any P[2] for an ideal orbit too (the sums are the same).
template <bool F, bool E>
cudaError_t go_geo(const BPParams& p, Geo geo, int zpt, int tx, cudaStream_t s) {
    if constexpr (!E) {
        if (geo == kGeoIdeal) return go_zpt<F, E, kGeoIdeal>(p, zpt, tx, s);
    }
    return geo == kGeoWZ ? go_zpt<F, E, kGeoWZ>(p, zpt, tx, s) : go_zpt<F, E, kGeoWConst>(p, zpt, tx, s);
}

}  // namespace
}  // namespace jfdk
