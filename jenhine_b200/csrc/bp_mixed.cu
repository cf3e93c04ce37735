// bp_mixed.cu -- the mixed form's backprojection.
#include "bp_body.cuh"

namespace jfdk {
namespace {

template <int ZPT, bool FINALIZE, int G, int TX, bool WV = false>
__global__ void __launch_bounds__(kBPThreads, bp_min_blocks(ZPT)) bp_mixed_kernel(BPParams p) {
    if constexpr (G == kGeoWZ)
        bp_mixed_block<ZPT, FINALIZE, G, GridTile<TX>, WV>(p, GridTile<TX>{});
    else
        bp_mixed_block<ZPT, FINALIZE, G, GridTileHeld<TX>, WV>(p, GridTileHeld<TX>{});
}

// The ideal orbit has its own loop where the weights come from the volume.
template <int ZPT, bool F, int G, int TX>
cudaError_t go_mixed(const BPParams& p, cudaStream_t s) {
    if constexpr (F) {
        if (p.wvol) {
            bp_mixed_kernel<ZPT, F, G, TX, true><<<bp_grid<TX>(p, ZPT), dim3(TX, kBPThreads / TX), 0, s>>>(p);
            return cudaGetLastError();
        }
    }
    constexpr int H = G == kGeoIdeal ? kGeoWConst : G;
    bp_mixed_kernel<ZPT, F, H, TX><<<bp_grid<TX>(p, ZPT), dim3(TX, kBPThreads / TX), 0, s>>>(p);
    return cudaGetLastError();
}

template <int ZPT, bool F, int G>
cudaError_t go_mixed_tx(const BPParams& p, int tx, cudaStream_t s) {
#ifndef DEV
    if constexpr (ZPT != 16) {
        if (tx == 8) return go_mixed<ZPT, F, G, 8>(p, s);
        if (tx == 32) return go_mixed<ZPT, F, G, 32>(p, s);
    }
#endif
    return go_mixed<ZPT, F, G, 4>(p, s);
}

template <bool F, int G>
cudaError_t go_mixed_zpt(const BPParams& p, int zpt, int tx, cudaStream_t s) {
    switch (zpt) {
        case 16: return go_mixed_tx<16, F, G>(p, tx, s);
        case 8: return go_mixed_tx<8, F, G>(p, tx, s);
        default: return go_mixed_tx<4, F, G>(p, tx, s);
    }
}

}  // namespace

cudaError_t launch_bp_mixed(const BPParams& p, bool finalize, Geo geo, int zpt, int tile_x, cudaStream_t s) {
    if ((long long)p.U * p.V > (1LL << 29)) return launch_bp_wide(p, finalize, false, true, geo, zpt, s);
    if (!finalize)
        return geo == kGeoWZ ? go_mixed_zpt<false, kGeoWZ>(p, zpt, tile_x, s)
                             : go_mixed_zpt<false, kGeoWConst>(p, zpt, tile_x, s);
    switch (geo) {
        case kGeoIdeal: return go_mixed_zpt<true, kGeoIdeal>(p, zpt, tile_x, s);
        case kGeoWConst: return go_mixed_zpt<true, kGeoWConst>(p, zpt, tile_x, s);
        default: return go_mixed_zpt<true, kGeoWZ>(p, zpt, tile_x, s);
    }
}

}  // namespace jfdk
