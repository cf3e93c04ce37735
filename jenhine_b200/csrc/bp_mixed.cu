// bp_mixed.cu -- the mixed form's backprojection.
#include "bp_body.cuh"

namespace jfdk {
namespace {

// B: resident CTAs per SM, and with them the registers a thread may use.
template <int ZPT, bool FINALIZE, int G, int TX, int B, bool WV = false>
__global__ void __launch_bounds__(kBPThreads, B) bp_mixed_kernel(BPParams p) {
    if constexpr (G == kGeoWZ)
        bp_mixed_block<ZPT, FINALIZE, G, GridTile<TX>, WV>(p, GridTile<TX>{});
    else
        bp_mixed_block<ZPT, FINALIZE, G, GridTileHeld<TX>, WV>(p, GridTileHeld<TX>{});
}

// The ideal orbit has its own loop where the weights come from the volume.
template <int ZPT, bool F, int G, int TX, int B>
cudaError_t go_mixed(const BPParams& p, cudaStream_t s) {
    if constexpr (F) {
        if (p.wvol) {
            bp_mixed_kernel<ZPT, F, G, TX, B, true><<<bp_grid<TX>(p, ZPT), dim3(TX, kBPThreads / TX), 0, s>>>(p);
            return cudaGetLastError();
        }
    }
    constexpr int H = G == kGeoIdeal ? kGeoWConst : G;
    bp_mixed_kernel<ZPT, F, H, TX, B><<<bp_grid<TX>(p, ZPT), dim3(TX, kBPThreads / TX), 0, s>>>(p);
    return cudaGetLastError();
}

// Resident CTAs per SM of a launch of 4-wide tiles.
//
// 16 slices (the default on large volumes when W does not depend on z): 128
// registers and 16 warps per SM on a flexing gantry, 75.9 ms a 640 x 640 x 480
// volume from 600 views against 76.2 with 96 registers and 20 warps, which spill in
// the loop; but launches of few views spend their time at its ends, where 20 warps
// are the better ones (512 x 512 x 400, finalised: 8 views 1398 against 1215 us, 40
// 3170 and 3064, 100 7059 and 7034; accumulated, 640 x 640 x 480: one view 1112
// and 1048, 8 2088 and 2023, while 320^3 from 16 takes 619 and 627).  On an ideal
// orbit, whose loop needs fewer, 20 always (61.9 against 64.6 ms from 600 views).
//
// 8 slices: 72 registers and 28 warps, 1070 us a 128^3 volume from 360 views (64
// and 32: 1103; 80 and 24: 1196); a launch that 16 warps per SM hold in one wave
// waits for its loads instead, and has the registers for more of them in flight
// (accumulating 16 views: 64^3 24.3 us with 72 registers and 14.0 with 128, 96 x
// 96 x 64 26.0 and 17.7).
template <int ZPT, bool F, int G>
cudaError_t go_mixed_4(const BPParams& p, int sms, cudaStream_t s) {
    if constexpr (ZPT == 16) {
        if constexpr (F && G == kGeoIdeal) {
            if (p.wvol) return go_mixed<16, F, G, 4, 5>(p, s);
        }
        constexpr int H = G == kGeoIdeal ? kGeoWConst : G, few = F ? 48 : 6;
        if constexpr (H == kGeoWConst) {
            if (p.nv < few) return go_mixed<16, F, H, 4, 5>(p, s);
        }
        return go_mixed<16, F, H, 4, 4>(p, s);
    } else if constexpr (ZPT == 8) {
        const dim3 g = bp_grid<4>(p, 8);
        return (long long)g.x * g.y * g.z <= 4LL * sms ? go_mixed<8, F, G, 4, 4>(p, s) : go_mixed<8, F, G, 4, 7>(p, s);
    } else {
        return go_mixed<ZPT, F, G, 4, 1>(p, s);
    }
}

template <int ZPT, bool F, int G>
cudaError_t go_mixed_tx(const BPParams& p, int tx, int sms, cudaStream_t s) {
    if constexpr (ZPT != 16) {
        constexpr int B = bp_min_blocks(ZPT);
        if (tx == 8) return go_mixed<ZPT, F, G, 8, B>(p, s);
        if (tx == 32) return go_mixed<ZPT, F, G, 32, B>(p, s);
    }
    return go_mixed_4<ZPT, F, G>(p, sms, s);
}

template <bool F, int G>
cudaError_t go_mixed_zpt(const BPParams& p, int zpt, int tx, int sms, cudaStream_t s) {
    switch (zpt) {
        case 16: return go_mixed_tx<16, F, G>(p, tx, sms, s);
        case 8: return go_mixed_tx<8, F, G>(p, tx, sms, s);
        default: return go_mixed_tx<4, F, G>(p, tx, sms, s);
    }
}

}  // namespace

cudaError_t launch_bp_mixed(const BPParams& p, bool finalize, Geo geo, int zpt, int tile_x, int sms, cudaStream_t s) {
    if ((long long)p.U * p.V > (1LL << 29)) return launch_bp_wide(p, finalize, false, true, geo, zpt, s);
    if (!finalize)
        return geo == kGeoWZ ? go_mixed_zpt<false, kGeoWZ>(p, zpt, tile_x, sms, s)
                             : go_mixed_zpt<false, kGeoWConst>(p, zpt, tile_x, sms, s);
    switch (geo) {
        case kGeoIdeal: return go_mixed_zpt<true, kGeoIdeal>(p, zpt, tile_x, sms, s);
        case kGeoWConst: return go_mixed_zpt<true, kGeoWConst>(p, zpt, tile_x, sms, s);
        default: return go_mixed_zpt<true, kGeoWZ>(p, zpt, tile_x, sms, s);
    }
}

}  // namespace jfdk
