// bp_weights.cu -- the volumes of normalisation weights, once per geometry.
#include "bp_body.cuh"

namespace jfdk {
namespace {

template <int ZPT, bool EXACT, bool WZ, int TX>
__global__ void __launch_bounds__(kBPThreads, bp_fp32_min_blocks(ZPT)) bp_weights_kernel(BPParams p, float* out) {
    bp_block<ZPT, true, EXACT, WZ ? kGeoWZ : kGeoWConst, GridTile<TX>, false, true>(p, GridTile<TX>{}, out);
}

// (once per geometry; with 16 slices at 128 registers.  Tiles inside the detector
// run without the range test as in the backprojection: 640 x 640 x 480 voxels from
// 600 views 53.0 ms, all tiles by the range test 82.6)
template <int ZPT, bool WZ, int TX>
__global__ void __launch_bounds__(kBPThreads, ZPT == 16 ? 4 : bp_min_blocks(ZPT))
    bp_mixed_weights_kernel(BPParams p, float* out) {
    bp_mixed_block<ZPT, true, WZ ? kGeoWZ : kGeoWConst, GridTile<TX>, false, true>(p, GridTile<TX>{}, out);
}

template <int ZPT, bool E, bool WZ>
cudaError_t go_weights(const BPParams& p, int tx, float* out, cudaStream_t s) {
    if constexpr (ZPT != 16) {
        if (tx == 8) {
            bp_weights_kernel<ZPT, E, WZ, 8><<<bp_grid<8>(p, ZPT), dim3(8, kBPThreads / 8), 0, s>>>(p, out);
            return cudaGetLastError();
        }
        if (tx == 32) {
            bp_weights_kernel<ZPT, E, WZ, 32><<<bp_grid<32>(p, ZPT), dim3(32, kBPThreads / 32), 0, s>>>(p, out);
            return cudaGetLastError();
        }
    }
    bp_weights_kernel<ZPT, E, WZ, 4><<<bp_grid<4>(p, ZPT), dim3(4, kBPThreads / 4), 0, s>>>(p, out);
    return cudaGetLastError();
}

template <bool E, bool WZ>
cudaError_t go_weights2(const BPParams& p, int zpt, int tx, float* out, cudaStream_t s) {
    switch (zpt) {
        case 16: return go_weights<16, E, WZ>(p, tx, out, s);
        case 8: return go_weights<8, E, WZ>(p, tx, out, s);
        default: return go_weights<4, E, WZ>(p, tx, out, s);
    }
}

template <int ZPT, bool WZ>
cudaError_t go_mixed_weights(const BPParams& p, int tx, float* out, cudaStream_t s) {
    if constexpr (ZPT != 16) {
        if (tx == 8) {
            bp_mixed_weights_kernel<ZPT, WZ, 8><<<bp_grid<8>(p, ZPT), dim3(8, kBPThreads / 8), 0, s>>>(p, out);
            return cudaGetLastError();
        }
        if (tx == 32) {
            bp_mixed_weights_kernel<ZPT, WZ, 32><<<bp_grid<32>(p, ZPT), dim3(32, kBPThreads / 32), 0, s>>>(p, out);
            return cudaGetLastError();
        }
    }
    bp_mixed_weights_kernel<ZPT, WZ, 4><<<bp_grid<4>(p, ZPT), dim3(4, kBPThreads / 4), 0, s>>>(p, out);
    return cudaGetLastError();
}

template <bool WZ>
cudaError_t go_mixed_weights2(const BPParams& p, int zpt, int tx, float* out, cudaStream_t s) {
    switch (zpt) {
        case 16: return go_mixed_weights<16, WZ>(p, tx, out, s);
        case 8: return go_mixed_weights<8, WZ>(p, tx, out, s);
        default: return go_mixed_weights<4, WZ>(p, tx, out, s);
    }
}

}  // namespace

cudaError_t launch_bp_weights(const BPParams& p, bool exact, bool w_depends_on_z, int zpt, int tile_x, float* out,
                              cudaStream_t s) {
    if (!out || p.v0 != 0) return cudaErrorInvalidValue;
    if (exact)
        return w_depends_on_z ? go_weights2<true, true>(p, zpt, tile_x, out, s)
                              : go_weights2<true, false>(p, zpt, tile_x, out, s);
    return w_depends_on_z ? go_weights2<false, true>(p, zpt, tile_x, out, s)
                          : go_weights2<false, false>(p, zpt, tile_x, out, s);
}

cudaError_t launch_bp_mixed_weights(const BPParams& p, bool w_depends_on_z, int zpt, int tile_x, float* out,
                                    cudaStream_t s) {
    if (!out || p.v0 != 0) return cudaErrorInvalidValue;
    return w_depends_on_z ? go_mixed_weights2<true>(p, zpt, tile_x, out, s)
                          : go_mixed_weights2<false>(p, zpt, tile_x, out, s);
}

}  // namespace jfdk
