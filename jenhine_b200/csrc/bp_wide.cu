// bp_wide.cu -- backprojection of frames with more than 4 GB of records, whose
// byte offsets need 64 bits.  FP32 tiles 4 slices deep (its volume does not
// depend on the depth), mixed ones as deep as asked for; 4 wide.
#include "bp_body.cuh"

namespace jfdk {
namespace {

template <int ZPT, bool FINALIZE, bool EXACT, bool MIXED, int G, bool WV>
__global__ void __launch_bounds__(kBPThreads) bp_wide_kernel(BPParams p) {
    if constexpr (MIXED)
        bp_mixed_block<ZPT, FINALIZE, G, GridTile<kBPTileX>, WV, false, false, true>(p, GridTile<kBPTileX>{});
    else
        bp_block<ZPT, FINALIZE, EXACT, G, GridTile<kBPTileX>, WV, false, false, true>(p, GridTile<kBPTileX>{});
}

template <int ZPT, bool E, bool M, int G>
cudaError_t go_wide(const BPParams& p, bool finalize, cudaStream_t s) {
    const dim3 grid = bp_grid<kBPTileX>(p, ZPT), cta(kBPTileX, kBPTileY);
    if (!finalize)
        bp_wide_kernel<ZPT, false, E, M, G, false><<<grid, cta, 0, s>>>(p);
    else if (p.wvol)
        bp_wide_kernel<ZPT, true, E, M, G, true><<<grid, cta, 0, s>>>(p);
    else
        bp_wide_kernel<ZPT, true, E, M, G, false><<<grid, cta, 0, s>>>(p);
    return cudaGetLastError();
}

template <int G>
cudaError_t go_wide_form(const BPParams& p, bool finalize, bool exact, bool mixed_form, int zpt, cudaStream_t s) {
    if (!mixed_form)
        return exact ? go_wide<4, true, false, G>(p, finalize, s) : go_wide<4, false, false, G>(p, finalize, s);
    switch (zpt) {
        case 16: return go_wide<16, false, true, G>(p, finalize, s);
        case 8: return go_wide<8, false, true, G>(p, finalize, s);
        default: return go_wide<4, false, true, G>(p, finalize, s);
    }
}

}  // namespace

cudaError_t launch_bp_wide(const BPParams& p, bool finalize, bool exact, bool mixed_form, Geo geo, int zpt,
                           cudaStream_t s) {
    return geo == kGeoWZ ? go_wide_form<kGeoWZ>(p, finalize, exact, mixed_form, zpt, s)
                         : go_wide_form<kGeoWConst>(p, finalize, exact, mixed_form, zpt, s);
}

}  // namespace jfdk
