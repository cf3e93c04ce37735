// bp_fast.cu -- the FP32 form's backprojection, lerps fused into FMAs.
#include "bp_fp32.cuh"

namespace jfdk {

cudaError_t launch_bp_fast(const BPParams& p, bool finalize, Geo geo, int zpt, int tile_x, cudaStream_t s) {
    return finalize ? go_geo<true, false>(p, geo, zpt, tile_x, s) : go_geo<false, false>(p, geo, zpt, tile_x, s);
}

}  // namespace jfdk
