// bp_exact.cu -- the FP32 form's backprojection, every step rounded like BPCore.
#include "bp_fp32.cuh"

namespace jfdk {

cudaError_t launch_bp_exact(const BPParams& p, bool finalize, Geo geo, int zpt, int tile_x, cudaStream_t s) {
    return finalize ? go_geo<true, true>(p, geo, zpt, tile_x, s) : go_geo<false, true>(p, geo, zpt, tile_x, s);
}

}  // namespace jfdk
