// bp_batch_fp32.cu -- the persistent backprojection kernels of the FP32 form.
#include "bp_batch.cuh"

namespace jfdk {

cudaError_t launch_bp_batch_fp32(const BatchSlots& t, int nscans, unsigned total, bool wz, bool wv, bool deep,
                               unsigned* counter, int ctas, cudaStream_t s) {
    return wz ? batch_go2<false, true>(t, nscans, total, counter, ctas, wv, deep, s)
              : batch_go2<false, false>(t, nscans, total, counter, ctas, wv, deep, s);
}

cudaError_t bp_batch_resident_fp32(bool wz, bool wv, bool deep, int* per_sm) {
    return wz ? batch_occ2<false, true>(wv, deep, per_sm) : batch_occ2<false, false>(wv, deep, per_sm);
}

}  // namespace jfdk
