// bp_batch_mixed.cu -- the persistent backprojection kernels of the mixed form.
#include "bp_batch.cuh"

namespace jfdk {

cudaError_t launch_bp_batch_mixed(const BatchSlots& t, int nscans, unsigned total, bool wz, bool wv, bool deep,
                               unsigned* counter, int ctas, cudaStream_t s) {
    return wz ? batch_go2<true, true>(t, nscans, total, counter, ctas, wv, deep, s)
              : batch_go2<true, false>(t, nscans, total, counter, ctas, wv, deep, s);
}

cudaError_t bp_batch_resident_mixed(bool wz, bool wv, bool deep, int* per_sm) {
    return wz ? batch_occ2<true, true>(wv, deep, per_sm) : batch_occ2<true, false>(wv, deep, per_sm);
}

}  // namespace jfdk
