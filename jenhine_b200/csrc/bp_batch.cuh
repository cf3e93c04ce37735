// bp_batch.cuh -- persistent backprojection over the tiles of several scans,
// for bp_batch_fp32.cu and bp_batch_mixed.cu (each takes minutes to compile).
#pragma once

#include "bp_body.cuh"

namespace jfdk {
namespace {

__shared__ unsigned g_batch_tile;   // the batch kernel's current work item

struct BatchTile {
    static constexpr int kX = kBPTileX, kY = kBPTileY;
    const BatchScan& b;
    __device__ unsigned local() const { return *static_cast<volatile unsigned*>(&g_batch_tile) - b.first_tile; }
    __device__ int bx() const { return (int)(local() % (unsigned)b.gx); }
    __device__ int by() const { return (int)((local() / (unsigned)b.gx) % (unsigned)b.gy); }
    __device__ int bz() const { return (int)(local() / ((unsigned)b.gx * (unsigned)b.gy)); }
};

// Persistent backprojection over the tiles of up to kBatchSlots scans: each
// CTA takes the next tile of the launch's work list (scans in order, tiles
// of a scan in the grid order x, y, z) until the list is exhausted, so the
// tail of one scan runs beside the start of the next.  Each scan's
// parameters sit at a fixed offset of the kernel's parameter space (slot S,
// a compile-time index), so the tile body reads them as constant operands
// exactly as the single-scan kernels do; a shared-memory or indexed copy of
// them measured 16-27 % slower (at a bound of 64 registers).  Each slot holds its
// scan's own tile depth (4 or 8 slices, a uniform branch per tile), so scans
// tuned to either depth share the launch.  DEEP: a launch of the mixed
// form's 16-slice tiles only, at that body's register bound (128 registers, four
// CTAs per SM; the mixed 4- and 8-slice bodies run at 72 and seven, the FP32 ones at
// 80 and six).  The next tile's index is fetched while the current one runs.
//
// Every tile runs the loop with the range test and 64-bit addresses, without the
// per-scan kernels' sorting of tiles: 16 scans of uneven size 688 GUPS (FP32; the
// per-scan launches of the pipelined schedule 882) and 986 (mixed; 1252).
// WV: every scan of the launch divides by its weight volume (p.wvol).
template <int S, bool MIXED, bool WZ, bool WV, bool DEEP>
__device__ __forceinline__ void batch_slot_tile(const BatchSlots& t) {
    constexpr int G = WZ ? kGeoWZ : kGeoWConst;
    const BatchTile tile{t.s[S]};
    if constexpr (DEEP) {
        static_assert(MIXED, "16-slice batch tiles are the mixed form's");
        bp_mixed_block<16, true, G, BatchTile, WV, false, false, true>(t.s[S].p, tile);
    } else if (t.s[S].zpt == 8) {
        if (MIXED)
            bp_mixed_block<8, true, G, BatchTile, WV, false, false, true>(t.s[S].p, tile);
        else
            bp_block<8, true, false, G, BatchTile, WV, false, false, true>(t.s[S].p, tile);
    } else {
        if (MIXED)
            bp_mixed_block<4, true, G, BatchTile, WV, false, false, true>(t.s[S].p, tile);
        else
            bp_block<4, true, false, G, BatchTile, WV, false, false, true>(t.s[S].p, tile);
    }
}

// The tile of slot si (si < kBatchSlots): a compile-time slot per case.
template <int S, bool MIXED, bool WZ, bool WV, bool DEEP>
__device__ __forceinline__ void batch_dispatch(const BatchSlots& t, int si) {
    if constexpr (S < kBatchSlots) {
        if (si == S)
            batch_slot_tile<S, MIXED, WZ, WV, DEEP>(t);
        else
            batch_dispatch<S + 1, MIXED, WZ, WV, DEEP>(t, si);
    }
}

template <bool MIXED, bool WZ, bool WV, bool DEEP>
__global__ void __launch_bounds__(kBPThreads, DEEP    ? bp_min_blocks(16)
                                              : MIXED ? bp_min_blocks(8)
                                                      : bp_fp32_min_blocks(8))
    bp_batch_kernel(const __grid_constant__ BatchSlots t, int nscans, unsigned* __restrict__ counter,
                    unsigned total) {
    __shared__ unsigned s_next;
    const int tid = threadIdx.y * kBPTileX + threadIdx.x;
    if (tid == 0) g_batch_tile = atomicAdd(counter, 1u);
    __syncthreads();
    for (;;) {
        const unsigned it = *static_cast<volatile unsigned*>(&g_batch_tile);
        if (it >= total) break;
        if (tid == 0) s_next = atomicAdd(counter, 1u);   // the next tile, while this one runs
        int si = 0;
        while (si + 1 < nscans && it >= t.s[si + 1].first_tile) ++si;
        batch_dispatch<0, MIXED, WZ, WV, DEEP>(t, si);
        __syncthreads();   // every thread is done with the current tile
        if (tid == 0) g_batch_tile = s_next;
        __syncthreads();
    }
}

template <bool M, bool W, bool V, bool D>
cudaError_t batch_go(const BatchSlots& t, int nscans, unsigned total, unsigned* counter, int ctas, cudaStream_t s) {
    bp_batch_kernel<M, W, V, D><<<ctas, dim3(kBPTileX, kBPTileY), 0, s>>>(t, nscans, counter, total);
    return cudaGetLastError();
}

template <bool M, bool W, bool V, bool D>
cudaError_t batch_occ(int* per) {
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(per, bp_batch_kernel<M, W, V, D>, kBPThreads, 0);
}

// deep: 16-slice tiles (the mixed form only)
template <bool M, bool W>
cudaError_t batch_go2(const BatchSlots& t, int nscans, unsigned total, unsigned* counter, int ctas, bool wv,
                      bool deep, cudaStream_t s) {
    if constexpr (M) {
        if (deep)
            return wv ? batch_go<M, W, true, true>(t, nscans, total, counter, ctas, s)
                      : batch_go<M, W, false, true>(t, nscans, total, counter, ctas, s);
    }
    return wv ? batch_go<M, W, true, false>(t, nscans, total, counter, ctas, s)
              : batch_go<M, W, false, false>(t, nscans, total, counter, ctas, s);
}

template <bool M, bool W>
cudaError_t batch_occ2(bool wv, bool deep, int* per) {
    if constexpr (M) {
        if (deep) return wv ? batch_occ<M, W, true, true>(per) : batch_occ<M, W, false, true>(per);
    }
    return wv ? batch_occ<M, W, true, false>(per) : batch_occ<M, W, false, false>(per);
}

}  // namespace
}  // namespace jfdk
