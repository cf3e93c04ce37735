// bp_body.cuh -- voxel-driven cone-beam backprojection with fused normalisation and
// CT numbers (sm_100a): the bodies of the kernels, which bp_fast.cu, bp_exact.cu,
// bp_weights.cu, bp_mixed.cu, bp_wide.cu and bp_batch.cuh instantiate (one file
// each, so that they compile side by side).
//
// Semantics follow the reference's CPU backprojector, BPCore
// (BPAgent/BPCore.cpp:115-220):
//   * per view the projection is multiplied by the view's u-taper and an
//     image of the taper is backprojected alongside it (the weight);
//   * for voxel (x, y, z): U = (x*P0 + (y*P1 + P3)) + z*P2, likewise V, W,
//     every product and sum rounded separately; u = U / W + 0.5,
//     v = V / W + 0.5 with the quotient correctly rounded (in the default form but
//     for a few in 10^9, bp_quotient2);
//   * bilinear sample with pixel centres at integers, taken only when
//     0 <= u <= cols-1 and 0 <= v <= rows-1 (ippiRemap leaves the destination
//     untouched otherwise, so the view then adds nothing to sum or weight);
//   * voxel = sum / weight, then CTNumCore (CTNumAgent/CTNumCore.cpp:22-36).
// The reference GPU kernel (BPCUDAAgent/BPCUDACore.cu:25-66) differs: it
// samples the taper without interpolation, checks only u and clamps v.
//
// Data layout.  The filtered, tapered projections are stored as "quads": for
// every view, row r and column c one float4 (p[r][c], p[r+1][c],
// RN(p[r][c+1] - p[r][c]), RN(p[r+1][c+1] - p[r+1][c])) -- the whole bilinear
// footprint of a sample point in one 16-byte load, with the column
// differences BPCore's lerp rounds already formed -- with zeros past the last
// row and column (pack_quads_kernel writes it).  The taper is stored as pairs
// (w[c], RN(w[c+1] - w[c])), w[U] = 0.  The volume is [z][y][x], x fastest.
//
// Work split.  A CTA is 128 threads over (x, y), TX x (128 / TX) (4 x 32 by
// default, 8 x 16 or 32 x 4 by option or autotuner); each thread owns ZPT
// consecutive slices of its (x, y) column and keeps (sum, weight) pairs in
// registers across all views of the launch, so a launch covering every view
// stores the volume once and never reads it.
//
// Arithmetic.  U, V are formed exactly as BPCore rounds them.  The quotients
// come from one reciprocal (bp_quotient2); when P[10] == 0 for every view W does
// not depend on z (BPCore adds z*0) and the reciprocal is computed once per
// (x, y, view).  EXACT additionally rounds the lerps step by step like
// BPCore (every product and sum separately) instead of fusing them.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "bp_common.cuh"
#include "jfdk_internal.h"

namespace jfdk {
namespace {

constexpr int kBPThreads = kBPTileX * kBPTileY;

// Resident CTAs per SM the compiler must allow for.  Small CTAs (4 warps)
// measured 4 % faster than 8-warp ones: a finishing CTA leaves fewer warps idle
// while the SM waits for the next.  Each warp covers 4 x 8 voxels in (x, y)
// rather than a row of 32: its sample points spread less on the detector
// (1.5-1.7 % faster than 32 x 1 in both forms).
//
// FP32, 8 slices: 80 registers and 24 warps per SM with two views in flight,
// 111.0 ms a c2 volume (96 registers and 20 warps 112.3; one view at a time
// 114.2).  Mixed: bp_mixed_kernel's launches choose (bp_mixed.cu); these are the
// weights' and the batch kernel's.
constexpr int bp_min_blocks(int zpt) { return zpt == 8 ? 7 : zpt == 16 ? 4 : 1; }
constexpr int bp_fp32_min_blocks(int zpt) { return zpt == 8 ? 6 : 1; }

// Least views of a launch that asks where its tiles lie (tile_inside): a CTA waits
// for the matrices before its first sample, which few views do not earn back
// (640 x 640 x 480 voxels from one view 1112 us with it and 1069 without, two 1301
// and 1250, four 1684 and 1696; mixed 8-slice tiles 256 x 256 x 160 from one 69.7
// and 67.7, two 76.5 and 81).  On an ideal orbit, and with 16 mixed slices a
// thread, the loops with the range test are the slower ones from the first view on;
// with W(z) the choice costs the loops of more views what it saves (one view 65.6
// and 63.6 us, 24 386 and 391).
constexpr int box_views_fp32(int geo) { return geo == kGeoWConst ? 4 : 0; }
constexpr int box_views_mixed(int zpt) { return zpt == 16 ? 0 : 2; }

// Where a CTA's tile lies: the launch grid's block index for the per-scan
// kernels, the current work item of the batch kernel.  The tile bodies ask
// for it at the start and again after the view loop: the batch kernel's
// tile is re-read from shared memory then rather than held in registers
// through the loop (at the 64-register bound that made the FP32 body spill).
// GridTile reads the block index with volatile moves, so the compiler reads
// it again after the loop instead of keeping x, y and z live through it:
// with the W(z) mixed body's U, V, W stepped per slice, that removed its
// spills (12 bytes stored, 360 bytes of reloads) and made it 6.5 % faster
// on a tilted c2 orbit; the FP32 kernels ran 0.8 % faster on c2.  The mixed
// body with z-independent W measured 1 % slower with it and keeps the plain
// read (GridTileHeld).  TX is the tile's width in x (threads along x); the
// CTA is TX x (128 / TX) threads, each warp 32 consecutive threads of it.
template <int TX>
struct GridTile {
    static constexpr int kX = TX, kY = kBPThreads / TX;
    __device__ static int ctaid(int d) {
        unsigned r;
        if (d == 0) asm volatile("mov.u32 %0, %%ctaid.x;" : "=r"(r));
        else if (d == 1) asm volatile("mov.u32 %0, %%ctaid.y;" : "=r"(r));
        else asm volatile("mov.u32 %0, %%ctaid.z;" : "=r"(r));
        return (int)r;
    }
    __device__ int bx() const { return ctaid(0); }
    __device__ int by() const { return ctaid(1); }
    __device__ int bz() const { return ctaid(2); }
};

template <int TX>
struct GridTileHeld {
    static constexpr int kX = TX, kY = kBPThreads / TX;
    __device__ int bx() const { return blockIdx.x; }
    __device__ int by() const { return blockIdx.y; }
    __device__ int bz() const { return blockIdx.z; }
};

// Whether every voxel of the CTA's tile samples every view of the launch
// inside the detector (box_place), so that the view loop may leave out the
// range test (two compares and two selects of a sample's 28 instructions in the
// FP32 form, two minima in the mixed one); and in `none` a bit for each of the
// first kNoneViews views that no voxel of the tile samples, which the loop with
// the range test passes over (an offset detector misses a voxel in up to half
// of its views: 360 x 360 x 200 voxels from 360 offset views 7.4 -> 5.4 ms, and
// 1.4 % of c2's FP32 time).  The views are dealt over the CTA's threads: under
// 1 % of the loop's work, whatever the sizes.  Frames of more
// than 2^23 records are never inside (their record index is not exact in a
// float).  Every thread of the CTA calls it.
constexpr int kNoneViews = 4096;

template <int ZPT, class Tile>
__device__ __forceinline__ bool tile_inside(const BPParams& p, const Tile& tile, unsigned* none) {
    const int x = tile.bx() * Tile::kX, y = tile.by() * Tile::kY, z = p.z_begin + tile.bz() * ZPT;
    const VoxelBox box(bp_axis(x, p.X, p.pxy), bp_axis(min(x + Tile::kX, p.X) - 1, p.X, p.pxy), bp_axis(y, p.Y, p.pxy),
                       bp_axis(min(y + Tile::kY, p.Y) - 1, p.Y, p.pxy), bp_axis(z, p.Z, p.pz),
                       bp_axis(z + ZPT - 1, p.Z, p.pz));   // all slices a thread walks
    const int tid = threadIdx.y * Tile::kX + threadIdx.x;
    bool ok = (long long)p.U * p.V <= (1LL << 23);
    for (int n0 = 0; n0 < p.nv; n0 += kBPThreads) {
        const int n = n0 + tid;
        const BoxPlace at = n < p.nv ? box_place(box, p.ptm + (size_t)(p.v0 + n) * 12, p.U, p.V) : kBoxInside;
        ok = ok && at == kBoxInside;
        const unsigned bits = __ballot_sync(0xffffffffu, at == kBoxOutside);
        if ((tid & 31) == 0 && n < kNoneViews) none[n >> 5] = bits;
    }
    return __syncthreads_and(ok);
}

// Whether any of the launch's views has its bit in none.
__device__ __forceinline__ bool any_none(const unsigned* none, int nv) {
    unsigned any = 0;
    for (int i = 0; i < (min(nv, kNoneViews) + 31) / 32; ++i) any |= none[i];
    return any != 0;
}

// The tile's (sum, weight) pairs: normalised, CT numbers, stored (FINALIZE),
// or stored as accumulators.  The coordinates are asked for again here.
// WV: the weights come from p.wvol (the whole volume, absolute slices).
template <int ZPT, bool FINALIZE, class Tile, bool WV = false>
__device__ __forceinline__ void epilogue(const BPParams& p, const Tile& tile, const float2 (&acc)[ZPT]) {
    const int x = tile.bx() * Tile::kX + threadIdx.x;
    const int y = tile.by() * Tile::kY + threadIdx.y;
    const int zb = p.z_begin + tile.bz() * ZPT;
#pragma unroll
    for (int k = 0; k < ZPT; ++k) {
        if (zb + k >= p.z_end) break;
        if (FINALIZE) {
            const size_t idx = ((size_t)(zb + k - p.out_z0) * p.Y + y) * p.X + x;
            const float wsum = WV ? __ldg(p.wvol + ((size_t)(zb + k) * p.Y + y) * p.X + x) : acc[k].y;
            float o = __fdiv_rn(acc[k].x, wsum);   // BPCore::DoneSlice
            if (p.apply_ct) o = ct_number(o, p.ct_scale, p.ct_norm1);
            if (p.out) p.out[idx] = o;
            if (p.out16) p.out16[idx] = to_i16(o);
        } else {
            const size_t idx = ((size_t)(zb + k - p.acc_z0) * p.Y + y) * p.X + x;
            p.sum[idx] = acc[k].x;
            p.cnt[idx] = acc[k].y;
        }
    }
}

// One sample's lerp of a quad, and its taper lerp: fused, or rounded step by
// step like BPCore (EXACT).
template <bool EXACT>
__device__ __forceinline__ float quad_lerp(const float4& Q, float2 fxy) {
    const float2 lo = f2(Q.x, Q.y), d = f2(Q.z, Q.w);    // column ix, RN(column ix+1 - ix)
    if (EXACT) {
        const float t0 = __fadd_rn(lo.x, __fmul_rn(fxy.x, d.x));
        const float t1 = __fadd_rn(lo.y, __fmul_rn(fxy.x, d.y));
        return __fadd_rn(t0, __fmul_rn(fxy.y, __fsub_rn(t1, t0)));
    }
    const float2 t = pfma(f2(fxy.x, fxy.x), d, lo);
    return fmaf(fxy.y, t.y - t.x, t.x);
}

template <bool EXACT>
__device__ __forceinline__ float taper_lerp(float2 w, float fx) {
    return EXACT ? __fadd_rn(w.x, __fmul_rn(fx, w.y)) : fmaf(fx, w.y, w.x);
}

// The view loop of a thread's ZPT slices.  INSIDE: no sample of the tile can
// leave the detector (tile_inside), so no range test.  G: how the sample's
// place depends on z (Geo in jfdk_internal.h).
//
// What bounds the loop is the FMA pipe: a packed operation takes it for two
// cycles, a scalar one for one (both measured), so packing saves issue slots
// only.  At G = kGeoWConst a sample takes 24 cycles of it (products and sums of
// U, V 4, quotients 4, + 0.5 2, floor and fraction 6, index 1, lerp and sum 5,
// the view's share 2) and about 20 issue slots; the 16-byte loads take the L1
// data pipe for as long (6 wavefronts a request: four, and one for each second
// quarter-warp whose records cross a 128-byte line).  c2, 1.18e11 samples:
// 127.9 ms with range tests, 64-bit addresses, Markstein's quotient and one
// view at a time, 102.8 now (33 cycles a sample and scheduler).  At kGeoIdeal
// u is the view's and V, v and the rest are formed for two slices at a time, 14
// cycles of the FMA pipe a sample.
// Measured and left out: floor on the conversion pipe (0.9 ms of 114 faster,
// more registers), the products z P[2], z P[6] from shared memory (9 slower).
template <int ZPT, bool EXACT, int G, bool WV, bool WEIGHTS, bool INSIDE, bool WIDE, bool SKIP = false>
__device__ __forceinline__ void bp_views(const BPParams& p, const unsigned* none, float ax, float ay,
                                         const float (&az)[ZPT], float2 (&acc)[ZPT]) {
    constexpr bool WZ = G == kGeoWZ;
    const unsigned umax_bits = __float_as_uint((float)(p.U - 1)), vmax_bits = __float_as_uint((float)(p.V - 1));
    const float Uf = (float)p.U;
    const float2 magic = f2(kMagic, kMagic);

    // Pointers step from view to view (index arithmetic on v0 and view_base
    // inside the loop measured over 10% slower at the 64-register bound).
    const float4* P4 = reinterpret_cast<const float4*>(p.ptm + (size_t)p.v0 * 12);
    const float4* __restrict__ q = p.q4 + (size_t)(p.v0 - p.view_base) * p.q4_frame;
    size_t qi = record_base(q);
    const float2* __restrict__ tw = p.tw + (size_t)p.v0 * p.U;
    constexpr int kUnroll = INSIDE ? 2 : 1;   // two views in flight where the registers allow it
#pragma unroll kUnroll
    for (int n = 0; n < p.nv; ++n, P4 += 3, q += p.q4_frame, qi += p.q4_frame * sizeof(float4), tw += p.U) {
        if (SKIP && n < kNoneViews && (none[n >> 5] >> (n & 31) & 1u)) continue;
        const float4 r0 = __ldg(P4), r1 = __ldg(P4 + 1), r2 = __ldg(P4 + 2);
        const XYTerms xy = bp_xy_terms(ax, ay, r0, r1, r2);
        const Recip rc = WZ ? Recip{0.0f, 0.0f} : bp_recip(xy.W);
        // the sums of (val, c) round as the packed add does
        auto sum = [&](int k, float val, float c) {
            if constexpr (WV) acc[k].x = __fadd_rn(acc[k].x, val);
            else if constexpr (WEIGHTS) acc[k].y = __fadd_rn(acc[k].y, c);
            else acc[k] = padd(acc[k], f2(val, c));
        };
        if constexpr (G == kGeoIdeal) {
            float u = bp_quotient<EXACT>(xy.U, xy.W, rc) + 0.5f;
            const bool inu = __float_as_uint(u) <= umax_bits;
            if (!INSIDE) u = inu ? u : 0.0f;
            const float tx = __fadd_rd(u, kMagic);
            const float fx = __fsub_rn(u, __fsub_rn(tx, kMagic));
            const unsigned ix = __float_as_uint(tx) - (unsigned)kMagicBits;
            float c = 0.0f;
            if constexpr (!WV) c = taper_lerp<EXACT>(load_at<false>(tw, ix), fx);
#pragma unroll
            for (int k = 0; k < ZPT; k += 2) {
                const float2 V = f2(__fadd_rn(xy.V, __fmul_rn(az[k], r1.z)), __fadd_rn(xy.V, __fmul_rn(az[k + 1], r1.z)));
                float2 v = padd(bp_quotient2<EXACT>(V, xy.W, rc), f2(0.5f, 0.5f));
                bool in0 = true, in1 = true;
                if constexpr (!INSIDE) {
                    in0 = inu & (__float_as_uint(v.x) <= vmax_bits);
                    in1 = inu & (__float_as_uint(v.y) <= vmax_bits);
                    v = f2(in0 ? v.x : 0.0f, in1 ? v.y : 0.0f);
                }
                const float2 t = padd_rm(v, magic);
                const float2 fl = psub(t, magic);
                const float2 fy = psub(v, fl);
                float val0 = 0.0f, val1 = 0.0f;
                if constexpr (!WEIGHTS) {
                    float4 Q0, Q1;
                    if constexpr (INSIDE) {
                        Q0 = load_record<float4>(qi, tx, fl.x, Uf);
                        Q1 = load_record<float4>(qi, tx, fl.y, Uf);
                    } else {
                        Q0 = load_at<WIDE>(q, (__float_as_uint(t.x) - (unsigned)kMagicBits) * (unsigned)p.U + ix);
                        Q1 = load_at<WIDE>(q, (__float_as_uint(t.y) - (unsigned)kMagicBits) * (unsigned)p.U + ix);
                    }
                    val0 = quad_lerp<EXACT>(Q0, f2(fx, fy.x));
                    val1 = quad_lerp<EXACT>(Q1, f2(fx, fy.y));
                }
                if (in0) sum(k, val0, c);
                if (in1) sum(k + 1, val1, c);
            }
        } else {
#pragma unroll
            for (int k = 0; k < ZPT; ++k) {
                float2 uv = bp_uv<EXACT, WZ>(xy, rc, az[k], r0.z, r1.z, r2.z);
                if constexpr (INSIDE) {
                    const float2 t = padd_rm(uv, magic);         // 2^23 + floor(uv)
                    const float2 fl = psub(t, magic);
                    const float2 fxy = psub(uv, fl);             // (u - fu, v - fv), exact
                    float val = 0.0f, c = 0.0f;
                    if constexpr (!WEIGHTS) val = quad_lerp<EXACT>(load_record<float4>(qi, t.x, fl.y, Uf), fxy);
                    if constexpr (!WV)
                        c = taper_lerp<EXACT>(load_at<false>(tw, __float_as_uint(t.x) - (unsigned)kMagicBits), fxy.x);
                    sum(k, val, c);
                } else {
                    // Branch-free so the loads of all ZPT slices can be in flight at
                    // once: a point off the detector reads quad (0, 0) and adds nothing.
                    // 0 <= u <= umax on the bit patterns: non-negative floats order like
                    // their bits, negatives and NaN have larger unsigned patterns (u is
                    // never -0: RN(U / W) + 0.5 rounds an exact zero to +0)
                    const bool in = (__float_as_uint(uv.x) <= umax_bits) & (__float_as_uint(uv.y) <= vmax_bits);
                    uv = in ? uv : f2(0.0f, 0.0f);
                    const float2 t = padd_rm(uv, magic);             // 2^23 + floor(uv)
                    const float2 fxy = psub(uv, psub(t, magic));     // (u - fu, v - fv), exact
                    const unsigned ix = __float_as_uint(t.x) - (unsigned)kMagicBits;
                    const unsigned idx = (__float_as_uint(t.y) - (unsigned)kMagicBits) * (unsigned)p.U + ix;
                    float val = 0.0f, c = 0.0f;
                    if constexpr (!WEIGHTS) val = quad_lerp<EXACT>(load_at<WIDE>(q, idx), fxy);
                    if constexpr (!WV) c = taper_lerp<EXACT>(load_at<false>(tw, ix), fxy.x);
                    if (in) sum(k, val, c);
                }
            }
        }
    }
}

// WV: the normalisation weights come from p.wvol (finalize over every view):
// the view loop loads and accumulates only the projection samples.
// WEIGHTS: the loop accumulates only the weights and stores them to out at
// absolute slices (launch_bp_weights).
// SPLIT: tiles that lie inside every view run their own copy of the loop.
template <int ZPT, bool FINALIZE, bool EXACT, int G, class Tile, bool WV = false, bool WEIGHTS = false,
          bool SPLIT = true, bool WIDE = false>
__device__ __forceinline__ void bp_block(const BPParams& p, const Tile& tile, float* wout = nullptr) {
    unsigned* none = nullptr;
    bool asked = false, inside = false;
    if constexpr (SPLIT) {
        __shared__ unsigned none_bits[kNoneViews / 32];
        none = none_bits;
        asked = box_views_fp32(G) == 0 || p.nv >= box_views_fp32(G);
        if (asked) inside = tile_inside<ZPT>(p, tile, none);
    }
    const int x = tile.bx() * Tile::kX + threadIdx.x;
    const int y = tile.by() * Tile::kY + threadIdx.y;
    const int zb = p.z_begin + tile.bz() * ZPT;
    if (x >= p.X || y >= p.Y) return;

    const float ax = bp_axis(x, p.X, p.pxy), ay = bp_axis(y, p.Y, p.pxy);
    float az[ZPT];
    float2 acc[ZPT];  // (sum, weight)
#pragma unroll
    for (int k = 0; k < ZPT; ++k) {
        az[k] = bp_axis(zb + k, p.Z, p.pz);
        acc[k] = f2(0.0f, 0.0f);
        if (!FINALIZE && p.load_acc && zb + k < p.z_end) {
            const size_t i = ((size_t)(zb + k - p.acc_z0) * p.Y + y) * p.X + x;
            acc[k] = f2(p.sum[i], p.cnt[i]);
        }
    }
    if (SPLIT && inside)
        bp_views<ZPT, EXACT, G, WV, WEIGHTS, true, WIDE>(p, none, ax, ay, az, acc);
    else if (SPLIT && asked && any_none(none, p.nv))
        bp_views<ZPT, EXACT, G, WV, WEIGHTS, false, WIDE, SPLIT>(p, none, ax, ay, az, acc);
    else
        bp_views<ZPT, EXACT, G, WV, WEIGHTS, false, WIDE>(p, none, ax, ay, az, acc);

    if constexpr (WEIGHTS) {
#pragma unroll
        for (int k = 0; k < ZPT; ++k)
            if (zb + k < p.z_end) wout[((size_t)(zb + k) * p.Y + y) * p.X + x] = acc[k].y;
        return;
    }
    // The output index is formed here, not before the view loop, so that it
    // holds no registers across the loop.
    epilogue<ZPT, FINALIZE, Tile, WV>(p, tile, acc);
}

// ---- mixed precision ---------------------------------------------------------
// Record per (slot, row r, column c), 8 bytes, the tapered footprint
// p00 = p[r][c], p01 = p[r][c+1], p10 = p[r+1][c], p11 = p[r+1][c+1] divided
// by the view's power-of-two scale s, in FP16, as the coefficients of the
// bilinear form  val = p00 + fx dx + fy (dy + fx dxy):
//   .x  half2 (p00, dx = p01 - p00)
//   .y  half2 (dy = p10 - p00, dxy = p11 - p10 - p01 + p00)
// each difference rounded against the already rounded coefficients, so every
// corner the form reproduces carries the rounding of one coefficient only.
// The records of the last row and the last column are zero: their samples
// are not taken (below), and an index clamped onto them reads nothing.
// The interpolation is two FP16 x FP16 + FP32 fused multiply-adds
// (fma.rn.f32.f16, products exact in FP32) and one FP32 one.
// The coordinates use an approximate reciprocal of W and fused
// multiply-adds; when W does not depend on z the slices of a thread are
// equally spaced on the detector and u, v advance by a constant per slice.
// A sample is taken when floor(u) <= cols-2 and floor(v) <= rows-2 (the
// same set as 0 <= u <= cols-1, 0 <= v <= rows-1 up to the measure-zero
// points u = cols-1, v = rows-1) and W > 0.  The lerps, the rescale by s and
// the (sum, weight) accumulation are FP32; the weight is the FP32 taper
// pair's lerp at the sample's FP32 fraction.
// WV: the weights come from p.wvol (finalize over every view), so the loop
// clamps the index onto the zero records instead of testing the range and
// loads one record per sample.  WEIGHTS: the loop accumulates only the
// weights and stores them to out at absolute slices.
__device__ __forceinline__ float rcp_approx(float x) {
    float r;
    asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// p00 + fx dx + fy (dy + fx dxy) of an 8-byte record (fx rounded to FP16).
__device__ __forceinline__ float mixed_lerp(uint2 rec, float2 f) {
    float v1, inner;
    asm("{\n .reg .f16 p0, dx, dy, dxy, fh;\n .reg .f32 p0f, dyf;\n"
        " mov.b32 {p0, dx}, %2;\n mov.b32 {dy, dxy}, %3;\n"
        " cvt.rn.f16.f32 fh, %4;\n cvt.f32.f16 p0f, p0;\n cvt.f32.f16 dyf, dy;\n"
        " fma.rn.f32.f16 %0, fh, dx, p0f;\n fma.rn.f32.f16 %1, fh, dxy, dyf;\n}"
        : "=f"(v1), "=f"(inner)
        : "r"(rec.x), "r"(rec.y), "f"(f.x));
    return fmaf(f.y, inner, v1);
}

template <int ZPT, int G, bool WV, bool WEIGHTS, bool INSIDE, bool WIDE, bool SKIP = false>
__device__ __forceinline__ void bp_mixed_views(const BPParams& p, const unsigned* none, float ax, float ay, float az0,
                                               float2 (&acc)[ZPT]) {
    constexpr bool WZ = G == kGeoWZ;
    const unsigned um1 = (unsigned)(p.U - 1), vm1 = (unsigned)(p.V - 1), uu = (unsigned)p.U;
    const float Uf = (float)p.U;
    const float2 magic = f2(kMagic, kMagic);

    const float4* P4 = reinterpret_cast<const float4*>(p.ptm + (size_t)p.v0 * 12);
    const float* sc = p.qscale + p.v0;
    const uint2* __restrict__ q = p.qh + (size_t)(p.v0 - p.view_base) * p.q4_frame;
    size_t qi = record_base(q);
    const float2* __restrict__ tw = p.tw + (size_t)p.v0 * p.U;
#pragma unroll 2   // two views in flight: 82.4 against 87.6 ms on c2
    for (int n = 0; n < p.nv; ++n, P4 += 3, ++sc, q += p.q4_frame, qi += p.q4_frame * sizeof(uint2), tw += p.U) {
        if (SKIP && n < kNoneViews && (none[n >> 5] >> (n & 31) & 1u)) continue;
        const float4 r0 = __ldg(P4), r1 = __ldg(P4 + 1), r2 = __ldg(P4 + 2);
        const float2 P26 = f2(r0.z, r1.z);
        // U, V, W at slice zb
        const float2 UV0 = pfma(f2(az0, az0), P26,
                                pfma(f2(ax, ax), f2(r0.x, r1.x), pfma(f2(ay, ay), f2(r0.y, r1.y), f2(r0.w, r1.w))));
        const float W0 = fmaf(az0, r2.z, fmaf(ax, r2.x, fmaf(ay, r2.y, r2.w)));
        if (!INSIDE && !WZ && !(W0 > 0.0f)) continue;   // a point at or behind the source plane samples nothing
        // !WZ: (u, v) itself steps from slice to slice.  WZ: U, V and W step
        // (one add each per slice, no per-slice offsets held through the loop)
        float2 uv = f2(0.f, 0.f), duv = f2(0.f, 0.f), UVk = UV0;
        float Wk = W0, dW = 0.f;
        if (!WZ) {
            const float r = rcp_approx(W0);
            uv = pfma(UV0, f2(r, r), f2(0.5f, 0.5f));
            const float rz = __fmul_rn(r, p.pz);
            duv = f2(__fmul_rn(P26.x, rz), __fmul_rn(P26.y, rz));
        } else {
            duv = f2(__fmul_rn(P26.x, p.pz), __fmul_rn(P26.y, p.pz));
            dW = __fmul_rn(p.pz, r2.z);
        }
        // (scalar products: a packed product feeding the packed adds below
        // may be fused into them, differently in each kernel built from here)
        const float s = __ldg(sc);
        if constexpr (G == kGeoIdeal && WV) {   // u and its fraction are the view's (duv.x = 0)
            const float tx = __fadd_rd(uv.x, kMagic);
            const float fx = __fsub_rn(uv.x, __fsub_rn(tx, kMagic));
            const unsigned iu = min(__float_as_uint(tx) - (unsigned)kMagicBits, um1);
            float v0 = uv.y;
#pragma unroll
            for (int k = 0; k < ZPT; k += 2) {
                const float v1 = __fadd_rn(v0, duv.y);
                const float2 cv = f2(v0, v1);
                v0 = __fadd_rn(v1, duv.y);
                const float2 t = padd_rm(cv, magic);
                const float2 fl = psub(t, magic);
                const float2 f = psub(cv, fl);
                uint2 rec0, rec1;
                if constexpr (INSIDE) {
                    rec0 = load_record<uint2>(qi, tx, fl.x, Uf);
                    rec1 = load_record<uint2>(qi, tx, fl.y, Uf);
                } else {
                    rec0 = load_at<WIDE>(q, min(__float_as_uint(t.x) - (unsigned)kMagicBits, vm1) * uu + iu);
                    rec1 = load_at<WIDE>(q, min(__float_as_uint(t.y) - (unsigned)kMagicBits, vm1) * uu + iu);
                }
                acc[k].x = fmaf(s, mixed_lerp(rec0, f2(fx, f.x)), acc[k].x);
                acc[k + 1].x = fmaf(s, mixed_lerp(rec1, f2(fx, f.y)), acc[k + 1].x);
            }
            continue;
        }
#pragma unroll
        for (int k = 0; k < ZPT; ++k) {
            float2 cuv;
            bool front = true;
            if (WZ) {
                const float r = rcp_approx(Wk);
                front = INSIDE || Wk > 0.0f;
                cuv = pfma(UVk, f2(r, r), f2(0.5f, 0.5f));
                UVk = padd(UVk, duv);
                Wk = __fadd_rn(Wk, dW);
            } else {
                cuv = uv;              // slice k: uv0 + k duv, stepped
                uv = padd(uv, duv);
            }
            const float2 t = padd_rm(cuv, magic);                     // 2^23 + floor(uv)
            const float2 fl = psub(t, magic);
            const float2 f = psub(cuv, fl);                           // fractions
            const unsigned iu = __float_as_uint(t.x) - (unsigned)kMagicBits;
            const unsigned iv = __float_as_uint(t.y) - (unsigned)kMagicBits;
            if constexpr (WV) {
                // out of range (negative / NaN wrap to large): a zero record
                const uint2 rec = INSIDE ? load_record<uint2>(qi, t.x, fl.y, Uf)
                                         : load_at<WIDE>(q, min(iv, vm1) * uu + min(iu, um1));
                const float val = mixed_lerp(rec, f);
                if (front) acc[k].x = fmaf(s, val, acc[k].x);
            } else {
                const bool in = INSIDE || ((iu < um1) & (iv < vm1) & front);
                const float2 w = load_at<false>(tw, in ? iu : 0u);
                const float c = fmaf(f.x, w.y, w.x);
                if constexpr (WEIGHTS) {
                    if (in) acc[k].y = __fadd_rn(acc[k].y, c);
                } else {
                    const uint2 rec = INSIDE ? load_record<uint2>(qi, t.x, fl.y, Uf)
                                             : load_at<WIDE>(q, in ? iv * uu + iu : 0u);
                    const float val = mixed_lerp(rec, f);
                    if (in) acc[k] = pfma(f2(s, 1.0f), f2(val, c), acc[k]);   // (s val + sum, c + weight)
                }
            }
        }
    }
}

template <int ZPT, bool FINALIZE, int G, class Tile, bool WV = false, bool WEIGHTS = false, bool SPLIT = true,
          bool WIDE = false>
__device__ __forceinline__ void bp_mixed_block(const BPParams& p, const Tile& tile, float* wout = nullptr) {
    unsigned* none = nullptr;
    bool asked = false, inside = false;
    if constexpr (SPLIT) {
        __shared__ unsigned none_bits[kNoneViews / 32];
        none = none_bits;
        asked = box_views_mixed(ZPT) == 0 || p.nv >= box_views_mixed(ZPT);
        if (asked) inside = tile_inside<ZPT>(p, tile, none);
    }
    const int x = tile.bx() * Tile::kX + threadIdx.x;
    const int y = tile.by() * Tile::kY + threadIdx.y;
    const int zb = p.z_begin + tile.bz() * ZPT;
    if (x >= p.X || y >= p.Y) return;
    // every rounding explicit, so that each kernel built from this body
    // (per-scan, batch, weights) forms the same coordinates
    const float ax = __fmul_rn(__fadd_rn((float)x, -0.5f * (float)(p.X - 1)), p.pxy);
    const float ay = __fmul_rn(__fadd_rn((float)y, -0.5f * (float)(p.Y - 1)), p.pxy);
    const float az0 = __fmul_rn(__fadd_rn((float)zb, -0.5f * (float)(p.Z - 1)), p.pz);
    float2 acc[ZPT];  // (sum, weight)
#pragma unroll
    for (int k = 0; k < ZPT; ++k) {
        acc[k] = f2(0.0f, 0.0f);
        if (!FINALIZE && p.load_acc && zb + k < p.z_end) {
            const size_t i = ((size_t)(zb + k - p.acc_z0) * p.Y + y) * p.X + x;
            acc[k] = f2(p.sum[i], p.cnt[i]);
        }
    }
    if (SPLIT && inside)
        bp_mixed_views<ZPT, G, WV, WEIGHTS, true, WIDE>(p, none, ax, ay, az0, acc);
    else if (SPLIT && asked && any_none(none, p.nv))
        bp_mixed_views<ZPT, G, WV, WEIGHTS, false, WIDE, SPLIT>(p, none, ax, ay, az0, acc);
    else
        bp_mixed_views<ZPT, G, WV, WEIGHTS, false, WIDE>(p, none, ax, ay, az0, acc);
    if constexpr (WEIGHTS) {
#pragma unroll
        for (int k = 0; k < ZPT; ++k)
            if (zb + k < p.z_end) wout[((size_t)(zb + k) * p.Y + y) * p.X + x] = acc[k].y;
        return;
    }
    epilogue<ZPT, FINALIZE, Tile, WV>(p, tile, acc);
}

// The launch grid covers the volume's columns with TX x (128 / TX) tiles and
// the launch's slices with ZPT-deep ones; threads outside the volume return
// at once, slices past z_end are skipped.
template <int TX>
dim3 bp_grid(const BPParams& p, int zpt) {
    constexpr int TY = kBPThreads / TX;
    const int nz = p.z_end - p.z_begin;
    return dim3((p.X + TX - 1) / TX, (p.Y + TY - 1) / TY, (nz + zpt - 1) / zpt);
}

}  // namespace
}  // namespace jfdk
