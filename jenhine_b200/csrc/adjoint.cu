// adjoint.cu -- derivatives of the FP32 FDK form (sm_100a):
//
//   * the adjoint of the backprojector, vol = S q / C: with the weights C
//     (the backprojected taper) fixed, q_bar = S^T (vol_bar / C) -- for every
//     voxel and view the transposed bilinear weights of its sample point, summed
//     per pixel and multiplied by the taper;
//   * the adjoint of the ramp filter, y = T (w o x) + c e(x) with
//     e(x) = (x0 + x1 + x2) / 3 (or the last three for a mirrored filter):
//     x_bar = w o (T^T y_bar) + (c . y_bar) / 3 on the edge samples;
//   * the gradient with respect to per-view projection-matrix parameters:
//     for a loss L(vol), dL/dtheta_j = sum over voxels of
//     vol_bar / C * [(dS/du - vol dC/du) du/dtheta_j + dS/dv dv/dtheta_j],
//     with u = U/W, du/dtheta_j = (dU_j - u dW_j) / W for (dU_j, dV_j, dW_j)
//     = (dP/dtheta_j) X; per-CTA partial sums in FP32, the reduction over
//     CTAs in FP64.
// Every kernel uses the default form's sample points and in-range decisions
// (bp_common.cuh), so the adjoint is the transpose of the forward as computed (of
// one with JFDK_OPT_BP_EXACT but for the quotients that bp_quotient2 rounds the
// other way).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>

#include "bp_common.cuh"
#include "jfdk_internal.h"

namespace jfdk {
namespace {

// rt = vol_bar / C (0 where no view saw the voxel).
__device__ __forceinline__ float residual(float vol_bar, float cnt) { return cnt != 0.0f ? vol_bar / cnt : 0.0f; }

constexpr int kAdjZpt = 8;

// rt times the bilinear weights at (u, v): lo on the upper row (left, right
// pixel), hi on the lower one.  Products of rt with each side's own weight, so
// that a small one is as exact as a large one (1 - f is exact) and an infinite
// rt gives infinities.
__device__ __forceinline__ void adjoint_weights(float2 uv, float rt, float2& lo, float2& hi) {
    const float2 magic = f2(kMagic, kMagic);
    const float2 f = psub(uv, psub(padd_rm(uv, magic), magic));
    const float2 g = psub(f2(1.0f, 1.0f), f);
    const float2 ab = pmul(f2(rt, rt), f2(g.x, f.x));
    hi = pmul(ab, f2(f.y, f.y));
    lo = pmul(ab, f2(g.y, g.y));
}

// Adjoint of the backprojection, q_bar[view][iv][iu] += w[iu] rt x (bilinear
// weights) over the voxels, in one of two ways (adjoint_by_patches chooses).
//
// By "quad space", the way of any scan and size: the forward's footprint records,
// one 16-byte vector reduction per sample, folded back to pixels and multiplied
// by the taper afterwards (unpack_adjoint_kernel).  A reduction takes 28 to 37
// cycles an SM and warp request, whatever the lanes' addresses, which is what
// bounds it; a thread per column and eight slices fills the GPU early.
__device__ __forceinline__ void red_add_v4(float4* p, float4 v) {
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w)
                 : "memory");
}

// (six CTAs per SM: with W(z) two registers more would leave five and a third wave
// of 256 x 256 x 48, 1010 against 885 us for 64 views)
template <bool WZ>
__global__ void __launch_bounds__(256, 6) bp_adjoint_quads_kernel(AdjParams p) {
    constexpr int ZPT = kAdjZpt;
    const int x = blockIdx.x * 32 + threadIdx.x;
    const int y = blockIdx.y * 8 + threadIdx.y;
    const int zb = blockIdx.z * ZPT;
    if (x >= p.X || y >= p.Y) return;
    const float ax = bp_axis(x, p.X, p.pxy), ay = bp_axis(y, p.Y, p.pxy);
    const size_t plane = (size_t)p.X * p.Y, base = (size_t)y * p.X + x;
    float az[ZPT], rt[ZPT];
    bool any = false;
#pragma unroll
    for (int k = 0; k < ZPT; ++k) {
        const size_t at = (size_t)(zb + k) * plane + base;
        az[k] = bp_axis(zb + k, p.Z, p.pz);
        rt[k] = zb + k < p.Z ? residual(p.vol_bar[at], p.cnt[at]) : 0.0f;
        any |= rt[k] != 0.0f;
    }
    if (!any) return;
    const unsigned umax_bits = __float_as_uint((float)(p.U - 1)), vmax_bits = __float_as_uint((float)(p.V - 1));
    const float4* P4 = reinterpret_cast<const float4*>(p.ptm + (size_t)p.v0 * 12);
    float4* __restrict__ qb = p.quads;
#pragma unroll 1
    for (int n = 0; n < p.nv; ++n, P4 += 3, qb += p.q_frame) {
        const float4 r0 = __ldg(P4), r1 = __ldg(P4 + 1), r2 = __ldg(P4 + 2);
        const XYTerms xy = bp_xy_terms(ax, ay, r0, r1, r2);
        const Recip rc = WZ ? Recip{0.0f, 0.0f} : bp_recip(xy.W);
#pragma unroll
        for (int k = 0; k < ZPT; ++k) {
            const float2 uv = bp_uv<false, WZ>(xy, rc, az[k], r0.z, r1.z, r2.z);
            if ((__float_as_uint(uv.x) <= umax_bits) & (__float_as_uint(uv.y) <= vmax_bits) & (rt[k] != 0.0f)) {
                float2 lo, hi;
                adjoint_weights(uv, rt[k], lo, hi);
                const float2 t = padd_rm(uv, f2(kMagic, kMagic));
                const unsigned iu = __float_as_uint(t.x) - (unsigned)kMagicBits;
                const unsigned iv = __float_as_uint(t.y) - (unsigned)kMagicBits;
                red_add_v4(qb + (size_t)iv * p.U + iu, make_float4(lo.x, hi.x, lo.y, hi.y));
            }
        }
    }
}

// Quad space -> detector pixels: p[r][c] appears in quads (r, c).x,
// (r-1, c).y, (r, c-1).z, (r-1, c-1).w, each times the taper w[c].
__global__ void __launch_bounds__(256) unpack_adjoint_kernel(AdjParams p) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= p.U) return;
    for (int f = blockIdx.z; f < p.nv; f += gridDim.z) {
        const float4* q = p.quads + (size_t)f * p.q_frame + c;
        float* out = p.qbar + (size_t)f * p.q_frame + c;
        const float w = p.tw[(size_t)((p.v0 + f) % p.num_views) * p.U + c].x;
        for (int r = blockIdx.y; r < p.V; r += gridDim.y) {
            const float4* at = q + (size_t)r * p.U;
            float s = at->x;
            if (r > 0) s += (at - p.U)->y;
            if (c > 0) s += (at - 1)->z;
            if (r > 0 && c > 0) s += (at - p.U - 1)->w;
            out[(size_t)r * p.U] = w * s;
        }
    }
}

// By patches: a warp sums the samples of a block of 8 x 8 columns and 32 slices
// in its own patch of the view, in shared memory (a load, an addition and a
// store there take 2.7 cycles a request, a scalar reduction to global memory over
// 32 neighbouring pixels 7.6), and adds the patch to global memory once per
// view, about half a pixel a sample.  The lanes are 32 slices of one column: they
// fall on different rows, and where consecutive slices are at least a row apart
// (checked per block and view) no two lanes hold the same pixel, so plain
// additions serve, first to the samples' upper rows, then to the lower ones;
// elsewhere shared-memory reductions (4.1 cycles each).  Samples outside the patch
// (it holds kPatch pixels; a sample on the last column has no right neighbour)
// go to global memory by themselves.  What bounds it is the shared memory: 20
// wavefronts a sample, eight of them bank conflicts (32 lanes spread over more
// than 32 rows).
constexpr int kPatch = 1024, kAdjCols = 64, kAdjWarps = 4, kAdjBatch = 4;
struct AdjWarp {
    float patch[kPatch];
    float rt[kAdjCols * 33];          // [column][slice], padded
    float4 xy[kAdjCols];              // U, V, W at z = 0 and RN(1 / W) of the view
};

template <bool WZ, bool INSIDE>
__device__ __forceinline__ void adjoint_views(const AdjParams& p, AdjWarp& m, const VoxelBox& box, int x0, int y0, int zb) {
    const int lane = threadIdx.x & 31;
    const unsigned umax_bits = __float_as_uint((float)(p.U - 1)), vmax_bits = __float_as_uint((float)(p.V - 1));
    const float az = bp_axis(zb + lane, p.Z, p.pz);
    // this lane's corner of the block
    const float xc = bp_axis(lane & 1 ? min(x0 + 8, p.X) - 1 : x0, p.X, p.pxy);
    const float yc = bp_axis(lane & 2 ? min(y0 + 8, p.Y) - 1 : y0, p.Y, p.pxy);
    const float zc = bp_axis(lane & 4 ? min(zb + 32, p.Z) - 1 : zb, p.Z, p.pz);
    const float2 magic = f2(kMagic, kMagic);
    const float4* P4 = reinterpret_cast<const float4*>(p.ptm + (size_t)p.v0 * 12);
    float* out = p.qbar;
#pragma unroll 1
    for (int n = 0; n < p.nv; ++n, P4 += 3, out += p.q_frame) {
        const float4 r0 = __ldg(P4), r1 = __ldg(P4 + 1), r2 = __ldg(P4 + 2);
        const float2* __restrict__ tw = p.tw + (size_t)((p.v0 + n) % p.num_views) * p.U;
        __syncwarp();   // the last view's columns and patch are done with
#pragma unroll
        for (int c = lane; c < kAdjCols; c += 32) {
            const XYTerms t = bp_xy_terms(bp_axis(min(x0 + (c & 7), p.X - 1), p.X, p.pxy),
                                          bp_axis(min(y0 + (c >> 3), p.Y - 1), p.Y, p.pxy), r0, r1, r2);
            m.xy[c] = make_float4(t.U, t.V, t.W, WZ ? 0.0f : rcp_rn_nr(t.W));
        }
        // the patch: the block's corners in the view, a little around them
        int c0 = 0, w = 0, row0 = 0, h = 0;
        bool apart = false;
        float wmin = 0.0f;
        {
            const float Vxy = fmaf(xc, r1.x, fmaf(yc, r1.y, r1.w)), Wxy = fmaf(xc, r2.x, fmaf(yc, r2.y, r2.w));
            const float U = fmaf(zc, r0.z, fmaf(xc, r0.x, fmaf(yc, r0.y, r0.w)));
            const float V = fmaf(zc, r1.z, Vxy), W = fmaf(zc, r2.z, Wxy);
            const float u = __fdividef(U, W) + 0.5f, v = __fdividef(V, W) + 0.5f;
            // dv/dz = (P6 W - P10 V) / W^2, its numerator the same in every slice
            const float d = fmaf(r1.z, Wxy, -r2.z * Vxy);
            float lo[4] = {u, v, W, d}, hi[4] = {u, v, W, d};
#pragma unroll
            for (int o = 1; o <= 4; o <<= 1)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    lo[i] = fminf(lo[i], __shfl_xor_sync(0xffffffffu, lo[i], o));
                    hi[i] = fmaxf(hi[i], __shfl_xor_sync(0xffffffffu, hi[i], o));
                }
            const float um = (float)(p.U - 1), vm = (float)(p.V - 1);
            // (comparisons false for NaN leave the patch empty)
            if (lo[2] > 0.0f && hi[0] >= 0.0f && lo[0] <= um && hi[1] >= 0.0f && lo[1] <= vm) {
                c0 = (int)fmaxf(lo[0] - 0.05f, 0.0f);
                row0 = (int)fmaxf(lo[1] - 0.05f, 0.0f);
                w = (int)fminf(hi[0] + 1.05f, um) - c0 + 1;
                h = (int)fminf(hi[1] + 1.05f, vm) - row0 + 1;
                const float dmin = lo[3] > 0.0f ? lo[3] : -hi[3];
                apart = p.pz * dmin > 1.01f * hi[2] * hi[2];
                wmin = lo[2];
            }
        }
        const int pitch = w | 1;   // odd: lanes a row apart use different banks
        const int full = h;
        h = min(h, kPatch / pitch);
        const unsigned wlim = (unsigned)max(w - 1, 0), hlim = (unsigned)max(h - 1, 0);
        // Every sample of the block's voxels lies in the patch, and consecutive
        // slices' rows differ: the rounded places are within 2^-22 of the sum of
        // the terms' moduli (over W), which has to be far below the 0.05 pixels
        // around the corners and the hundredth of a row above one; and the
        // patch's index below is exact in a float.
        const float lim = (float)(p.U + p.V);
        const float moduli = fmaf(box.mx, fabsf(r0.x) + fabsf(r1.x) + lim * fabsf(r2.x),
                                  fmaf(box.my, fabsf(r0.y) + fabsf(r1.y) + lim * fabsf(r2.y),
                                       fmaf(box.mz, fabsf(r0.z) + fabsf(r1.z) + lim * fabsf(r2.z),
                                            fabsf(r0.w) + fabsf(r1.w) + lim * fabsf(r2.w))));
        const bool whole = INSIDE && w > 0 && h == full && moduli * 0x1p-22f < 0.004f * wmin &&
                           (long long)(row0 + h) * pitch + c0 + w < (1LL << 23);
        const float pf = (float)pitch;
        const int first = row0 * pitch + c0;
        const bool zin = zb + lane < p.Z;
        __syncwarp();
        if (whole && apart) {
#pragma unroll 1
            for (int cb = 0; cb < kAdjCols; cb += kAdjBatch) {
                // the places and weights of kAdjBatch columns first, side by
                // side: the additions below follow one another
                float* s[kAdjBatch];
                float2 lo[kAdjBatch], hi[kAdjBatch];
#pragma unroll
                for (int k = 0; k < kAdjBatch; ++k) {
                    const float4 xw = m.xy[cb + k];
                    const Recip rc{xw.w, WZ ? 0.0f : __fmul_rn(fmaf(-xw.z, xw.w, 1.0f), xw.w)};
                    const float2 uv = bp_uv<false, WZ>(XYTerms{xw.x, xw.y, xw.z}, rc, az, r0.z, r1.z, r2.z);
                    adjoint_weights(uv, m.rt[(cb + k) * 33 + lane], lo[k], hi[k]);
                    const float2 t = padd_rm(uv, magic);
                    const int at = __float_as_int(fmaf(__fsub_rn(t.y, kMagic), pf, t.x)) - kMagicBits - first;
                    // (a lane past the last slice has no place in the patch)
                    s[k] = m.patch + (zin ? at : 0);
                }
#pragma unroll
                for (int k = 0; k < kAdjBatch; ++k) {
                    if (zin) { s[k][0] += lo[k].x; s[k][1] += lo[k].y; }
                    __syncwarp();
                    if (zin) { s[k][pitch] += hi[k].x; s[k][pitch + 1] += hi[k].y; }
                    __syncwarp();
                }
            }
        } else {
#pragma unroll 1
            for (int c = 0; c < kAdjCols; ++c) {
                const float4 xw = m.xy[c];
                const float rt = m.rt[c * 33 + lane];
                const Recip rc{xw.w, WZ ? 0.0f : __fmul_rn(fmaf(-xw.z, xw.w, 1.0f), xw.w)};
                float2 uv = bp_uv<false, WZ>(XYTerms{xw.x, xw.y, xw.z}, rc, az, r0.z, r1.z, r2.z);
                const bool in = (rt != 0.0f) & (INSIDE || ((__float_as_uint(uv.x) <= umax_bits) & (__float_as_uint(uv.y) <= vmax_bits)));
                uv = in ? uv : f2(0.0f, 0.0f);
                float2 lo, hi;
                adjoint_weights(uv, rt, lo, hi);
                const float2 t = padd_rm(uv, magic);
                const int iu = __float_as_int(t.x) - kMagicBits, iv = __float_as_int(t.y) - kMagicBits;
                const bool inner = ((unsigned)(iu - c0) < wlim) & ((unsigned)(iv - row0) < hlim);
                if (in & inner) {
                    float* s = m.patch + (iv * pitch + iu - first);
                    atomicAdd(s, lo.x); atomicAdd(s + 1, lo.y);
                    atomicAdd(s + pitch, hi.x); atomicAdd(s + pitch + 1, hi.y);
                } else if (in) {   // pixels past the last row and column do not exist (their weight is 0)
                    float* g = out + (size_t)iv * p.U + iu;
                    const bool right = iu + 1 < p.U, down = iv + 1 < p.V;
                    const float wl = tw[iu].x, wr = right ? tw[iu + 1].x : 0.0f;
                    atomicAdd(g, wl * lo.x);
                    if (right) atomicAdd(g + 1, wr * lo.y);
                    if (down) atomicAdd(g + p.U, wl * hi.x);
                    if (right && down) atomicAdd(g + p.U + 1, wr * hi.y);
                }
            }
        }
        __syncwarp();
        // add the patch to the view, and clear it for the next one
        const int dr = 32 / pitch, dc = 32 % pitch;
        int row = lane / pitch, col = lane % pitch;
        for (int i = lane; i < pitch * h; i += 32) {
            const float v = m.patch[i];
            if (v != 0.0f) {   // (true for NaN)
                m.patch[i] = 0.0f;
                atomicAdd(out + (size_t)(row0 + row) * p.U + c0 + col, v * tw[c0 + col].x);
            }
            row += dr;
            col += dc;
            if (col >= pitch) { col -= pitch; ++row; }
        }
    }
}

template <bool WZ>
__global__ void __launch_bounds__(32 * kAdjWarps, 4) bp_adjoint_kernel(AdjParams p) {
    extern __shared__ AdjWarp adj_warps[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    AdjWarp& m = adj_warps[warp];
    const int x0 = blockIdx.x * 16 + (warp & 1) * 8, y0 = blockIdx.y * 16 + (warp >> 1) * 8, zb = blockIdx.z * 32;
    if (x0 >= p.X || y0 >= p.Y) return;   // (the warps do not wait for each other)
    for (int i = lane; i < kPatch; i += 32) m.patch[i] = 0.0f;
    const size_t plane = (size_t)p.X * p.Y;
    bool any = false;
    // 8 voxels in x by 4 slices to a load
    const int x = x0 + (lane & 7);
    for (int i = 0; i < 64; ++i) {
        const int y = y0 + (i & 7), z = (i >> 3) * 4 + (lane >> 3);
        float r = 0.0f;
        if (x < p.X && y < p.Y && zb + z < p.Z) {
            const size_t at = (size_t)(zb + z) * plane + (size_t)y * p.X + x;
            r = residual(p.vol_bar[at], p.cnt[at]);
        }
        m.rt[((i & 7) * 8 + (lane & 7)) * 33 + z] = r;
        any |= r != 0.0f;
    }
    if (!__any_sync(0xffffffffu, any)) return;
    bool ok = true;
    // (lanes past the last slice add nothing: thin volumes are inside too)
    const VoxelBox box(bp_axis(x0, p.X, p.pxy), bp_axis(min(x0 + 8, p.X) - 1, p.X, p.pxy), bp_axis(y0, p.Y, p.pxy),
                       bp_axis(min(y0 + 8, p.Y) - 1, p.Y, p.pxy), bp_axis(zb, p.Z, p.pz),
                       bp_axis(min(zb + 32, p.Z) - 1, p.Z, p.pz));
    for (int n = lane; n < p.nv; n += 32) ok = ok && box_place(box, p.ptm + (size_t)(p.v0 + n) * 12, p.U, p.V) == kBoxInside;
    if (__all_sync(0xffffffffu, ok))
        adjoint_views<WZ, true>(p, m, box, x0, y0, zb);
    else
        adjoint_views<WZ, false>(p, m, box, x0, y0, zb);
}

// Geometry gradient: per (CTA, view) partial sums of the 6 components.
//
// For a sample with a_u = rt (dS/du - vol dC/du) / W, a_v = rt dS/dv / W and
// s = a_u u + a_v v, the contribution to component j is
// a_u dU_j + a_v dV_j - s dW_j with (dU_j, dV_j, dW_j) = dP_j (x, y, z, 1).
// That is linear in dP_j, so a thread only sums, over its slices, the six
// moments a_u, a_u z, a_v, a_v z, s, s z; per view they become the twelve
// coefficients m of the 3x4 matrix dP_j (m = (x A, y A, A_z, A) for the U
// row, likewise B for V and -C for W); the CTA sums m over its threads
// (a transposing butterfly in each warp, then shared memory), and six
// threads form sum_i dP_j[i] m[i].  dP is read once per CTA and view.
//
// What bounds it is instruction issue and the latency of its loads (52
// instructions a sample, the place's exact rounding and the W(z) reciprocal
// among them).  The reduction costs about 65 instructions a thread and view, so
// a thread walks J = 4 columns of kAdjZpt slices before each, rt and vol of its
// voxels waiting in shared memory (one 8-byte load a sample); warps of 4 x 8
// voxels rather than 32 x 1 sample fewer records (L1 hits 84 %); tiles inside
// the detector run without the range test.  Eight samples in flight at 128
// registers and 16 warps measured faster than more warps: a 64-view chunk of
// 256^3 from 512^2 takes 2.1 ms, 2.3 with W(z) (96 registers and 20 warps 2.9, 80
// and 24 3.2; 3.26 with the reduction every 8 samples, 32 x 1 warps and 64
// registers).
// J is 1 where 4 would leave less than a full wave of CTAs.
constexpr int kGradThreads = 128, kGradRows = kGradThreads / 8;   // 8 columns x kGradRows of warps of 4 x 8
constexpr int kGradRed = 2 * (kGradThreads / 32) * 16;           // floats the CTA's reduction takes, double buffered

template <int J, bool WZ, bool INSIDE>
__device__ __forceinline__ void gradient_views(const AdjParams& p, const float2* vox, float* red, int x0, int y, int zb) {
    constexpr int ZPT = kAdjZpt;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const unsigned umax_bits = __float_as_uint((float)(p.U - 1)), vmax_bits = __float_as_uint((float)(p.V - 1));
    const float ay = bp_axis(y, p.Y, p.pxy), Uf = (float)p.U;
    float az[ZPT];
#pragma unroll
    for (int k = 0; k < ZPT; ++k) az[k] = bp_axis(zb + k, p.Z, p.pz);
    const size_t cta = ((size_t)blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x;
    const size_t ncta = (size_t)gridDim.x * gridDim.y * gridDim.z;
    const float4* P4 = reinterpret_cast<const float4*>(p.ptm + (size_t)p.v0 * 12);
    const float4* __restrict__ q = p.q4;
    size_t qi = record_base(q);
    const float2 magic = f2(kMagic, kMagic);
#pragma unroll 1
    for (int n = 0; n < p.nv; ++n, P4 += 3, q += p.q_frame, qi += p.q_frame * sizeof(float4)) {
        const float4 r0 = __ldg(P4), r1 = __ldg(P4 + 1), r2 = __ldg(P4 + 2);
        const float2* __restrict__ tw = p.tw + (size_t)((p.v0 + n) % p.num_views) * p.U;
        // sums over the thread's voxels of a, a x, a z (a = a_u, a_v, s)
        float A = 0.f, Ax = 0.f, Az = 0.f, B = 0.f, Bx = 0.f, Bz = 0.f, C = 0.f, Cx = 0.f, Cz = 0.f;
#pragma unroll 1
        for (int j = 0; j < J; ++j) {
            const float ax = bp_axis(min(x0 + 8 * j, p.X - 1), p.X, p.pxy);
            const XYTerms xy = bp_xy_terms(ax, ay, r0, r1, r2);
            const Recip rc = WZ ? Recip{0.0f, 0.0f} : bp_recip(xy.W);
            const float2* vx = vox + j * ZPT * kGradThreads + tid;
            float A0 = 0.f, B0 = 0.f, C0 = 0.f;
#pragma unroll
            for (int k = 0; k < ZPT; ++k) {
                float2 wr, uv0;                                        // W, RN(1 / W); U / W, V / W
                float2 uv = bp_uv<false, WZ>(xy, rc, az[k], r0.z, r1.z, r2.z, &wr, &uv0);
                const float2 rv = vx[k * kGradThreads];                         // (rt, vol)
                bool use = rv.x != 0.0f;
                if (!INSIDE) {
                    use = use & (__float_as_uint(uv.x) <= umax_bits) & (__float_as_uint(uv.y) <= vmax_bits);
                    uv = use ? uv : f2(0.0f, 0.0f);
                }
                const float2 t = padd_rm(uv, magic);                   // 2^23 + floor
                const float2 fl = psub(t, magic);
                const float2 f = psub(uv, fl);
                const unsigned iu = __float_as_uint(t.x) - (unsigned)kMagicBits;
                const float4 Q = INSIDE ? load_record<float4>(qi, t.x, fl.y, Uf)
                                        : __ldg(q + ((size_t)(__float_as_uint(t.y) - (unsigned)kMagicBits) * (unsigned)p.U + iu));
                const float2 w = load_at<false>(tw, iu);
                // quads: (t00, t10, t01 - t00, t11 - t10); taper pairs (w0, w1 - w0)
                const float cross = Q.w - Q.z;
                const float dSu = fmaf(f.y, cross, Q.z);
                const float dSv = fmaf(f.x, cross, Q.y - Q.x);
                const float ri = rv.x * wr.y;                          // rt RN(1 / W)
                const float au = ri * fmaf(-rv.y, w.y, dSu), av = ri * dSv;
                const float sk = fmaf(au, uv0.x, av * uv0.y);
                if (use) {
                    A0 += au; Az = fmaf(au, az[k], Az);
                    B0 += av; Bz = fmaf(av, az[k], Bz);
                    C0 += sk; Cz = fmaf(sk, az[k], Cz);
                }
            }
            A += A0; Ax = fmaf(ax, A0, Ax);
            B += B0; Bx = fmaf(ax, B0, Bx);
            C += C0; Cx = fmaf(ax, C0, Cx);
        }
        // the coefficients of dP_j's twelve entries (padded to 16)
        float m[16] = {Ax, ay * A, Az, A, Bx, ay * B, Bz, B, -Cx, -ay * C, -Cz, -C, 0.f, 0.f, 0.f, 0.f};
        // transposing butterfly: after the steps at 16, 8, 4, 2 lanes apart
        // lane l holds one coefficient, index (l >> 1) & 15, summed over 16
        // lanes; the step at 1 completes the warp's sum
#pragma unroll
        for (int o = 16, h = 8; o >= 2; o >>= 1, h >>= 1) {
            const bool upper = (lane & o) != 0;
#pragma unroll
            for (int i = 0; i < h; ++i) {
                const float send = upper ? m[i] : m[i + h];
                const float keep = upper ? m[i + h] : m[i];
                m[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
            }
        }
        m[0] += __shfl_xor_sync(0xffffffffu, m[0], 1);
        float* buf = red + (n & 1) * (kGradThreads / 32) * 16;
        if ((lane & 1) == 0) buf[warp * 16 + (lane >> 1)] = m[0];
        __syncthreads();
        if (tid < 6) {
            float mc[12];
#pragma unroll
            for (int i = 0; i < 12; ++i) {
                float t = 0.0f;
#pragma unroll
                for (int w = 0; w < kGradThreads / 32; ++w) t += buf[w * 16 + i];
                mc[i] = t;
            }
            const float* d = p.dptm + (size_t)n * 72 + tid * 12;
            float g = 0.0f;
#pragma unroll
            for (int i = 0; i < 12; ++i) g = fmaf(__ldg(d + i), mc[i], g);
            p.partial[((size_t)n * ncta + cta) * 6 + tid] = g;
        }
    }
}

template <int J, bool WZ>
__global__ void __launch_bounds__(kGradThreads, 4) geometry_gradient_kernel(AdjParams p) {
    constexpr int ZPT = kAdjZpt;
    extern __shared__ float2 vox[];            // [J][ZPT][kGradThreads] (rt, vol)
    __shared__ float red[kGradRed];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int xb = blockIdx.x * 8 * J, yb = blockIdx.y * kGradRows, zb = blockIdx.z * ZPT;
    const int x0 = xb + (warp & 1) * 4 + (lane & 3), y = yb + (warp >> 1) * 8 + (lane >> 2);
    const size_t plane = (size_t)p.X * p.Y;
    for (int j = 0; j < J; ++j)
#pragma unroll
        for (int k = 0; k < ZPT; ++k) {
            float2 rv = f2(0.0f, 0.0f);
            if (x0 + 8 * j < p.X && y < p.Y && zb + k < p.Z) {
                const size_t i = (size_t)(zb + k) * plane + (size_t)y * p.X + x0 + 8 * j;
                rv = f2(residual(p.vol_bar[i], p.cnt[i]), p.vol[i]);
                if (!(rv.y == rv.y)) rv = f2(0.0f, 0.0f);   // unseen voxel: no contribution
            }
            vox[(j * ZPT + k) * kGradThreads + tid] = rv;            // read by this thread only
        }
    bool ok = (long long)p.U * p.V <= (1LL << 23);
    const VoxelBox box(bp_axis(xb, p.X, p.pxy), bp_axis(min(xb + 8 * J, p.X) - 1, p.X, p.pxy), bp_axis(yb, p.Y, p.pxy),
                       bp_axis(min(yb + kGradRows, p.Y) - 1, p.Y, p.pxy), bp_axis(zb, p.Z, p.pz),
                       bp_axis(zb + ZPT - 1, p.Z, p.pz));
    for (int n = tid; n < p.nv; n += kGradThreads) ok = ok && box_place(box, p.ptm + (size_t)(p.v0 + n) * 12, p.U, p.V) == kBoxInside;
    // threads past the volume's edge walk its last row and column with rt = 0
    const int yc = min(y, p.Y - 1);
    if (__syncthreads_and(ok))
        gradient_views<J, WZ, true>(p, vox, red, x0, yc, zb);
    else
        gradient_views<J, WZ, false>(p, vox, red, x0, yc, zb);
}

// grad[view][j] = sum over CTAs of the partials, in FP64: 192 threads read a
// view's partials as they lie (32 CTAs of 6 at a time, so a thread keeps to
// one component), then 32 per component are summed.
__global__ void __launch_bounds__(192) reduce_partials_kernel(const float* __restrict__ partial, size_t ncta, double* grad) {
    const size_t n = blockIdx.x;
    const float* src = partial + n * ncta * 6;
    double s = 0.0;
    for (size_t i = threadIdx.x; i < ncta * 6; i += 192) s += (double)src[i];
    __shared__ double part[192];
    part[threadIdx.x] = s;
    __syncthreads();
    if (threadIdx.x < 6) {
        s = 0.0;
        for (int c = 0; c < 32; ++c) s += part[c * 6 + threadIdx.x];
        grad[n * 6 + threadIdx.x] = s;
    }
}

// Filter adjoint, after out = T^T y_bar (rows of in_w): out *= w (the
// pre-weight of the row), then (c . y_bar) / 3 added to the edge samples.
__global__ void __launch_bounds__(256) filter_adjoint_finish_kernel(const float* __restrict__ ybar, int out_w,
                                                                    float* __restrict__ xbar, int in_w, int rows,
                                                                    int v0, int num_views,
                                                                    const float* __restrict__ pw,
                                                                    const float* __restrict__ c, int mirror) {
    const size_t m = (size_t)blockIdx.y * rows + blockIdx.x;
    const int row = blockIdx.x, view = (v0 + blockIdx.y) % num_views, g = view / 9;
    const float* yb = ybar + m * out_w;
    float* xb = xbar + m * in_w;
    const float* w = pw + ((size_t)g * rows + row) * in_w;
    float dot = 0.0f;
    for (int j = threadIdx.x; j < out_w; j += blockDim.x) dot = fmaf(c[j], yb[j], dot);
    __shared__ float part[8];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = dot;
    __syncthreads();
    float e = 0.0f;
    for (int i = 0; i < (int)(blockDim.x >> 5); ++i) e += part[i];
    e /= 3.0f;
    for (int i = threadIdx.x; i < in_w; i += blockDim.x) {
        float v = xb[i] * w[i];
        if (mirror ? (i >= in_w - 3) : (i < 3)) v += e;
        xb[i] = v;
    }
}

// y_bar [M][out_w] -> A operand rows [M][pitch], zero padded.
__global__ void pad_rows_kernel(const float* __restrict__ src, int w, float* __restrict__ dst, int pitch) {
    const size_t m = blockIdx.x;
    for (int i = threadIdx.x; i < pitch; i += blockDim.x) dst[m * pitch + i] = i < w ? src[m * w + i] : 0.0f;
}

}  // namespace

// Whether a call's views go by patches: where that is the faster way, which is
// where its plain additions run throughout.  The matrices (host copies, p.nv
// views from h_ptm) tell for the whole volume that
//   * it lies inside the detector (a block across the border runs without the
//     plain additions: 256^3 with a fifth of its slices off the detector 3.7
//     against 2.9 ms a 64-view chunk);
//   * slices are more than a row apart (256^3 at 0.9 rows a slice at the far
//     side: 5.4 against 3.7 ms, at 1.03 2.8 against 3.6);
//   * a block fits its patch, or a sixteenth more than that by the extents
//     below, which are those of the voxels nearest to the source: up to about
//     1.4 pixels a voxel (1.45: 3.0 against 3.7 ms, 1.6: 4.1 against 3.8; 128^3
//     0.58 against 0.60 and 0.92 against 0.62).
// And the blocks, a warp each, have to be enough (6.5 per SM) and full (5/6): a
// warp walks its views one after another, 0.43 ms for 64 however few the warps.
// Where all hold, a chunk of 64 views takes 2.84 against 3.66 ms at 256^3, 1.31
// against 1.64 at 192^3 and 0.53 against 0.59 at 128^3 (1.3 pixels a voxel); 96^3
// (432 blocks) would take 0.45 against 0.26.
bool adjoint_by_patches(const AdjParams& p, const float* h_ptm) {
    const long long voxels = (long long)p.X * p.Y * p.Z, block = kAdjCols * 32;
    const long long blocks = (long long)((p.X + 7) / 8) * ((p.Y + 7) / 8) * ((p.Z + 31) / 32);
    if (2 * voxels < 13LL * p.sms * block || 6 * voxels < 5 * blocks * block) return false;
    const float hx = 0.5f * (float)(p.X - 1) * p.pxy, hy = 0.5f * (float)(p.Y - 1) * p.pxy, hz = 0.5f * (float)(p.Z - 1) * p.pz;
    const float ul = (float)(p.U - 1), vl = (float)(p.V - 1);
    for (int n = 0; n < p.nv; ++n, h_ptm += 12) {
        const float *r0 = h_ptm, *r1 = h_ptm + 4, *r2 = h_ptm + 8;
        // least and largest of k r + l r2 over the volume
        auto least = [&](const float* r, float k, float l) {
            return k * r[3] + l * r2[3] - std::fabs(k * r[0] + l * r2[0]) * hx - std::fabs(k * r[1] + l * r2[1]) * hy -
                   std::fabs(k * r[2] + l * r2[2]) * hz;
        };
        const float wmin = least(r2, 1.0f, 0.0f), wmax = -least(r2, -1.0f, 0.0f);
        // (comparisons false for NaN)
        if (!(wmin > 0.0f && least(r0, 1.0f, 0.49f) > 0.0f && least(r0, -1.0f, ul - 0.51f) > 0.0f &&
              least(r1, 1.0f, 0.49f) > 0.0f && least(r1, -1.0f, vl - 0.51f) > 0.0f))
            return false;
        // du/dx = (P[0] - u P[8]) / W and its like, u over the detector
        auto slope = [&](const float* r, int i, float lim) {
            return std::max(std::fabs(r[i]), std::fabs(r[i] - lim * r2[i])) / wmin;
        };
        const float w = 7.0f * p.pxy * (slope(r0, 0, ul) + slope(r0, 1, ul)) + 31.0f * p.pz * slope(r0, 2, ul) + 2.1f;
        const float h = 7.0f * p.pxy * (slope(r1, 0, vl) + slope(r1, 1, vl)) + 31.0f * p.pz * slope(r1, 2, vl) + 2.1f;
        if (!(w * h <= 1.0625f * (float)kPatch)) return false;
        if (!(p.pz * (std::fabs(r1[2]) - vl * std::fabs(r2[2])) > 1.01f * wmax)) return false;
    }
    return true;
}

cudaError_t launch_bp_adjoint_quads(const AdjParams& p, bool wz, cudaStream_t s) {
    cudaError_t e = cudaMemsetAsync(p.quads, 0, sizeof(float4) * (size_t)p.nv * p.q_frame, s);
    if (e != cudaSuccess) return e;
    const dim3 grid((p.X + 31) / 32, (p.Y + 7) / 8, (p.Z + kAdjZpt - 1) / kAdjZpt);
    if (wz)
        bp_adjoint_quads_kernel<true><<<grid, dim3(32, 8), 0, s>>>(p);
    else
        bp_adjoint_quads_kernel<false><<<grid, dim3(32, 8), 0, s>>>(p);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    unpack_adjoint_kernel<<<dim3((p.U + 255) / 256, std::min(p.V, 65535), std::min(p.nv, 65535)), 256, 0, s>>>(p);
    return cudaGetLastError();
}

cudaError_t launch_bp_adjoint_patches(const AdjParams& p, bool wz, cudaStream_t s) {
    constexpr int smem = kAdjWarps * (int)sizeof(AdjWarp);
    // (per call: the attribute belongs to the current device)
    cudaError_t e = wz ? cudaFuncSetAttribute(bp_adjoint_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem)
                       : cudaFuncSetAttribute(bp_adjoint_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e == cudaSuccess) e = cudaMemsetAsync(p.qbar, 0, sizeof(float) * (size_t)p.nv * p.q_frame, s);
    if (e != cudaSuccess) return e;
    const dim3 grid((p.X + 15) / 16, (p.Y + 15) / 16, (p.Z + 31) / 32);
    if (wz)
        bp_adjoint_kernel<true><<<grid, 32 * kAdjWarps, smem, s>>>(p);
    else
        bp_adjoint_kernel<false><<<grid, 32 * kAdjWarps, smem, s>>>(p);
    return cudaGetLastError();
}

namespace {

template <int J>
dim3 gradient_grid(const AdjParams& p) {
    return dim3((p.X + 8 * J - 1) / (8 * J), (p.Y + kGradRows - 1) / kGradRows, (p.Z + kAdjZpt - 1) / kAdjZpt);
}

size_t blocks_of(const dim3& g) { return (size_t)g.x * g.y * g.z; }

// Columns a thread walks: 4 if that leaves a full wave of CTAs (4 per SM).
bool gradient_deep(const AdjParams& p) { return blocks_of(gradient_grid<4>(p)) >= 4u * (unsigned)p.sms; }

template <int J, bool WZ>
cudaError_t go_gradient(const AdjParams& p, cudaStream_t s) {
    constexpr int smem = J * kAdjZpt * kGradThreads * (int)sizeof(float2);
    static_assert(smem + kGradRed * (int)sizeof(float) <= 48 * 1024, "shared memory without an attribute");
    geometry_gradient_kernel<J, WZ><<<gradient_grid<J>(p), kGradThreads, smem, s>>>(p);
    return cudaGetLastError();
}

}  // namespace

size_t geometry_gradient_ctas(const AdjParams& p) {
    return gradient_deep(p) ? blocks_of(gradient_grid<4>(p)) : blocks_of(gradient_grid<1>(p));
}

cudaError_t launch_geometry_gradient(const AdjParams& p, bool wz, double* grad, cudaStream_t s) {
    const cudaError_t e = gradient_deep(p) ? (wz ? go_gradient<4, true>(p, s) : go_gradient<4, false>(p, s))
                                           : (wz ? go_gradient<1, true>(p, s) : go_gradient<1, false>(p, s));
    if (e != cudaSuccess) return e;
    reduce_partials_kernel<<<p.nv, 192, 0, s>>>(p.partial, geometry_gradient_ctas(p), grad);
    return cudaGetLastError();
}

cudaError_t launch_pad_rows(const float* src, size_t rows, int w, float* dst, int pitch, cudaStream_t s) {
    pad_rows_kernel<<<(unsigned)rows, 256, 0, s>>>(src, w, dst, pitch);
    return cudaGetLastError();
}

cudaError_t launch_filter_adjoint_finish(const float* ybar, int out_w, float* xbar, int in_w, int rows, int nv, int v0,
                                         int num_views, const float* pw, const float* c, int mirror, cudaStream_t s) {
    filter_adjoint_finish_kernel<<<dim3(rows, nv), 256, 0, s>>>(ybar, out_w, xbar, in_w, rows, v0, num_views, pw, c,
                                                                mirror);
    return cudaGetLastError();
}

}  // namespace jfdk
