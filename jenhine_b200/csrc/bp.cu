// bp.cu -- the kernels around the backprojection (sm_100a): packing of filtered
// frames into its records, the per-view maxima of the mixed form, the
// finalisation of accumulated volumes, CT numbers and the z-filter.  The
// backprojection itself is in bp_body.cuh.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "bp_common.cuh"
#include "jfdk_internal.h"

namespace jfdk {
namespace {

// Largest |value| of each frame as float bits; for non-negative floats the
// bit patterns order like the values, so an integer atomicMax reduces them.
// out[] must be zero before the launch.
__global__ void __launch_bounds__(256) frame_absmax_kernel(const float* __restrict__ plain, long long frame,
                                                           unsigned* __restrict__ out) {
    const float* fr = plain + (size_t)blockIdx.y * frame;
    float m = 0.0f;
    for (long long i = blockIdx.x * 256LL + threadIdx.x; i < frame; i += (long long)gridDim.x * 256)
        m = fmaxf(m, fabsf(__ldg(fr + i)));   // fmaxf drops NaN operands
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) atomicMax(out + blockIdx.y, __float_as_uint(m));
}

// Power-of-two scale of a view: max |q| / s lies in [2^12, 2^13), so every
// coefficient of the bilinear form (|dxy| < 4 max) stays inside the FP16
// range (65504), and dividing by s is exact.  An all-zero (or non-finite)
// view gets 1.
__device__ __forceinline__ float view_scale(unsigned maxbits) {
    const float m = __uint_as_float(maxbits);
    if (!(m > 0.0f) || !(m <= 3.0e38f)) return 1.0f;
    return ldexpf(1.0f, ilogbf(m) - 12);
}

// The packers write 16 or 8 bytes a pixel and are bound by that: a thread walks
// kPackRows rows of its column, so that a row's samples serve as the upper
// ones of one record and the lower ones of the one before, and the taper is
// read once (a chunk of 32 frames of 768 x 768: 84.6 -> 57.4 us, 302 MB written at
// 5.3 TB/s; mixed 99.4 -> 51.0).
constexpr int kPackRows = 8;

// Filtered frames -> mixed-precision records in slots [slot0, slot0 + nv),
// tapered with the taper of rotation view (view0 + f) mod num_views; writes
// that view's scale to scale[view].
__global__ void __launch_bounds__(256) pack_mixed_kernel(const float* __restrict__ plain, long long plain_frame,
                                                         int rows, int U, const float2* __restrict__ tw, int view0,
                                                         int num_views, const unsigned* __restrict__ absmax,
                                                         float* __restrict__ scale, uint2* __restrict__ qh,
                                                         long long q_frame, int slot0) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    const int r0 = blockIdx.y * kPackRows, f = blockIdx.z;
    if (c >= U) return;
    const int view = (view0 + f) % num_views;
    const float s = view_scale(absmax[f]);
    const float inv = __fdiv_rn(1.0f, s);
    if (r0 == 0 && c == 0) scale[view] = s;
    const bool right = c + 1 < U;
    const float* src = plain + (size_t)f * plain_frame + (size_t)r0 * U + c;
    uint2* dst = qh + (size_t)(slot0 + f) * q_frame + (size_t)r0 * U + c;
    const float w0 = tw[(size_t)view * U + c].x, w1 = right ? tw[(size_t)view * U + c + 1].x : 0.0f;
    // the tapered footprint over the view's scale (exact: inv a power of two)
    float p[kPackRows + 1], q[kPackRows + 1];
#pragma unroll
    for (int i = 0; i <= kPackRows; ++i) {
        const bool in = r0 + i < rows;
        p[i] = in ? (src[(size_t)i * U] * w0) * inv : 0.0f;
        q[i] = in && right ? (src[(size_t)i * U + 1] * w1) * inv : 0.0f;
    }
#pragma unroll
    for (int i = 0; i < kPackRows; ++i) {
        if (r0 + i >= rows) break;
        uint2 rec = make_uint2(0u, 0u);   // the last row and column: samples not taken
        if (right && r0 + i + 1 < rows) {
            const __half hp = __float2half_rn(p[i]);
            const float ap = __half2float(hp);
            const __half hdx = __float2half_rn(q[i] - ap), hdy = __float2half_rn(p[i + 1] - ap);
            const __half hdxy = __float2half_rn(q[i + 1] - (ap + __half2float(hdx) + __half2float(hdy)));
            const __half2 h1 = __halves2half2(hp, hdx), h2 = __halves2half2(hdy, hdxy);
            rec.x = *reinterpret_cast<const unsigned*>(&h1);
            rec.y = *reinterpret_cast<const unsigned*>(&h2);
        }
        dst[(size_t)i * U] = rec;
    }
}

// Filtered frames -> tapered quads: the tapered values w[c] p[r][c],
// w[c] p[r+1][c], w[c+1] p[r][c+1], w[c+1] p[r+1][c+1], each product rounded as
// InitView's in-place multiply (BPCore.cpp:147-151), stored as (t00, t10,
// RN(t01 - t00), RN(t11 - t10)).
__global__ void __launch_bounds__(256) pack_quads_kernel(const float* __restrict__ plain, long long plain_frame,
                                                         int rows, int U, const float2* __restrict__ tw,
                                                         int view0, int num_views, int apply_taper,
                                                         float4* __restrict__ q4, long long q4_frame, int slot0) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    const int r0 = blockIdx.y * kPackRows, f = blockIdx.z;
    if (c >= U) return;
    const bool right = c + 1 < U;
    const float* src = plain + (size_t)f * plain_frame + (size_t)r0 * U + c;
    float4* dst = q4 + (size_t)(slot0 + f) * q4_frame + (size_t)r0 * U + c;
    float w0 = 1.0f, w1 = 1.0f;
    if (apply_taper) {
        const float2* wv = tw + (size_t)((view0 + f) % num_views) * U;
        w0 = wv[c].x;
        w1 = right ? wv[c + 1].x : 0.0f;
    }
    float p[kPackRows + 1], q[kPackRows + 1];
#pragma unroll
    for (int i = 0; i <= kPackRows; ++i) {
        const bool in = r0 + i < rows;
        p[i] = in ? src[(size_t)i * U] : 0.0f;
        q[i] = in && right ? src[(size_t)i * U + 1] : 0.0f;
        if (apply_taper) {
            p[i] = __fmul_rn(p[i], w0);
            q[i] = __fmul_rn(q[i], w1);
        }
    }
#pragma unroll
    for (int i = 0; i < kPackRows; ++i) {
        if (r0 + i >= rows) break;
        dst[(size_t)i * U] = make_float4(p[i], p[i + 1], __fsub_rn(q[i], p[i]), __fsub_rn(q[i + 1], p[i + 1]));
    }
}

__global__ void finalize_kernel(const float* __restrict__ sum, const float* __restrict__ cnt, size_t n,
                                int apply_ct, float s, float n1, float* out, int16_t* out16) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        float o = __fdiv_rn(sum[i], cnt[i]);
        if (apply_ct) o = ct_number(o, s, n1);
        if (out) out[i] = o;
        if (out16) out16[i] = to_i16(o);
    }
}

__global__ void ctnum_kernel(float* d, size_t n, float s, float n1) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        d[i] = ct_number(d[i], s, n1);
}

// ZFilterAgent::ProcessTask (FilterAgent/ZFilterAgent.cpp:49-71): out[v] =
// 0.5 in[v] + 0.25 in[max(v-1,0)] + 0.25 in[min(v+1,rows-1)], each product
// and sum rounded in the reference's order.  One thread walks one column of
// one frame top to bottom, in place: the previous and current input rows in
// registers, and the next kZRows input rows loaded together before any of
// them is overwritten, so kZRows loads are in flight instead of one (a
// column walked row by row waited out one load latency per row: 349 us per
// 32-view chunk of 768 x 768).
constexpr int kZRows = 16;

__global__ void __launch_bounds__(128) zfilter_kernel(float* frames, int nv, int rows, int width, long long stride,
                                                      int pitch) {
    const int col = blockIdx.x * blockDim.x + threadIdx.x, f = blockIdx.y;
    if (col >= width || f >= nv) return;
    float* c = frames + (size_t)f * stride + col;
    float prev = c[0], cur = c[0];
    for (int r0 = 0; r0 < rows; r0 += kZRows) {
        float nxt[kZRows];
#pragma unroll
        for (int i = 0; i < kZRows; ++i) nxt[i] = c[(size_t)min(r0 + 1 + i, rows - 1) * pitch];
#pragma unroll
        for (int i = 0; i < kZRows; ++i) {
            if (r0 + i >= rows) break;
            float o = __fmul_rn(cur, 0.5f);
            o = __fadd_rn(o, __fmul_rn(prev, 0.25f));
            o = __fadd_rn(o, __fmul_rn(nxt[i], 0.25f));
            c[(size_t)(r0 + i) * pitch] = o;
            prev = cur;
            cur = nxt[i];
        }
    }
}

}  // namespace

cudaError_t launch_bp(const BPParams& p, bool finalize, bool exact, Geo geo, int zpt, int tile_x, cudaStream_t s) {
    if ((long long)p.U * p.V > (1LL << 28)) return launch_bp_wide(p, finalize, exact, false, geo, zpt, s);
    return exact ? launch_bp_exact(p, finalize, geo, zpt, tile_x, s) : launch_bp_fast(p, finalize, geo, zpt, tile_x, s);
}

cudaError_t launch_bp_batch(const BatchSlots& t, int nscans, unsigned total_tiles, bool mixed_form, bool wz,
                            bool wv, unsigned* counter, int ctas, cudaStream_t s) {
    if (nscans < 1 || nscans > kBatchSlots) return cudaErrorInvalidValue;
    const bool deep = t.s[0].zpt == 16;   // a launch of 16-slice tiles holds those only
    if (deep && !mixed_form) return cudaErrorInvalidValue;
    for (int i = 0; i < nscans; ++i) {
        const int z = t.s[i].zpt;
        if ((deep ? z != 16 : (z != 4 && z != 8)) || (wv && !t.s[i].p.wvol)) return cudaErrorInvalidValue;
    }
    cudaError_t e = cudaMemsetAsync(counter, 0, sizeof(unsigned), s);
    if (e != cudaSuccess) return e;
    return mixed_form ? launch_bp_batch_mixed(t, nscans, total_tiles, wz, wv, deep, counter, ctas, s)
                      : launch_bp_batch_fp32(t, nscans, total_tiles, wz, wv, false, counter, ctas, s);
}

cudaError_t bp_batch_ctas(bool mixed_form, bool wz, bool wv, bool deep, int* ctas) {
    int dev = 0, sms = 0, per = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess)
        e = mixed_form ? bp_batch_resident_mixed(wz, wv, deep, &per) : bp_batch_resident_fp32(wz, wv, false, &per);
    *ctas = sms * (per > 0 ? per : 1);
    return e;
}

cudaError_t launch_frame_absmax(const float* plain, long long frame, int nv, unsigned* absmax, cudaStream_t s) {
    cudaError_t e = cudaMemsetAsync(absmax, 0, sizeof(unsigned) * nv, s);
    if (e != cudaSuccess) return e;
    const int bx = (int)std::min<long long>((frame + 255) / 256, 64);
    frame_absmax_kernel<<<dim3(bx, nv), 256, 0, s>>>(plain, frame, absmax);
    return cudaGetLastError();
}

namespace {
// Columns a packing CTA covers: 256, 128 or 64, the widest that leaves under a
// quarter of the threads past the last column where one does.
int pack_cta(int U) {
    for (int t : {256, 128})
        if ((U + t - 1) / t * t * 3 <= U * 4) return t;
    return 64;
}
}  // namespace

cudaError_t launch_pack_mixed(const float* plain, long long plain_frame, int nv, int rows, int U, const float2* tw,
                              int view0, int num_views, const unsigned* absmax, float* scale, uint2* qh,
                              long long q_frame, int slot0, cudaStream_t s) {
    const int cta = pack_cta(U);
    dim3 grid((U + cta - 1) / cta, (rows + kPackRows - 1) / kPackRows, nv);
    pack_mixed_kernel<<<grid, cta, 0, s>>>(plain, plain_frame, rows, U, tw, view0, num_views, absmax, scale, qh,
                                           q_frame, slot0);
    return cudaGetLastError();
}

cudaError_t launch_pack_quads(const float* plain, long long plain_frame, int nv, int rows, int U, const float2* tw,
                              int view0, int num_views, int apply_taper, float4* q4, long long q4_frame, int slot0,
                              cudaStream_t s) {
    const int cta = pack_cta(U);
    dim3 grid((U + cta - 1) / cta, (rows + kPackRows - 1) / kPackRows, nv);
    pack_quads_kernel<<<grid, cta, 0, s>>>(plain, plain_frame, rows, U, tw, view0, num_views, apply_taper, q4,
                                           q4_frame, slot0);
    return cudaGetLastError();
}

cudaError_t launch_finalize(const float* sum, const float* cnt, size_t n, int apply_ct, float ct_scale,
                            float norm1, float* out, int16_t* out16, cudaStream_t s) {
    const int blocks = (int)std::min<size_t>((n + 255) / 256, 148 * 16);
    finalize_kernel<<<blocks, 256, 0, s>>>(sum, cnt, n, apply_ct, ct_scale, norm1, out, out16);
    return cudaGetLastError();
}

cudaError_t launch_ctnum(float* d, size_t n, float ct_scale, float norm1, cudaStream_t s) {
    const int blocks = (int)std::min<size_t>((n + 255) / 256, 148 * 16);
    ctnum_kernel<<<blocks, 256, 0, s>>>(d, n, ct_scale, norm1);
    return cudaGetLastError();
}

cudaError_t launch_zfilter(float* frames, int nv, int rows, int width, long long frame_stride, int pitch,
                           cudaStream_t s) {
    dim3 grid((width + 127) / 128, nv);
    zfilter_kernel<<<grid, 128, 0, s>>>(frames, nv, rows, width, frame_stride, pitch);
    return cudaGetLastError();
}

}  // namespace jfdk
