// adjoint.cu -- derivatives of the FP32 FDK form (sm_100a):
//
//   * the adjoint of the backprojector, vol = S q / C: with the weights C
//     (the backprojected taper) fixed, q_bar = S^T (vol_bar / C) -- for every
//     voxel and view the transposed bilinear weights of its sample point,
//     scattered into "quad space" (the forward's tapered footprint records,
//     one 16-byte vector atomic per sample) and folded back to detector
//     pixels and multiplied by the taper;
//   * the adjoint of the ramp filter, y = T (w o x) + c e(x) with
//     e(x) = (x0 + x1 + x2) / 3 (or the last three for a mirrored filter):
//     x_bar = w o (T^T y_bar) + (c . y_bar) / 3 on the edge samples;
//   * the gradient with respect to per-view projection-matrix parameters:
//     for a loss L(vol), dL/dtheta_j = sum over voxels of
//     vol_bar / C * [(dS/du - vol dC/du) du/dtheta_j + dS/dv dv/dtheta_j],
//     with u = U/W, du/dtheta_j = (dU_j - u dW_j) / W for (dU_j, dV_j, dW_j)
//     = (dP/dtheta_j) X; per-CTA partial sums in FP32, the reduction over
//     CTAs in FP64.
// Every kernel uses the forward's sample points and in-range decisions
// (bp_common.cuh), so the adjoint is the transpose of the forward as computed.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "bp_common.cuh"
#include "jfdk_internal.h"

namespace jfdk {
namespace {

__device__ __forceinline__ void red_add_v4(float4* p, float4 v) {
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w)
                 : "memory");
}

// rt = vol_bar / C (0 where no view saw the voxel).
__device__ __forceinline__ float residual(float vol_bar, float cnt) { return cnt != 0.0f ? vol_bar / cnt : 0.0f; }

constexpr int kAdjZpt = 8;

// Quad-space adjoint: Qbar[view - v0][iv][iu] += rt * (bilinear weights).
template <int ZPT, bool WZ>
__global__ void __launch_bounds__(256) bp_adjoint_kernel(AdjParams p) {
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
        az[k] = bp_axis(zb + k, p.Z, p.pz);
        rt[k] = zb + k < p.Z ? residual(p.vol_bar[(size_t)(zb + k) * plane + base], p.cnt[(size_t)(zb + k) * plane + base]) : 0.0f;
        any |= rt[k] != 0.0f;
    }
    if (!any) return;
    const float umax = (float)(p.U - 1), vmax = (float)(p.V - 1);
    const float4* P4 = reinterpret_cast<const float4*>(p.ptm + (size_t)p.v0 * 12);
    float4* __restrict__ qb = p.qbar;
#pragma unroll 1
    for (int n = 0; n < p.nv; ++n, P4 += 3, qb += p.q_frame) {
        const float4 r0 = __ldg(P4), r1 = __ldg(P4 + 1), r2 = __ldg(P4 + 2);
        const XYTerms xy = bp_xy_terms(ax, ay, r0, r1, r2);
        const Recip rc = WZ ? Recip{0.0f, 0.0f} : bp_recip(xy.W);
#pragma unroll
        for (int k = 0; k < ZPT; ++k) {
            const float2 uv = bp_uv<false, WZ>(xy, rc, az[k], r0.z, r1.z, r2.z);
            const bool in = (uv.x >= 0.0f) & (uv.x <= umax) & (uv.y >= 0.0f) & (uv.y <= vmax);
            if (in && rt[k] != 0.0f) {
                // floor by the 2^23 add rounded toward -inf (exact for 0 <= u, v < 2^23)
                const float2 t = padd_rm(uv, f2(kMagic, kMagic));
                const float2 f = psub(uv, psub(t, f2(kMagic, kMagic)));
                const unsigned iu = __float_as_uint(t.x) - (unsigned)kMagicBits;
                const unsigned iv = __float_as_uint(t.y) - (unsigned)kMagicBits;
                const float a = rt[k] * (1.0f - f.x), b = rt[k] * f.x;
                red_add_v4(qb + (size_t)iv * p.U + iu, make_float4(a * (1.0f - f.y), a * f.y, b * (1.0f - f.y), b * f.y));
            }
        }
    }
}

// Quad space -> detector pixels: p[r][c] appears in quads (r, c).x,
// (r-1, c).y, (r, c-1).z, (r-1, c-1).w, each times the taper w[c].
__global__ void __launch_bounds__(256) unpack_adjoint_kernel(const float4* __restrict__ qbar, long long q_frame,
                                                             int rows, int U, const float2* __restrict__ tw,
                                                             int view0, int num_views, float* __restrict__ out) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    const int r = blockIdx.y, f = blockIdx.z;
    if (c >= U) return;
    const float4* q = qbar + (size_t)f * q_frame;
    float s = q[(size_t)r * U + c].x;
    if (r > 0) s += q[(size_t)(r - 1) * U + c].y;
    if (c > 0) s += q[(size_t)r * U + c - 1].z;
    if (r > 0 && c > 0) s += q[(size_t)(r - 1) * U + c - 1].w;
    const float w = tw[(size_t)((view0 + f) % num_views) * U + c].x;
    out[(size_t)f * rows * U + (size_t)r * U + c] = w * s;
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
// 256^3 from 512^2 takes 2.1 ms (96 registers and 20 warps 2.9, 80 and 24
// 3.2; 3.26 with the reduction every 8 samples, 32 x 1 warps and 64 registers).
// J is 1 where 4 would leave less than a full wave of CTAs.
constexpr int kGradThreads = 128, kGradRows = kGradThreads / 8;   // 8 columns x kGradRows of warps of 4 x 8

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
    __shared__ float red[2 * (kGradThreads / 32) * 16];
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
    for (int n = tid; n < p.nv; n += kGradThreads) ok = ok && box_inside(box, p.ptm + (size_t)(p.v0 + n) * 12, p.U, p.V);
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

template <int ZPT>
dim3 bp_grid(const AdjParams& p) {
    return dim3((p.X + 31) / 32, (p.Y + 7) / 8, (p.Z + ZPT - 1) / ZPT);
}

}  // namespace

cudaError_t launch_bp_adjoint(const AdjParams& p, bool wz, cudaStream_t s) {
    cudaError_t e = cudaMemsetAsync(p.qbar, 0, sizeof(float4) * (size_t)p.nv * p.q_frame, s);
    if (e != cudaSuccess) return e;
    const dim3 g = bp_grid<kAdjZpt>(p);
    if (wz)
        bp_adjoint_kernel<kAdjZpt, true><<<g, dim3(32, 8), 0, s>>>(p);
    else
        bp_adjoint_kernel<kAdjZpt, false><<<g, dim3(32, 8), 0, s>>>(p);
    return cudaGetLastError();
}

cudaError_t launch_unpack_adjoint(const float4* qbar, long long q_frame, int nv, int rows, int U, const float2* tw,
                                  int view0, int num_views, float* out, cudaStream_t s) {
    dim3 grid((U + 255) / 256, rows, nv);
    unpack_adjoint_kernel<<<grid, 256, 0, s>>>(qbar, q_frame, rows, U, tw, view0, num_views, out);
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
    if constexpr (smem > 32 * 1024) {   // per call: the attribute belongs to the current device
        const cudaError_t e = cudaFuncSetAttribute(geometry_gradient_kernel<J, WZ>,
                                                   cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return e;
    }
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
