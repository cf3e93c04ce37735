// bp_common.cuh -- device helpers shared by the backprojector (bp_body.cuh) and its
// adjoint / geometry gradient (adjoint.cu): packed f32x2 arithmetic, the
// floor trick, CT numbers, and the sample coordinates of the FP32 form, so the
// adjoint sees exactly the forward's sample points and in-range decisions.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace jfdk {
namespace {

__device__ __forceinline__ float ct_number(float mu, float s, float n1) {
    // CTNumCore::Process: h = mu * s - 1000; above 300 HU the slope is norm1,
    // capped at 8191.  Separately rounded, no contraction.
    float h = __fsub_rn(__fmul_rn(mu, s), 1000.f);
    if (h > 300.0f) {
        const float t = __fadd_rn(__fmul_rn(__fsub_rn(h, 300.0f), n1), 300.0f);
        h = (t < 8191.f) ? t : 8191.f;
    }
    return h;
}

__device__ __forceinline__ int16_t to_i16(float f) {
    if (f != f) return 0;
    const float t = truncf(f);
    return t >= 32767.0f ? (int16_t)32767 : (t <= -32768.0f ? (int16_t)-32768 : (int16_t)t);
}

__device__ __forceinline__ float2 f2(float a, float b) { return make_float2(a, b); }

// Packed f32x2 arithmetic.  Each lane of a single mul / add / fma rounds like
// the scalar operation, but a packed multiply whose result feeds a packed add
// can be fused into one fma by the compiler (measured on sm_100a with this
// toolchain, for both the intrinsics and inline PTX with .rn), so every
// product that BPCore rounds before adding is computed with scalar
// __fmul_rn / __fadd_rn, which are never contracted.
#define JFDK_PACKED_OP(name, op)                                                              \
    __device__ __forceinline__ float2 name(float2 a, float2 b) {                              \
        float2 d;                                                                             \
        asm("{\n .reg .b64 ra, rb, rd;\n mov.b64 ra, {%2, %3};\n mov.b64 rb, {%4, %5};\n " op \
            " rd, ra, rb;\n mov.b64 {%0, %1}, rd;\n}"                                          \
            : "=f"(d.x), "=f"(d.y)                                                            \
            : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));                                        \
        return d;                                                                             \
    }
JFDK_PACKED_OP(pmul, "mul.rn.f32x2")
JFDK_PACKED_OP(padd, "add.rn.f32x2")
JFDK_PACKED_OP(psub, "sub.rn.f32x2")
#undef JFDK_PACKED_OP

// a * b + c per lane, one rounding (fma.rn.f32x2).
__device__ __forceinline__ float2 pfma(float2 a, float2 b, float2 c) {
    float2 d;
    asm("{\n .reg .b64 ra, rb, rc, rd;\n mov.b64 ra, {%2, %3};\n mov.b64 rb, {%4, %5};\n"
        " mov.b64 rc, {%6, %7};\n fma.rn.f32x2 rd, ra, rb, rc;\n mov.b64 {%0, %1}, rd;\n}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return d;
}

// add.rm.f32x2: the lanewise sum rounded toward -infinity.
__device__ __forceinline__ float2 padd_rm(float2 a, float2 b) {
    float2 d;
    asm("{\n .reg .b64 ra, rb, rd;\n mov.b64 ra, {%2, %3};\n mov.b64 rb, {%4, %5};\n"
        " add.rm.f32x2 rd, ra, rb;\n mov.b64 {%0, %1}, rd;\n}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}

// Floor without the conversion unit: for 0 <= x < 2^23 the sum 2^23 + x has
// a unit in the last place of 1, so rounding it toward -infinity gives
// 2^23 + floor(x) exactly; its bit pattern minus that of 2^23 is floor(x) as
// an integer, and subtracting 2^23 back gives floor(x) as a float.
constexpr float kMagic = 8388608.0f;   // 2^23
constexpr int kMagicBits = 0x4B000000;  // bit pattern of 2^23

// Sample point of the FP32 form, as BPCore rounds it (BPCore.cpp:120-145,
// 207-220): Uxy = x*P0 + (y*P1 + P3), likewise V, W; U = Uxy + z*P2 etc.,
// every product and sum rounded separately; u = RN(U / W) + 0.5
// (bp_quotient2).
struct XYTerms { float U, V, W; };

__device__ __forceinline__ XYTerms bp_xy_terms(float ax, float ay, const float4& r0, const float4& r1,
                                               const float4& r2) {
    XYTerms t;
    t.U = __fadd_rn(__fmul_rn(ax, r0.x), __fadd_rn(__fmul_rn(ay, r0.y), r0.w));
    t.V = __fadd_rn(__fmul_rn(ax, r1.x), __fadd_rn(__fmul_rn(ay, r1.y), r1.w));
    t.W = __fadd_rn(__fmul_rn(ax, r2.x), __fadd_rn(__fmul_rn(ay, r2.y), r2.w));
    return t;
}

// RN(1/w) from the approximate reciprocal (rcp.approx, at most 1 ulp off)
// and one Newton-Raphson step with a fused residual, y' = RN(y + y RN(1 - w y))
// (Markstein, IBM J. Res. Dev. 34(1), 1990).  Equal to __frcp_rn for every
// float w whose reciprocal is a normal float, both signs (all 4.2e9 of them,
// tests/cuda/reciprocal_check.cu); W of a voxel lies far inside that range.
__device__ __forceinline__ float rcp_rn_nr(float w) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(w));
    return fmaf(fmaf(-w, y, 1.0f), y, y);
}

// 1/W as a float r = RN(1/W) and the float nearest to what r lacks, rl =
// RN(e r) with e = 1 - W r, which is exact and at most 2^-24: r + rl is within
// 2^-47 of 1/W, e^2 left out and rl rounded being 2^-48 each.
struct Recip { float r, rl; };

__device__ __forceinline__ Recip bp_recip(float W) {
    const float r = rcp_rn_nr(W);
    return {r, __fmul_rn(fmaf(-W, r, 1.0f), r)};
}

// U / W of both lanes.  EXACT: correctly rounded, from r and Markstein's
// correction q = RN(q0 + RN(U - W q0) r), q0 = RN(U r).  Otherwise
// RN(U r + RN(U rl)), one operation less (5 % of the FP32 loop): the sum is
// within 3 2^-48 of U / W before its one rounding (a third 2^-48 from RN(U rl)), so
// it is the correctly rounded quotient but where U / W lies that close to the
// middle between two floats, and then the other of the two, off by half a unit in
// the last place like the one it stands for: 5 of 2.1e9 random quotients
// (tests/cuda/quotient_check.cu).  This holds while rl and U rl stay normal: |W|
// from 2^-78 to 2^78, |U / W| above 2^-78, far below what the 0.5 that a place adds
// leaves of it.
template <bool EXACT>
__device__ __forceinline__ float2 bp_quotient2(float2 U, float W, const Recip& rc) {
    const float2 rr = f2(rc.r, rc.r);
    if constexpr (EXACT) {
        const float2 q0 = pmul(U, rr);
        const float2 rem = pfma(f2(-W, -W), q0, U);           // exact remainder
        return pfma(rem, rr, q0);
    }
    return pfma(U, rr, pmul(U, f2(rc.rl, rc.rl)));
}

template <bool EXACT>
__device__ __forceinline__ float bp_quotient(float U, float W, const Recip& rc) {
    if constexpr (EXACT) {
        const float q0 = __fmul_rn(U, rc.r);
        return fmaf(fmaf(-W, q0, U), rc.r, q0);
    }
    return fmaf(U, rc.r, __fmul_rn(U, rc.rl));
}

// W and RN(1/W) at slice coordinate az (W independent of z unless WZ).
template <bool WZ>
__device__ __forceinline__ float2 bp_w_r(const XYTerms& t, const Recip& rc, float az, float P10) {
    if (WZ) {
        const float W = __fadd_rn(t.W, __fmul_rn(az, P10));
        return f2(W, rcp_rn_nr(W));
    }
    return f2(t.W, rc.r);
}

// (u, v) of the sample at slice coordinate az.  WZ: W and its reciprocal are
// the slice's, and the quotient is Markstein's (rl would cost two operations
// a sample to save one).  w_r, quot: also W with its
// reciprocal, and the quotients.
template <bool EXACT, bool WZ>
__device__ __forceinline__ float2 bp_uv(const XYTerms& t, const Recip& rc, float az, float P2, float P6, float P10,
                                        float2* w_r = nullptr, float2* quot = nullptr) {
    const float2 UV = f2(__fadd_rn(t.U, __fmul_rn(az, P2)), __fadd_rn(t.V, __fmul_rn(az, P6)));
    const float2 wr = bp_w_r<WZ>(t, rc, az, P10);
    if (w_r) *w_r = wr;
    const float2 q = WZ ? bp_quotient2<true>(UV, wr.x, Recip{wr.y, 0.0f}) : bp_quotient2<EXACT>(UV, t.W, rc);
    if (quot) *quot = q;
    return padd(q, f2(0.5f, 0.5f));
}

// The BPCore axis value (i - (n-1)/2) * pitch (BPCore.cpp:47-66).
__device__ __forceinline__ float bp_axis(int i, int n, float pitch) {
    return __fmul_rn(__fadd_rn(-((float)n - 1.0f) / 2.0f, (float)i), pitch);
}

// Record loads.  The address is formed from a 32-bit byte offset, a shift on
// the integer pipe, beside the view's base address: a 64-bit multiply-add
// (IMAD.WIDE) instead takes two cycles of the FMA pipe, which is what bounds
// the view loop (71 % busy; c2: 125.3 -> 119.3 ms FP32, 91.4 -> 82.3 ms
// mixed).  WIDE: frames of more than 4 GB of records, and the batch kernel,
// keep the 64-bit form.
template <bool WIDE, class T>
__device__ __forceinline__ T load_at(const T* frame, unsigned idx) {
    if constexpr (WIDE) return __ldg(frame + idx);
    return __ldg(reinterpret_cast<const T*>(reinterpret_cast<size_t>(frame) + idx * (unsigned)sizeof(T)));
}

// The record of integer column and row (as floats; tx = 2^23 + column) in a
// frame of at most 2^23 records: 2^23 + row U + column is exact in a float,
// and its bit pattern is the record's index above that of 2^23.  One FFMA in
// place of two integer subtractions and a multiply-add; the constant part of
// the shifted pattern is taken off the frame's address (record_base).
template <class T>
__device__ __forceinline__ T load_record(size_t base, float tx, float row, float Uf) {
    const unsigned off = __float_as_uint(fmaf(row, Uf, tx)) * (unsigned)sizeof(T);   // mod 2^32
    return __ldg(reinterpret_cast<const T*>(base + off));
}

template <class T>
__device__ __forceinline__ size_t record_base(const T* frame) {
    return reinterpret_cast<size_t>(frame) - (unsigned)kMagicBits * (unsigned)sizeof(T);
}

// A box of voxels: centre, half extents and largest moduli of its coordinates.
struct VoxelBox {
    float cx, cy, cz, hx, hy, hz, mx, my, mz;
    __device__ VoxelBox(float x0, float x1, float y0, float y1, float z0, float z1)
        : cx(0.5f * (x0 + x1)), cy(0.5f * (y0 + y1)), cz(0.5f * (z0 + z1)), hx(0.5f * fabsf(x1 - x0)),
          hy(0.5f * fabsf(y1 - y0)), hz(0.5f * fabsf(z1 - z0)), mx(fmaxf(fabsf(x0), fabsf(x1))),
          my(fmaxf(fabsf(y0), fabsf(y1))), mz(fmaxf(fabsf(z0), fabsf(z1))) {}
};

// Where the voxels of the box sample the view of matrix P on a U x V detector:
// kBoxInside, every one at 0 <= u <= U - 1, 0 <= v <= V - 1 in front of the
// source (W > 0); kBoxOutside, none; kBoxAcross, not known.  The conditions
// are linear in the voxel's place once multiplied by W, so the least and the
// largest value over the box are the one at its centre minus and plus the
// coefficients' moduli times the half extents: five linear forms.  The margin,
// 2^-16 of the sum of the terms' moduli, is far above what the rounded
// coordinates can be off (a few 2^-24 of that sum, 16 steps of it in the mixed
// form), so the range test would take every sample of a box inside and none of
// a box outside.
enum BoxPlace { kBoxAcross = 0, kBoxInside = 1, kBoxOutside = 2 };

__device__ __forceinline__ BoxPlace box_place(const VoxelBox& b, const float* P, int U, int V) {
    const float4* P4 = reinterpret_cast<const float4*>(P);
    const float4 r0 = __ldg(P4), r1 = __ldg(P4 + 1), r2 = __ldg(P4 + 2);
    bool inside = true, outside = false;
    // k r + l r2 (rows of the matrix) over the box, against the margin
    auto clear = [&](const float4& r, float k, float l, float lim) {
        const float kx = fmaf(k, r.x, l * r2.x), ky = fmaf(k, r.y, l * r2.y), kz = fmaf(k, r.z, l * r2.z);
        const float f = fmaf(kx, b.cx, fmaf(ky, b.cy, fmaf(kz, b.cz, fmaf(k, r.w, l * r2.w))));
        const float h = fmaf(fabsf(kx), b.hx, fmaf(fabsf(ky), b.hy, fabsf(kz) * b.hz));
        const float m = fmaf(fmaf(lim, fabsf(r2.x), fabsf(r.x)), b.mx,
                             fmaf(fmaf(lim, fabsf(r2.y), fabsf(r.y)), b.my,
                                  fmaf(fmaf(lim, fabsf(r2.z), fabsf(r.z)), b.mz, fmaf(lim, fabsf(r2.w), fabsf(r.w)))));
        inside = inside && f - h > 0x1p-16f * m;     // both false for NaN
        outside = outside || f + h < -0x1p-16f * m;
    };
    const float ul = (float)U, vl = (float)V;
    clear(r2, 1.0f, 0.0f, 1.0f);
    // u and v have the signs of these forms in front of the source only
    const bool front = inside;
    outside = false;
    clear(r0, 1.0f, 0.5f, ul);
    clear(r0, -1.0f, ul - 1.5f, ul);
    clear(r1, 1.0f, 0.5f, vl);
    clear(r1, -1.0f, vl - 1.5f, vl);
    return inside ? kBoxInside : front && outside ? kBoxOutside : kBoxAcross;
}

}  // namespace
}  // namespace jfdk
