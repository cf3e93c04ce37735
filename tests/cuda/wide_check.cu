// The backprojection's launch for frames of more than 4 GB of records
// (launch_bp_wide in jenhine_b200/csrc/bp_wide.cu) against the ordinary one on
// small frames, where both give an answer: the same sums, weights and volumes bit
// for bit, in both forms, EXACT, for each way a place depends on the slice, with
// and without a weight volume, each mixed tile depth.  Built and run by
// tests/test_wide.py, linked with libjfdk.so.
#include <cmath>
#include <cstdio>
#include <cstring>
#include <vector>

#include <cuda_fp16.h>

#include "jfdk_internal.h"

using namespace jfdk;

template <class T>
T* upload(const std::vector<T>& v) {
    T* p = nullptr;
    if (cudaMalloc(&p, v.size() * sizeof(T)) != cudaSuccess) return nullptr;
    cudaMemcpy(p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice);
    return p;
}

int main() {
    constexpr int N = 7, U = 41, V = 33, X = 21, Y = 37, Z = 19;
    constexpr size_t px = (size_t)U * V, vox = (size_t)X * Y * Z;
    unsigned s = 12345;
    auto rnd = [&] { s = s * 1664525u + 1013904223u; return (float)(s >> 8) / 16777216.0f; };
    std::vector<float4> quads(N * px);
    std::vector<uint2> records(N * px);
    std::vector<float2> taper(N * U);
    std::vector<float> scale(N), weights(vox), zero(vox, 0.0f);
    for (auto& q : quads) q = make_float4(rnd(), rnd(), rnd() - 0.5f, rnd() - 0.5f);
    for (size_t i = 0; i < records.size(); ++i) {
        const int c = (int)(i % U), r = (int)(i / U % V);
        if (c == U - 1 || r == V - 1) { records[i] = make_uint2(0u, 0u); continue; }
        __half h[4] = {__float2half(rnd()), __float2half(rnd()), __float2half(rnd()), __float2half(rnd())};
        std::memcpy(&records[i], h, 8);
    }
    for (auto& t : taper) t = make_float2(0.5f + rnd(), 0.1f * rnd());
    for (auto& w : weights) w = 1.0f + rnd();
    for (auto& x : scale) x = std::ldexp(1.0f, (int)(4 * rnd()));
    BPParams p{};
    p.q4 = upload(quads); p.qh = upload(records); p.tw = upload(taper); p.qscale = upload(scale);
    const float* wvol = upload(weights);
    float* sum[2] = {upload(zero), upload(zero)};
    float* cnt[2] = {upload(zero), upload(zero)};
    float* out[2] = {upload(zero), upload(zero)};
    p.q4_frame = (long long)px;
    p.view_base = 0; p.v0 = 0; p.nv = N;
    p.U = U; p.V = V; p.X = X; p.Y = Y; p.Z = Z;
    p.pxy = 1.0f; p.pz = 1.0f;
    p.z_begin = 0; p.z_end = Z;
    p.apply_ct = 1; p.ct_scale = 50.0f; p.ct_norm1 = 1.0f;
    long long runs = 0, differ = 0;
    for (int geo = 0; geo < 3; ++geo) {
        std::vector<float> ptm(N * 12);
        for (int v = 0; v < N; ++v) {
            const double b = 6.283185307179586 * v / N, c = std::cos(b), t = std::sin(b), f = 1.3, d = 100.0;
            // magnification f at the centre, the principal point a little off it; some voxels leave the detector
            double r0[4] = {-f * t, f * c, geo == kGeoIdeal ? 0.0 : 0.01, 0.0}, r1[4] = {0.003, 0.002, f, 0.0};
            double r2[4] = {-c / d, -t / d, geo == kGeoWZ ? 0.004 : 0.0, 1.0};
            for (int k = 0; k < 4; ++k) {
                ptm[v * 12 + k] = (float)(r0[k] + (U / 2 - 1.3) * r2[k]);
                ptm[v * 12 + 4 + k] = (float)(r1[k] + (V / 2 - 0.7) * r2[k]);
                ptm[v * 12 + 8 + k] = (float)r2[k];
            }
            if (geo == kGeoIdeal) ptm[v * 12 + 2] = 0.0f;
        }
        float* d_ptm = upload(ptm);
        p.ptm = d_ptm;
        for (int form = 0; form < 5; ++form) {   // FP32, EXACT, mixed of 4, 8 and 16 slices
            const bool mix = form >= 2;
            const int zpt = mix ? 4 << (form - 2) : 8;
            for (int way = 0; way < 3; ++way) {   // accumulate; finalise with per-sample weights, with the volume
                for (int k = 0; k < 2; ++k) {
                    for (float* a : {sum[k], cnt[k], out[k]}) cudaMemset(a, 0, vox * sizeof(float));
                    BPParams q = p;
                    q.sum = sum[k]; q.cnt = cnt[k]; q.out = out[k];
                    q.load_acc = way == 0; q.wvol = way == 2 ? wvol : nullptr;
                    const cudaError_t e = k ? launch_bp_wide(q, way != 0, form == 1, mix, (Geo)geo, zpt, nullptr)
                                        : mix ? launch_bp_mixed(q, way != 0, (Geo)geo, zpt, 4, 148, nullptr)
                                              : launch_bp(q, way != 0, form == 1, (Geo)geo, zpt, 4, nullptr);
                    if (e != cudaSuccess || cudaDeviceSynchronize() != cudaSuccess) {
                        std::printf("CUDA error: %s\n", cudaGetErrorString(e != cudaSuccess ? e : cudaGetLastError()));
                        return 2;
                    }
                }
                size_t bad = 0, seen = 0;
                for (float* const* pair : {sum, cnt, out}) {
                    std::vector<float> a(vox), b(vox);
                    cudaMemcpy(a.data(), pair[0], vox * sizeof(float), cudaMemcpyDeviceToHost);
                    cudaMemcpy(b.data(), pair[1], vox * sizeof(float), cudaMemcpyDeviceToHost);
                    for (size_t i = 0; i < vox; ++i) {
                        const bool nan = std::isnan(a[i]) && std::isnan(b[i]);
                        bad += !nan && std::memcmp(&a[i], &b[i], 4) != 0;
                        seen += a[i] != 0.0f;
                    }
                }
                ++runs;
                if (bad || seen < vox / 4) {
                    std::printf("geometry %d form %d way %d: %zu values differ, %zu not zero\n", geo, form, way, bad, seen);
                    ++differ;
                }
            }
        }
        cudaFree(d_ptm);
    }
    std::printf("%lld launches, %lld differ\n", runs, differ);
    return differ ? 1 : 0;
}
