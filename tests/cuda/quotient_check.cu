// The FP32 form's quotient RN(U r + RN(U rl)) (bp_quotient2 in
// jenhine_b200/csrc/bp_common.cuh) against CUDA's correctly rounded __fdiv_rn, on
// random mantissas: |W| and |U| from 2^-60 to 2^60, and from the scales of projection
// matrices (1/2 .. 2, U to 4096).  Where the two differ, the quotient has to be the
// float next to the right one with U / W within 3 2^-48 of the middle between them
// (three roundings of 2^-48 before the last one; 3.01 for what the bound itself
// leaves out, 2^-53 for U / W in double) -- unless U rl is below the normal floats,
// which takes |U / W| < 2^-78 (a place adds 0.5 to it).  The scalar form and both lanes have to
// agree, and the EXACT form never differs.  Prints the counts; exit status 0 when
// all holds.  Built and run by tests/test_quotient.py.
#include <cstdio>

#include "bp_common.cuh"

__device__ unsigned mix(unsigned long long x) {   // splitmix64
    x += 0x9E3779B97F4A7C15ull;
    x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
    x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
    return (unsigned)((x ^ (x >> 31)) >> 16);
}

// counts: [0] quotients that differ from __fdiv_rn, [1] differ by more than allowed, [2] forms that disagree
__global__ void check(unsigned long long n, int wide, unsigned long long* counts) {
    const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
    for (unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        float v[3];
        for (int k = 0; k < 3; ++k) {   // W, two U
            const unsigned m = mix(6 * i + 2 * k + (wide ? 1ull << 60 : 0ull)), e = mix(6 * i + 2 * k + 1);
            const int exponent = wide ? (int)(e % 121u) - 60 : k == 0 ? -(int)(e & 1u) : (int)(e % 13u);
            v[k] = ldexpf(__uint_as_float(0x3F800000u | (m & 0x7FFFFFu)), exponent) * ((e >> 20 & 1u) && (wide || k) ? -1.0f : 1.0f);
        }
        const float W = v[0];
        const jfdk::Recip rc = jfdk::bp_recip(W);
        const float2 U = make_float2(v[1], v[2]);
        const float2 fast = jfdk::bp_quotient2<false>(U, W, rc), exact = jfdk::bp_quotient2<true>(U, W, rc);
        const float u[2] = {U.x, U.y}, f[2] = {fast.x, fast.y}, x[2] = {exact.x, exact.y};
        for (int k = 0; k < 2; ++k) {
            const float right = __fdiv_rn(u[k], W);
            if (x[k] != right || jfdk::bp_quotient<true>(u[k], W, rc) != right || jfdk::bp_quotient<false>(u[k], W, rc) != f[k])
                atomicAdd(counts + 2, 1ull);
            if (f[k] == right) continue;
            atomicAdd(counts, 1ull);
            const int apart = __float_as_int(f[k]) - __float_as_int(right);
            const double q = (double)u[k] / (double)W, middle = 0.5 * ((double)f[k] + (double)right);
            const bool normal = fabs((double)u[k] * (double)rc.rl) >= 0x1p-126;
            if ((apart != 1 && apart != -1) || (normal && fabs(q - middle) > (3.01 * 0x1p-48 + 0x1p-53) * fabs(q))) atomicAdd(counts + 1, 1ull);
        }
    }
}

int main() {
    unsigned long long* counts = nullptr;
    if (cudaMalloc(&counts, 3 * sizeof(*counts)) != cudaSuccess) {
        std::printf("allocation failed\n");
        return 2;
    }
    int status = 0;
    for (int wide = 0; wide < 2; ++wide) {
        const unsigned long long n = 1ull << 30;   // two quotients each
        cudaMemset(counts, 0, 3 * sizeof(*counts));
        check<<<148 * 8, 256>>>(n, wide, counts);
        const cudaError_t e = cudaDeviceSynchronize();
        if (e != cudaSuccess) {
            std::printf("CUDA error: %s\n", cudaGetErrorString(e));
            return 2;
        }
        unsigned long long h[3] = {0};
        cudaMemcpy(h, counts, sizeof(h), cudaMemcpyDeviceToHost);
        std::printf("%s: %llu quotients, %llu differ, %llu outside the bound, %llu forms disagree\n",
                    wide ? "wide" : "matrices", 2 * n, h[0], h[1], h[2]);
        if (h[1] || h[2]) status = 1;
    }
    cudaFree(counts);
    return status;
}
