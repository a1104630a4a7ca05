// Counts, over all significands, where the shared-root evaluation of physics.cuh differs from
// the IEEE operations it stands for (tests/test_gpu_rounding.py). Test infrastructure only.
#include <cuda_runtime.h>

#include "../hidem_b200/csrc/physics.cuh"

using namespace hidem;

__device__ unsigned long long g_bad[4];

__device__ void count(int k, bool bad) {
    if (bad) atomicAdd(g_bad + k, 1ull);
}

// v runs over two binades from `base` (every significand with both exponent parities)
__global__ void k_roundings(unsigned base, unsigned salt) {
    const unsigned m = blockIdx.x * blockDim.x + threadIdx.x;
    const float v = __uint_as_float(base + m);
    const float r = rsqrt_start(v);
    const float s = root_from(v, r);
    count(0, s != __fsqrt_rn(v));
    count(1, !tie_root(v) && recip_from(s, r) != __frcp_rn(s));
    // reciprocals of v from starts up to 16 units off, then quotients of random numerators
    unsigned h = (m + salt) * 2654435761u;
    for (int k = -16; k <= 16; k += 2) {
        const float y0 = __uint_as_float(__float_as_uint(__frcp_rn(v)) + k);
        const float y = recip_from(v, y0);
        count(2, !all_ones(v) && y != __frcp_rn(v));
        for (int j = 0; j < 2; ++j) {
            h = h * 1664525u + 1013904223u;
            const float n = __uint_as_float((j ? 0x4c000000u : 0x3f800000u) | (h >> 9));
            count(3, !all_ones(v) && quotient_from(n, v, y) != __fdiv_rn(n, v));
        }
    }
}

// v = 1.0 .. with numerators whose quotient ends next to a tie: n = RN(v * (q + ulp/2))
__global__ void k_hard_quotients(unsigned base, unsigned qbase) {
    const unsigned m = blockIdx.x * blockDim.x + threadIdx.x;
    const float v = __uint_as_float(base + m);
    const float y = recip_from(v, __frcp_rn(v));
    unsigned h = m * 2246822519u + qbase;
    for (int k = 0; k < 32; ++k) {
        h = h * 1664525u + 1013904223u;
        const float q = __uint_as_float(0x3f800000u | (h >> 9));
        const double mid = (double)q + 0.5 * ((double)__uint_as_float(__float_as_uint(q) + 1) - (double)q);
        const float n = (float)((double)v * mid);
        count(3, !all_ones(v) && (quotient_from(n, v, y) != __fdiv_rn(n, v) || quotient_from(q, v, y) != __fdiv_rn(q, v)));
    }
}

extern "C" int rounding_mismatches(unsigned base, unsigned salt, unsigned long long *out) {
    void *p = nullptr;
    if (cudaGetSymbolAddress(&p, g_bad) != cudaSuccess) return 1;
    if (cudaMemset(p, 0, sizeof(unsigned long long) * 4) != cudaSuccess) return 2;
    k_roundings<<<(1 << 24) / 256, 256>>>(base, salt);
    k_hard_quotients<<<(1 << 24) / 256, 256>>>(base, salt);
    if (cudaDeviceSynchronize() != cudaSuccess) return 3;
    return cudaMemcpy(out, p, sizeof(unsigned long long) * 4, cudaMemcpyDeviceToHost) == cudaSuccess ? 0 : 4;
}
