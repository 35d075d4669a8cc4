// Test-only: compares fwi::div4_by_const (fwi_gb300/csrc/fwi_div.cuh) bit for
// bit with CUDA's IEEE division over pseudo-random quads whose four dividends
// are drawn from zeros, denormals, tiny, ordinary, huge and non-finite values.
#include <cstdint>

#include "fwi_div.cuh"

namespace {

__device__ unsigned mix(uint64_t x) {  // splitmix64
    x += 0x9e3779b97f4a7c15ull;
    x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ull;
    x = (x ^ (x >> 27)) * 0x94d049bb133111ebull;
    return (unsigned)(x >> 32);
}

__global__ void k_check(float b, float y, unsigned quads, unsigned long long* bad) {
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < quads; i += gridDim.x * blockDim.x) {
        float a[4], q[4];
        const unsigned kinds = mix(2 * (uint64_t)i);
        for (int e = 0; e < 4; ++e) {
            unsigned u = mix(0x100000000ull + 4 * (uint64_t)i + e);
            switch ((kinds >> (8 * e)) & 7u) {
                case 0: u &= 0x80000000u; break;                                 // zeros
                case 1: u &= 0x80003fffu; break;                                 // the smallest denormals
                case 2: u &= 0x807fffffu; break;                                 // denormals
                case 3: u = (u & 0x80ffffffu) | ((u >> 8 & 0x0cu) << 24); break;  // tiny and small
                case 4: u |= 0x70000000u; break;                                 // huge, infinities, NaN
                default: break;
            }
            a[e] = q[e] = __uint_as_float(u);
        }
        fwi::div4_by_const(q, b, y);
        for (int e = 0; e < 4; ++e) {
            const float ref = __fdiv_rn(a[e], b);
            if (__float_as_uint(ref) != __float_as_uint(q[e]) && (ref == ref || q[e] == q[e])) atomicAdd(bad, 1ull);
        }
    }
}

}  // namespace

extern "C" int div4_check(float b, float y, unsigned quads, unsigned long long* mismatches) {
    unsigned long long* d_bad = nullptr;
    if (cudaMalloc(&d_bad, sizeof *d_bad) != cudaSuccess) return 1;
    cudaMemset(d_bad, 0, sizeof *d_bad);
    k_check<<<152 * 8, 256>>>(b, y, quads, d_bad);
    const cudaError_t e = cudaDeviceSynchronize();
    cudaMemcpy(mismatches, d_bad, sizeof *d_bad, cudaMemcpyDeviceToHost);
    cudaFree(d_bad);
    return e == cudaSuccess ? 0 : 1;
}
