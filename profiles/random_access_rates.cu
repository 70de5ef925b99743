/*
 * Random accesses by array size: the rates that the floors of the workload
 * table are made of.  Four independent accesses per thread, 8 blocks of 256
 * threads per SM, every address drawn by a hash of the access's number.
 *
 *   nvcc -gencode arch=compute_100a,code=sm_100a -O3 -o rates random_access_rates.cu && ./rates
 */
#include <cstdint>
#include <cstdio>
#include <cuda_runtime.h>

enum Kind { kRed, kAdd, kCas64, kCas128, kLoad8, kStore8, kStore16 };

__device__ __forceinline__ uint64_t mix(uint64_t x)
{
    x ^= x >> 33;
    x *= 0xff51afd7ed558ccdull;
    x ^= x >> 33;
    x *= 0xc4ceb9fe1a85ec53ull;
    return x ^ (x >> 33);
}

/* n accesses to 16-byte units of an array of `units` */
template <Kind kind>
__global__ void __launch_bounds__(256) access(unsigned long long *p, uint64_t units, uint64_t n,
                                              unsigned long long *sink)
{
    using ull = unsigned long long;
    const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
    ull sum = 0;
    for (uint64_t i0 = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; i0 < n; i0 += 4 * stride) {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const uint64_t i = i0 + u * stride;
            if (i >= n) continue;
            ull *const q = p + 2 * __umul64hi(mix(i), units);
            if constexpr (kind == kRed) {
                atomicAdd(q, 1ull);
            } else if constexpr (kind == kAdd) {
                sum += atomicAdd(q, 1ull);
            } else if constexpr (kind == kCas64) {
                sum += atomicCAS(q, 0ull, ull(i | 1));
            } else if constexpr (kind == kCas128) {
                ull lo, hi;
                asm volatile("{\n.reg .b128 c, n, o;\nmov.b128 c, {%2, %3};\nmov.b128 n, {%4, %5};\n"
                             "atom.global.cas.b128 o, [%6], c, n;\nmov.b128 {%0, %1}, o;\n}"
                             : "=l"(lo), "=l"(hi)
                             : "l"(0ull), "l"(0ull), "l"(ull(i | 1)), "l"(ull(i)), "l"(q)
                             : "memory");
                sum += lo;
            } else if constexpr (kind == kLoad8) {
                sum += __ldcg(q);
            } else if constexpr (kind == kStore8) {
                *reinterpret_cast<volatile ull *>(q) = i;
            } else {
                __stcg(reinterpret_cast<ulonglong2 *>(q), make_ulonglong2(i, i));
            }
        }
    }
    if (sum == 0x1234567) *sink = sum;
}

/* G accesses per second, best of three */
template <Kind kind>
double rate(unsigned long long *p, uint64_t bytes, unsigned long long *sink)
{
    const uint64_t n = 1ull << 25;
    cudaEvent_t a, b;
    cudaEventCreate(&a);
    cudaEventCreate(&b);
    float best = 1e9f;
    for (int r = 0; r < 3; ++r) {
        cudaMemset(p, 0, bytes);
        cudaEventRecord(a);
        access<kind><<<148 * 8, 256>>>(p, bytes / 16, n, sink);
        cudaEventRecord(b);
        cudaEventSynchronize(b);
        float ms = 0;
        cudaEventElapsedTime(&ms, a, b);
        if (ms < best) best = ms;
    }
    return double(n) / best / 1e6;
}

int main()
{
    unsigned long long *p = nullptr, *sink = nullptr;
    if (cudaMalloc(&p, 2400ull << 20) != cudaSuccess || cudaMalloc(&sink, 8) != cudaSuccess) return 1;
    std::printf("   MB red.add atom.add cas.64 cas.128 load 8 store 8 store 16\n");
    for (uint64_t mb : {16, 48, 96, 168, 256, 600, 2400}) {
        const uint64_t bytes = mb << 20;
        std::printf("%5lu %7.0f %8.0f %6.0f %7.0f %6.0f %7.0f %8.0f\n", (unsigned long)mb,
                    rate<kRed>(p, bytes, sink), rate<kAdd>(p, bytes, sink),
                    rate<kCas64>(p, bytes, sink), rate<kCas128>(p, bytes, sink),
                    rate<kLoad8>(p, bytes, sink), rate<kStore8>(p, bytes, sink),
                    rate<kStore16>(p, bytes, sink));
    }
    const cudaError_t e = cudaDeviceSynchronize();
    std::printf("%s\n", cudaGetErrorString(e));
    return e != cudaSuccess;
}
