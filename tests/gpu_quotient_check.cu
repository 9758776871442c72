// Built and run by test_gpu_quotient.py: quotient(a, b, 1 / b) and over255(v)
// against __ddiv_rn on random operands (full mantissas, few-bit mantissas and
// mantissas next to all ones, exponents over the range that quotient_range
// admits). Prints the operands tried and the number of different results.
#include <cstdio>

#include "quotient.cuh"

using namespace stitch::b200;

__device__ unsigned long long mix(unsigned long long v) {
    v += 0x9e3779b97f4a7c15ull;
    v = (v ^ (v >> 30)) * 0xbf58476d1ce4e5b9ull;
    v = (v ^ (v >> 27)) * 0x94d049bb133111ebull;
    return v ^ (v >> 31);
}

__device__ double operand(unsigned long long h, int spread) {
    unsigned long long m = h & 0xfffffffffffffull;
    if ((h >> 60) == 0) m = ~0ull >> 12 ^ (m & 7);       // next to all ones
    else if ((h >> 60) == 1) m &= 0xfff0000000000ull;    // few bits
    const long long e = 1023 + static_cast<long long>((h >> 52 & 0xffull) * spread / 128) - spread;
    return __longlong_as_double(static_cast<long long>(m | static_cast<unsigned long long>(e) << 52));
}

__global__ void count(unsigned long long n, unsigned long long* bad) {
    unsigned long long q = 0, v = 0;
    for (unsigned long long i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const unsigned long long ha = mix(2 * i), hb = mix(2 * i + 1);
        const int spread = i & 1 ? 8 : 390;
        const double a = operand(ha, spread), b = (hb & 1 ? -1.0 : 1.0) * operand(hb, spread);
        q += !quotient_range(a, b) || quotient(a, b, __drcp_rn(b)) != __ddiv_rn(a, b);
        const double c = i % 3 ? operand(ha, 60) : static_cast<double>(i & 0xffff) / 256.0;
        v += over255(c) != __ddiv_rn(c, 255.0);
        const double w = static_cast<double>(1 + (hb >> 40)), x = static_cast<double>(ha >> 30) / 1048576.0 + 0.5;
        q += quotient(x, w, __ddiv_rn(1.0, w)) != __ddiv_rn(x, w);
    }
    atomicAdd(&bad[0], q);
    atomicAdd(&bad[1], v);
}

int main() {
    unsigned long long *bad = nullptr, host[2] = {~0ull, ~0ull};
    const unsigned long long n = 1ull << 28;
    if (cudaMalloc(&bad, sizeof(host)) != cudaSuccess || cudaMemset(bad, 0, sizeof(host)) != cudaSuccess) return 1;
    count<<<148 * 8, 256>>>(n, bad);
    if (cudaMemcpy(host, bad, sizeof(host), cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
    std::printf("operands %llu quotient %llu over255 %llu\n", n, host[0], host[1]);
    cudaFree(bad);
    return 0;
}
