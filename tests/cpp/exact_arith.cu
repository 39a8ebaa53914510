// Compares the correctly rounded root and quotient of mps_exact.cuh with the compiler's, on the
// device. Prints one count of differing results per check.
#include <cstdio>

#include "../../mps_cuda_b200/csrc/mps_exact.cuh"

using namespace mps;
__device__ unsigned long long bad[8];

// every significand of a root's operand, at both parities of the exponent, near 1 and near 2^-63
__global__ void f32_root() {
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    for (unsigned e : {0x3f800000u, 0x20000000u}) {
        const float x = __uint_as_float(e + i);
        if (sqrt_in(x) != sqrtf(x)) atomicAdd(&bad[0], 1ull);
    }
}
// every significand of a divisor: its reciprocal, 64 quotients, and 64 quotients by it given
// its rounded reciprocal
__global__ void f32_div() {
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    const float b = __uint_as_float(0x3f800000u + i), c = 1.0f / b;
    if (rcp_in(b) != c) atomicAdd(&bad[1], 1ull);
    unsigned h = i * 2654435761u + 12345u;
    for (int k = 0; k < 64; ++k) {
        h ^= h << 13;
        h ^= h >> 17;
        h ^= h << 5;
        const float a = __uint_as_float(0x3f800000u | (h & 0x7fffffu));
        if (div_in(a, b) != a / b) atomicAdd(&bad[2], 1ull);
        if (div_by(a, b, c) != a / b) atomicAdd(&bad[3], 1ull);
    }
}
// random doubles over 32 binades
__global__ void f64_all() {
    unsigned long long h = 99 + (blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x) *
                                    0x9E3779B97F4A7C15ull;
    for (int k = 0; k < 32; ++k) {
        h ^= h << 13;
        h ^= h >> 7;
        h ^= h << 17;
        const double x = __longlong_as_double(0x3f00000000000000ull + (h >> 6) % 0x0200000000000000ull);
        const unsigned long long g = h * 0xD1342543DE82EF95ull + 1;
        const double a = __longlong_as_double(0x3f00000000000000ull + (g >> 6) % 0x0200000000000000ull);
        if (sqrt_in(x) != sqrt(x)) atomicAdd(&bad[4], 1ull);
        if (rcp_in(x) != 1.0 / x) atomicAdd(&bad[5], 1ull);
        if (div_in(a, x) != a / x) atomicAdd(&bad[6], 1ull);
        if (div_by(a, x, 1.0 / x) != a / x) atomicAdd(&bad[7], 1ull);
    }
}

int main() {
    f32_root<<<(1 << 24) / 256, 256>>>();
    f32_div<<<(1 << 23) / 256, 256>>>();
    f64_all<<<4096, 256>>>();
    unsigned long long b[8];
    if (cudaDeviceSynchronize() != cudaSuccess || cudaMemcpyFromSymbol(b, bad, sizeof b) != cudaSuccess)
        return 1;
    for (int i = 0; i < 8; ++i) printf("%llu ", b[i]);
    printf("\n");
    return 0;
}
