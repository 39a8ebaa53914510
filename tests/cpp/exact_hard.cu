// The root and quotient of mps_exact.cuh in double, on the operands whose exact results lie nearest
// to the middle of two doubles, against the compiler's. Prints one count of differing results per
// check, then the number of operands of each.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <random>
#include <vector>

#include "../../mps_cuda_b200/csrc/mps_exact.cuh"

using namespace mps;
using u64 = unsigned long long;
using u128 = unsigned __int128;
struct Pair { double a, b; };

__global__ void roots(const Pair* v, int n, u64* bad) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n && sqrt_in(v[i].a) != sqrt(v[i].a)) atomicAdd(bad, 1ull);
}
__global__ void quotients(const Pair* v, int n, u64* bad) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double a = v[i].a, b = v[i].b;
    if (rcp_in(b) != 1.0 / b) atomicAdd(bad, 1ull);
    if (div_in(a, b) != a / b) atomicAdd(bad + 1, 1ull);
    if (div_by(a, b, 1.0 / b) != a / b) atomicAdd(bad + 2, 1ull);
}

// r with r^2 = c modulo 2^bits (c = 1 modulo 8), digit by digit
static u64 root_2adic(u64 c, int bits) {
    u64 r = 1;
    for (int k = 3; k < bits; ++k)
        if (((r * r - c) >> k) & 1) r += 1ull << (k - 1);
    return r;
}
// 1 / b modulo 2^64, b odd
static u64 inverse(u64 b) {
    u64 x = b;
    for (int k = 0; k < 6; ++k) x *= 2 - b * x;
    return x;
}
// m 2^e
static double scaled(u64 m, int e) { return ldexp(double(m), e); }

int main() {
    std::mt19937_64 rng(7);
    auto exponent = [&] { return int(rng() % 40) - 20; };
    // A root's middle is an odd M over 2^53, and x - M^2 / 2^106 = c / 2^106 with c = 1 modulo 8:
    // every operand within 2000 of a middle's square, at both parities of the exponent
    std::vector<Pair> x;
    for (long long c = -1999; c <= 2001; c += 8)
        for (int odd = 0; odd < 2; ++odd) {
            const int bits = 54 + odd;
            const u64 r = root_2adic(u64(c), bits), mask = (1ull << bits) - 1;
            for (u64 m : {r, 0 - r, r + (1ull << (bits - 1)), (1ull << (bits - 1)) - r}) {
                m &= mask;
                if (m < (1ull << 53) || m >= (1ull << 54)) continue;
                const u128 k = (u128(m) * m - u128((__int128)c)) >> bits;
                if (k >= (u128(1) << 53) || k < (u128(1) << 52)) continue;
                x.push_back({scaled(u64(k), -52 + odd + 2 * exponent()), 0});
            }
        }
    // A quotient's middle is an odd m of 54 bits, and a 2^s - b m = c: divisors at random and at
    // the ends of the binade, small c
    std::vector<Pair> q;
    auto nearest = [&](u64 b, u64 want) {
        for (int c = -9; c <= 9; c += 2)
            for (int s : {53, 54}) {
                const u64 mask = (1ull << s) - 1;
                u64 m = (0 - u64((long long)c)) * inverse(b) & mask;  // b m + c = 0 modulo 2^s
                if (s == 53) m |= 1ull << 53;                     // 54 bits: add the leading one
                if (!(m >> 53)) continue;
                const u128 a = (u128(b) * m + u128((__int128)c)) >> s;
                if (((u128(b) * m + u128((__int128)c)) & mask) != 0) continue;
                if (a < (u128(1) << 52) || a >= (u128(1) << 53)) continue;
                q.push_back({scaled(u64(a), exponent() - 52), scaled(b, exponent() - 52)});
            }
        for (u64 a : {1ull << 52, (1ull << 52) + 1, (1ull << 53) - 1, (1ull << 52) | (want >> 12)})
            q.push_back({scaled(a, exponent() - 52), scaled(b, exponent() - 52)});
    };
    for (u64 k = 0; k < 200000; ++k) {
        const u64 one = 1ull << 52;
        nearest((2 * one - 1) - 2 * k, rng());           // all ones downward: the reciprocal's middles
        nearest(one + 2 * k + 1, rng());
        nearest(one | (rng() >> 12) | 1, rng());
    }
    u64 bad[4] = {}, *d_bad;
    Pair* d;
    if (cudaMalloc(&d_bad, sizeof bad) != cudaSuccess ||
        cudaMemcpy(d_bad, bad, sizeof bad, cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMalloc(&d, sizeof(Pair) * std::max(x.size(), q.size())) != cudaSuccess ||
        cudaMemcpy(d, x.data(), sizeof(Pair) * x.size(), cudaMemcpyHostToDevice) != cudaSuccess)
        return 1;
    roots<<<int(x.size() + 255) / 256, 256>>>(d, int(x.size()), d_bad);
    if (cudaMemcpy(d, q.data(), sizeof(Pair) * q.size(), cudaMemcpyHostToDevice) != cudaSuccess) return 1;
    quotients<<<int(q.size() + 255) / 256, 256>>>(d, int(q.size()), d_bad + 1);
    if (cudaMemcpy(bad, d_bad, sizeof bad, cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
    for (u64 v : bad) printf("%llu ", v);
    printf("%zu %zu\n", x.size(), q.size());
    return 0;
}
