// Check of mvs::quotients (csrc/quot.cuh) against the IEEE division, bit for bit:
// random operands over the exponents that the sweep's projections can have, and
// operands whose quotient lies as close to the middle of two floats as floats
// allow (a 2^25 = m b + e for odd 25-bit m and small e).  Prints one line per kind
// and exits 1 on any difference.
#include <cstdint>
#include <cstdio>

#include "../../plane-sweep-cuda_b200/csrc/quot.cuh"

__device__ uint64_t mix(uint64_t x)   // splitmix64
{
    x += 0x9e3779b97f4a7c15ull;
    x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ull;
    x = (x ^ (x >> 27)) * 0x94d049bb133111ebull;
    return x ^ (x >> 31);
}

// kind 0: |b| from 2^-25 to 2^60, |a / b| from 2^-26 to 2^40; 1: the same with b's significand all ones or zeros
// 2: next to a midpoint
__device__ bool operands(int kind, uint64_t i, float &a, float &b)
{
    const uint64_t r = mix(i), t = mix(r);
    uint32_t ma = (uint32_t)r & 0x7fffffu, mb = (uint32_t)(r >> 24) & 0x7fffffu;
    int eb = (int)(t % 86) - 25, ea = eb + (int)((t >> 16) % 67) - 26;
    if (kind == 1) mb = (r >> 60) & 1 ? 0x7fffffu - (uint32_t)((r >> 50) & 3) : (uint32_t)((r >> 50) & 3);
    if (kind == 2) {
        const uint32_t B = 0x800000u | mb | 1u;   // odd, 24 bits
        uint32_t inv = B;                         // B^-1 mod 2^32, by Newton
        for (int k = 0; k < 5; ++k) inv *= 2u - B * inv;
        const int e = (int)(t >> 40) % 9 - 4;
        const uint32_t m = ((uint32_t)(-e) * inv) & 0x1ffffffu;   // m B = -e (mod 2^25)
        if (!(m & 0x1000000u) || !(m & 1u) || e == 0) return false;   // a 25-bit odd number: a midpoint
        const uint64_t A = ((uint64_t)m * B + (int64_t)e) >> 25;  // m B + e = A 2^25
        if (A < 0x400000u || A >= 0x1000000u) return false;
        a = ldexpf((float)(uint32_t)A, ea - 23);
        b = ldexpf((float)B, eb - 23);
    } else {
        a = ldexpf((float)(0x800000u | ma), ea - 23);
        b = ldexpf((float)(0x800000u | mb), eb - 23);
    }
    if (r >> 63) a = -a;
    if ((t >> 62) & 1) b = -b;
    return true;
}

__global__ void check(int kind, uint64_t n, unsigned long long *bad, unsigned long long *done)
{
    unsigned long long nb = 0, nd = 0;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        float a, b, q0, q1;
        if (!operands(kind, i + (uint64_t)kind * 0x123456789ull, a, b)) continue;
        mvs::quotients(a, 3.f * a, b, q0, q1);
        nb += __float_as_uint(q0) != __float_as_uint(__fdiv_rn(a, b));
        nb += __float_as_uint(q1) != __float_as_uint(__fdiv_rn(3.f * a, b));
        ++nd;
    }
    atomicAdd(bad, nb);
    atomicAdd(done, nd);
}

int main()
{
    unsigned long long *c = nullptr, total = 0;
    if (cudaMalloc(&c, 2 * sizeof(*c)) != cudaSuccess) return 2;
    for (int kind = 0; kind < 3; ++kind) {
        cudaMemset(c, 0, 2 * sizeof(*c));
        check<<<148 * 16, 256>>>(kind, 1ull << 32, c, c + 1);
        unsigned long long h[2] = {~0ull, 0};
        cudaMemcpy(h, c, sizeof(h), cudaMemcpyDeviceToHost);
        const cudaError_t e = cudaGetLastError();
        printf("kind %d: %llu differences in %llu pairs %s\n", kind, h[0], h[1], cudaGetErrorString(e));
        total += e == cudaSuccess && h[1] > (1ull << 24) ? h[0] : 1;
    }
    cudaFree(c);
    return total == 0 ? 0 : 1;
}
