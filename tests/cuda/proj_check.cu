// Check of mvs::project (csrc/proj.cuh) against the IEEE double square root and
// divisions of the reference's projections, bit for bit, for 2 and 3
// components: generic values, values where one component is zero (whose norm
// is a short sum of floats, often the middle of two floats), norms next to 1,
// short sums on both sides of 1, tiny and huge components, infinities and NaN.
// Prints one line per kind and exits 1 on any difference.
#include <cstdint>
#include <cstdio>

#include <cuda_runtime.h>

#include "../../plane-sweep-cuda_b200/csrc/proj.cuh"

__device__ uint64_t mix(uint64_t x)   // splitmix64
{
    x += 0x9e3779b97f4a7c15ull;
    x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ull;
    x = (x ^ (x >> 27)) * 0x94d049bb133111ebull;
    return x ^ (x >> 31);
}
__device__ double unit(uint64_t r) { return (double)(r >> 11) * 0x1p-53; }

__device__ double value(int kind, uint64_t r)
{
    const double u = 2 * unit(mix(r)) - 1;
    const float a = (float)(2 * unit(mix(r ^ 0x1111)) - 1), b = (float)(2 * unit(mix(r ^ 0x2222)) - 1);
    switch (kind) {
    case 0: return 3 * u;                                   // generic doubles
    case 1: return (r & 3) ? 0.0 : (double)a + 6.0 * b;     // mostly one component, a short sum of floats
    case 2: return 0.70710678118654752 * (1 + 0x1p-20 * u) * ((r & 1) ? 1 : -1);   // norms next to 1
    case 3: return (double)a + 1.5 * (double)b;             // short sums
    case 4: return ldexp(u, -(int)(mix(r ^ 7) % 200)) * ((r & 4) ? 2 : 1);         // down to below the normal floats
    case 5: return ldexp(u, (int)(mix(r ^ 7) % 126));       // up to the largest floats
    default: {
        const unsigned k = (unsigned)(mix(r ^ 9) % 8);
        return k == 0 ? INFINITY : k == 1 ? -INFINITY : k == 2 ? NAN : k == 3 ? -0.0 : 2 * u;
    }
    }
}

template <int M, int N>
__global__ void check(int kind, uint64_t n, unsigned long long *bad)
{
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        double s[M], x[M][N];
        float out[M][N];
        for (int m = 0; m < M; ++m) {
            for (int c = 0; c < N; ++c) x[m][c] = value(kind, mix(i * 16 + m * 4 + c + (uint64_t)kind * 0x1234567));
            s[m] = __dadd_rn(__dmul_rn(x[m][0], x[m][0]), __dmul_rn(x[m][1], x[m][1]));
            if (N == 3) {   // dz counts twice, as in the reference's q
                const double z = __dmul_rn(x[m][N - 1], x[m][N - 1]);
                s[m] = __dadd_rn(__dadd_rn(s[m], z), z);
            }
        }
        mvs::project(s, x, out);
        for (int m = 0; m < M; ++m) {
            const double d = (double)fmaxf(1.f, (float)sqrt(s[m]));
            for (int c = 0; c < N; ++c) {
                const float want = (float)(x[m][c] / d);
                if (!(want != want && out[m][c] != out[m][c]) && want != out[m][c]) atomicAdd(bad, 1ull);
            }
        }
    }
}

int main()
{
    unsigned long long *bad = nullptr, total = 0;
    if (cudaMalloc(&bad, sizeof(*bad)) != cudaSuccess) return 2;
    for (int kind = 0; kind < 7; ++kind) {
        const uint64_t n = 1ull << 27;
        cudaMemset(bad, 0, sizeof(*bad));
        check<2, 2><<<148 * 8, 256>>>(kind, n, bad);
        check<1, 3><<<148 * 8, 256>>>(kind, n, bad);
        unsigned long long hb = ~0ull;
        cudaMemcpy(&hb, bad, sizeof(hb), cudaMemcpyDeviceToHost);
        const cudaError_t e = cudaGetLastError();
        printf("kind %d: %llu differences %s\n", kind, hb, cudaGetErrorString(e));
        total += e == cudaSuccess ? hb : 1;
    }
    cudaFree(bad);
    return total == 0 ? 0 : 1;
}
