// Check of mvs::project (csrc/proj.cuh) where components are zero, by the bits of the
// results: a zero keeps the sign that the division x / d gives it, beside generic values,
// short sums of floats (whose norms are often the middle of two floats) and projections that
// are the identity.  Prints one line per count of components and projections; exits 1 on any
// difference.
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
__device__ double unit(uint64_t r) { return (double)(mix(r) >> 11) * 0x1p-52 - 1; }   // [-1, 1)

__device__ double value(uint64_t r)
{
    const float a = (float)unit(r ^ 0x1111), b = (float)unit(r ^ 0x2222);
    switch (r & 7) {
    case 0: case 1: return 0.0;
    case 2: case 3: return -0.0;
    case 4: return 3 * unit(r ^ 0x3333);
    case 5: return 0.5 * unit(r ^ 0x4444);
    case 6: return (double)a + 6.0 * (double)b;
    default: return (double)a;
    }
}

template <int M, int N>
__global__ void check(uint64_t n, unsigned long long *bad)
{
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        double s[M], x[M][N];
        float out[M][N];
        for (int m = 0; m < M; ++m) {
            for (int c = 0; c < N; ++c) x[m][c] = value(mix(i * 16 + m * 4 + c + N * 0x1234567ull + M));
            s[m] = __dadd_rn(__dmul_rn(x[m][0], x[m][0]), __dmul_rn(x[m][1], x[m][1]));
            if (N == 3) {   // dz counts twice, as in the reference's q
                const double z = __dmul_rn(x[m][N - 1], x[m][N - 1]);
                s[m] = __dadd_rn(__dadd_rn(s[m], z), z);
            }
        }
        mvs::project(s, x, out);
        for (int m = 0; m < M; ++m) {
            const double d = (double)fmaxf(1.f, (float)sqrt(s[m]));
            for (int c = 0; c < N; ++c)
                if (__float_as_uint((float)(x[m][c] / d)) != __float_as_uint(out[m][c])) atomicAdd(bad, 1ull);
        }
    }
}

template <int M, int N>
bool report(unsigned long long *bad)
{
    unsigned long long hb = ~0ull;
    cudaMemset(bad, 0, sizeof(*bad));
    check<M, N><<<148 * 8, 256>>>(1ull << 25, bad);
    cudaMemcpy(&hb, bad, sizeof(hb), cudaMemcpyDeviceToHost);
    const cudaError_t e = cudaGetLastError();
    printf("%d x %d: %llu differences %s\n", M, N, hb, cudaGetErrorString(e));
    return e == cudaSuccess && hb == 0;
}

int main()
{
    unsigned long long *bad = nullptr;
    if (cudaMalloc(&bad, sizeof(*bad)) != cudaSuccess) return 2;
    bool ok = report<1, 2>(bad);
    ok = report<2, 2>(bad) && ok;
    ok = report<1, 3>(bad) && ok;
    ok = report<2, 3>(bad) && ok;
    cudaFree(bad);
    return ok ? 0 : 1;
}
