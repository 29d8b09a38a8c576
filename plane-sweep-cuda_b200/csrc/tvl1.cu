// TV-L1 depth denoising (PlaneSweep::CudaDenoise, planesweep.cpp:297-379) for
// sm_100a.
//
// The reference alternates two full-image launches per iteration:
// denoising_TVL1_calculateP_tensor_weighed (kernels.cu:283-307) and
// denoising_TVL1_update (kernels.cu:342-370).  Here one launch runs several
// iterations on a region of the image held on chip (tvl1_block_kernel).
// Arithmetic follows the reference statement for statement (compiled with
// -fmad=false); its projections are formed by project() (proj.cuh), the same
// floats.
#include <math.h>

#include "blocked.cuh"
#include "common.cuh"
#include "proj.cuh"

namespace mvs {
namespace {

constexpr float kInv255 = 1.f / 255.f;
constexpr int TX = 32, TY = 8;

// ref/255 and its diffusion tensor (Anisotropic_diffusion_tensor_kernel,
// TGV2_kernels.cu:257-298), and the scaled start (planesweep.cpp:334-344):
// out = (d - znear) * xscale.
__global__ void tvl1_setup_kernel(const float *__restrict__ ref255, const float *__restrict__ depth, int w, int h,
                                  float beta, float gamma, float znear, float xscale,
                                  float *__restrict__ T11, float *__restrict__ T12, float *__restrict__ T22,
                                  float *__restrict__ out, float *__restrict__ R,
                                  float *__restrict__ Px, float *__restrict__ Py)
{
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= w || y >= h) return;
    const int i = y * w + x, xn = min(x + 1, w - 1), yn = min(y + 1, h - 1);
    const float r = ref255[i] * kInv255;
    float gx = ref255[y * w + xn] * kInv255 - r;
    float gy = ref255[yn * w + x] * kInv255 - r;
    const float d = sqrtf(gx * gx + gy * gy);
    if (d > 0.f) {
        gx = gx / d;
        gy = gy / d;
        const float k = expf(-beta * powf(d, gamma));
        T11[i] = k * gx * gx + gy * gy;
        T12[i] = (k - 1) * gx * gy;
        T22[i] = k * gy * gy + gx * gx;
    } else {
        T11[i] = 1.f;
        T12[i] = 0.f;
        T22[i] = 1.f;
    }
    const float s = depth[i] + -znear;
    out[i] = s * xscale;
    R[i] = 0.f;
    Px[i] = 0.f;
    Py[i] = 0.f;
}

struct Bufs {
    const float *T11, *T12, *T22, *depth;
    const float *in, *R_in, *Px_in, *Py_in;
    float *out, *R_out, *Px_out, *Py_out;
    int w, h;
    int iters;          // iterations of this launch
    int halo;           // block_halo(iters)
    int first;          // 1: this launch starts the run
    float sigma_first, sigma_p, tau, theta, lambda, sigma, znear, inputscale;
};

// `iters` iterations in one launch on the regions of blocked.cuh: primal, px,
// py, r and the data term in registers, the tensor, as the doubles the update
// wants, in shared memory.  Neighbours in x come by warp shuffles, in y from
// the thread's own rows or, across warps, from one row per warp and direction
// in shared memory, so an iteration is two barriers and no global access.
// Nothing that another CTA reads is written in place (primal, p and r are
// double-buffered).
//
// What bounds it: instruction issue and the FP64 and conversion pipes (about
// 120 instructions, 30 of them FP64 and 6 conversions, per cell and
// iteration), then the 4 us that a launch costs with its loads.  One launch per
// iteration was bound by that chain of launch, loads and barriers alone: 7.2 us
// an iteration at 640x480, of which the IEEE double square root and divisions
// of the projections were a third; 3.0 us in this form (B200).
constexpr int BW = kBlockW, RPT = kBlockRows, MAXWARPS = 32;
constexpr size_t kWarpBytes = (size_t)3 * RPT * 32 * sizeof(double2);   // dynamic shared memory per warp: the tensor

template <bool THETA1>
__global__ void __launch_bounds__(32 * MAXWARPS) tvl1_block_kernel(Bufs b)
{
    extern __shared__ double2 sT[];   // [3][rows][32]: T11, T12, T22 of the region
    // the rows that neighbouring warps read: each warp's first row of the
    // primal and last row of py (with a row of zeros below the last and above
    // the first warp: their values only reach halo cells)
    __shared__ float2 sTop[MAXWARPS + 1][32], sBot[MAXWARPS + 1][32];
    const int w = b.w, h = b.h, K = b.halo;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const int xa = (int)blockIdx.x * (BW - 2 * K) - K + 2 * lane;
    const int y0 = (int)blockIdx.y * (RPT * warps - 2 * K) - K + RPT * warp;
    bool in[RPT][2];
#pragma unroll
    for (int j = 0; j < RPT; ++j)
#pragma unroll
        for (int c = 0; c < 2; ++c) in[j][c] = xa + c >= 0 && xa + c < w && y0 + j >= 0 && y0 + j < h;
    float o[RPT][2], px[RPT][2], py[RPT][2], r[RPT][2], raw[RPT][2];
    const int rows = RPT * warps;
    if (b.first) wait_for_previous_grid();   // the set-up is complete
#pragma unroll
    for (int j = 0; j < RPT; ++j) {
        double2 t[3];
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            const size_t i = (size_t)(y0 + j) * w + (xa + c);
            // constant through the run: read before the wait in the later launches
            const float a = in[j][c] ? ldg(b.T11 + i) : 0.f, d = in[j][c] ? ldg(b.T12 + i) : 0.f;
            const float e = in[j][c] ? ldg(b.T22 + i) : 0.f;
            (c ? t[0].y : t[0].x) = a;
            (c ? t[1].y : t[1].x) = d;
            (c ? t[2].y : t[2].x) = e;
            raw[j][c] = in[j][c] ? (ldg(b.depth + i) + -b.znear) * b.inputscale : 0.f;
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) sT[(k * rows + RPT * warp + j) * 32 + lane] = t[k];   // read by this thread only
    }
    if (!b.first) wait_for_previous_grid();   // dependent launch: the previous iterations are complete
    allow_next_grid();   // after the wait: the next launch reads the set-up's data before its own
#pragma unroll
    for (int j = 0; j < RPT; ++j)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            const size_t i = (size_t)(y0 + j) * w + (xa + c);
            o[j][c] = in[j][c] ? b.in[i] : 0.f;
            px[j][c] = in[j][c] ? b.Px_in[i] : 0.f;
            py[j][c] = in[j][c] ? b.Py_in[i] : 0.f;
            r[j][c] = in[j][c] ? b.R_in[i] : 0.f;
        }
    const bool right0 = xa + 1 <= w - 1, right1 = xa + 2 <= w - 1;   // has a right neighbour
    if (warp == 0) sTop[warps][lane] = sBot[0][lane] = make_float2(0.f, 0.f);
    const double sigma = b.sigma_p;
    double sp = b.first ? (double)b.sigma_first : sigma;
    for (int k = 0; k < b.iters; ++k) {
        sTop[warp][lane] = make_float2(o[0][0], o[0][1]);
        // denoising_TVL1_calculateP_tensor_weighed_kernel (kernels.cu:283-307) of one row, `d0`, `d1`: the row below
        auto p_row = [&](int j, float d0, float d1) {
            const float nr = __shfl_down_sync(0xffffffffu, o[j][0], 1);
            const bool down = y0 + j + 1 <= h - 1;
            const float rt[2] = {right0 ? o[j][1] : o[j][0], right1 ? nr : o[j][1]};
            const float dn[2] = {down ? d0 : o[j][0], down ? d1 : o[j][1]};
            double d2[2][2], s2[2];
            float q[2][2];
            const double2 *tr = sT + (RPT * warp + j) * 32 + lane;
            const double2 u11 = tr[0], u12 = tr[rows * 32], u22 = tr[2 * rows * 32];
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const double x = rt[c] - o[j][c], y = dn[c] - o[j][c];
                const double a11 = c ? u11.y : u11.x, a12 = c ? u12.y : u12.x, a22 = c ? u22.y : u22.x;
                d2[c][0] = (double)px[j][c] + sp * (a11 * x + a12 * y);
                d2[c][1] = (double)py[j][c] + sp * (a12 * x + a22 * y);
                s2[c] = d2[c][0] * d2[c][0] + d2[c][1] * d2[c][1];
            }
            project(s2, d2, q);
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                px[j][c] = q[c][0];
                py[j][c] = q[c][1];
            }
        };
        // denoising_TVL1_update_kernel (kernels.cu:342-370) of one row, `u0`, `u1`: py of the row above
        auto d_row = [&](int j, float u0, float u1) {
            const float nl = __shfl_up_sync(0xffffffffu, px[j][1], 1);
            // at x = 0 the reference leaves the difference in x out: (px - px) + cpy is cpy
            const float pl[2] = {xa == 0 ? px[j][0] : nl, px[j][0]};
            const float pu[2] = {y0 + j > 0 ? u0 : py[j][0], y0 + j > 0 ? u1 : py[j][1]};
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                float q = r[j][c];
                q += raw[j][c];
                const float ov = o[j][c];
                q += b.sigma * ov;
                // if (q > lambda) q = lambda; if (q < -lambda) q = -lambda; a NaN stays
                asm("min.NaN.f32 %0, %0, %1;" : "+f"(q) : "f"(b.lambda));
                asm("max.NaN.f32 %0, %0, %1;" : "+f"(q) : "f"(-b.lambda));
                r[j][c] = q;
                const float cpx = px[j][c], cpy = py[j][c];
                const float xn = ov + b.tau * (cpx - pl[c] + cpy - pu[c]) - b.tau * q;
                // The reference forms xn + theta (xn - o) in double.  For theta = 1 that
                // is 2 xn - o, whose double sum is exact unless one term is below 2^-28
                // of the other, where the float result is the larger term either way:
                // one fused multiply-add gives the same float.
                o[j][c] = THETA1 ? __fmaf_rn(2.f, xn, -ov)
                                         : (float)((double)xn + (double)b.theta * ((double)xn - (double)ov));
            }
        };
#pragma unroll
        for (int j = 0; j + 1 < RPT; ++j) p_row(j, o[j + 1][0], o[j + 1][1]);
        __syncthreads();
        const float2 below = sTop[warp + 1][lane];
        p_row(RPT - 1, below.x, below.y);
        sBot[warp + 1][lane] = make_float2(py[RPT - 1][0], py[RPT - 1][1]);
#pragma unroll
        for (int j = RPT - 1; j > 0; --j) d_row(j, py[j - 1][0], py[j - 1][1]);
        __syncthreads();
        const float2 above = sBot[warp][lane];
        d_row(0, above.x, above.y);
        sp = sigma;
    }
    const int xl = 2 * lane, yl = RPT * warp;
#pragma unroll
    for (int j = 0; j < RPT; ++j)
#pragma unroll
        for (int c = 0; c < 2; ++c)
            if (in[j][c] && xl + c >= K && xl + c < BW - K && yl + j >= K && yl + j < RPT * warps - K) {
                const size_t i = (size_t)(y0 + j) * w + (xa + c);
                b.out[i] = o[j][c];
                b.Px_out[i] = px[j][c];
                b.Py_out[i] = py[j][c];
                b.R_out[i] = r[j][c];
            }
}

// element_scale(d, zfar - znear) then element_add(d, znear) (planesweep.cpp:355-356)
__global__ void tvl1_finish_kernel(const float *__restrict__ in, int n, float scale, float znear, float *__restrict__ out)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        out[i] = in[i] * scale + znear;
}

struct Layout {
    float *T11, *T12, *T22, *D[2], *R[2], *Px[2], *Py[2];
    size_t bytes;
};

Layout layout(void *base, int w, int h)
{
    Layout L{};
    const size_t n = (size_t)w * h;
    char *p = (char *)base;
    size_t off = 0;
    auto take = [&]() {
        float *q = (float *)(p + off);
        off += ((n * sizeof(float) + 255) / 256) * 256;
        return q;
    };
    L.T11 = take();
    L.T12 = take();
    L.T22 = take();
    for (int k = 0; k < 2; ++k) {
        L.D[k] = take();
        L.R[k] = take();
        L.Px[k] = take();
        L.Py[k] = take();
    }
    L.bytes = off;
    return L;
}

}  // namespace

size_t tvl1_workspace_bytes(int w, int h) { return layout(nullptr, w, h).bytes; }

int tvl1_run(int w, int h, const float *ref255, float *depth, float znear, float zfar, const mvs_tvl1_params *prm,
             void *ws, cudaStream_t st)
{
    Layout L = layout(ws, w, h);
    const int n = w * h;
    // xscale = 1.f/(zfar - znear) in float; inputscale = -sigma/(zfar - znear)
    // in double, both handed to float kernel parameters (planesweep.cpp:340-344)
    const float xscale = 1.f / (zfar - znear);
    const float inputscale = (float)(-(double)prm->sigma / (double)(zfar - znear));
    const dim3 b2(TX, TY), g2(ceil_div(w, TX), ceil_div(h, TY));
    tvl1_setup_kernel<<<g2, b2, 0, st>>>(ref255, depth, w, h, prm->beta, prm->gamma, znear, xscale, L.T11, L.T12, L.T22,
                                        L.D[0], L.R[0], L.Px[0], L.Py[0]);
    int cur = 0;
    Bufs b;
    b.T11 = L.T11;
    b.T12 = L.T12;
    b.T22 = L.T22;
    b.depth = depth;
    b.w = w;
    b.h = h;
    b.tau = prm->tau;
    b.theta = prm->theta;
    b.lambda = prm->lambda;
    b.sigma = prm->sigma;
    b.znear = znear;
    b.inputscale = inputscale;
    // first dual step uses sigma + 1 (planesweep.cpp:347)
    b.sigma_first = (float)(1.0 + (double)prm->sigma);
    b.sigma_p = (float)(double)prm->sigma;
    // Measured on the B200 over 97x73 to 1242x375: 4.2 us a launch plus 0.08 us an
    // iteration and warp, within 10% (640x480: 4 iterations and 24 warps, 284 us
    // per 100 iterations, against 324 us for 4 and 14 and 389 us for 2 and 24;
    // 320x240: 6 and 12, 176 us; 1242x375: 400 us)
    const BlockPlan plan = block_plan(w, h, prm->niters, MAXWARPS, 4.2, 0.08);
    const size_t smem = kWarpBytes * plan.warps;
    auto kernel = b.theta == 1.f ? tvl1_block_kernel<true> : tvl1_block_kernel<false>;
    MVS_TRY_CUDA(allow_shared_memory(kernel, kWarpBytes * MAXWARPS));
    for (int it = 0; it < prm->niters; it += b.iters) {
        b.iters = min(plan.iters, prm->niters - it);
        b.halo = block_halo(b.iters);
        b.first = it == 0;
        b.in = L.D[cur];
        b.R_in = L.R[cur];
        b.Px_in = L.Px[cur];
        b.Py_in = L.Py[cur];
        b.out = L.D[cur ^ 1];
        b.R_out = L.R[cur ^ 1];
        b.Px_out = L.Px[cur ^ 1];
        b.Py_out = L.Py[cur ^ 1];
        MVS_TRY_CUDA(launch_dependent(kernel, block_grid(w, h, b.iters, plan.warps), dim3(32 * plan.warps), smem, st, b));
        cur ^= 1;
    }
    tvl1_finish_kernel<<<min(ceil_div(n, 256), 8 * kSMs), 256, 0, st>>>(L.D[cur], n, zfar - znear, znear, depth);
    return check_launch("tvl1 denoise");
}

}  // namespace mvs
