// Warm-start network for TGV2 (no counterpart in the reference): a 4-level
// U-Net (16/32/64/128 channels) that maps the sweep's winner-take-all depth,
// its matching confidence and the reference image to a prediction of the
// converged TGV2 primal (u, v).  Training and inference run on the kernels of
// this file.
//
// Activations are NHWC bf16 with channel counts that are multiples of 16.  A
// 3x3 convolution is an implicit GEMM on the 5th-generation tensor cores:
//   D[128 pixels][Cout] += A_tap[128 pixels][16 ch] * B_tap[Cout][16 ch]
// for every tap and 16-channel slice, one tcgen05.mma (kind::f16, BF16 in,
// FP32 accumulator in tensor memory) each.  A CTA owns an 8 x 16 pixel tile;
// its (8+2) x (16+2) input halo sits in shared memory as two planes of 8
// channels, 16 bytes per pixel, which is exactly the "no swizzle, K-major"
// operand layout (8 rows x 16 bytes per core matrix), so every tap's A operand
// is the same halo addressed from a different start: no im2col copy.  The
// weights of a slice are staged as [tap][8-ch plane][Cout][8].  Up to three
// stages form a ring: the copies of the next two slices overlap the MMAs of a
// slice, and an mbarrier signalled by tcgen05.commit says when a stage may be
// refilled.
// The epilogue reads the accumulator with tcgen05.ld (one pixel per thread),
// adds the bias, applies ReLU or the ReLU mask of the backward pass and
// stores bf16.
//
// The backward pass w.r.t. the input is the same kernel with the weights
// flipped and transposed.  The weight gradient is a second tensor-core kernel
// with K = pixels (and a per-tap reduction on the CUDA cores that it is tested
// against), the bias gradient a reduction over pixels.
#include <math.h>
#include <string.h>

#include <algorithm>
#include <vector>

#include "common.cuh"

namespace mvs {
namespace unet {

typedef uint16_t bf16;   // raw bits

constexpr int TW = 8, TH = 16;               // output tile (M = 128 pixels)
constexpr int HW_ = TW + 2, HH_ = TH + 2;     // halo
constexpr int HALO_PIX = HW_ * HH_;           // 180
constexpr int HALO_BYTES = 2 * HALO_PIX * 16; // two 8-channel planes
constexpr int CONV_THREADS = 128;
constexpr int kSmemSM = 228 * 1024, kSmemReserved = 1024;   // shared memory of an SM, and of it per CTA
// output tiles per CTA of the convolution at 16 and 32 output channels
constexpr int CONV_MT16 = 2, CONV_MT32 = 2;

// ---------------------------------------------------------------------------
// tcgen05 / mbarrier helpers (inline PTX, sm_100a)
// ---------------------------------------------------------------------------


// shared-memory matrix descriptor: no swizzle, K-major core matrices of 8 rows
// x 16 bytes; lbo = byte distance between the two 8-element K halves, sbo =
// byte distance between consecutive 8-row groups; version 1 (sm_100)
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo)
{
    return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

// instruction descriptor of kind::f16: D f32, A and B bf16, both K-major
__host__ __device__ constexpr uint32_t idesc_bf16(int M, int N)
{
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}


__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void tmem_alloc(uint32_t *dst, uint32_t ncols)
{
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst)),
                 "r"(ncols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols)
{
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

__device__ __forceinline__ void mma_bf16(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accum)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(a), "l"(b), "r"(idesc), "r"(accum)
        : "memory");
}

__device__ __forceinline__ void mma_commit(uint64_t *bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16])
{
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int k = 0; k < 16; ++k) v[k] = __uint_as_float(r[k]);
}

__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src, bool valid)
{
    // src-size 0 zero-fills the 16 bytes (padding outside the image)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(valid ? 16 : 0)
                 : "memory");
}
// untiled bulk copy (16-byte aligned, a multiple of 16 bytes), counted on `bar`
__device__ __forceinline__ void bulk_copy(uint32_t dst, const void *src, uint32_t bytes, uint64_t *bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait_group() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// a in the low half, both rounded to nearest even (NaN stays NaN)
__device__ __forceinline__ uint32_t pack_bf16x2(float a, float b)
{
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(b), "f"(a));
    return r;
}

// ---------------------------------------------------------------------------
// 3x3 convolution, zero padding, on tensor cores
// ---------------------------------------------------------------------------

// An activation tensor of `channels` channels at H x W: one tensor [B][H][W][channels],
// or (up > 0) the concatenation that a decoder level reads, never stored: the
// first `up` channels are the next coarser level's [B][H/2][W/2][up], nearest
// upsampled, the others `skip` [B][H][W][channels - up].  H and W are even there.
struct Act {
    const bf16 *p, *skip;
    int channels, up;
};

// Where 16 channels of an Act lie, from channel `c` on (a multiple of 16; `up`
// is one too): base pointer, channels per pixel, and 1 for the coarser level.
struct Source {
    const bf16 *p;
    int pitch, half;
};
__device__ __forceinline__ Source act_source(const Act &a, int c)
{
    if (a.up == 0) return Source{a.p + c, a.channels, 0};
    if (c < a.up) return Source{a.p + c, a.up, 1};
    return Source{a.skip + (c - a.up), a.channels - a.up, 0};
}
// Offset (in elements) of pixel (y + dy, x + dx) from pixel (y, x) of image b, y and
// x even, and of that pixel itself.
__device__ __forceinline__ int source_delta(const Source &s, int W, int dy, int dx)
{
    return ((dy >> s.half) * (W >> s.half) + (dx >> s.half)) * s.pitch;
}
__device__ __forceinline__ size_t source_at(const Source &s, int H, int W, int b, int y, int x)
{
    return (((size_t)b * (H >> s.half) + (y >> s.half)) * (W >> s.half) + (x >> s.half)) * s.pitch;
}

struct Norm {
    float depth_scale, depth_shift;   // channel 0 = depth * scale + shift
    float cost_clip;                  // channel 1 = 1 - min(cost, clip)
    float u_scale, v_scale;           // u = wta + u_scale * out0, v = v_scale * out{1,2}
    float w_u, w_v;                   // loss weights of (u - u*)^2 and |v - v*|^2
};

// The 1x1 head on the last activation (16 channels), formed in that
// convolution's epilogue; u null: no head.
struct Head {
    const float *w, *b, *wta;   // [3][16], [3], [B][H][W]
    float *u, *v;               // [B][H][W], [B][2][H][W]
    Norm nm;
};

struct ConvArgs {
    Act in;             // cin channels
    const bf16 *wpack;  // [9][cin/8][COUT][8]
    const float *bias;  // [COUT] or null
    Act mask;           // COUT channels, or p null; out *= (mask > 0)
    bf16 *out;          // [B][H][W][COUT]
    int *err;           // set to 1 when a bounded wait gives up
    int H, W, cin, relu, tiles_x;
    Head head;
};

constexpr uint64_t kWaitNs = 1000000000ull;   // 1 s

#define MVS_RC_(x)                \
    do {                          \
        int rc__ = (x);           \
        if (rc__) return rc__;    \
    } while (0)

// MT output tiles of 8 x 16 pixels stacked vertically per CTA: they share
// one (MT * 16 + 2)-row halo and one copy of the weights, and accumulate in
// MT column blocks of COUT in tensor memory.
template <int COUT, int MT = 1>
struct ConvSmem {
    static constexpr int HALO_ROWS = MT * TH + 2;
    static constexpr int HPIX = HW_ * HALO_ROWS;          // halo pixels
    static constexpr int HBYTES = 2 * HPIX * 16;          // two 8-channel planes
    static constexpr int W_BYTES = 9 * 2 * COUT * 16;
    static constexpr int STAGE = (HBYTES + W_BYTES + 127) / 128 * 128;
    static constexpr int bytes(int stages) { return stages * STAGE + 64 + COUT * (int)sizeof(float); }
    static constexpr int TMEM_COLS = MT * COUT <= 32 ? 32 : MT * COUT <= 64 ? 64 : MT * COUT <= 128 ? 128 : 256;
};

// CTAs per SM that the registers are bounded for, by stages of the ring.
constexpr int conv_min_ctas(int stages) { return stages == 1 ? 12 : stages == 2 ? 6 : 4; }

// NST: stages of the ring, at most the number of 16-channel slices.
template <int COUT, int MT, int NST>
__global__ void __launch_bounds__(CONV_THREADS, conv_min_ctas(NST)) conv3x3_tc_kernel(ConvArgs a)
{
    using S = ConvSmem<COUT, MT>;
    extern __shared__ __align__(128) unsigned char smem[];
    const int H = a.H, W = a.W, cin = a.cin;
    const int nslices = cin >> 4;
    uint64_t *bars = (uint64_t *)(smem + NST * S::STAGE);   // the MMAs that read a stage are done
    uint64_t *wbars = bars + NST;                           // a stage's weights have landed
    uint32_t *tmem_slot = (uint32_t *)(bars + 2 * NST);
    float *sbias = (float *)(smem + NST * S::STAGE + 64);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int b = blockIdx.y;
    const int tx = blockIdx.x % a.tiles_x, ty = blockIdx.x / a.tiles_x;
    const int x0 = tx * TW, y0 = ty * (MT * TH);
    const size_t img = (size_t)H * W;
    const uint32_t sbase = smem_u32(smem);

    // Each thread's halo copies are the same for every slice: 16-byte halves
    // tid, tid + 128, ... of the halo pixels.
    constexpr int HI = (2 * S::HPIX + CONV_THREADS - 1) / CONV_THREADS;
    const bool inner = y0 > 0 && x0 > 0 && y0 + MT * TH < H && x0 + TW < W;   // the halo lies inside the image
    // stage slice c in stage c % NST: halo pixels (2 x 16 B) by cp.async (one
    // commit group), the 9 taps' weights by bulk copies (contiguous per tap)
    // that signal the stage's wbar
    auto load = [&](int c) {
        const int s = c % NST;
        const uint32_t hb = sbase + s * S::STAGE, wb = hb + S::HBYTES;
        const Source sr = act_source(a.in, 16 * c);
        const bf16 *src0 = sr.p + source_at(sr, H, W, b, y0, x0) + 8 * (tid & 1);
#pragma unroll
        for (int i = 0; i < HI; ++i) {
            const int k = tid + i * CONV_THREADS;
            if (k >= 2 * S::HPIX) break;
            const int pix = k >> 1, half = k & 1;
            const int hy = pix / HW_ - 1, hx = pix - (hy + 1) * HW_ - 1;
            const bool ok = inner || (y0 + hy >= 0 && y0 + hy < H && x0 + hx >= 0 && x0 + hx < W);
            cp_async16(hb + (half * S::HPIX + pix) * 16, ok ? src0 + source_delta(sr, W, hy, hx) : a.in.p, ok);
        }
        cp_async_commit();
        if (warp == 1) {
            constexpr uint32_t WB = 2 * COUT * 16;   // bytes per tap
            if (lane == 0)
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(&wbars[s])),
                             "r"(9 * WB)
                             : "memory");
            __syncwarp();
            if (lane < 9)
                bulk_copy(wb + lane * WB, a.wpack + ((size_t)(lane * (cin >> 3) + 2 * c) * COUT) * 8, WB, &wbars[s]);
        }
    };

    if (warp == 0) tmem_alloc(tmem_slot, S::TMEM_COLS);
    if (tid == 32) {
        for (int k = 0; k < NST; ++k) mbar_init(&wbars[k], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) __syncwarp();
    if (tid == 0) {
        for (int k = 0; k < NST; ++k) mbar_init(&bars[k], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    constexpr int AHEAD = NST > 1 ? NST - 1 : 1;   // slices in flight before the first MMAs
    // dependent launch: the previous kernels are complete.  (The next grid is let
    // in only here, once this CTA holds its tensor memory: CTAs that wait must not
    // take it from CTAs that run.)
    __syncthreads();
    wait_for_previous_grid();
    allow_next_grid();
#pragma unroll
    for (int k = 0; k < AHEAD; ++k) load(k);
    if (a.bias && tid < COUT) sbias[tid] = a.bias[tid];
    if (COUT > CONV_THREADS && a.bias && tid + CONV_THREADS < COUT) sbias[tid + CONV_THREADS] = a.bias[tid + CONV_THREADS];
    tc_fence_before();

    constexpr uint32_t idesc = idesc_bf16(128, COUT);
    bool failed = false;
    int last = -1;   // the last slice whose MMAs were due (the same in every thread)
    for (int c = 0; c < nslices; ++c) {
        cp_async_wait_group<AHEAD - 1>();   // slice c's halo landed
        fence_async_smem();
        failed = __syncthreads_or(failed) != 0;   // (the first one also publishes barriers, tensor memory and bias)
        if (failed) break;
        const int s = c % NST;
        // (a weight copy that never lands leaves the MMAs out: the waits on
        // bars[s] below then give up)
        if (tid == 0 && mbar_wait_bounded(&wbars[s], (uint32_t)((c / NST) & 1), kWaitNs)) {
            tc_fence_after();
            const uint32_t tmem = *tmem_slot;
            // descriptors differ only in their start address (16-byte units)
            const uint32_t hb = sbase + s * S::STAGE, wb = hb + S::HBYTES;
            const uint64_t ad = smem_desc(hb, S::HPIX * 16, HW_ * 16), bd = smem_desc(wb, COUT * 16, 128);
#pragma unroll
            for (int t = 0; t < 9; ++t) {
                const int ky = t / 3, kx = t - 3 * ky;
#pragma unroll
                for (int mt = 0; mt < MT; ++mt)
                    mma_bf16(tmem + (uint32_t)(mt * COUT), ad + (mt * TH + ky) * HW_ + kx, bd + t * 2 * COUT, idesc,
                             (c > 0 || t > 0) ? 1u : 0u);
            }
            mma_commit(&bars[s]);
        }
        last = c;
        if (NST > 1 && c + AHEAD < nslices) {
            // stage (c - 1) % NST takes slice c + NST - 1 once slice c - 1's MMAs have read it
            failed = c >= 1 && !mbar_wait_bounded(&bars[(c - 1) % NST], (uint32_t)(((c - 1) / NST) & 1), kWaitNs);
            if (!failed) load(c + AHEAD);
        } else {
            cp_async_commit();   // empty groups keep the group count per slice fixed
        }
    }
    // one thread waits for the last MMAs, the others at the barrier (a wait of
    // all of them took issue slots from the CTAs that share the SM)
    if (tid == 0 && !failed) failed = !mbar_wait_bounded(&bars[last % NST], (uint32_t)((last / NST) & 1), kWaitNs);
    failed = __syncthreads_or(failed) != 0;
    const uint32_t tmem = *tmem_slot;
    if (failed) {
        if (tid == 0) atomicExch(a.err, 1);
        // give the tensor core and the copies a second bounded chance to finish
        // before the accumulator columns are released
        cp_async_wait_all();
        if (last >= 0) mbar_wait_bounded(&bars[last % NST], (uint32_t)((last / NST) & 1), kWaitNs);
        if (tid == 32)
            for (int c = max(0, last); c < min(nslices, last + NST); ++c)
                mbar_wait_bounded(&wbars[c % NST], (uint32_t)((c / NST) & 1), kWaitNs);
        tc_fence_before();
        __syncthreads();
        if (warp == 0) {
            tc_fence_after();
            tmem_dealloc(tmem, S::TMEM_COLS);
        }
        return;
    }
    tc_fence_after();

    // epilogue: thread = accumulator row = pixel (of each of the MT tiles)
    const int m = warp * 32 + lane;
#pragma unroll 1
    for (int mt = 0; mt < MT; ++mt) {
    const int py = y0 + mt * TH + (m >> 3), px = x0 + (m & 7);
    const bool inside = py < H && px < W;
    const size_t pidx = (size_t)b * img + (size_t)min(py, H - 1) * W + min(px, W - 1);
#pragma unroll 1
    for (int c0 = 0; c0 < COUT; c0 += 16) {
        float v[16];
        tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(mt * COUT + c0), v);
        if (a.bias) {
#pragma unroll
            for (int k = 0; k < 16; ++k) v[k] += sbias[c0 + k];
        }
        if (a.relu) {
#pragma unroll
            for (int k = 0; k < 16; ++k) v[k] = fmaxf(v[k], 0.f);
        }
        if (a.mask.p && inside) {
            const Source sm = act_source(a.mask, c0);
            const uint4 *mp = (const uint4 *)(sm.p + source_at(sm, H, W, b, py, px));
            const uint4 m0 = mp[0], m1 = mp[1];
            const uint32_t mw[8] = {m0.x, m0.y, m0.z, m0.w, m1.x, m1.y, m1.z, m1.w};
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                if (!(bf2f((uint16_t)(mw[k] & 0xffffu)) > 0.f)) v[2 * k] = 0.f;
                if (!(bf2f((uint16_t)(mw[k] >> 16)) > 0.f)) v[2 * k + 1] = 0.f;
            }
        }
        if (inside) {
            uint4 *op = (uint4 *)(a.out + pidx * COUT + c0);
            const uint4 o0 = make_uint4(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]), pack_bf16x2(v[4], v[5]),
                                        pack_bf16x2(v[6], v[7]));
            const uint4 o1 = make_uint4(pack_bf16x2(v[8], v[9]), pack_bf16x2(v[10], v[11]), pack_bf16x2(v[12], v[13]),
                                        pack_bf16x2(v[14], v[15]));
            op[0] = o0;
            op[1] = o1;
            if (COUT == 16 && a.head.u) {
                // the head reads the stored (rounded) activation
                const uint32_t ow[8] = {o0.x, o0.y, o0.z, o0.w, o1.x, o1.y, o1.z, o1.w};
                float o[3];
#pragma unroll
                for (int k = 0; k < 3; ++k) o[k] = __ldg(a.head.b + k);
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const float lo = bf2f((uint16_t)(ow[j] & 0xffffu)), hi = bf2f((uint16_t)(ow[j] >> 16));
#pragma unroll
                    for (int k = 0; k < 3; ++k) {
                        o[k] = fmaf(__ldg(a.head.w + 16 * k + 2 * j), lo, o[k]);
                        o[k] = fmaf(__ldg(a.head.w + 16 * k + 2 * j + 1), hi, o[k]);
                    }
                }
                float dw = __ldg(a.head.wta + pidx);
                if (!(dw == dw)) dw = 0.f;
                a.head.u[pidx] = dw + a.head.nm.u_scale * o[0];
                float *vv = a.head.v + pidx + (size_t)b * img;   // [b][2][H][W]
                vv[0] = a.head.nm.v_scale * o[1];
                vv[img] = a.head.nm.v_scale * o[2];
            }
        }
    }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(tmem, S::TMEM_COLS);
    }
}

template <int COUT, int MT, int NST>
int launch_conv_n(const ConvArgs &a, int B, cudaStream_t st)
{
    using S = ConvSmem<COUT, MT>;
    auto kernel = conv3x3_tc_kernel<COUT, MT, NST>;
    MVS_TRY_CUDA(allow_shared_memory(kernel, S::bytes(NST)));
    MVS_TRY_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                                      (int)cudaSharedmemCarveoutMaxShared));
    const int tiles = a.tiles_x * ceil_div(a.H, MT * TH);
    MVS_TRY_CUDA(launch_dependent(kernel, dim3(tiles, B), dim3(CONV_THREADS), S::bytes(NST), st, a));
    return MVS_OK;
}

// Stages of the ring: at most the 16-channel slices, two or three.  A third stage
// hides more of a slice's copies, but leaves fewer CTAs per SM, and those hide them
// too: it is taken only where the grid needs no more waves for it.  Batch 4, with the
// weight pack, three and two stages (B200): 48->16 at 640x480 76 and 66 us, 128->128
// at 320x240 171 and 123 us, 96->32 43 and 40 us, 128->128 at 80x60 (160 CTAs, one or
// two per SM) 22 and 16 us; with equal waves 192->64 at 160x120 34 and 39 us, 64->64
// at 320x240, batch 2, 26.0 and 26.8 us.  One slice, 16->16 at 640x480: 37 us.
template <int COUT, int MT, int NST>
int conv_waves(long long ctas)
{
    using S = ConvSmem<COUT, MT>;
    const int per_sm = std::min({kSmemSM / (S::bytes(NST) + kSmemReserved), 512 / S::TMEM_COLS, conv_min_ctas(NST)});
    return (int)((ctas + kSMs * per_sm - 1) / (kSMs * per_sm));
}

template <int COUT, int MT = 1>
int launch_conv_t(const ConvArgs &a, int B, cudaStream_t st)
{
    static_assert(ConvSmem<COUT, MT>::bytes(3) <= kSmemMax, "three stages fit a CTA");
    const long long ctas = (long long)a.tiles_x * ceil_div(a.H, MT * TH) * B;
    if (a.cin <= 16) return launch_conv_n<COUT, MT, 1>(a, B, st);
    if (a.cin <= 32 || conv_waves<COUT, MT, 3>(ctas) > conv_waves<COUT, MT, 2>(ctas))
        return launch_conv_n<COUT, MT, 2>(a, B, st);
    return launch_conv_n<COUT, MT, 3>(a, B, st);
}

int launch_conv(const Act &in, const bf16 *wpack, const float *bias, const Act &mask, bf16 *out, int cout, int B, int H,
                int W, int relu, int *err, cudaStream_t st, const Head &head = Head{})
{
    const int cin = in.channels;
    if (cin <= 0 || cin % 16 || cin > 512) return set_error(MVS_ERR_ARG, "conv input channels %d (multiple of 16)", cin);
    ConvArgs a{in, wpack, bias, mask, out, err, H, W, cin, relu, ceil_div(W, TW), head};
    switch (cout) {
    case 16: return launch_conv_t<16, CONV_MT16>(a, B, st);
    case 32: return launch_conv_t<32, CONV_MT32>(a, B, st);
    case 48: return launch_conv_t<48>(a, B, st);
    case 64: return launch_conv_t<64>(a, B, st);
    case 96: return launch_conv_t<96>(a, B, st);
    case 128: return launch_conv_t<128>(a, B, st);
    case 192: return launch_conv_t<192>(a, B, st);
    default: return set_error(MVS_ERR_ARG, "conv output channels %d not built (16/32/48/64/96/128/192)", cout);
    }
}

// ---------------------------------------------------------------------------
// weight gradient on tensor cores: for every tap (ky, kx),
//   D[co][kx][ky][ci] += sum_p dz[p][co] * x[p + (ky, kx)][ci]
// with K = pixels, for chunks of NC = 16, 32 or 48 input channels (G = NC / 8
// groups).  A = dz^T (M = 64 or 128 output channels) is MN-major, [co / 8][pixel][8].
// B is the tile's input halo itself, stored so that one descriptor reaches three
// taps: rows of 10 pixels x 16 bytes ordered [halo row][8-channel group], so the
// (ky, group) neighbour of a core matrix (8 pixels of a tile row x 8 channels) lies
// 160 bytes further for each step of G ky + group, the next tile row 160 G bytes
// further, and tap kx starts 16 kx bytes later.  A K-step of 16 pixels (two tile
// rows) is then three MMAs with N = 3 ky x NC channels, straight from the bytes
// that cp.async brought: nothing is expanded or copied in shared memory.
// ---------------------------------------------------------------------------

struct WgArgs {
    Act x;            // cin channels
    const bf16 *dz;   // [B][H][W][cout]
    float *dW;        // [cout][cin][9]
    int *err;
    int B, H, W, cin, cout, tiles_x, tiles_y, tiles_per_cta, n_tiles;
    int vec;          // dW is 16-byte aligned
};

constexpr int WG_COPY = 256, WG_TC_THREADS = WG_COPY + 32;   // eight copying warps and one that issues the MMAs
constexpr int WG_NC = 16;                                      // input channels of a chunk, or 2 or 3 times as many
constexpr int WG_HALO_W = TW + 2, WG_HALO_H = TH + 2;          // 10 x 18 input pixels around an 8 x 16 tile
constexpr int WG_HALO_BYTES = 2 * WG_HALO_H * WG_HALO_W * 16;  // 5760 per 16 channels
constexpr int WG_MAX_STAGES = 8;
// tiles a CTA sums at least: each adds its 9 x 16 x cout sums to dW atomically
constexpr int WG_MIN_TILES = 8;

// Shared memory for `cg` groups of 8 output channels: `stages` x (dz tile [cg]
// [128 pixels][16 B], input halo), then room for what an A descriptor of M rows
// spans past the last stage's groups.  (The groups past cg read other bytes of
// the ring and only fill accumulator rows co >= cout, which are never stored.)
struct WgLayout {
    int a_bytes, stage_bytes, bytes;
};

__host__ __device__ inline WgLayout wg_layout(int m, int stages, int cg, int nc)
{
    WgLayout L;
    L.a_bytes = cg * 128 * 16;
    L.stage_bytes = L.a_bytes + nc / WG_NC * WG_HALO_BYTES;
    L.bytes = stages * L.stage_bytes + (m / 8) * 128 * 16 + 128;
    return L;
}

// MN-major descriptors have the instruction descriptor's transpose bits set
__host__ __device__ constexpr uint32_t idesc_bf16_mn(int M, int N) { return idesc_bf16(M, N) | (1u << 15) | (1u << 16); }

__device__ __forceinline__ void tmem_ld4(uint32_t taddr, float (&v)[4])
{
    uint32_t r[4];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(taddr)
                 : "memory");
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = __uint_as_float(r[k]);
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

__device__ __forceinline__ void red_add4(float *dst, float a, float b, float c, float d)
{
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}

// A CTA sums a run of 8 x 16 tiles for one chunk of NC input channels
// (blockIdx.y) and one block of M output channels (blockIdx.z) in tensor memory:
// a ring of R stages is filled by cp.async R - 1 tiles ahead, one thread issues
// the 24 MMAs of a tile, and tcgen05.commit on the stage's mbarrier frees it.
// Every wait is bounded.  M = 64 keeps rows 16 q .. 16 q + 15 of the accumulator
// in lanes 32 q .. 32 q + 15.
//
// What bounds it: shared-memory reads of the MMAs (24 per tile and chunk, each 2 KB
// of dz at M = 64, of which 16 output channels use a quarter, and 0.1 KB per input
// channel; 48 input channels take 115 cycles an MMA, 16 take 65) and, on the inner
// levels, the latency of few tiles per CTA.
template <int M, int R, int NC>
__global__ void __launch_bounds__(WG_TC_THREADS) wgrad_tc_kernel(WgArgs a)
{
    static_assert(R >= 2 && R <= WG_MAX_STAGES, "at least two stages");
    constexpr int SUB = NC / WG_NC, G = NC / 8;   // 16-channel parts, 8-channel groups
    constexpr int N = 3 * NC;                     // columns of one MMA: (ky, channel)
    constexpr int TMEM_COLS = 3 * N <= 256 ? 256 : 512;
    extern __shared__ __align__(128) unsigned char smem[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int ci0 = blockIdx.y * NC, co0 = blockIdx.z * M;
    const int cg = min(a.cout - co0, M) >> 3;
    const WgLayout L = wg_layout(M, R, cg, NC);
    uint64_t *bars = (uint64_t *)(smem + L.bytes - 128);
    uint32_t *tmem_slot = (uint32_t *)(smem + L.bytes - 128 + 8 * WG_MAX_STAGES);
    const int t_begin = blockIdx.x * a.tiles_per_cta;
    const int t_end = min(t_begin + a.tiles_per_cta, a.n_tiles);
    const int H = a.H, W = a.W, cin = a.cin, cout = a.cout;
    const size_t img = (size_t)H * W;

    if (warp == 0) tmem_alloc(tmem_slot, TMEM_COLS);
    if (tid == 0) {
        for (int k = 0; k < R; ++k) mbar_init(&bars[k], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    // dependent launch: the previous kernels are complete.  (The next grid is let
    // in only here, once this CTA holds its tensor memory, as in the convolution.)
    wait_for_previous_grid();
    allow_next_grid();
    const uint32_t tmem = *tmem_slot;
    const uint32_t sbase = smem_u32(smem);

    // Each copying thread's copies are the same for every tile: dz pixel
    // (tid & 127) of the groups tid >> 7, + 2, ...; halo items tid, tid + 256
    // (halo pixel, then channel group), worked out once here.
    constexpr int HALO_ITEMS = 2 * WG_HALO_H * WG_HALO_W;
    constexpr int HI = (HALO_ITEMS + WG_COPY - 1) / WG_COPY;
    const bool copies = tid < WG_COPY;
    const int dz_m = tid & 127, dz_y = dz_m >> 3, dz_x = dz_m & 7, dz_g0 = tid >> 7;
    int h_y[HI], h_x[HI], h_dst[HI];
#pragma unroll
    for (int i = 0; i < HI; ++i) {
        const int k = tid + i * WG_COPY;
        const int pix = k >> 1, g = k & 1, y = pix / WG_HALO_W, x = pix - y * WG_HALO_W;
        h_y[i] = y - 1;
        h_x[i] = x - 1;
        h_dst[i] = k < HALO_ITEMS ? ((y * G + g) * WG_HALO_W + x) * 16 : -1;
    }
    Source sx[SUB];
    int h_off[SUB][HI];
#pragma unroll
    for (int q = 0; q < SUB; ++q) {
        sx[q] = act_source(a.x, ci0 + q * WG_NC);
        sx[q].p += 8 * (tid & 1);
#pragma unroll
        for (int i = 0; i < HI; ++i) h_off[q][i] = source_delta(sx[q], W, h_y[i], h_x[i]);
    }
    const int dz_off = (dz_y * W + dz_x) * cout;
    const bf16 *zg = a.dz + co0 + 8 * dz_g0;
    // the next tile to copy: image lb, tile row and column lty, ltx
    const int per_img = a.tiles_x * a.tiles_y;
    int lb = t_begin / per_img, lty = (t_begin - lb * per_img) / a.tiles_x,
        ltx = t_begin - lb * per_img - lty * a.tiles_x;
    // cp.async of the next tile's dz and input halo into stage s (one commit group)
    auto load = [&](int s) {
        const int y0 = lty * TH, x0 = ltx * TW;
        const uint32_t ab = sbase + s * L.stage_bytes, hb = ab + L.a_bytes;
        const size_t pb = (size_t)lb * img + (size_t)y0 * W + x0;
        const bf16 *zt = zg + pb * cout + dz_off;
        uint32_t zd = ab + (dz_g0 * 128 + dz_m) * 16;
        if (y0 > 0 && x0 > 0 && y0 + TH < H && x0 + TW < W) {   // halo and all inside the image
            for (int g = dz_g0; g < cg; g += 2, zt += 16, zd += 2 * 128 * 16) cp_async16(zd, zt, true);
#pragma unroll
            for (int q = 0; q < SUB; ++q) {
                const bf16 *xt = sx[q].p + source_at(sx[q], H, W, lb, y0, x0);
#pragma unroll
                for (int i = 0; i < HI; ++i)
                    if (h_dst[i] >= 0) cp_async16(hb + h_dst[i] + q * 2 * WG_HALO_W * 16, xt + h_off[q][i], true);
            }
        } else {
            const bool ok = y0 + dz_y < H && x0 + dz_x < W;
            if (!ok) zt = a.dz;
            for (int g = dz_g0; g < cg; g += 2, zt += ok ? 16 : 0, zd += 2 * 128 * 16) cp_async16(zd, zt, ok);
#pragma unroll
            for (int q = 0; q < SUB; ++q) {
                const bf16 *xt = sx[q].p + source_at(sx[q], H, W, lb, y0, x0);
#pragma unroll
                for (int i = 0; i < HI; ++i) {
                    const int gy = y0 + h_y[i], gx = x0 + h_x[i];
                    const bool in = gy >= 0 && gy < H && gx >= 0 && gx < W;
                    if (h_dst[i] >= 0)
                        cp_async16(hb + h_dst[i] + q * 2 * WG_HALO_W * 16, in ? xt + h_off[q][i] : a.x.p, in);
                }
            }
        }
        cp_async_commit();
        if (++ltx == a.tiles_x) {
            ltx = 0;
            if (++lty == a.tiles_y) lty = 0, ++lb;
        }
    };

    constexpr uint32_t idesc = idesc_bf16_mn(M, N);
    const int n = t_end - t_begin;
    bool failed = false;
    int last = -1;   // the last tile whose MMAs were issued (the same in every thread)
    for (int k = 0; k < R - 1; ++k) {
        if (k < n && copies) load(k);
        else cp_async_commit();   // empty groups keep the group count per tile fixed
    }
    // tile c's MMAs read stage c % R and signal bars[c % R]: that barrier's
    // (c / R)-th completion, of parity (c / R) & 1
    for (int c = 0; c < n; ++c) {
        cp_async_wait_group<R - 2>();   // tile c's group landed (R - 2 newer ones may be in flight)
        fence_async_smem();             // visible to the MMAs
        failed = __syncthreads_or(failed) != 0;
        if (failed) break;
        if (tid == WG_COPY) {
            tc_fence_after();
            // descriptors differ only in their start address (16-byte units)
            const uint32_t ab = sbase + (c % R) * L.stage_bytes, hb = ab + L.a_bytes;
            const uint64_t ad = smem_desc(ab, 128, 128 * 16), bd = smem_desc(hb, G * WG_HALO_W * 16, WG_HALO_W * 16);
#pragma unroll
            for (int ks = 0; ks < 8; ++ks)
#pragma unroll
                for (int kx = 0; kx < 3; ++kx)
                    mma_bf16(tmem + kx * N, ad + 16 * ks, bd + 2 * G * ks * WG_HALO_W + kx, idesc,
                             (c > 0 || ks > 0) ? 1u : 0u);
            mma_commit(&bars[c % R]);
        }
        last = c;
        if (c + R - 1 < n && copies) {
            // stage (c - 1) % R takes tile c + R - 1 once tile c - 1's MMAs have read it
            failed = c >= 1 && !mbar_wait_bounded(&bars[(c - 1) % R], (uint32_t)(((c - 1) / R) & 1), kWaitNs);
            if (!failed) load((c + R - 1) % R);
        } else {
            cp_async_commit();
        }
    }
    failed = __syncthreads_or(failed) != 0;
    if (!failed && last >= 0) {
        const bool ok = mbar_wait_bounded(&bars[last % R], (uint32_t)((last / R) & 1), kWaitNs);
        failed = __syncthreads_or(!ok) != 0;
    }
    cp_async_wait_group<0>();
    if (failed) {
        if (tid == 0) atomicExch(a.err, 1);
        if (last >= 0)   // the MMAs in flight (they complete in order)
            mbar_wait_bounded(&bars[last % R], (uint32_t)((last / R) & 1), kWaitNs);
        tc_fence_before();
        __syncthreads();
        if (warp == 0) {
            tc_fence_after();
            tmem_dealloc(tmem, TMEM_COLS);
        }
        return;
    }
    tc_fence_after();
    if (n > 0) {
        // D[co][kx][ky][ci]; warps w and w + 4 read lanes 32 (w % 4) .. + 31, the
        // even and the odd groups of four channels: 36 consecutive values of dW
        const int quarter = warp & 3;
        const int row = M == 128 ? quarter * 32 + lane : quarter * 16 + lane;
        const bool own = (M == 128 || lane < 16) && co0 + row < cout;
        float *dst = a.dW + ((size_t)(co0 + row) * cin + ci0) * 9;
#pragma unroll 1
        for (int cq = warp >> 2; cq < NC / 4 && copies; cq += 2) {
            float v[9][4];
#pragma unroll
            for (int t = 0; t < 9; ++t)
                tmem_ld4(tmem + ((uint32_t)(quarter * 32) << 16) + (t % 3) * N + (t / 3) * NC + 4 * cq, v[t]);
            tmem_ld_wait();
            if (!own) continue;
            if (a.vec) {
#pragma unroll
                for (int k = 0; k < 9; ++k)   // value 4k + e is channel (4k + e) / 9, tap (4k + e) % 9
                    red_add4(dst + 36 * cq + 4 * k, v[(4 * k) % 9][(4 * k) / 9], v[(4 * k + 1) % 9][(4 * k + 1) / 9],
                             v[(4 * k + 2) % 9][(4 * k + 2) / 9], v[(4 * k + 3) % 9][(4 * k + 3) / 9]);
            } else {
#pragma unroll
                for (int k = 0; k < 36; ++k) atomicAdd(dst + 36 * cq + k, v[k % 9][k / 9]);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(tmem, TMEM_COLS);
    }
}

// One launch in one wave: the CTAs of every (chunk, output block) split the tiles
// evenly (a last wave of a few CTAs would cost a whole run of tiles), with at
// least WG_MIN_TILES each.
template <int M, int R, int NC>
int launch_wgrad_tc_t(WgArgs a, cudaStream_t st)
{
    const WgLayout L = wg_layout(M, R, std::min(a.cout, M) >> 3, NC);
    const int chunks = a.cin / NC, coblocks = ceil_div(a.cout, M);
    const int xctas = std::max(1, (NC == WG_NC ? 2 : 1) * kSMs / (chunks * coblocks));
    a.tiles_per_cta = std::max(ceil_div(a.n_tiles, xctas), WG_MIN_TILES);
    auto kernel = wgrad_tc_kernel<M, R, NC>;
    // (one kernel serves several counts of output channels, whose rings differ in size)
    MVS_TRY_CUDA(allow_shared_memory(kernel, kSmemMax));
    MVS_TRY_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                                      (int)cudaSharedmemCarveoutMaxShared));
    MVS_TRY_CUDA(launch_dependent(kernel, dim3(ceil_div(a.n_tiles, a.tiles_per_cta), chunks, coblocks),
                                  dim3(WG_TC_THREADS), L.bytes, st, a));
    return MVS_OK;
}

// The deepest ring of which two CTAs (one with wide chunks, whose sums take all of
// the tensor memory) fit an SM.
template <int M, int NC>
int launch_wgrad_tc_m(const WgArgs &a, cudaStream_t st)
{
    const int room = (NC == WG_NC ? kSmemSM / 2 : kSmemSM) - kSmemReserved;
    int r = WG_MAX_STAGES;
    while (r > 2 && wg_layout(M, r, std::min(a.cout, M) >> 3, NC).bytes > room) --r;
    switch (r) {
    case 8: return launch_wgrad_tc_t<M, 8, NC>(a, st);
    case 7: return launch_wgrad_tc_t<M, 7, NC>(a, st);
    case 6: return launch_wgrad_tc_t<M, 6, NC>(a, st);
    case 5: return launch_wgrad_tc_t<M, 5, NC>(a, st);
    case 4: return launch_wgrad_tc_t<M, 4, NC>(a, st);
    case 3: return launch_wgrad_tc_t<M, 3, NC>(a, st);
    default: return launch_wgrad_tc_t<M, 2, NC>(a, st);
    }
}

int launch_wgrad_tc(const Act &x, const bf16 *dz, int cout, int B, int H, int W, float *dW, int *err, cudaStream_t st)
{
    const int cin = x.channels;
    if (cout % 8 || cin % WG_NC) return set_error(MVS_ERR_ARG, "wgrad: cin %d, cout %d", cin, cout);
    WgArgs a{x, dz, dW, err, B, H, W, cin, cout, ceil_div(W, TW), ceil_div(H, TH), 1, 0, ((uintptr_t)dW & 15) == 0};
    a.n_tiles = B * a.tiles_x * a.tiles_y;
    // Wide chunks read dz once for 48 or 32 input channels and issue a third or half of
    // the MMAs, but leave one CTA per SM: only where the runs of WG_MIN_TILES tiles
    // still make a CTA for every SM (4 x 640 x 480, 48 -> 16 channels: 130 us in chunks
    // of 16, 93 of 48; 32 -> 32: 34 and 31; a training step of it 2025 and 1937 us, of
    // 2 x 320 x 240 940 and 907; below that size the rule keeps 16 nearly everywhere).
    const int coblocks = cout <= 64 ? 1 : ceil_div(cout, 128);
    auto fills = [&](int nc) {
        return cin % nc == 0 && a.n_tiles / WG_MIN_TILES * (cin / nc) * coblocks >= kSMs;
    };
    const int nc = fills(3 * WG_NC) ? 3 * WG_NC : fills(2 * WG_NC) ? 2 * WG_NC : WG_NC;
    if (nc == 3 * WG_NC)
        return cout <= 64 ? launch_wgrad_tc_m<64, 3 * WG_NC>(a, st) : launch_wgrad_tc_m<128, 3 * WG_NC>(a, st);
    if (nc == 2 * WG_NC)
        return cout <= 64 ? launch_wgrad_tc_m<64, 2 * WG_NC>(a, st) : launch_wgrad_tc_m<128, 2 * WG_NC>(a, st);
    return cout <= 64 ? launch_wgrad_tc_m<64, WG_NC>(a, st) : launch_wgrad_tc_m<128, WG_NC>(a, st);
}

// ---------------------------------------------------------------------------
// weight gradient (CUDA cores, FP32): dW[co][ci][t] += sum_p x[p + off_t][ci] dz[p][co]
// (the reference formulation the tensor-core kernel is tested against)
// ---------------------------------------------------------------------------

constexpr int WG_THREADS = 256;

// Each thread owns a 4 (ci) x 4 (co) block of one tap; a CTA covers a
// TCI x TCO tile of one tap, G = 256 / ((TCI/4)(TCO/4)) thread groups split
// the CTA's pixels, and the groups' sums meet in shared memory before one
// atomic add per weight.
template <int TCI, int TCO>
__global__ void __launch_bounds__(WG_THREADS) wgrad_kernel(const bf16 *__restrict__ x, const bf16 *__restrict__ dz,
                                                           int B, int H, int W, int cin, int cout, int px_per_cta,
                                                           float *__restrict__ dW)
{
    constexpr int TPG = (TCI / 4) * (TCO / 4);   // threads per group
    constexpr int G = WG_THREADS / TPG;
    __shared__ float red[WG_THREADS][17];
    const int tid = threadIdx.x, g = tid / TPG, r = tid - g * TPG;
    const int ci4 = (r % (TCI / 4)) * 4, co4 = (r / (TCI / 4)) * 4;
    const int t = blockIdx.y, ky = t / 3, kx = t - 3 * ky;
    const int ntile_ci = cin / TCI;
    const int ci0 = (blockIdx.z % ntile_ci) * TCI + ci4, co0 = (blockIdx.z / ntile_ci) * TCO + co4;
    const long long npix = (long long)B * H * W;
    const long long p0 = (long long)blockIdx.x * px_per_cta;
    const long long p1 = min(p0 + px_per_cta, npix);
    float acc[4][4] = {};
    for (long long p = p0 + g; p < p1; p += G) {
        const int bb = (int)(p / ((long long)H * W));
        const int rem = (int)(p - (long long)bb * H * W);
        const int y = rem / W, xx = rem - y * W;
        const int sy = y + ky - 1, sx = xx + kx - 1;
        if (sy < 0 || sy >= H || sx < 0 || sx >= W) continue;
        const uint2 xv = *(const uint2 *)(x + (((size_t)bb * H + sy) * W + sx) * cin + ci0);
        const uint2 dv = *(const uint2 *)(dz + (size_t)p * cout + co0);
        const float xf[4] = {bf2f((uint16_t)(xv.x & 0xffffu)), bf2f((uint16_t)(xv.x >> 16)),
                             bf2f((uint16_t)(xv.y & 0xffffu)), bf2f((uint16_t)(xv.y >> 16))};
        const float df[4] = {bf2f((uint16_t)(dv.x & 0xffffu)), bf2f((uint16_t)(dv.x >> 16)),
                             bf2f((uint16_t)(dv.y & 0xffffu)), bf2f((uint16_t)(dv.y >> 16))};
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(xf[i], df[j], acc[i][j]);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) red[tid][4 * i + j] = acc[i][j];
    __syncthreads();
    if (g == 0) {
        for (int q = 1; q < G; ++q)
#pragma unroll
            for (int k = 0; k < 16; ++k) red[tid][k] += red[q * TPG + r][k];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) atomicAdd(&dW[((size_t)(co0 + j) * cin + ci0 + i) * 9 + t], red[tid][4 * i + j]);
    }
}

// bias gradient: db[co] += sum_p dz[p][co].  HBM-bound: a thread sums 16-byte
// groups of 8 channels of every `rows`-th pixel of its block's run, four loads
// in flight; runs are sized for four blocks per SM (at least 256 pixels).
// Against one channel per thread and 2048 pixels per block (cold caches, B200):
// 640x480 x 4, 16 channels, 22 -> 11 us; 80x60 x 4, 128 channels, which gave
// only 10 blocks, 134 -> 8 us.
__global__ void __launch_bounds__(256) bgrad_kernel(const bf16 *__restrict__ dz, long long npix, int cout,
                                                    int px_per_cta, float *__restrict__ db)
{
    wait_for_previous_grid();   // dependent launch
    allow_next_grid();
    __shared__ float red[256][9];   // 9: no bank conflicts
    const int tid = threadIdx.x, groups = cout >> 3;
    const long long p0 = (long long)blockIdx.x * px_per_cta, p1 = min(p0 + px_per_cta, npix);
    for (int g0 = 0; g0 < groups; g0 += 256) {   // one pass up to 2048 channels
        const int gn = min(groups - g0, 256), rows = 256 / gn;
        const int g = tid % gn, row = tid / gn;
        float s[8] = {};
        if (row < rows) {
            const uint4 *q = (const uint4 *)dz + g0 + g;
#pragma unroll 4
            for (long long p = p0 + row; p < p1; p += rows) {
                const uint4 v = __ldg(q + (size_t)p * groups);
                const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    s[2 * k] += bf2f((uint16_t)(w[k] & 0xffffu));
                    s[2 * k + 1] += bf2f((uint16_t)(w[k] >> 16));
                }
            }
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < 8; ++k) red[tid][k] = s[k];
        __syncthreads();
        for (int c = tid; c < 8 * gn; c += 256) {
            float t = 0.f;
            for (int r = 0; r < rows; ++r) t += red[r * gn + (c >> 3)][c & 7];
            atomicAdd(&db[8 * g0 + c], t);
        }
    }
}

int launch_wgrad_cuda_cores(const bf16 *x, int cin, const bf16 *dz, int cout, int B, int H, int W, float *dW,
                            cudaStream_t st);

// (the CUDA-core form takes one tensor only)
int launch_wgrad(const Act &x, const bf16 *dz, int cout, int B, int H, int W, float *dW, float *db, int *err,
                 cudaStream_t st, bool tensor_cores = true)
{
    const long long npix = (long long)B * H * W;
    if (tensor_cores) {
        MVS_RC_(launch_wgrad_tc(x, dz, cout, B, H, W, dW, err, st));
    } else {
        MVS_RC_(launch_wgrad_cuda_cores(x.p, x.channels, dz, cout, B, H, W, dW, st));
    }
    if (db) {
        const int px = (int)std::max<long long>(256, (npix + 4 * kSMs - 1) / (4 * kSMs));
        MVS_TRY_CUDA(launch_dependent(bgrad_kernel, dim3((unsigned)((npix + px - 1) / px)), dim3(256), 0, st, dz, npix,
                                      cout, px, db));
    }
    return MVS_OK;
}

int launch_wgrad_cuda_cores(const bf16 *x, int cin, const bf16 *dz, int cout, int B, int H, int W, float *dW,
                            cudaStream_t st)
{
    const long long npix = (long long)B * H * W;
    const int px = 4096;
    const int chunks = (int)((npix + px - 1) / px);
    const int tci = cin % 64 == 0 ? 64 : cin % 32 == 0 ? 32 : 16;
    const int tco = cout % 64 == 0 ? 64 : cout % 32 == 0 ? 32 : 16;
    const dim3 g(chunks, 9, (cin / tci) * (cout / tco));
#define MVS_WG(A, B_)                                                                              \
    if (tci == A && tco == B_) wgrad_kernel<A, B_><<<g, WG_THREADS, 0, st>>>(x, dz, B, H, W, cin, cout, px, dW); \
    else
    MVS_WG(16, 16) MVS_WG(16, 32) MVS_WG(16, 64) MVS_WG(32, 16) MVS_WG(32, 32) MVS_WG(32, 64) MVS_WG(64, 16)
    MVS_WG(64, 32) MVS_WG(64, 64) return set_error(MVS_ERR_ARG, "wgrad tile %dx%d", tci, tco);
#undef MVS_WG
    return MVS_OK;
}

// ---------------------------------------------------------------------------
// elementwise layers (8 channels = 16 bytes per thread)
// ---------------------------------------------------------------------------

__device__ __forceinline__ void unpack8(const uint4 &q, float (&f)[8])
{
    const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        f[2 * k] = bf2f((uint16_t)(w[k] & 0xffffu));
        f[2 * k + 1] = bf2f((uint16_t)(w[k] >> 16));
    }
}
__device__ __forceinline__ uint4 pack8(const float (&f)[8])
{
    return make_uint4(pack_bf16x2(f[0], f[1]), pack_bf16x2(f[2], f[3]), pack_bf16x2(f[4], f[5]),
                      pack_bf16x2(f[6], f[7]));
}

// The kernels below move 8 channels (16 bytes) per thread and are bound by memory.
// A thread's row (of all images: H is even, so row r of the half-size map lies on
// rows 2 r and 2 r + 1) comes from the block's y, its column and channel group from
// x: with one flat index three 64-bit divisions came before the first load
// (4 x 640 x 480: gradient into the first level 30.4 us, now 29.2, gradient of its
// upsampled half 21.0 and 19.8; all of a 640 x 480 prediction 172.5 and 170.6 us).
struct RowGrid {
    dim3 grid, block;
};
inline RowGrid row_grid(long long rows, int items)
{
    int bx = 32;
    while (bx < 256 && bx < items) bx *= 2;
    const int by = 256 / bx;
    return RowGrid{dim3((items + bx - 1) / bx, (unsigned)std::min<long long>((rows + by - 1) / by, 65535)), dim3(bx, by)};
}

// 2x2 average pool: out [B][H/2][W/2][C] (rows = B * H / 2, Wo = W / 2)
__global__ void __launch_bounds__(256) pool_kernel(const bf16 *__restrict__ in, int rows, int Wo, int C,
                                                   bf16 *__restrict__ out)
{
    wait_for_previous_grid();   // dependent launch
    allow_next_grid();
    const int k = blockIdx.x * blockDim.x + threadIdx.x, pitch = Wo * C;
    if (8 * k >= pitch) return;
    const unsigned x = (unsigned)(8 * k) / (unsigned)C;
    for (int r = blockIdx.y * blockDim.y + threadIdx.y; r < rows; r += gridDim.y * blockDim.y) {
        const bf16 *src = in + (size_t)r * 4 * pitch + 8 * k + (size_t)x * C;   // pixel 2 x of row 2 r
        uint4 q[4];
#pragma unroll
        for (int d = 0; d < 4; ++d) q[d] = *(const uint4 *)(src + (d >> 1) * 2 * pitch + (d & 1) * C);
        float s[8] = {}, f[8];
#pragma unroll
        for (int d = 0; d < 4; ++d) {
            unpack8(q[d], f);
#pragma unroll
            for (int j = 0; j < 8; ++j) s[j] += f[j];
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) s[j] *= 0.25f;
        *(uint4 *)(out + (size_t)r * pitch + 8 * k) = pack8(s);
    }
}

// gradient into an encoder output e (C channels, rows = B * H rows of W) from the
// pool that read it (dp, H/2 x W/2) and from the skip half of a concat gradient
// (dc with ctot channels, the skip starting at coff), masked by e > 0
__global__ void __launch_bounds__(256) pool_back_kernel(const bf16 *__restrict__ dp, const bf16 *__restrict__ dc,
                                                        int ctot, int coff, const bf16 *__restrict__ e, int rows,
                                                        int W, int C, bf16 *__restrict__ de)
{
    wait_for_previous_grid();   // dependent launch
    allow_next_grid();
    const int k = blockIdx.x * blockDim.x + threadIdx.x, pitch = W * C;
    if (8 * k >= pitch) return;
    const unsigned x = (unsigned)(8 * k) / (unsigned)C;
    const int c = 8 * k - (int)x * C;
    for (int r = blockIdx.y * blockDim.y + threadIdx.y; r < rows; r += gridDim.y * blockDim.y) {
        const size_t at = (size_t)r * pitch + 8 * k;
        const uint4 qg = *(const uint4 *)(dp + (size_t)(r >> 1) * (pitch >> 1) + (x >> 1) * C + c);
        const uint4 qe = *(const uint4 *)(e + at);
        float g[8], f[8], m[8];
        unpack8(qg, g);
#pragma unroll
        for (int j = 0; j < 8; ++j) g[j] *= 0.25f;
        if (dc) {
            unpack8(*(const uint4 *)(dc + ((size_t)r * W + x) * ctot + coff + c), f);
#pragma unroll
            for (int j = 0; j < 8; ++j) g[j] += f[j];
        }
        unpack8(qe, m);
#pragma unroll
        for (int j = 0; j < 8; ++j)
            if (!(m[j] > 0.f)) g[j] = 0.f;
        *(uint4 *)(de + at) = pack8(g);
    }
}

// gradient of the upsampled half: dprev[y][x] = sum of the 2x2 block of dc
// (already masked by the concat's ReLU mask, which is prev's); rows = B * H / 2 of Wp = W / 2
__global__ void __launch_bounds__(256) upcat_back_kernel(const bf16 *__restrict__ dc, int ctot, int rows, int Wp,
                                                         int cp, bf16 *__restrict__ dprev)
{
    wait_for_previous_grid();   // dependent launch
    allow_next_grid();
    const int k = blockIdx.x * blockDim.x + threadIdx.x, pitch = Wp * cp;
    if (8 * k >= pitch) return;
    const unsigned x = (unsigned)(8 * k) / (unsigned)cp;
    const int c = 8 * k - (int)x * cp;
    for (int r = blockIdx.y * blockDim.y + threadIdx.y; r < rows; r += gridDim.y * blockDim.y) {
        const bf16 *src = dc + ((size_t)r * 4 * Wp + 2 * x) * ctot + c;   // pixel 2 x of row 2 r
        uint4 q[4];
#pragma unroll
        for (int d = 0; d < 4; ++d) q[d] = *(const uint4 *)(src + ((size_t)(d >> 1) * 2 * Wp + (d & 1)) * ctot);
        float s[8] = {}, f[8];
#pragma unroll
        for (int d = 0; d < 4; ++d) {
            unpack8(q[d], f);
#pragma unroll
            for (int j = 0; j < 8; ++j) s[j] += f[j];
        }
        *(uint4 *)(dprev + (size_t)r * pitch + 8 * k) = pack8(s);
    }
}

// ---------------------------------------------------------------------------
// input features, prediction head and loss
// ---------------------------------------------------------------------------

__global__ void features_kernel(const float *__restrict__ wta, const float *__restrict__ cost,
                                const float *__restrict__ ref255, long long npix, Norm nm, bf16 *__restrict__ x0)
{
    wait_for_previous_grid();   // dependent launch
    allow_next_grid();
    for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < npix; p += (long long)gridDim.x * blockDim.x) {
        float d = wta[p];
        if (!(d == d)) d = 0.f;
        float c = cost ? cost[p] : 0.f;
        if (!(c == c)) c = nm.cost_clip;
        float f[8] = {d * nm.depth_scale + nm.depth_shift, 1.f - fminf(fmaxf(c, 0.f), nm.cost_clip),
                      ref255[p] * (1.f / 255.f) - 0.5f, 0.f, 0.f, 0.f, 0.f, 0.f};
        const float z[8] = {};
        uint4 *o = (uint4 *)(x0 + (size_t)p * 16);
        o[0] = pack8(f);
        o[1] = pack8(z);
    }
}

// loss = mean_p [w_u (u - u*)^2 + w_v |v - v*|^2] and its gradient down to
// the last decoder activation (masked by its ReLU), the head's weight and bias
// gradients; partial sums per block, one atomic add per quantity.  A thread takes
// 8 of a pixel's 16 channels (even lanes the first 8, and the loss and bias
// terms), which leaves registers for four blocks per SM: bound by memory latency,
// 4 x 640 x 480 pixels 46.3 us with whole pixels per thread, now 42.8 us.
__global__ void __launch_bounds__(256, 4) head_back_kernel(const bf16 *__restrict__ d, const float *__restrict__ Wh,
                                                           const float *__restrict__ u, const float *__restrict__ v,
                                                           const float *__restrict__ ut, const float *__restrict__ vt,
                                                           int B, long long img, Norm nm, bf16 *__restrict__ dz,
                                                           float *__restrict__ dWh, float *__restrict__ dbh,
                                                           double *__restrict__ loss)
{
    __shared__ float w[48];
    __shared__ float red[8][52];
    __shared__ double lred[8];
    if (threadIdx.x < 48) w[threadIdx.x] = Wh[threadIdx.x];
    __syncthreads();
    const int half = threadIdx.x & 1;
    float gw[24] = {}, gb[3] = {};
    double ls = 0.0;
    const long long npix = img * B;
    const float inv_n = 1.f / (float)npix;
    for (int b = blockIdx.y; b < B; b += gridDim.y) {
        const size_t p0 = (size_t)b * img;
        for (long long q = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 1; q < img;
             q += ((long long)gridDim.x * blockDim.x) >> 1) {
            const size_t p = p0 + q, iv0 = p0 + p, iv1 = iv0 + img;
            const uint4 qa = *(const uint4 *)(d + p * 16 + 8 * half);
            const float eu = u[p] - ut[p], ex = v[iv0] - vt[iv0], ey = v[iv1] - vt[iv1];
            const float go[3] = {2.f * nm.w_u * eu * nm.u_scale * inv_n, 2.f * nm.w_v * ex * nm.v_scale * inv_n,
                                 2.f * nm.w_v * ey * nm.v_scale * inv_n};
            if (half == 0) {
                ls += (double)nm.w_u * eu * eu + (double)nm.w_v * (ex * ex + ey * ey);
#pragma unroll
                for (int k = 0; k < 3; ++k) gb[k] += go[k];
            }
            float a[8], g[8];
            unpack8(qa, a);
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                const float *wc = w + 8 * half + c;
                const float s = go[0] * wc[0] + go[1] * wc[16] + go[2] * wc[32];
                g[c] = a[c] > 0.f ? s : 0.f;
#pragma unroll
                for (int k = 0; k < 3; ++k) gw[8 * k + c] = fmaf(go[k], a[c], gw[8 * k + c]);
            }
            *(uint4 *)(dz + p * 16 + 8 * half) = pack8(g);
        }
    }
    // block reduction of 48 + 3 floats (over the lanes of one parity) and the loss
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
    for (int k = 0; k < 27; ++k) {
        float s = k < 24 ? gw[k] : gb[k - 24];
        for (int o = 16; o > 1; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
        if (k < 24) {
            if (lane < 2) red[warp][(k >> 3) * 16 + 8 * half + (k & 7)] = s;
        } else if (lane == 0) {
            red[warp][24 + k] = s;
        }
    }
    for (int o = 16; o > 1; o >>= 1) ls += __shfl_down_sync(0xffffffffu, ls, o);
    if (lane == 0) lred[warp] = ls;
    __syncthreads();
    if (threadIdx.x < 51) {
        float s = 0.f;
        for (int q = 0; q < 8; ++q) s += red[q][threadIdx.x];
        atomicAdd(threadIdx.x < 48 ? &dWh[threadIdx.x] : &dbh[threadIdx.x - 48], s);
    }
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int q = 0; q < 8; ++q) s += lred[q];
        atomicAdd(loss, s / (double)npix);
    }
}

// ---------------------------------------------------------------------------
// parameters: FP32 master copy, Adam, bf16 packs for the tensor cores
// ---------------------------------------------------------------------------

__global__ void adam_kernel(float *__restrict__ w, const float *__restrict__ g, float *__restrict__ m,
                            float *__restrict__ v, long long n, float lr, float b1, float b2, float eps, float c1,
                            float c2)
{
    for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x) {
        const float gk = g[k];
        const float mk = b1 * m[k] + (1.f - b1) * gk;
        const float vk = b2 * v[k] + (1.f - b2) * gk * gk;
        m[k] = mk;
        v[k] = vk;
        w[k] -= lr * (mk / c1) / (sqrtf(vk / c2) + eps);
    }
}

// W [cout][cin][9] (FP32) -> forward pack [9][cin/8][cout][8] and the
// backward-data pack [9][cout/8][cin][8] of the flipped, transposed kernel;
// one grid row per layer.
struct PackLayer {
    const float *w;
    bf16 *fwd, *bwd;   // bwd may be null
    int cin, cout;
};
constexpr int PACK_LAYERS = 14;
struct PackArgs {
    PackLayer l[PACK_LAYERS];
};
__global__ void pack_kernel(PackArgs a)
{
    wait_for_previous_grid();   // dependent launch
    allow_next_grid();
    const PackLayer &L = a.l[blockIdx.y];
    const int cin = L.cin, cout = L.cout, n = 9 * cin * cout;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        const int t = k % 9, ci = (k / 9) % cin, co = k / (9 * cin);
        const uint16_t b = f2bf(L.w[k]);
        L.fwd[(((size_t)t * (cin >> 3) + (ci >> 3)) * cout + co) * 8 + (ci & 7)] = b;
        if (L.bwd) L.bwd[(((size_t)(8 - t) * (cout >> 3) + (co >> 3)) * cin + ci) * 8 + (co & 7)] = b;
    }
}

// the packs of one layer
int launch_pack(const float *w, int cin, int cout, bf16 *fwd, bf16 *bwd, cudaStream_t st)
{
    PackArgs p{};
    p.l[0] = PackLayer{w, fwd, bwd, cin, cout};
    MVS_TRY_CUDA(launch_dependent(pack_kernel, dim3(ceil_div(9 * cin * cout, 256)), dim3(256), 0, st, p));
    return MVS_OK;
}

}  // namespace unet
}  // namespace mvs

// ===========================================================================
// network driver
// ===========================================================================

namespace {

using namespace mvs;
using namespace mvs::unet;

struct ConvLayer {
    int cin, cout;
    size_t w_off, b_off;   // offsets into the FP32 parameter array
    bf16 *wf, *wb;         // packs
};

// layer indices
enum {
    E0A, E0B, E1A, E1B, E2A, E2B, E3A, E3B, D2A, D2B, D1A, D1B, D0A, D0B, NCONV
};

}  // namespace

struct mvs_unet {
    int B, H, W;
    Norm nm;
    ConvLayer L[NCONV];
    size_t n_params, head_w, head_b;
    float *params = nullptr, *grads = nullptr, *adam_m = nullptr, *adam_v = nullptr;
    bf16 *packs = nullptr;
    // activations (and their gradients, prefixed g)
    bf16 *x0, *e0a, *e0, *p0, *e1a, *e1, *p1, *e2a, *e2, *p2, *e3a, *e3, *d2a, *d2, *d1a, *d1, *d0a, *d0;
    bf16 *gd0, *gd0a, *gc0, *gd1, *gd1a, *gc1, *gd2, *gd2a, *gc2, *ge3, *ge3a, *gp2, *ge2, *ge2a, *gp1, *ge1, *ge1a,
        *gp0, *ge0, *ge0a;
    float *u = nullptr, *v = nullptr;   // predictions
    double *loss = nullptr;
    int *err = nullptr;
    void *act_mem = nullptr;
    long long step = 0;
};

namespace {

int alloc_net(mvs_unet *n)
{
    static const int spec[NCONV][2] = {{16, 16},  {16, 16}, {16, 32}, {32, 32}, {32, 64},  {64, 64}, {64, 128},
                                       {128, 128}, {192, 64}, {64, 64}, {96, 32}, {32, 32}, {48, 16}, {16, 16}};
    size_t off = 0, pack = 0;
    for (int l = 0; l < NCONV; ++l) {
        n->L[l].cin = spec[l][0];
        n->L[l].cout = spec[l][1];
        n->L[l].w_off = off;
        off += (size_t)9 * spec[l][0] * spec[l][1];
        n->L[l].b_off = off;
        off += spec[l][1];
        pack += (size_t)2 * 9 * spec[l][0] * spec[l][1];
    }
    n->head_w = off;
    off += 48;
    n->head_b = off;
    off += 3;
    n->n_params = off;
    MVS_TRY_CUDA(cudaMalloc(&n->params, off * sizeof(float)));
    MVS_TRY_CUDA(cudaMalloc(&n->grads, off * sizeof(float)));
    MVS_TRY_CUDA(cudaMalloc(&n->adam_m, off * sizeof(float)));
    MVS_TRY_CUDA(cudaMalloc(&n->adam_v, off * sizeof(float)));
    MVS_TRY_CUDA(cudaMemset(n->adam_m, 0, off * sizeof(float)));
    MVS_TRY_CUDA(cudaMemset(n->adam_v, 0, off * sizeof(float)));
    MVS_TRY_CUDA(cudaMalloc(&n->packs, pack * sizeof(bf16)));
    bf16 *pp = n->packs;
    for (int l = 0; l < NCONV; ++l) {
        const size_t s = (size_t)9 * n->L[l].cin * n->L[l].cout;
        n->L[l].wf = pp;
        n->L[l].wb = pp + s;
        pp += 2 * s;
    }
    // activations
    const size_t B = n->B, H = n->H, W = n->W;
    auto px = [&](int lvl) { return B * (H >> lvl) * (W >> lvl); };
    struct Item {
        bf16 **p;
        size_t elems;
    };
    std::vector<Item> items = {
        {&n->x0, px(0) * 16},   {&n->e0a, px(0) * 16},  {&n->e0, px(0) * 16},   {&n->p0, px(1) * 16},
        {&n->e1a, px(1) * 32},  {&n->e1, px(1) * 32},   {&n->p1, px(2) * 32},   {&n->e2a, px(2) * 64},
        {&n->e2, px(2) * 64},   {&n->p2, px(3) * 64},   {&n->e3a, px(3) * 128}, {&n->e3, px(3) * 128},
        {&n->d2a, px(2) * 64},  {&n->d2, px(2) * 64},   {&n->d1a, px(1) * 32},  {&n->d1, px(1) * 32},    {&n->d0a, px(0) * 16},
        {&n->d0, px(0) * 16},   {&n->gd0, px(0) * 16},  {&n->gd0a, px(0) * 16}, {&n->gc0, px(0) * 48},
        {&n->gd1, px(1) * 32},  {&n->gd1a, px(1) * 32}, {&n->gc1, px(1) * 96},  {&n->gd2, px(2) * 64},
        {&n->gd2a, px(2) * 64}, {&n->gc2, px(2) * 192}, {&n->ge3, px(3) * 128}, {&n->ge3a, px(3) * 128},
        {&n->gp2, px(3) * 64},  {&n->ge2, px(2) * 64},  {&n->ge2a, px(2) * 64}, {&n->gp1, px(2) * 32},
        {&n->ge1, px(1) * 32},  {&n->ge1a, px(1) * 32}, {&n->gp0, px(1) * 16},  {&n->ge0, px(0) * 16},
        {&n->ge0a, px(0) * 16}};
    size_t bytes = 0;
    for (auto &it : items) bytes += (it.elems * sizeof(bf16) + 255) / 256 * 256;
    const size_t fbytes = (B * H * W * 3 * sizeof(float) + 255) / 256 * 256;
    MVS_TRY_CUDA(cudaMalloc(&n->act_mem, bytes + fbytes + 256));
    char *q = (char *)n->act_mem;
    for (auto &it : items) {
        *it.p = (bf16 *)q;
        q += (it.elems * sizeof(bf16) + 255) / 256 * 256;
    }
    n->u = (float *)q;
    n->v = n->u + B * H * W;
    q += fbytes;
    n->loss = (double *)q;
    n->err = (int *)(q + 8);
    MVS_TRY_CUDA(cudaMemset(q, 0, 256));
    return MVS_OK;
}

int repack(mvs_unet *n, cudaStream_t st)
{
    static_assert(NCONV == PACK_LAYERS, "one pack entry per layer");
    PackArgs p{};
    int most = 0;
    for (int l = 0; l < NCONV; ++l) {
        const ConvLayer &c = n->L[l];
        most = std::max(most, 9 * c.cin * c.cout);
        p.l[l] = PackLayer{n->params + c.w_off, c.wf, l == E0A ? nullptr : c.wb, c.cin, c.cout};
    }
    MVS_TRY_CUDA(launch_dependent(pack_kernel, dim3(std::min(ceil_div(most, 256), kSMs), NCONV), dim3(256), 0, st, p));
    return check_launch("unet weight pack");
}

#define MVS_RC(x)                 \
    do {                          \
        int rc__ = (x);           \
        if (rc__) return rc__;    \
    } while (0)

inline int grid_for(long long n) { return (int)std::min<long long>((n + 255) / 256, 16LL * kSMs); }

// one tensor, or the concatenation of `prev` (nearest upsampled) and `skip`
Act act(const bf16 *p, int channels) { return Act{p, nullptr, channels, 0}; }
Act cat(const bf16 *prev, int cp, const bf16 *skip, int cs) { return Act{prev, skip, cp + cs, cp}; }

int conv_fwd(mvs_unet *n, int l, const Act &in, bf16 *out, int lvl, cudaStream_t st, const Head &head = Head{})
{
    const ConvLayer &c = n->L[l];
    return launch_conv(in, c.wf, n->params + c.b_off, Act{}, out, c.cout, n->B, n->H >> lvl, n->W >> lvl, 1, n->err, st,
                       head);
}
int conv_fwd(mvs_unet *n, int l, const bf16 *in, bf16 *out, int lvl, cudaStream_t st)
{
    return conv_fwd(n, l, act(in, n->L[l].cin), out, lvl, st);
}

// what the decoder levels read
Act cat2(const mvs_unet *n) { return cat(n->e3, 128, n->e2, 64); }
Act cat1(const mvs_unet *n) { return cat(n->d2, 64, n->e1, 32); }
Act cat0(const mvs_unet *n) { return cat(n->d1, 32, n->e0, 16); }

int forward(mvs_unet *n, const float *wta, const float *cost, const float *ref255, cudaStream_t st)
{
    const long long npix = (long long)n->B * n->H * n->W;
    MVS_TRY_CUDA(launch_dependent(features_kernel, dim3(grid_for(npix)), dim3(256), 0, st, wta, cost, ref255, npix, n->nm,
                                  n->x0));
    const int B = n->B, H = n->H, W = n->W;
    auto pool = [&](const bf16 *in, int lvl, int C, bf16 *out) -> int {
        const int rows = B * (H >> (lvl + 1)), wo = W >> (lvl + 1);
        const RowGrid g = row_grid(rows, wo * C / 8);
        MVS_TRY_CUDA(launch_dependent(pool_kernel, g.grid, g.block, 0, st, in, rows, wo, C, out));
        return MVS_OK;
    };
    MVS_RC(conv_fwd(n, E0A, n->x0, n->e0a, 0, st));
    MVS_RC(conv_fwd(n, E0B, n->e0a, n->e0, 0, st));
    MVS_RC(pool(n->e0, 0, 16, n->p0));
    MVS_RC(conv_fwd(n, E1A, n->p0, n->e1a, 1, st));
    MVS_RC(conv_fwd(n, E1B, n->e1a, n->e1, 1, st));
    MVS_RC(pool(n->e1, 1, 32, n->p1));
    MVS_RC(conv_fwd(n, E2A, n->p1, n->e2a, 2, st));
    MVS_RC(conv_fwd(n, E2B, n->e2a, n->e2, 2, st));
    MVS_RC(pool(n->e2, 2, 64, n->p2));
    MVS_RC(conv_fwd(n, E3A, n->p2, n->e3a, 3, st));
    MVS_RC(conv_fwd(n, E3B, n->e3a, n->e3, 3, st));
    MVS_RC(conv_fwd(n, D2A, cat2(n), n->d2a, 2, st));
    MVS_RC(conv_fwd(n, D2B, n->d2a, n->d2, 2, st));
    MVS_RC(conv_fwd(n, D1A, cat1(n), n->d1a, 1, st));
    MVS_RC(conv_fwd(n, D1B, n->d1a, n->d1, 1, st));
    MVS_RC(conv_fwd(n, D0A, cat0(n), n->d0a, 0, st));
    const Head head{n->params + n->head_w, n->params + n->head_b, wta, n->u, n->v, n->nm};
    MVS_RC(conv_fwd(n, D0B, act(n->d0a, 16), n->d0, 0, st, head));
    return check_launch("unet forward");
}

// backward of conv layer l: dz = gradient at its (pre-ReLU-masked) output;
// weight/bias gradients from its input x; dx (optional) masked by x > 0 when
// mask_x
int conv_bwd(mvs_unet *n, int l, const Act &x, const bf16 *dz, bf16 *dx, bool mask_x, int lvl, cudaStream_t st)
{
    const ConvLayer &c = n->L[l];
    const int H = n->H >> lvl, W = n->W >> lvl;
    MVS_RC(launch_wgrad(x, dz, c.cout, n->B, H, W, n->grads + c.w_off, n->grads + c.b_off, n->err, st));
    if (dx)
        MVS_RC(launch_conv(act(dz, c.cout), c.wb, nullptr, mask_x ? x : Act{}, dx, c.cin, n->B, H, W, 0, n->err, st));
    return MVS_OK;
}
int conv_bwd(mvs_unet *n, int l, const bf16 *x, const bf16 *dz, bf16 *dx, bool mask_x, int lvl, cudaStream_t st)
{
    return conv_bwd(n, l, act(x, n->L[l].cin), dz, dx, mask_x, lvl, st);
}

int backward(mvs_unet *n, const float *ut, const float *vt, cudaStream_t st)
{
    const int B = n->B, H = n->H, W = n->W;
    MVS_TRY_CUDA(cudaMemsetAsync(n->grads, 0, n->n_params * sizeof(float), st));
    MVS_TRY_CUDA(cudaMemsetAsync(n->loss, 0, sizeof(double), st));
    const long long img = (long long)H * W;
    const dim3 hg((unsigned)std::min<long long>((2 * img + 255) / 256, std::max(1, 4 * kSMs / B)), std::min(B, 65535));
    head_back_kernel<<<hg, 256, 0, st>>>(n->d0, n->params + n->head_w, n->u, n->v, ut, vt, B, img, n->nm, n->gd0,
                                         n->grads + n->head_w, n->grads + n->head_b, n->loss);
    auto upback = [&](const bf16 *dc, int ctot, int lvl, int cp, bf16 *dprev) -> int {
        const int rows = B * (H >> (lvl + 1)), wp = W >> (lvl + 1);
        const RowGrid g = row_grid(rows, wp * cp / 8);
        MVS_TRY_CUDA(launch_dependent(upcat_back_kernel, g.grid, g.block, 0, st, dc, ctot, rows, wp, cp, dprev));
        return MVS_OK;
    };
    auto poolback = [&](const bf16 *dp, const bf16 *dc, int ctot, int coff, const bf16 *e, int lvl, int C,
                        bf16 *de) -> int {
        const int rows = B * (H >> lvl), wl = W >> lvl;
        const RowGrid g = row_grid(rows, wl * C / 8);
        MVS_TRY_CUDA(launch_dependent(pool_back_kernel, g.grid, g.block, 0, st, dp, dc, ctot, coff, e, rows, wl, C, de));
        return MVS_OK;
    };
    // decoder level 0
    MVS_RC(conv_bwd(n, D0B, n->d0a, n->gd0, n->gd0a, true, 0, st));
    MVS_RC(conv_bwd(n, D0A, cat0(n), n->gd0a, n->gc0, true, 0, st));
    MVS_RC(upback(n->gc0, 48, 0, 32, n->gd1));
    // decoder level 1
    MVS_RC(conv_bwd(n, D1B, n->d1a, n->gd1, n->gd1a, true, 1, st));
    MVS_RC(conv_bwd(n, D1A, cat1(n), n->gd1a, n->gc1, true, 1, st));
    MVS_RC(upback(n->gc1, 96, 1, 64, n->gd2));
    // decoder level 2
    MVS_RC(conv_bwd(n, D2B, n->d2a, n->gd2, n->gd2a, true, 2, st));
    MVS_RC(conv_bwd(n, D2A, cat2(n), n->gd2a, n->gc2, true, 2, st));
    MVS_RC(upback(n->gc2, 192, 2, 128, n->ge3));
    // bottleneck
    MVS_RC(conv_bwd(n, E3B, n->e3a, n->ge3, n->ge3a, true, 3, st));
    MVS_RC(conv_bwd(n, E3A, n->p2, n->ge3a, n->gp2, false, 3, st));
    // encoder level 2
    MVS_RC(poolback(n->gp2, n->gc2, 192, 128, n->e2, 2, 64, n->ge2));
    MVS_RC(conv_bwd(n, E2B, n->e2a, n->ge2, n->ge2a, true, 2, st));
    MVS_RC(conv_bwd(n, E2A, n->p1, n->ge2a, n->gp1, false, 2, st));
    // encoder level 1
    MVS_RC(poolback(n->gp1, n->gc1, 96, 64, n->e1, 1, 32, n->ge1));
    MVS_RC(conv_bwd(n, E1B, n->e1a, n->ge1, n->ge1a, true, 1, st));
    MVS_RC(conv_bwd(n, E1A, n->p0, n->ge1a, n->gp0, false, 1, st));
    // encoder level 0
    MVS_RC(poolback(n->gp0, n->gc0, 48, 32, n->e0, 0, 16, n->ge0));
    MVS_RC(conv_bwd(n, E0B, n->e0a, n->ge0, n->ge0a, true, 0, st));
    MVS_RC(conv_bwd(n, E0A, n->x0, n->ge0a, nullptr, false, 0, st));
    return check_launch("unet backward");
}

int read_err(mvs_unet *n, cudaStream_t st)
{
    int e = 0;
    MVS_TRY_CUDA(cudaMemcpyAsync(&e, n->err, sizeof(int), cudaMemcpyDeviceToHost, st));
    MVS_TRY_CUDA(cudaStreamSynchronize(st));
    if (e) return set_error(MVS_ERR_TIMEOUT, "unet: a tensor-core wait gave up");
    return MVS_OK;
}

}  // namespace

// ===========================================================================
// C ABI
// ===========================================================================

extern "C" {

int mvs_unet_create(mvs_unet **out, int32_t batch, int32_t height, int32_t width, const float *norm7)
{
    if (!out) return set_error(MVS_ERR_ARG, "null output");
    *out = nullptr;
    if (batch <= 0 || height <= 0 || width <= 0 || height % 8 || width % 8)
        return set_error(MVS_ERR_ARG, "unet needs batch > 0 and height, width multiples of 8 (got %d, %dx%d)", batch,
                         width, height);
    mvs_unet *n = new mvs_unet();
    n->B = batch;
    n->H = height;
    n->W = width;
    const float def[7] = {0.25f, -1.f, 2.f, 1.f, 0.01f, 1.f, 1.f};
    const float *s = norm7 ? norm7 : def;
    n->nm = Norm{s[0], s[1], s[2], s[3], s[4], s[5], s[6]};
    int rc = alloc_net(n);
    if (rc) {
        mvs_unet_destroy(n);
        return rc;
    }
    *out = n;
    return MVS_OK;
}

int mvs_unet_destroy(mvs_unet *n)
{
    if (!n) return MVS_OK;
    cudaFree(n->params);
    cudaFree(n->grads);
    cudaFree(n->adam_m);
    cudaFree(n->adam_v);
    cudaFree(n->packs);
    cudaFree(n->act_mem);
    delete n;
    return MVS_OK;
}

int64_t mvs_unet_param_count(const mvs_unet *n) { return n ? (int64_t)n->n_params : 0; }

int mvs_unet_layer_info(const mvs_unet *n, int32_t layer, int32_t *cin, int32_t *cout, int64_t *w_off, int64_t *b_off)
{
    if (!n || layer < 0 || layer > NCONV) return set_error(MVS_ERR_ARG, "layer %d", layer);
    if (layer == NCONV) {   // the 1x1 head
        if (cin) *cin = 16;
        if (cout) *cout = 3;
        if (w_off) *w_off = (int64_t)n->head_w;
        if (b_off) *b_off = (int64_t)n->head_b;
        return MVS_OK;
    }
    if (cin) *cin = n->L[layer].cin;
    if (cout) *cout = n->L[layer].cout;
    if (w_off) *w_off = (int64_t)n->L[layer].w_off;
    if (b_off) *b_off = (int64_t)n->L[layer].b_off;
    return MVS_OK;
}

int mvs_unet_set_params(mvs_unet *n, const float *h_params)
{
    if (!n || !h_params) return set_error(MVS_ERR_ARG, "null argument");
    MVS_TRY_CUDA(cudaMemcpy(n->params, h_params, n->n_params * sizeof(float), cudaMemcpyHostToDevice));
    MVS_TRY_CUDA(cudaMemset(n->adam_m, 0, n->n_params * sizeof(float)));
    MVS_TRY_CUDA(cudaMemset(n->adam_v, 0, n->n_params * sizeof(float)));
    n->step = 0;
    MVS_RC(repack(n, 0));
    MVS_TRY_CUDA(cudaDeviceSynchronize());
    return MVS_OK;
}

int mvs_unet_get_params(mvs_unet *n, float *h_params, float *h_grads)
{
    if (!n) return set_error(MVS_ERR_ARG, "null net");
    MVS_TRY_CUDA(cudaDeviceSynchronize());
    if (h_params) MVS_TRY_CUDA(cudaMemcpy(h_params, n->params, n->n_params * sizeof(float), cudaMemcpyDeviceToHost));
    if (h_grads) MVS_TRY_CUDA(cudaMemcpy(h_grads, n->grads, n->n_params * sizeof(float), cudaMemcpyDeviceToHost));
    return MVS_OK;
}

int mvs_unet_forward(mvs_unet *n, const float *d_wta, const float *d_cost, const float *d_ref255, float *d_u,
                     float *d_v, void *stream)
{
    if (!n || !d_wta || !d_ref255) return set_error(MVS_ERR_ARG, "null argument");
    cudaStream_t st = (cudaStream_t)stream;
    MVS_RC(forward(n, d_wta, d_cost, d_ref255, st));
    const size_t img = (size_t)n->B * n->H * n->W;
    if (d_u) MVS_TRY_CUDA(cudaMemcpyAsync(d_u, n->u, img * sizeof(float), cudaMemcpyDeviceToDevice, st));
    if (d_v) MVS_TRY_CUDA(cudaMemcpyAsync(d_v, n->v, 2 * img * sizeof(float), cudaMemcpyDeviceToDevice, st));
    return MVS_OK;
}

int mvs_unet_backward(mvs_unet *n, const float *d_u_target, const float *d_v_target, double *loss_out, void *stream)
{
    if (!n || !d_u_target || !d_v_target) return set_error(MVS_ERR_ARG, "null argument");
    cudaStream_t st = (cudaStream_t)stream;
    MVS_RC(backward(n, d_u_target, d_v_target, st));
    if (loss_out) {
        MVS_TRY_CUDA(cudaMemcpyAsync(loss_out, n->loss, sizeof(double), cudaMemcpyDeviceToHost, st));
        MVS_RC(read_err(n, st));
    }
    return MVS_OK;
}

int mvs_unet_adam_step(mvs_unet *n, float lr, float beta1, float beta2, float eps, void *stream)
{
    if (!n) return set_error(MVS_ERR_ARG, "null net");
    cudaStream_t st = (cudaStream_t)stream;
    n->step += 1;
    const float c1 = 1.f - powf(beta1, (float)n->step), c2 = 1.f - powf(beta2, (float)n->step);
    adam_kernel<<<grid_for((long long)n->n_params), 256, 0, st>>>(n->params, n->grads, n->adam_m, n->adam_v,
                                                                  (long long)n->n_params, lr, beta1, beta2, eps, c1,
                                                                  c2);
    MVS_RC(repack(n, st));
    return MVS_OK;
}

int mvs_unet_train_step(mvs_unet *n, const float *d_wta, const float *d_cost, const float *d_ref255,
                        const float *d_u_target, const float *d_v_target, float lr, double *loss_out, void *stream)
{
    MVS_RC(mvs_unet_forward(n, d_wta, d_cost, d_ref255, nullptr, nullptr, stream));
    MVS_RC(mvs_unet_backward(n, d_u_target, d_v_target, nullptr, stream));
    MVS_RC(mvs_unet_adam_step(n, lr, 0.9f, 0.999f, 1e-8f, stream));
    if (loss_out) {
        cudaStream_t st = (cudaStream_t)stream;
        MVS_TRY_CUDA(cudaMemcpyAsync(loss_out, n->loss, sizeof(double), cudaMemcpyDeviceToHost, st));
        MVS_RC(read_err(n, st));
    }
    return MVS_OK;
}

int mvs_unet_check(mvs_unet *n, void *stream)
{
    if (!n) return set_error(MVS_ERR_ARG, "null net");
    return read_err(n, (cudaStream_t)stream);
}

// single layers, for gradient checks against the CPU restatement
int mvs_conv3x3_forward(const uint16_t *d_in, int32_t cin, const float *d_w, const float *d_bias, int32_t cout,
                        int32_t batch, int32_t height, int32_t width, int32_t relu, uint16_t *d_out,
                        uint16_t *d_wpack, int32_t *d_err, void *stream)
{
    if (!d_in || !d_w || !d_out || !d_wpack || !d_err) return set_error(MVS_ERR_ARG, "null argument");
    cudaStream_t st = (cudaStream_t)stream;
    MVS_RC(launch_pack(d_w, cin, cout, d_wpack, nullptr, st));
    MVS_RC(launch_conv(act(d_in, cin), d_wpack, d_bias, Act{}, d_out, cout, batch, height, width, relu, d_err, st));
    return check_launch("conv3x3 forward");
}

int mvs_conv3x3_backward(const uint16_t *d_x, int32_t cin, const float *d_w, const uint16_t *d_dz, int32_t cout,
                         int32_t batch, int32_t height, int32_t width, int32_t mask_x, uint16_t *d_dx, float *d_dw,
                         float *d_db, uint16_t *d_wpack, int32_t *d_err, int32_t tensor_cores, void *stream)
{
    if (!d_x || !d_w || !d_dz || !d_dw || !d_wpack || !d_err) return set_error(MVS_ERR_ARG, "null argument");
    if (cout % 16 || cin % 16) return set_error(MVS_ERR_ARG, "channels must be multiples of 16");
    cudaStream_t st = (cudaStream_t)stream;
    const size_t s = (size_t)9 * cin * cout;
    MVS_RC(launch_pack(d_w, cin, cout, d_wpack, d_wpack + s, st));
    MVS_RC(launch_wgrad(act(d_x, cin), d_dz, cout, batch, height, width, d_dw, d_db, d_err, st, tensor_cores != 0));
    if (d_dx)
        MVS_RC(launch_conv(act(d_dz, cout), d_wpack + s, nullptr, mask_x ? act(d_x, cin) : Act{}, d_dx, cin, batch,
                           height, width, 0, d_err, st));
    return check_launch("conv3x3 backward");
}

}  // extern "C"
