// The learned warm start of the pressure solve: a small convolutional network
// that predicts the change of the pressure correction from the same RK stage
// one time step earlier, trained on pairs the solver itself produces.  No
// counterpart in the reference.
//
// Network (fixed): six 3x3 convolutions, 3 -> 32 -> 32 -> 32 -> 32 -> 32 -> 1
// channels, zero padding, ReLU after all but the last; weights held in FP32
// for training and used in BF16 by the forward pass, every product
// accumulated in FP32.  Activations are channel-major planes [C][H][W].
//
// Inputs of a sample (all on the physical cells of the solve range):
//   x0 = rho, x1 = r0 / rms(r0) with r0 = rhs - A phi_prev the residual the
//   previous correction leaves, x2 = phi_prev / rms(phi_prev);
// output y, the predicted change of the correction over rms(phi_prev); the
// warm start takes the Galerkin step along it from phi_prev (k_cnn_apply);
// training target t = (phi - phi_prev) / rms(phi_prev).
//
// Kernels: the four hidden 32 -> 32 layers run on the tensor cores
// (k_conv_umma: tcgen05.mma on tiles staged once in shared memory, BF16
// activations and weights, FP32 accumulation in tensor memory), forward and
// input gradient, and their weight gradients (k_wgrad_umma, the pixels as the
// GEMM's K); the first (3 -> 32) and last (32 -> 1) layers, too narrow for an
// MMA tile, run on the FP32 pipes (k_conv3x3, k_conv_last, and k_last_back and
// k_first_wgrad backwards).  Weight gradients are per-CTA partial sums that
// one kernel adds for all layers; then the mean-square loss, Adam, and the
// input assembly with the two root mean squares.
#include <cuda_bf16.h>
#include <cstdint>
#include <cstring>
#include <vector>

#include "../../include/pvof.h"
#include "pvof_device.cuh"
#include "pvof_kernels.cuh"

namespace pvof {

namespace {

constexpr int CNN_TILE = 16;             // output tile edge of a block
constexpr int CNN_HALO = CNN_TILE + 2;   // with the 3x3 halo
constexpr int CNN_CMAX = 32;             // channels of the hidden layers

// forward: out[co][p] = b[co] + sum_ci sum_tap w[co][ci][tap] * in[ci][p + tap]
// (zero outside the H x W plane), then ReLU if relu
template <int COUT>
__global__ void __launch_bounds__(CNN_TILE * CNN_TILE) k_conv3x3(const float *__restrict__ in, int cin,
                                                                 const __nv_bfloat16 *__restrict__ w,
                                                                 const float *__restrict__ b, float *__restrict__ out,
                                                                 int H, int W, int relu)
{
    extern __shared__ float cnn_smem[];
    float (*tile)[CNN_HALO][CNN_HALO] = reinterpret_cast<float (*)[CNN_HALO][CNN_HALO]>(cnn_smem);
    float *ws = cnn_smem + cin * CNN_HALO * CNN_HALO;   // the layer's weights, COUT * cin * 9
    const int tx = threadIdx.x % CNN_TILE, ty = threadIdx.x / CNN_TILE;
    const int i0 = blockIdx.x * CNN_TILE, j0 = blockIdx.y * CNN_TILE;
    const size_t plane = (size_t)H * W;
    for (int q = threadIdx.x; q < cin * CNN_HALO * CNN_HALO; q += blockDim.x) {
        const int c = q / (CNN_HALO * CNN_HALO), r = q % (CNN_HALO * CNN_HALO);
        const int i = i0 + r % CNN_HALO - 1, j = j0 + r / CNN_HALO - 1;
        tile[c][r / CNN_HALO][r % CNN_HALO] = (i >= 0 && i < W && j >= 0 && j < H) ? in[c * plane + (size_t)j * W + i] : 0.0f;
    }
    for (int q = threadIdx.x; q < COUT * cin * 9; q += blockDim.x) ws[q] = __bfloat162float(w[q]);
    __syncthreads();
    const int i = i0 + tx, j = j0 + ty;
    if (i >= W || j >= H) return;
    float acc[COUT];
#pragma unroll
    for (int co = 0; co < COUT; co++) acc[co] = b ? b[co] : 0.0f;
    for (int ci = 0; ci < cin; ci++)
#pragma unroll
        for (int t = 0; t < 9; t++) {
            const float x = tile[ci][ty + t / 3][tx + t % 3];
#pragma unroll
            for (int co = 0; co < COUT; co++) acc[co] += x * ws[(co * cin + ci) * 9 + t];
        }
#pragma unroll
    for (int co = 0; co < COUT; co++) {
        float v = acc[co];
        if (relu && v < 0.0f) v = 0.0f;
        out[co * plane + (size_t)j * W + i] = v;
    }
}

// ---------------------------------------------------------------------------
// 32 -> 32 channel 3x3 convolutions on the tensor cores (tcgen05, kind::f16)
// ---------------------------------------------------------------------------
// A CTA takes a tile of TH rows x TW <= 128 pixels of the plane and stages it
// with its one-pixel halo in shared memory once, rounded to BF16: 16-byte
// units of 8 channels of one pixel, [row][group of 8 channels][pixel], with
// TP = TW + 2 pixels a row.  Read as a matrix without swizzle (core matrices
// of 8 x 16 bytes) that layout is both
//   K-major, rows = pixels, K = channels (8-pixel groups 128 bytes apart,
//     channel groups 16 TP bytes apart): A of the forward and input-gradient
//     convolutions, and
//   MN-major, rows = channels, K = pixels (channel groups 16 TP bytes apart,
//     8-pixel groups 128 bytes apart), four rows of the tile one more run of
//     channel groups: both operands of the weight gradient,
// and a tap (dy, dx) of the convolution is only another start address, so no
// im2col copy is made (it was read and stored nine times per pixel before).
//
// k_conv_umma: D[pixel][co] over K = tap * 32 + ci, per tile row one 128 x 32
// FP32 accumulator in tensor memory and 18 MMAs of K = 16 in tap order.  One
// thread issues them all and commits to an mbarrier; the warps read the
// accumulators back and write the 32 channels with the bias and the ReLU
// (forward) or through the ReLU mask of the layer below (input gradient, the
// same convolution with the flipped, transposed weights).
// Bound by the FP32 planes in HBM (256 MB per layer at 1000x1000): forward
// 383 -> 130 us, input gradient with its mask 480 -> 158 us.
constexpr int UM_M = 128;                          // pixels of an accumulator (MMA M)
constexpr int UM_N = 32;                           // output channels (MMA N)
constexpr int UM_KSTEPS = 9 * CNN_CMAX / 16;       // 18 MMAs of K = 16
constexpr int UM_B_STEP = UM_N * 16 * 2;           // bytes of B per MMA: 1024
constexpr int UM_B_BYTES = UM_KSTEPS * UM_B_STEP;
constexpr int UM_THREADS = 256;
constexpr long long UM_WAIT_LIMIT = 1LL << 26;     // bounded wait on the MMAs' mbarrier

// tcgen05.mma instruction descriptor: D F32 (bits 4-5 = 1), A and B BF16
// (bits 7-9, 10-12 = 1), A / B MN-major at bits 15 / 16, N >> 3 at bits
// 17-22, M >> 4 at bits 24-28
__host__ __device__ constexpr uint32_t um_idesc(int n, int mn_major)
{
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)mn_major << 15) | ((uint32_t)mn_major << 16) |
           ((uint32_t)(n >> 3) << 17) | ((uint32_t)(UM_M >> 4) << 24);
}

// shared-memory matrix descriptor without swizzle: start address, leading and
// stride byte offsets, each in 16-byte units (K-major: the K halves and the
// 8-row groups; MN-major: the 8-deep K groups and the 8-channel groups);
// version 1 at bit 46; layout type 0 (no swizzle) at bits 61-63
__device__ __forceinline__ uint64_t um_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo)
{
    return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

__device__ __forceinline__ uint32_t um_pack(float a, float b)
{
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);   // a in the low half: the lower address
    return *reinterpret_cast<const uint32_t *>(&h);
}

__device__ __forceinline__ uint32_t um_smem(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

template <int COLS>
__device__ __forceinline__ void um_begin(uint32_t *holder, uint64_t *mbar)
{
    if (threadIdx.x < 32) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(um_smem(holder)), "n"(COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (threadIdx.x == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(um_smem(mbar)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
}

template <int COLS>
__device__ __forceinline__ void um_end(uint32_t tmem)
{
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (threadIdx.x < 32) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(COLS) : "memory");
}

// the CTA's generic-proxy stores become visible to the tensor cores' async proxy
__device__ __forceinline__ void um_publish()
{
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

__device__ __forceinline__ void um_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(acc)
                 : "memory");
}

__device__ __forceinline__ void um_commit(uint64_t *mbar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(um_smem(mbar)) : "memory");
}

// bounded wait of the whole CTA for the committed MMAs; 0 if it gave up
__device__ __forceinline__ int um_wait(uint64_t *mbar, uint32_t parity)
{
    int done = 0;
    for (long long it = 0; it < UM_WAIT_LIMIT && !done; it++) {
        uint32_t ok;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                     "selp.u32 %0, 1, 0, p;\n\t}" : "=r"(ok) : "r"(um_smem(mbar)), "r"(parity) : "memory");
        done = (int)ok;
    }
    done = __syncthreads_and(done);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    return done;
}

__device__ __forceinline__ void um_read32(uint32_t taddr, uint32_t (&r)[32])
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, "
                 "%12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, "
                 "%30, %31}, [%32];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]),
                   "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]),
                   "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]),
                   "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
                 : "r"(taddr)
                 : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// strips of a row of W pixels: at most 128 each, a multiple of 16 wide (the
// weight gradient's K = 16 pixels stay within a row)
__host__ __device__ inline int um_strips(int W) { return (W + UM_M - 1) / UM_M; }
__host__ __device__ inline int um_width(int W)
{
    const int n = um_strips(W), w = (W + n - 1) / n;
    return (w + 15) / 16 * 16;
}

// `rows` rows of `width` pixels from (x0, y0) of the 32 planes of `in`, zero
// outside the plane, as 16-byte units [row][channel group][pixel] at dst; a
// warp takes one channel group, neighbouring lanes neighbouring pixels.  sum:
// the FP32 sums of the warp's 8 channels over the staged pixels, if not null.
__device__ __forceinline__ void um_stage(const float *__restrict__ in, int H, int W, int x0, int y0, int rows, int width,
                                         unsigned char *dst, float *sum)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, cg = warp & 3;
    const size_t plane = (size_t)H * W;
    const float *src = in + (size_t)(8 * cg) * plane;
    const int n = rows * width, step = UM_THREADS / 4;
    constexpr int U = 4;   // units in flight per thread: 32 loads before the first is used
    for (int q0 = (warp >> 2) * 32 + lane; q0 < n; q0 += U * step) {
        float v[U][8];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int q = q0 + u * step, r = (int)((unsigned)q / (unsigned)width);
            const int y = y0 + r, x = x0 + q - r * width;
            const bool ok = q < n && y >= 0 && y < H && x >= 0 && x < W;
            const float *p = src + (ok ? (size_t)y * W + x : 0);
#pragma unroll
            for (int e = 0; e < 8; e++) v[u][e] = ok ? p[(size_t)e * plane] : 0.0f;
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int q = q0 + u * step, r = (int)((unsigned)q / (unsigned)width);
            if (q < n)
                *reinterpret_cast<uint4 *>(dst + ((size_t)(r * 4 + cg) * width + (q - r * width)) * 16) =
                    make_uint4(um_pack(v[u][0], v[u][1]), um_pack(v[u][2], v[u][3]), um_pack(v[u][4], v[u][5]),
                               um_pack(v[u][6], v[u][7]));
            if (sum)
#pragma unroll
                for (int e = 0; e < 8; e++) sum[e] += v[u][e];
        }
    }
}

template <int TH>
constexpr size_t um_conv_smem(int TP)
{
    return (size_t)(TH + 2) * 4 * TP * 16 + 16 * UM_M + UM_B_BYTES;   // the last rows' 128-pixel reads run past the tile
}

template <int TH, bool DGRAD>
__global__ void __launch_bounds__(UM_THREADS) k_conv_umma(const float *__restrict__ in, const __nv_bfloat16 *__restrict__ w,
                                                          const float *__restrict__ b, float *__restrict__ out,
                                                          const float *__restrict__ mask, int H, int W, int relu,
                                                          int *__restrict__ err)
{
    extern __shared__ __align__(128) unsigned char um_raw[];
    __shared__ __align__(8) uint64_t mbar;
    __shared__ uint32_t tmem_holder;
    constexpr int COLS = TH * UM_N;
    const int TW = um_width(W), TP = TW + 2, ns = um_strips(W);
    const int x0 = (int)(blockIdx.x % ns) * TW, y0 = (int)(blockIdx.x / ns) * TH;
    unsigned char *Bs = um_raw, *As = um_raw + UM_B_BYTES;
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    um_begin<COLS>(&tmem_holder, &mbar);
    // B: rows of the output channel, K = tap * 32 + input channel, 16-byte
    // chunks (step, row, half), written as 4-byte words in their order in
    // shared memory; the input gradient's weights are w flipped and
    // transposed
    for (int q = t; q < UM_B_BYTES / 4; q += UM_THREADS) {
        const int s = q >> 8, n = (q >> 6 & 3) * 8 + (q >> 2 & 7), ci = (s & 1) * 16 + (q >> 5 & 1) * 8 + (q & 3) * 2;
        const int tap = DGRAD ? 8 - (s >> 1) : s >> 1;
        __nv_bfloat162 v;   // w[c0][c1][tap]
        v.x = DGRAD ? w[(ci * CNN_CMAX + n) * 9 + tap] : w[(n * CNN_CMAX + ci) * 9 + tap];
        v.y = DGRAD ? w[((ci + 1) * CNN_CMAX + n) * 9 + tap] : w[(n * CNN_CMAX + ci + 1) * 9 + tap];
        reinterpret_cast<__nv_bfloat162 *>(Bs)[q] = v;
    }
    um_stage(in, H, W, x0 - 1, y0 - 1, TH + 2, TP, As, nullptr);
    um_publish();
    const uint32_t tmem = tmem_holder;
    if (t == 0) {
        const uint32_t a0 = um_smem(As), b0 = um_smem(Bs);
#pragma unroll 1
        for (int r = 0; r < TH; r++)
#pragma unroll 1
            for (int s = 0; s < UM_KSTEPS; s++) {
                const int tap = s >> 1, dy = tap / 3, dx = tap - 3 * dy;
                const uint32_t a = a0 + (uint32_t)((((r + dy) * 4 + 2 * (s & 1)) * TP + dx) * 16);
                um_mma(tmem + (uint32_t)(r * UM_N), um_desc(a, (uint32_t)TP * 16, 128), um_desc(b0 + s * UM_B_STEP, 128, 256),
                       um_idesc(UM_N, 0), s > 0 ? 1u : 0u);
            }
        um_commit(&mbar);
    }
    if (um_wait(&mbar, 0)) {
        const size_t plane = (size_t)H * W;
        const int px = (warp & 3) * 32 + lane, x = x0 + px;
#pragma unroll 1
        for (int r = warp >> 2; r < TH; r += UM_THREADS / 128) {
            const int y = y0 + r;
            const bool live = px < TW && x < W && y < H;
            const size_t p = live ? (size_t)y * W + x : 0;
            uint32_t pass = 0xffffffffu;   // the ReLU mask of the layer below, by channel
            if (DGRAD && live) {
                pass = 0;
#pragma unroll
                for (int co = 0; co < UM_N; co++) pass |= (mask[(size_t)co * plane + p] > 0.0f ? 1u : 0u) << co;
            }
            uint32_t v[32];
            um_read32(tmem + (uint32_t)(r * UM_N) + ((uint32_t)((warp & 3) * 32) << 16), v);
            if (live) {
#pragma unroll
                for (int co = 0; co < UM_N; co++) {
                    float f = __uint_as_float(v[co]);
                    if (DGRAD) {
                        if (!(pass >> co & 1u)) f = 0.0f;
                    } else {
                        f += b ? b[co] : 0.0f;
                        if (relu && f < 0.0f) f = 0.0f;
                    }
                    out[(size_t)co * plane + p] = f;
                }
            }
        }
    } else if (t == 0) {
        atomicExch(err, 1);
    }
    um_end<COLS>(tmem);
}

// Weight and bias gradient of a 32 -> 32 layer: dw[co][ci][tap] = sum_p
// in[ci][p + tap] g[co][p], the pixels as K.  Per pair of output rows and 16
// pixels one MMA for each dx: M = four input rows x 32 ci, N = the two rows x
// 32 co, so every vertical tap of the pair is a block of the 128 x 64
// accumulator (input row minus output row).  A CTA walks its tiles of UW_TH
// rows, the three accumulators staying in tensor memory, and writes its
// partial sums in dw's order, the bias sums (FP32, of the unrounded g) behind
// them; k_grad_reduce adds the CTAs' partials in a fixed order.  Two CTAs per
// SM, one staging while the other multiplies.  1000x1000: 1645 -> 102 us.
constexpr int UW_TH = 4;
constexpr int UW_COLS = 256;                                  // 3 x 64 accumulator columns
constexpr int GRAD32 = 9 * CNN_CMAX * CNN_CMAX + CNN_CMAX;    // weights and biases of a hidden layer

size_t um_wgrad_smem(int TW)   // the staged tiles, later the sums of the nine taps
{
    const size_t tiles = (size_t)((UW_TH + 2) * 4 * (TW + 2) + UW_TH * 4 * TW) * 16, sums = sizeof(float) * 9 * CNN_CMAX * CNN_CMAX;
    return tiles > sums ? tiles : sums;
}

__global__ void __launch_bounds__(UM_THREADS) k_wgrad_umma(const float *__restrict__ in, const float *__restrict__ g, int H,
                                                           int W, float *__restrict__ partial, int *__restrict__ err)
{
    extern __shared__ __align__(128) unsigned char um_raw[];
    __shared__ __align__(8) uint64_t mbar;
    __shared__ uint32_t tmem_holder;
    __shared__ float bsum[UM_THREADS / 32][8];
    const int TW = um_width(W), TP = TW + 2, ns = um_strips(W), ntile = ns * ((H + UW_TH - 1) / UW_TH);
    unsigned char *As = um_raw, *Gs = um_raw + (UW_TH + 2) * 4 * TP * 16;
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    um_begin<UW_COLS>(&tmem_holder, &mbar);
    float bs[8];
#pragma unroll
    for (int e = 0; e < 8; e++) bs[e] = 0.0f;
    uint32_t phase = 0, tmem = 0;
    int ok = 1;
#pragma unroll 1
    for (int tile = blockIdx.x; tile < ntile && ok; tile += gridDim.x) {
        const int x0 = (tile % ns) * TW, y0 = (tile / ns) * UW_TH;
        um_stage(in, H, W, x0 - 1, y0 - 1, UW_TH + 2, TP, As, nullptr);
        um_stage(g, H, W, x0, y0, UW_TH, TW, Gs, bs);
        um_publish();
        tmem = tmem_holder;
        if (t == 0) {
            const uint32_t a0 = um_smem(As), g0 = um_smem(Gs);
#pragma unroll 1
            for (int pr = 0; pr < UW_TH / 2; pr++)
#pragma unroll 1
                for (int k = 0; k < TW / 16; k++)
#pragma unroll
                    for (int dx = 0; dx < 3; dx++)
                        um_mma(tmem + (uint32_t)(dx * 64),
                               um_desc(a0 + (uint32_t)((2 * pr * 4 * TP + 16 * k + dx) * 16), 128, (uint32_t)TP * 16),
                               um_desc(g0 + (uint32_t)((2 * pr * 4 * TW + 16 * k) * 16), 128, (uint32_t)TW * 16),
                               um_idesc(64, 1), (tile != (int)blockIdx.x || pr > 0 || k > 0) ? 1u : 0u);
            um_commit(&mbar);
        }
        ok = um_wait(&mbar, phase);   // the MMAs read the staged tiles
        phase ^= 1u;
    }
    float *out = partial + (size_t)blockIdx.x * GRAD32;
    if (ok) {
        // lanes ra * 32 + ci (input row ra), columns dx * 64 + rb * 32 + co
        // (output row rb): vertical tap dy = ra - rb in 0..2; the two output
        // rows' blocks are added through shared memory
        float *acc = reinterpret_cast<float *>(um_raw);   // [tap][ci][co], co rotated by ci against bank conflicts
#pragma unroll 1
        for (int rb = 0; rb < 2; rb++) {
            if (warp < 4 && warp - rb >= 0 && warp - rb < 3)
#pragma unroll 1
                for (int dx = 0; dx < 3; dx++) {
                    uint32_t v[32];
                    um_read32(tmem + (uint32_t)(dx * 64 + rb * 32) + ((uint32_t)(warp * 32) << 16), v);
                    float *p = acc + (((warp - rb) * 3 + dx) * CNN_CMAX + lane) * CNN_CMAX;
#pragma unroll
                    for (int co = 0; co < CNN_CMAX; co++) {
                        const int q = (co + lane) & 31;
                        p[q] = rb == 0 ? __uint_as_float(v[co]) : p[q] + __uint_as_float(v[co]);
                    }
                }
            __syncthreads();
        }
        for (int q = t; q < 9 * CNN_CMAX * CNN_CMAX; q += UM_THREADS) {
            const int tap = q % 9, ci = (q / 9) & 31, co = q / (9 * CNN_CMAX);
            out[q] = acc[(tap * CNN_CMAX + ci) * CNN_CMAX + ((co + ci) & 31)];
        }
    } else if (t == 0) {
        atomicExch(err, 1);
    }
#pragma unroll
    for (int e = 0; e < 8; e++) {
        for (int o = 16; o > 0; o >>= 1) bs[e] += __shfl_down_sync(0xffffffffu, bs[e], o);
        if (lane == 0) bsum[warp][e] = bs[e];
    }
    __syncthreads();
    if (t < CNN_CMAX) out[9 * CNN_CMAX * CNN_CMAX + t] = bsum[t >> 3][t & 7] + bsum[4 + (t >> 3)][t & 7];
    um_end<UW_COLS>(tmem_holder);
}

// ---------------------------------------------------------------------------
// the narrow layers (3 -> 32 and 32 -> 1) on the FP32 pipes
// ---------------------------------------------------------------------------

// the last layer forward: 32 planes to one, every thread LAST_ROWS pixels of a
// column (4, or 1 where that leaves SMs idle: 64x64 19.6 -> 13.8 us), its accumulators in k_conv3x3's order (ci, then tap).  y2: a second
// copy of the output, if not null.  1000x1000: 181 -> 113 us (read of 128 MB).
template <int LAST_ROWS>
__global__ void __launch_bounds__(256) k_conv_last(const float *__restrict__ in, const __nv_bfloat16 *__restrict__ w,
                                                   const float *__restrict__ b, float *__restrict__ y1,
                                                   float *__restrict__ y2, int H, int W)
{
    __shared__ float ws[CNN_CMAX * 9];
    for (int q = threadIdx.x; q < CNN_CMAX * 9; q += 256) ws[q] = __bfloat162float(w[q]);
    __syncthreads();
    const int x = blockIdx.x * 32 + (threadIdx.x & 31), y0 = (blockIdx.y * 8 + (threadIdx.x >> 5)) * LAST_ROWS;
    if (x >= W || y0 >= H) return;
    const size_t plane = (size_t)H * W;
    float acc[LAST_ROWS];
#pragma unroll
    for (int k = 0; k < LAST_ROWS; k++) acc[k] = b[0];
#pragma unroll(LAST_ROWS == 1 ? 4 : 2)
    for (int ci = 0; ci < CNN_CMAX; ci++) {
        const float *p = in + (size_t)ci * plane;
        float v[LAST_ROWS + 2][3];
#pragma unroll
        for (int r = 0; r < LAST_ROWS + 2; r++)
#pragma unroll
            for (int c = 0; c < 3; c++) {
                const int yy = y0 + r - 1, xx = x + c - 1;
                v[r][c] = (yy >= 0 && yy < H && xx >= 0 && xx < W) ? p[(size_t)yy * W + xx] : 0.0f;
            }
#pragma unroll
        for (int tp = 0; tp < 9; tp++) {
            const float wv = ws[ci * 9 + tp];
#pragma unroll
            for (int k = 0; k < LAST_ROWS; k++) acc[k] += v[k + tp / 3][tp % 3] * wv;
        }
    }
#pragma unroll
    for (int k = 0; k < LAST_ROWS; k++)
        if (y0 + k < H) {
            const size_t q = (size_t)(y0 + k) * W + x;
            y1[q] = acc[k];
            if (y2) y2[q] = acc[k];
        }
}

// the last layer backward in one pass over its 32 input planes: the gradient
// at its input through that layer's ReLU (gout) and the partial weight and
// bias gradients.  A pixel needs the nine values of dy around it for both; a
// warp takes 8 channels, so a thread holds 72 weight-gradient sums.  Partials
// [block][w (32 x 9), b].  1000x1000: 4.7 ms in three kernels -> 135 us.
constexpr int GRAD_LAST = CNN_CMAX * 9 + 1;
constexpr int LB_THREADS = 256;
__global__ void __launch_bounds__(LB_THREADS) k_last_back(const float *__restrict__ act, const float *__restrict__ dy,
                                                          const __nv_bfloat16 *__restrict__ w, int H, int W,
                                                          float *__restrict__ gout, float *__restrict__ partial)
{
    __shared__ float ws[CNN_CMAX * 9];
    __shared__ float red[LB_THREADS / 32][73];
    for (int q = threadIdx.x; q < CNN_CMAX * 9; q += LB_THREADS) ws[q] = __bfloat162float(w[q]);
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, cg = warp & 3;
    const int plane = H * W;
    float acc[8][9], bacc = 0.0f;
#pragma unroll
    for (int e = 0; e < 8; e++)
#pragma unroll
        for (int t = 0; t < 9; t++) acc[e][t] = 0.0f;
    for (int p = (blockIdx.x * 2 + (warp >> 2)) * 32 + lane; p < plane; p += gridDim.x * 64) {
        const int x = p % W, y = p / W;
        float n[9];
#pragma unroll
        for (int t = 0; t < 9; t++) {
            const int xx = x + t % 3 - 1, yy = y + t / 3 - 1;
            n[t] = (xx >= 0 && xx < W && yy >= 0 && yy < H) ? dy[(size_t)yy * W + xx] : 0.0f;
        }
        bacc += n[4];
#pragma unroll
        for (int e = 0; e < 8; e++) {
            const int ci = 8 * cg + e;
            const size_t q = (size_t)ci * plane + p;
            const float a = act[q];
            float g = 0.0f;
#pragma unroll
            for (int t = 0; t < 9; t++) g += n[t] * ws[ci * 9 + 8 - t];
            gout[q] = a > 0.0f ? g : 0.0f;
#pragma unroll
            for (int t = 0; t < 9; t++) acc[e][t] += a * n[8 - t];
        }
    }
#pragma unroll
    for (int e = 0; e < 8; e++)
#pragma unroll
        for (int t = 0; t < 9; t++) {
            float v = acc[e][t];
            for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
            if (lane == 0) red[warp][e * 9 + t] = v;
        }
    for (int o = 16; o > 0; o >>= 1) bacc += __shfl_down_sync(0xffffffffu, bacc, o);
    if (lane == 0) red[warp][72] = bacc;
    __syncthreads();
    float *out = partial + (size_t)blockIdx.x * GRAD_LAST;
    for (int q = threadIdx.x; q < GRAD_LAST; q += LB_THREADS)
        out[q] = q < CNN_CMAX * 9 ? red[q / 72][q % 72] + red[4 + q / 72][q % 72] : red[0][72] + red[4][72];
}

// the first layer's weight and bias gradient: a warp takes FW_CO of the 32
// output channels, so a thread holds 54 weight sums and reads the 27 inputs
// around its pixel (through L1, without bounds checks where the whole warp is
// inside the plane).  Partials [block][w (32 x 3 x 9), b (32)].  1000x1000:
// 2.3 ms -> 285 us.
constexpr int CNN_IN = 3;
constexpr int GRAD_FIRST = CNN_CMAX * CNN_IN * 9 + CNN_CMAX;
constexpr int FW_CO = 2, FW_THREADS = 32 * CNN_CMAX / FW_CO;
__global__ void __launch_bounds__(FW_THREADS) k_first_wgrad(const float *__restrict__ in, const float *__restrict__ g, int H,
                                                            int W, float *__restrict__ partial)
{
    const int lane = threadIdx.x & 31, c0 = (threadIdx.x >> 5) * FW_CO;
    const int plane = H * W;
    float acc[FW_CO][27], bacc[FW_CO];
#pragma unroll
    for (int e = 0; e < FW_CO; e++) {
        bacc[e] = 0.0f;
#pragma unroll
        for (int t = 0; t < 27; t++) acc[e][t] = 0.0f;
    }
    const int step = gridDim.x * 32, sy = step / W, sx = step - sy * W;
    int p = blockIdx.x * 32 + lane, y = p / W, x = p - y * W;
    for (; p - lane < plane; p += step) {
        const bool live = p < plane;
        float gv[FW_CO];
#pragma unroll
        for (int e = 0; e < FW_CO; e++) {
            gv[e] = live ? g[(size_t)(c0 + e) * plane + p] : 0.0f;
            bacc[e] += gv[e];
        }
        float v[27];
        if (__all_sync(0xffffffffu, live && x > 0 && x < W - 1 && y > 0 && y < H - 1)) {
#pragma unroll
            for (int t = 0; t < 27; t++) v[t] = in[(ptrdiff_t)(t / 9) * plane + p + (ptrdiff_t)(t % 9 / 3 - 1) * W + t % 3 - 1];
        } else {
#pragma unroll
            for (int t = 0; t < 27; t++) {
                const int xx = x + t % 3 - 1, yy = y + t % 9 / 3 - 1;
                v[t] = (live && xx >= 0 && xx < W && yy >= 0 && yy < H) ? in[(size_t)(t / 9) * plane + (size_t)yy * W + xx] : 0.0f;
            }
        }
#pragma unroll
        for (int t = 0; t < 27; t++)
#pragma unroll
            for (int e = 0; e < FW_CO; e++) acc[e][t] += v[t] * gv[e];
        x += sx;
        y += sy;
        if (x >= W) { x -= W; y++; }
    }
    float *out = partial + (size_t)blockIdx.x * GRAD_FIRST;
#pragma unroll
    for (int e = 0; e < FW_CO; e++) {
#pragma unroll
        for (int t = 0; t < 27; t++) {
            float v = acc[e][t];
            for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
            if (lane == 0) out[(c0 + e) * 27 + t] = v;
        }
        for (int o = 16; o > 0; o >>= 1) bacc[e] += __shfl_down_sync(0xffffffffu, bacc[e], o);
        if (lane == 0) out[CNN_CMAX * 27 + c0 + e] = bacc[e];
    }
}

// grad += the partials of every layer, a layer's parts added in a fixed order:
// 8 threads per value take every 8th part each, their sums added in order
struct GradPart {
    const float *p;
    int n, parts, at;   // values, parts, first index in grad
};
struct GradParts {
    GradPart l[6];
};
__global__ void __launch_bounds__(256) k_grad_reduce(const __grid_constant__ GradParts G, float *__restrict__ grad, int total)
{
    __shared__ float sh[8][32];
    const int q = blockIdx.x * 32 + (threadIdx.x & 31), s = threadIdx.x >> 5;
    float v = 0.0f;
    if (q < total) {
        int l = 0;
        while (l < 5 && q >= G.l[l + 1].at) l++;
        const float *p = G.l[l].p + (q - G.l[l].at);
        const int n = G.l[l].n, parts = G.l[l].parts;
#pragma unroll 8
        for (int c = s; c < parts; c += 8) v += p[(size_t)c * n];
    }
    sh[s][threadIdx.x & 31] = v;
    __syncthreads();
    if (s == 0 && q < total) {
        for (int k = 1; k < 8; k++) v += sh[k][threadIdx.x & 31];
        grad[q] += v;
    }
}

// mean-square loss and its gradient: dy = 2 (y - t) / n, loss partials per block
__global__ void k_mse(const float *__restrict__ y, const float *__restrict__ t, size_t n, float *__restrict__ dy,
                      double *__restrict__ loss)
{
    double s = 0.0;
    for (size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (size_t)gridDim.x * blockDim.x) {
        const float e = y[q] - t[q];
        dy[q] = 2.0f * e / (float)n;
        s += (double)e * (double)e;
    }
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) atomicAdd(loss, s / (double)n);
}

// Adam (Kingma & Ba) on the FP32 master weights, then their BF16 copy
__global__ void k_adam(float *__restrict__ w, const float *__restrict__ g, float *__restrict__ m, float *__restrict__ v,
                       __nv_bfloat16 *__restrict__ wb, int n, float lr, float b1, float b2, float c1, float c2,
                       float eps)
{
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n) return;
    const float gq = g[q];
    const float mq = b1 * m[q] + (1.0f - b1) * gq;
    const float vq = b2 * v[q] + (1.0f - b2) * gq * gq;
    m[q] = mq;
    v[q] = vq;
    const float wq = w[q] - lr * (mq / c1) / (sqrtf(vq / c2) + eps);
    w[q] = wq;
    wb[q] = __float2bfloat16(wq);
}

__global__ void k_to_bf16(const float *__restrict__ w, __nv_bfloat16 *__restrict__ wb, int n)
{
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q < n) wb[q] = __float2bfloat16(w[q]);
}

// layer shapes of the fixed network and their offsets in the flat parameter
// array [w0, b0, w1, b1, ..., w5, b5] (w: [cout][cin][3][3])
struct Layer {
    int cin, cout;
    size_t w, b;   // offsets
};

constexpr int CNN_LAYERS = 6;

void layers(Layer (&L)[CNN_LAYERS])
{
    size_t off = 0;
    for (int l = 0; l < CNN_LAYERS; l++) {
        L[l].cin = l == 0 ? CNN_IN : CNN_CMAX;
        L[l].cout = l == CNN_LAYERS - 1 ? 1 : CNN_CMAX;
        L[l].w = off;
        off += (size_t)L[l].cout * L[l].cin * 9;
        L[l].b = off;
        off += (size_t)L[l].cout;
    }
}

size_t param_count()
{
    Layer L[CNN_LAYERS];
    layers(L);
    return L[CNN_LAYERS - 1].b + 1;
}

// work buffer: the five hidden layers' outputs (32 planes each), the output
// plane, two gradient buffers of 32 planes, and the backward pass's partial
// sums of every layer
__device__ int g_cnn_err;   // set when a tensor-core convolution gave up waiting for its MMAs

constexpr int GRAD_CTAS = 296;   // most blocks of a weight gradient (two per SM of a B200)

int wgrad_ctas(int H, int W)   // tensor-core layers: every CTA gets a tile
{
    const long long n = (long long)um_strips(W) * ((H + UW_TH - 1) / UW_TH);
    return (int)(n < GRAD_CTAS ? n : GRAD_CTAS);
}
int pixel_ctas(int H, int W, int per)   // narrow layers: a block takes `per` pixels a trip
{
    const long long n = ((long long)H * W + per - 1) / per;
    return (int)(n < GRAD_CTAS ? n : GRAD_CTAS);
}

size_t work_floats(int H, int W)
{
    const size_t plane = (size_t)H * W;
    return (5 * CNN_CMAX + 1 + 2 * CNN_CMAX) * plane + 4 * (size_t)wgrad_ctas(H, W) * GRAD32 +
           (size_t)pixel_ctas(H, W, 64) * GRAD_LAST + (size_t)pixel_ctas(H, W, 32) * GRAD_FIRST;
}

int *cnn_error()
{
    int *err = nullptr;
    return cudaGetSymbolAddress((void **)&err, g_cnn_err) == cudaSuccess ? err : nullptr;
}

// multiprocessors of the current device
int device_sms()
{
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 148;
    return n;
}

// A hidden layer's convolution, forward (mask null) or input gradient through
// the ReLU mask of the layer below.  Tiles of 8 rows where they fill the SMs,
// else of 4 or 2 (more CTAs; a tile's halo rows are read again by its
// neighbours: 10 rows for 8, 4 for 2).
template <int TH, bool DGRAD>
int conv32_launch(const float *in, const __nv_bfloat16 *w, const float *b, float *out, const float *mask, int H, int W, int relu,
                  cudaStream_t st)
{
    const size_t sm = um_conv_smem<TH>(um_width(W) + 2);
    int *err = cnn_error();
    if (!err || !raise_dynamic_smem((const void *)k_conv_umma<TH, DGRAD>, sm)) return -1;
    k_conv_umma<TH, DGRAD><<<(unsigned)(um_strips(W) * ((H + TH - 1) / TH)), UM_THREADS, sm, st>>>(in, w, b, out, mask, H, W, relu, err);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

template <bool DGRAD>
int conv32(const float *in, const __nv_bfloat16 *w, const float *b, float *out, const float *mask, int H, int W, int relu,
           cudaStream_t st)
{
    const long long ns = um_strips(W), sms = device_sms();
    if (ns * (H / 8) >= sms) return conv32_launch<8, DGRAD>(in, w, b, out, mask, H, W, relu, st);
    if (ns * (H / 4) >= sms) return conv32_launch<4, DGRAD>(in, w, b, out, mask, H, W, relu, st);
    return conv32_launch<2, DGRAD>(in, w, b, out, mask, H, W, relu, st);
}

// the first layer, 3 -> 32 planes
int conv_first(const float *in, const __nv_bfloat16 *w, const float *b, float *out, int H, int W, cudaStream_t st)
{
    const size_t sm = sizeof(float) * ((size_t)CNN_IN * CNN_HALO * CNN_HALO + (size_t)CNN_CMAX * CNN_IN * 9);
    const dim3 grd((unsigned)((W + CNN_TILE - 1) / CNN_TILE), (unsigned)((H + CNN_TILE - 1) / CNN_TILE));
    k_conv3x3<CNN_CMAX><<<grd, CNN_TILE * CNN_TILE, sm, st>>>(in, CNN_IN, w, b, out, H, W, 1);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

}  // namespace

// sums of squares over the physical cells (W x H) of two planes, per block
__global__ void k_cnn_sumsq(Dom d, const double *__restrict__ a, const double *__restrict__ b,
                            double *__restrict__ partials)
{
    const int W = d.NX - 1, H = d.NY - 1, P = d.P;
    double sa = 0.0, sb = 0.0;
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < W * H; q += gridDim.x * blockDim.x) {
        const int i = q % W, j = q / W;
        const double x = AT_(a, i, j), y = AT_(b, i, j);
        sa += x * x;
        sb += y * y;
    }
    __shared__ double sh[2][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int o = 16; o > 0; o >>= 1) {
        sa += __shfl_down_sync(0xffffffffu, sa, o);
        sb += __shfl_down_sync(0xffffffffu, sb, o);
    }
    if (lane == 0) { sh[0][warp] = sa; sh[1][warp] = sb; }
    __syncthreads();
    if (threadIdx.x < 2) {
        double t = 0.0;
        for (int q = 0; q < (int)(blockDim.x >> 5); q++) t += sh[threadIdx.x][q];
        partials[threadIdx.x * gridDim.x + blockIdx.x] = t;
    }
}

// the residual of the previous correction under this substep's right-hand
// side, r0 = rhs - A phi_prev (A: the variable-density operator of the
// pressure solve with its ghost update), on the physical cells
__global__ void k_cnn_residual(Dom d, BcMap mp, const double *__restrict__ rho, const double *__restrict__ rhs,
                               const double *__restrict__ phi_prev, double *__restrict__ r0)
{
    const int W = d.NX - 1, H = d.NY - 1, P = d.P;
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= W * H) return;
    const int i = q % W, j = q / W;
    const double a = pressure_op(d, rho, i, j, [&](int x, int y) { return remap(mp, phi_prev, P, d.NX, d.NY, x, y); });
    // the right-hand side with the operator's axisymmetric row weight, as the solve forms its residual
    AT_(r0, i, j) = (d.axisym ? AT_(rhs, i, j) * d.m.r_c[i] : AT_(rhs, i, j)) - a;
}

// network inputs x = [rho, r0 / rms(r0), phi_prev / rms(phi_prev)] and, if
// phi is given, the target t = (phi - phi_prev) / rms(phi_prev)
__global__ void k_cnn_assemble(Dom d, const double *__restrict__ rho, const double *__restrict__ rhs,
                               const double *__restrict__ phi_prev, const double *__restrict__ phi,
                               const DevScalars *__restrict__ sc, float *__restrict__ x, float *__restrict__ t)
{
    const int W = d.NX - 1, H = d.NY - 1, P = d.P;
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= W * H) return;
    const int i = q % W, j = q / W;
    const double n = (double)W * H;
    const double rr = sqrt(sc->cnn_ms[0] / n) + 1e-300, rp = sqrt(sc->cnn_ms[1] / n) + 1e-300;
    const size_t plane = (size_t)W * H;
    x[q] = (float)AT_(rho, i, j);
    x[plane + q] = (float)(AT_(rhs, i, j) / rr);
    x[2 * plane + q] = (float)(AT_(phi_prev, i, j) / rp);
    if (phi) t[q] = (float)((AT_(phi, i, j) - AT_(phi_prev, i, j)) / rp);
}

// the network's change as a plane of the solve's layout: e = y (ghosts zero)
__global__ void k_cnn_expand(Dom d, const float *__restrict__ y, double *__restrict__ e)
{
    const int W = d.NX - 1, H = d.NY - 1, P = d.P;
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= W * H) return;
    AT_(e, q % W, q / W) = (double)y[q];
}

// the two inner products of the step along e that minimises the residual in
// the solve's stopping norm (r . M r, M the Jacobi preconditioner): per block
// sum (A e) M r0 and sum (A e) M (A e) over the physical cells
__global__ void k_cnn_galerkin(Dom d, BcMap mp, const double *__restrict__ rho, const double *__restrict__ e,
                               const double *__restrict__ r0, const double *__restrict__ M, double *__restrict__ partials)
{
    const int W = d.NX - 1, H = d.NY - 1, P = d.P;
    double s0 = 0.0, s1 = 0.0;
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < W * H; q += gridDim.x * blockDim.x) {
        const int i = q % W, j = q / W;
        const double ae = pressure_op(d, rho, i, j, [&](int x, int y) { return remap(mp, e, P, d.NX, d.NY, x, y); });
        const double m = AT_(M, i, j);
        s0 += ae * m * AT_(r0, i, j);
        s1 += ae * m * ae;
    }
    __shared__ double sh[2][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int o = 16; o > 0; o >>= 1) {
        s0 += __shfl_down_sync(0xffffffffu, s0, o);
        s1 += __shfl_down_sync(0xffffffffu, s1, o);
    }
    if (lane == 0) { sh[0][warp] = s0; sh[1][warp] = s1; }
    __syncthreads();
    if (threadIdx.x < 2) {
        double t = 0.0;
        for (int q = 0; q < (int)(blockDim.x >> 5); q++) t += sh[threadIdx.x][q];
        partials[threadIdx.x * gridDim.x + blockIdx.x] = t;
    }
}

// the warm start phi = phi_prev + alpha e with alpha = (A e . M r0) /
// (A e . M A e): of the corrections along e it leaves the smallest residual
// in the solve's stopping norm, so the solve never starts further from its
// stopping test than from phi_prev
__global__ void k_cnn_apply(Dom d, const double *__restrict__ e, const double *__restrict__ phi_prev,
                            const DevScalars *__restrict__ sc, double *__restrict__ phi)
{
    const int W = d.NX - 1, H = d.NY - 1, P = d.P;
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= W * H) return;
    const int i = q % W, j = q / W;
    const double den = sc->cnn_ms[1];
    const double alpha = (den != 0.0) ? sc->cnn_ms[0] / den : 0.0;
    AT_(phi, i, j) = AT_(phi_prev, i, j) + alpha * AT_(e, i, j);
}

}  // namespace pvof

using namespace pvof;

extern "C" {

size_t pvof_cnn_param_count(void) { return param_count(); }

size_t pvof_cnn_work_floats(int H, int W) { return (H > 0 && W > 0) ? work_floats(H, W) : 0; }

int pvof_cnn_forward(const float *params, const uint16_t *params_bf16, const float *x, float *y, int H, int W,
                     float *work, void *stream)
{
    if (!params || !params_bf16 || !x || !work || H <= 0 || W <= 0) return PVOF_EINVAL;
    cudaStream_t st = (cudaStream_t)stream;
    Layer L[CNN_LAYERS];
    layers(L);
    const size_t plane = (size_t)H * W;
    const __nv_bfloat16 *wb = reinterpret_cast<const __nv_bfloat16 *>(params_bf16);
    if (conv_first(x, wb + L[0].w, params + L[0].b, work, H, W, st)) return PVOF_ECUDA;
    const float *in = work;
    for (int l = 1; l < CNN_LAYERS - 1; l++) {
        float *out = work + (size_t)l * CNN_CMAX * plane;   // layer l's output
        if (conv32<false>(in, wb + L[l].w, params + L[l].b, out, nullptr, H, W, 1, st)) return PVOF_ECUDA;
        in = out;
    }
    const Layer &Z = L[CNN_LAYERS - 1];   // the last: one plane, and y
    float *y0 = work + (size_t)(CNN_LAYERS - 1) * CNN_CMAX * plane;
    const unsigned gx = (unsigned)((W + 31) / 32), gy4 = (unsigned)((H + 31) / 32);
    if (gx * gy4 >= (unsigned)device_sms()) k_conv_last<4><<<dim3(gx, gy4), 256, 0, st>>>(in, wb + Z.w, params + Z.b, y0, y, H, W);
    else k_conv_last<1><<<dim3(gx, (unsigned)((H + 7) / 8)), 256, 0, st>>>(in, wb + Z.w, params + Z.b, y0, y, H, W);
    return cudaGetLastError() == cudaSuccess ? PVOF_OK : PVOF_ECUDA;
}

int pvof_cnn_backward(const float *params, const uint16_t *params_bf16, const float *x, const float *dy, float *grad,
                      int H, int W, float *work, void *stream)
{
    if (!params || !params_bf16 || !x || !dy || !grad || !work || H <= 0 || W <= 0) return PVOF_EINVAL;
    (void)params;
    cudaStream_t st = (cudaStream_t)stream;
    Layer L[CNN_LAYERS];
    layers(L);
    const size_t plane = (size_t)H * W;
    const __nv_bfloat16 *wb = reinterpret_cast<const __nv_bfloat16 *>(params_bf16);
    float *gbuf[2] = {work + (5 * CNN_CMAX + 1) * plane, work + (6 * CNN_CMAX + 1) * plane};
    float *part = work + (7 * CNN_CMAX + 1) * plane;   // every layer's partial sums, added at the end
    GradParts G;
    auto parts = [&](int l, int n, int ctas) {
        float *p = part;
        G.l[l] = GradPart{p, n, ctas, (int)L[l].w};
        part += (size_t)n * ctas;
        return p;
    };
    int *err = cnn_error();
    const size_t wsm = um_wgrad_smem(um_width(W));
    if (!err || !raise_dynamic_smem((const void *)k_wgrad_umma, wsm)) return PVOF_ECUDA;
    // the last layer: its gradients and the gradient at its input, through the ReLU
    const int last = CNN_LAYERS - 1, nl = pixel_ctas(H, W, 64);
    k_last_back<<<(unsigned)nl, LB_THREADS, 0, st>>>(work + (size_t)(last - 1) * CNN_CMAX * plane, dy, wb + L[last].w, H, W,
                                                    gbuf[0], parts(last, GRAD_LAST, nl));
    int cur = 0;
    const int nw = wgrad_ctas(H, W);
    for (int l = last - 1; l >= 1; l--) {   // the tensor-core layers
        const float *lin = work + (size_t)(l - 1) * CNN_CMAX * plane;
        k_wgrad_umma<<<(unsigned)nw, UM_THREADS, wsm, st>>>(lin, gbuf[cur], H, W, parts(l, GRAD32, nw), err);
        if (conv32<true>(gbuf[cur], wb + L[l].w, nullptr, gbuf[1 - cur], lin, H, W, 0, st)) return PVOF_ECUDA;
        cur = 1 - cur;
    }
    const int nf = pixel_ctas(H, W, 32);
    k_first_wgrad<<<(unsigned)nf, FW_THREADS, 0, st>>>(x, gbuf[cur], H, W, parts(0, GRAD_FIRST, nf));
    const int total = (int)param_count();
    k_grad_reduce<<<(unsigned)((total + 31) / 32), 256, 0, st>>>(G, grad, total);
    return cudaGetLastError() == cudaSuccess ? PVOF_OK : PVOF_ECUDA;
}

int pvof_cnn_mse(const float *y, const float *t, float *dy, size_t n, double *loss, void *stream)
{
    if (!y || !t || !dy || !loss || n == 0) return PVOF_EINVAL;
    k_mse<<<296, 256, 0, (cudaStream_t)stream>>>(y, t, n, dy, loss);
    return cudaGetLastError() == cudaSuccess ? PVOF_OK : PVOF_ECUDA;
}

int pvof_cnn_adam(float *params, const float *grad, float *m, float *v, uint16_t *params_bf16, int step, float lr,
                  void *stream)
{
    if (!params || !grad || !m || !v || !params_bf16 || step < 1) return PVOF_EINVAL;
    const int n = (int)param_count();
    const float b1 = 0.9f, b2 = 0.999f;
    const float c1 = 1.0f - powf(b1, (float)step), c2 = 1.0f - powf(b2, (float)step);
    k_adam<<<(n + 255) / 256, 256, 0, (cudaStream_t)stream>>>(params, grad, m, v,
                                                             reinterpret_cast<__nv_bfloat16 *>(params_bf16), n, lr, b1,
                                                             b2, c1, c2, 1e-8f);
    return cudaGetLastError() == cudaSuccess ? PVOF_OK : PVOF_ECUDA;
}

int pvof_cnn_conv32(const float *x, const uint16_t *w_bf16, const float *b, float *y, int H, int W, int relu,
                    void *stream)
{
    if (!x || !w_bf16 || !y || H <= 0 || W <= 0) return PVOF_EINVAL;
    return conv32<false>(x, reinterpret_cast<const __nv_bfloat16 *>(w_bf16), b, y, nullptr, H, W, relu, (cudaStream_t)stream)
               ? PVOF_ECUDA
               : PVOF_OK;
}

int pvof_cnn_status(void *stream)
{
    int *err = nullptr, h = 0;
    if (cudaGetSymbolAddress((void **)&err, g_cnn_err) != cudaSuccess) return PVOF_ECUDA;
    cudaStream_t st = (cudaStream_t)stream;
    if (cudaMemcpyAsync(&h, err, sizeof(int), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess)
        return PVOF_ECUDA;
    if (h && cudaMemsetAsync(err, 0, sizeof(int), st) != cudaSuccess) return PVOF_ECUDA;
    return h ? PVOF_ECUDA : PVOF_OK;
}

int pvof_cnn_to_bf16(const float *params, uint16_t *params_bf16, void *stream)
{
    if (!params || !params_bf16) return PVOF_EINVAL;
    const int n = (int)param_count();
    k_to_bf16<<<(n + 255) / 256, 256, 0, (cudaStream_t)stream>>>(params, reinterpret_cast<__nv_bfloat16 *>(params_bf16),
                                                                 n);
    return cudaGetLastError() == cudaSuccess ? PVOF_OK : PVOF_ECUDA;
}

}  // extern "C"
