// hydro_train.cu -- one training step of the 64 -> 256 -> 256 -> 256 -> 64
// surrogate network in three launches (hydro_nn.cu holds the general
// kernels, which train networks of other widths layer by layer).
//
// Step by step the layers' products, epilogues, transposes, column sums and
// parameter updates are 36 launches of 3 to 15 us whose operands travel
// through memory between them: 228 us at batch 4096, of which the tensor
// cores need about 3; the fused step takes 41 us.  Here
//   1. train_rows_kernel: 32 rows of the batch go through the four layers,
//      the loss gradient and back to the first layer's pre-activations in
//      one CTA.  No row needs another one, so the activations stay in shared
//      memory and the FP32 pre-activations in registers; only the BF16
//      layer inputs and gradients that the weight gradients need are written
//      (in a call's last step the pre-activations too).
//   2. train_grads_kernel: every layer's weight-gradient product (split
//      along the batch), bias column sums and the loss, side by side.  The
//      transposed operand is formed by ldmatrix.trans, not by a transpose
//      in memory.
//   3. train_update_kernel: the slices' partial products summed in slice
//      order, AdamW and the BF16 copies of weights and biases.
// Every product is accumulated over the same k16 steps by the same mma.sync
// instruction and every sum runs in the order of the general kernels, so
// the trained weights are the same bits.
#include <algorithm>
#include <cstdint>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "../../include/stonefish_hydro.h"
#include "hydro_chain.cuh"
#include "hydro_mma.cuh"
#include "hydro_train.h"

namespace sfh {

namespace train {

constexpr int kRows = 32;        // batch rows per CTA of the row kernel
constexpr int kH = 256;
constexpr int kLdA = kH + 8;     // activation row stride in shared memory (an odd number of 16-byte units)
// Sixteen warps, each 32 rows x 16 columns: with eight warps of 32 x 32 the
// kernel issued an instruction in 23% of its cycles (two warps per scheduler
// waiting on mma and ldmatrix results) and took 29 us; with sixteen 22 us.
constexpr int kThreads = 512;
// Chunks of 128 weight rows, the next one in flight: eleven CTA barriers for
// the seven products.  With chunks of 64 and two in flight there were 22, and a
// step took 1.4 us longer.
constexpr int kStages = 2;
constexpr int kStageBytes = 128 * kH * 2;   // 128 weight rows
constexpr int kChunks = 11;      // weight chunks of the seven products
constexpr size_t kRowsSmem = (size_t)kStages * kStageBytes + 2 * kRows * kLdA * 2 + (3 * kH + 64) * 4;

__device__ __forceinline__ void cp16(void* dst, const void* src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;"
                 :: "r"(static_cast<uint32_t>(__cvta_generic_to_shared(dst))), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" :: "n"(N) : "memory"); }

// Chunk i of the weights in the order the row kernel multiplies by them:
// 128 rows of the layers' weights going forward, of their transposes going
// back (64 or 256 where the layer is narrow), 16-byte unit c of row r stored at unit c ^ (r % 8) so that ldmatrix
// reads eight rows without bank conflicts.  One commit group per chunk.
__device__ __forceinline__ void load_weights(const RowsParams& P, unsigned char* smem, int i)
{
    if (i < kChunks) {
        const bf16* src;
        int rows = 128;
        if (i < 1) { src = P.w16[0]; rows = 64; }
        else if (i < 3) src = P.w16[1] + (i - 1) * 128 * kH;
        else if (i < 5) src = P.w16[2] + (i - 3) * 128 * kH;
        else if (i < 6) { src = P.w16[3]; rows = 0; }   // 256 rows of 64
        else if (i < 7) { src = P.wt16[3]; rows = 64; }
        else if (i < 9) src = P.wt16[2] + (i - 7) * 128 * kH;
        else src = P.wt16[1] + (i - 9) * 128 * kH;
        unsigned char* st = smem + (i % kStages) * kStageBytes;
        if (rows == 0) {
#pragma unroll
            for (int j = 0; j < 256 * 8 / kThreads; ++j) {
                const int u = threadIdx.x + j * kThreads, r = u >> 3, c = u & 7;
                cp16(st + r * 128 + ((c ^ (r & 7)) << 4), src + r * 64 + c * 8);
            }
        } else {
#pragma unroll 4
            for (int j = 0; j < rows * 32 / kThreads; ++j) {
                const int u = threadIdx.x + j * kThreads, r = u >> 5, c = u & 31;
                cp16(st + r * 512 + ((c ^ (r & 7)) << 4), src + r * kH + c * 8);
            }
        }
    }
    cp_commit();
}

// 32 rows x `cols` BF16 from shared to global memory, 16 bytes per thread.
__device__ __forceinline__ void store_rows(const bf16* buf, bf16* dst, int cols)
{
    const int units = cols >> 3;
    for (int u = threadIdx.x; u < kRows * units; u += kThreads) {
        const int r = u / units, c = u % units;
        *reinterpret_cast<uint4*>(dst + (size_t)r * cols + c * 8) =
            *reinterpret_cast<const uint4*>(buf + r * kLdA + c * 8);
    }
}

// One warp's 32 x 16 accumulators of a 256-column product.
typedef float Tile[2][2][4];

// One product of the row kernel: N = 256, warp w's 32 x 16 tile at column
// 16 w.  A (32 x 64 n_chunks) is in `buf`, whose contents also go to `out`
// once they are visible; the weights arrive as chunks first, first + 1, ...
__device__ __forceinline__ void product256(const RowsParams& P, unsigned char* smem, const bf16* buf, int first,
                                           int n_chunks, bf16* out, int out_cols, Tile& acc)
{
    const int lane = threadIdx.x & 31, wn = (threadIdx.x >> 5) * 16;
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int k = 0; k < 4; ++k) acc[i][j][k] = 0.f;
    const int rows = n_chunks == 1 ? 64 : 128;
#pragma unroll 1
    for (int q = 0; q < n_chunks; ++q) {
        const int i = first + q;
        cp_wait<0>();
        __syncthreads();   // chunk i is visible, and chunk i - 1's stage is free
        load_weights(P, smem, i + 1);
        const unsigned char* st = smem + (i % kStages) * kStageBytes;
#pragma unroll 8
        for (int kk = 0; kk < rows; kk += 16) {
            uint32_t a[2][4], t[4];
#pragma unroll
            for (int mi = 0; mi < 2; ++mi)
                ldsm_x4(a[mi], buf + (mi * 16 + (lane & 15)) * kLdA + q * 128 + kk + (lane >> 4) * 8);
            const int j = lane >> 3, r = kk + (lane & 7) + 8 * (j & 1), c = (wn >> 3) + (j >> 1);
            ldsm_x4_t(t, st + r * 512 + ((c ^ (r & 7)) << 4));
#pragma unroll
            for (int mi = 0; mi < 2; ++mi) {
                mma_bf16(acc[mi][0], a[mi], t[0], t[1]);
                mma_bf16(acc[mi][1], a[mi], t[2], t[3]);
            }
        }
        // behind the first chunk's products: in front of them a step took 0.4 us longer
        if (q == 0 && out) store_rows(buf, out, out_cols);
    }
}

// Hidden layer: z = acc + bias, SiLU(z) into `y`; acc keeps SiLU'(z), all
// that the way back needs of z (one sigmoid serves both).  KEEP: z to memory
// as well.
template <bool KEEP>
__device__ __forceinline__ void epilogue_silu(Tile& acc, const float* bias, bf16* y, float* z)
{
    const int lane = threadIdx.x & 31, wn = (threadIdx.x >> 5) * 16;
#pragma unroll
    for (int ni = 0; ni < 2; ++ni) {
        const int c = wn + ni * 8 + (lane & 3) * 2;
        const float2 b = *reinterpret_cast<const float2*>(bias + c);
#pragma unroll
        for (int mi = 0; mi < 2; ++mi)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int r = mi * 16 + (lane >> 2) + 8 * h;
                const float z0 = acc[mi][ni][2 * h] + b.x, z1 = acc[mi][ni][2 * h + 1] + b.y;
                if (KEEP) *reinterpret_cast<float2*>(z + (size_t)r * kH + c) = make_float2(z0, z1);
                const float s0 = sigmoidf_(z0), s1 = sigmoidf_(z1);
                *reinterpret_cast<__nv_bfloat162*>(y + r * kLdA + c) =
                    __nv_bfloat162(__float2bfloat16(z0 * s0), __float2bfloat16(z1 * s1));
                acc[mi][ni][2 * h] = s0 + z0 * s0 * (1.f - s0);
                acc[mi][ni][2 * h + 1] = s1 + z1 * s1 * (1.f - s1);
            }
    }
}

// Gradient through a hidden layer's SiLU, d its derivative.
__device__ __forceinline__ void epilogue_grad(const Tile& acc, const Tile& d, bf16* y)
{
    const int lane = threadIdx.x & 31, wn = (threadIdx.x >> 5) * 16;
#pragma unroll
    for (int ni = 0; ni < 2; ++ni)
#pragma unroll
        for (int mi = 0; mi < 2; ++mi)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int r = mi * 16 + (lane >> 2) + 8 * h, c = wn + ni * 8 + (lane & 3) * 2;
                *reinterpret_cast<__nv_bfloat162*>(y + r * kLdA + c) =
                    __nv_bfloat162(__float2bfloat16(acc[mi][ni][2 * h] * d[mi][ni][2 * h]),
                                   __float2bfloat16(acc[mi][ni][2 * h + 1] * d[mi][ni][2 * h + 1]));
            }
}

}  // namespace train

// KEEP: the call's last step, which leaves every pre-activation in memory.
template <bool KEEP>
__global__ void __launch_bounds__(train::kThreads, 1) train_rows_kernel(const RowsParams P)
{
    using namespace train;
    extern __shared__ __align__(128) unsigned char smem[];
    bf16* buf0 = reinterpret_cast<bf16*>(smem + kStages * kStageBytes);
    bf16* buf1 = buf0 + kRows * kLdA;
    float* bias = reinterpret_cast<float*>(buf1 + kRows * kLdA);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const size_t row0 = (size_t)blockIdx.x * kRows;
    dependency_wait();
    launch_dependents();
    load_weights(P, smem, 0);
    if (tid < 256) {
        const int r = tid >> 3, c = tid & 7;
        *reinterpret_cast<uint4*>(buf0 + r * kLdA + c * 8) =
            *reinterpret_cast<const uint4*>(P.x0 + (row0 + r) * 64 + c * 8);
    }
    for (int i = tid; i < 3 * kH + 64; i += kThreads) bias[i] = P.bias[i >> 8][i & 255];
    Tile d0, d1, d2;   // products, then SiLU derivatives, of the hidden layers
    product256(P, smem, buf0, 0, 1, nullptr, 0, d0);
    epilogue_silu<KEEP>(d0, bias, buf1, P.z[0] + row0 * kH);
    product256(P, smem, buf1, 1, 2, P.x[0] + row0 * kH, kH, d1);
    epilogue_silu<KEEP>(d1, bias + kH, buf0, P.z[1] + row0 * kH);
    product256(P, smem, buf0, 3, 2, P.x[1] + row0 * kH, kH, d2);
    epilogue_silu<KEEP>(d2, bias + 2 * kH, buf1, P.z[2] + row0 * kH);
    // output layer, N = 64: warp w's 16 x 8 tile; then the loss gradient
    {
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
        const int wm = (warp >> 3) * 16, wn = (warp & 7) * 8;
        cp_wait<0>();
        __syncthreads();
        load_weights(P, smem, 6);
        const unsigned char* st = smem + (5 % kStages) * kStageBytes;
#pragma unroll 2
        for (int kk = 0; kk < kH; kk += 32) {
            uint32_t a[4], t[4];
            const int r = kk + lane;   // four 8 x 8 matrices along k
            ldsm_x4_t(t, st + r * 128 + (((wn >> 3) ^ (r & 7)) << 4));
            ldsm_x4(a, buf1 + (wm + (lane & 15)) * kLdA + kk + (lane >> 4) * 8);
            mma_bf16(acc, a, t[0], t[1]);
            ldsm_x4(a, buf1 + (wm + (lane & 15)) * kLdA + kk + 16 + (lane >> 4) * 8);
            mma_bf16(acc, a, t[2], t[3]);
        }
        store_rows(buf1, P.x[2] + row0 * kH, kH);
        const float scale = 1.f / (float)((size_t)P.batch * P.n_out);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int r = wm + (lane >> 2) + 8 * h, c = wn + (lane & 3) * 2;
            float g[2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                g[e] = 0.f;
                const float z = acc[2 * h + e] + bias[3 * kH + c + e];
                if (KEEP || c + e < P.n_out) P.z[3][(row0 + r) * 64 + c + e] = z;   // for the loss
                if (c + e < P.n_out) {
                    float tv = P.target[(row0 + r) * P.n_out + c + e];
                    if (P.tmean) tv = (tv - P.tmean[c + e]) * P.tistd[c + e];
                    const float d = z - tv;
                    g[e] = 2.f * d * scale;
                }
            }
            *reinterpret_cast<__nv_bfloat162*>(buf0 + r * kLdA + c) =
                __nv_bfloat162(__float2bfloat16(g[0]), __float2bfloat16(g[1]));
        }
    }
    Tile acc;
    product256(P, smem, buf0, 6, 1, P.dz[3] + row0 * 64, 64, acc);
    epilogue_grad(acc, d2, buf1);
    product256(P, smem, buf1, 7, 2, P.dz[2] + row0 * kH, kH, acc);
    epilogue_grad(acc, d1, buf0);
    product256(P, smem, buf0, 9, 2, P.dz[1] + row0 * kH, kH, acc);
    epilogue_grad(acc, d0, buf1);
    __syncthreads();
    store_rows(buf1, P.dz[0] + row0 * kH, kH);
}

// ------------------------------------------------------------- gradients
namespace train {

constexpr int kGradThreads = 128;
// Three stages and 72 registers let seven CTAs run per SM: with four stages,
// and so six CTAs, a step took 1 us longer; eight CTAs spill.
constexpr int kGradStages = 3;
constexpr int kGradLd = 64 + 8;

struct GradSmem {
    bf16 a[kGradStages][32][kGradLd];
    bf16 b[kGradStages][32][kGradLd];
};

// A 64 x 64 tile of in^T dz over batch rows [r0, r0 + len): the k16 steps,
// tiles and accumulators of gemm_kernel<EPI_F32> on the transposed input.
__device__ __forceinline__ void weight_tile(GradSmem& S, const GradLayer& L, int m0, int n0, int slice)
{
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wm = (warp >> 1) * 32, wn = (warp & 1) * 32;
    const bf16* A = L.in + (size_t)slice * L.slice_rows * L.k + m0;
    const bf16* B = L.dz + (size_t)slice * L.slice_rows * L.n + n0;
    const int steps = L.slice_rows / 32;
    auto load = [&](int s) {
        if (s < steps) {
            const int st = s % kGradStages;
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const int u = tid + j * kGradThreads, r = u >> 3, c = (u & 7) * 8;
                cp16(&S.a[st][r][c], A + (size_t)(s * 32 + r) * L.k + c);
                cp16(&S.b[st][r][c], B + (size_t)(s * 32 + r) * L.n + c);
            }
        }
        cp_commit();
    };
    float acc[2][4][4];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int k = 0; k < 4; ++k) acc[i][j][k] = 0.f;
#pragma unroll
    for (int s = 0; s < kGradStages - 1; ++s) load(s);
#pragma unroll 1
    for (int s = 0; s < steps; ++s) {
        cp_wait<kGradStages - 2>();
        __syncthreads();
        load(s + kGradStages - 1);
        const int st = s % kGradStages;
#pragma unroll
        for (int kk = 0; kk < 32; kk += 16) {
            uint32_t a[2][4], b[4][2];
            const int j = lane >> 3;
#pragma unroll
            for (int mi = 0; mi < 2; ++mi)
                ldsm_x4_t(a[mi], &S.a[st][kk + (lane & 7) + 8 * (j >> 1)][wm + mi * 16 + 8 * (j & 1)]);
#pragma unroll
            for (int nj = 0; nj < 2; ++nj) {
                uint32_t t[4];
                ldsm_x4_t(t, &S.b[st][kk + (lane & 7) + 8 * (j & 1)][wn + nj * 16 + 8 * (j >> 1)]);
                b[2 * nj][0] = t[0];
                b[2 * nj][1] = t[1];
                b[2 * nj + 1][0] = t[2];
                b[2 * nj + 1][1] = t[3];
            }
#pragma unroll
            for (int mi = 0; mi < 2; ++mi)
#pragma unroll
                for (int ni = 0; ni < 4; ++ni) mma_bf16(acc[mi][ni], a[mi], b[ni][0], b[ni][1]);
        }
    }
    float* out = L.part + (size_t)slice * L.k * L.n;
#pragma unroll
    for (int mi = 0; mi < 2; ++mi)
#pragma unroll
        for (int ni = 0; ni < 4; ++ni)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int r = m0 + wm + mi * 16 + (lane >> 2) + 8 * h, c = n0 + wn + ni * 8 + (lane & 3) * 2;
                *reinterpret_cast<float2*>(out + (size_t)r * L.n + c) =
                    make_float2(acc[mi][ni][2 * h], acc[mi][ni][2 * h + 1]);
            }
}

// Column sums of 32 columns of dz over one row slab, in colsum_slab_kernel's
// order: 32 strided row groups, then the groups in order.
__device__ __forceinline__ void column_slab(float (&part)[32][33], const GradLayer& L, int c0, int slab, int batch)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int r0 = slab * L.slab_rows, r1 = min(batch, r0 + L.slab_rows);
    const int c = c0 + lane;
    float s[8];   // row groups warp, warp + 4, ...
#pragma unroll
    for (int g = 0; g < 8; ++g) s[g] = 0.f;
#pragma unroll 2
    for (int r = r0 + warp; r < r1; r += 32)
#pragma unroll
        for (int g = 0; g < 8; ++g)
            if (r + 4 * g < r1) s[g] += __bfloat162float(L.dz[(size_t)(r + 4 * g) * L.n + c]);
#pragma unroll
    for (int g = 0; g < 8; ++g) part[warp + 4 * g][lane] = s[g];
    __syncthreads();
    if (warp == 0) {
        float t = 0.f;
        for (int k = 0; k < 32; ++k) t += part[k][lane];
        L.col[(size_t)slab * L.n + c] = t;
    }
}

// Block b of mse_grad_kernel's 256 blocks of 256 threads: its FP32 sum of
// squared errors in the same order (threads t and t + 128 here are one),
// added to the loss in FP64.
__device__ __forceinline__ void loss_block(float* red, const GradsParams& P, int b)
{
    const uint32_t n = (uint32_t)P.batch * 64u;
    const float scale = 1.f / (float)((size_t)P.batch * P.n_out);
    float a[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        a[h] = 0.f;
        for (uint32_t i = (uint32_t)b * 256u + threadIdx.x + 128u * h; i < n; i += 65536u) {
            const uint32_t r = i >> 6, c = i & 63u;
            if (c < (uint32_t)P.n_out) {
                float tv = P.target[(size_t)r * P.n_out + c];
                if (P.tmean) tv = (tv - P.tmean[c]) * P.tistd[c];
                const float d = P.z3[i] - tv;
                a[h] += d * d;
            }
        }
    }
    red[threadIdx.x] = a[0] + a[1];
    __syncthreads();
    for (int w = 64; w > 0; w >>= 1) {
        if ((int)threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) atomicAdd(P.loss, (double)red[0] * (double)scale);
}

}  // namespace train

__global__ void __launch_bounds__(train::kGradThreads, 7) train_grads_kernel(const GradsParams P)
{
    using namespace train;
    __shared__ __align__(16) union {
        GradSmem g;
        float part[32][33];
        float red[kGradThreads];
    } S;
    dependency_wait();
    launch_dependents();
    // the products first: behind the short CTAs their last wave is emptier (a step 1 us longer)
    int b = (int)blockIdx.x;
#pragma unroll 1
    for (int l = 0; l < 4; ++l) {
        const GradLayer& L = P.layer[l];
        const int tn = L.n / 64, tiles = (L.k / 64) * tn, count = tiles * L.splits;
        if (b < count) {
            const int t = b % tiles;
            weight_tile(S.g, L, (t / tn) * 64, (t % tn) * 64, b / tiles);
            return;
        }
        b -= count;
    }
    if (b < 256) {
        loss_block(S.red, P, b);
        return;
    }
    b -= 256;
#pragma unroll 1
    for (int l = 0; l < 4; ++l) {
        const GradLayer& L = P.layer[l];
        const int groups = L.n / 32, count = groups * L.slabs;
        if (b < count) {
            column_slab(S.part, L, (b % groups) * 32, b / groups, P.batch);
            return;
        }
        b -= count;
    }
}

// ---------------------------------------------------------------- update
namespace train {
struct Moments {
    float w, m, v;
};

__device__ __forceinline__ float adamw(const UpdateParams& P, const Moments& o, float* w, float* m, float* v, size_t i,
                                       float g, float wd)
{
    const float mi = P.b1 * o.m + (1.f - P.b1) * g;
    const float vi = P.b2 * o.v + (1.f - P.b2) * g * g;
    m[i] = mi;
    v[i] = vi;
    const float mh = mi / P.bc1, vh = vi / P.bc2;
    const float wi = o.w * (1.f - P.lr * wd) - P.lr * mh / (sqrtf(vh) + P.eps);
    w[i] = wi;
    return wi;
}

// p[0] + p[stride] + ... (n terms, summed in order), the terms' loads sixteen
// at a time in flight: one at a time the sum waits for L2 n times.
__device__ __forceinline__ float ordered_sum(const float* p, size_t stride, int n)
{
    float s = 0.f;
    for (int z0 = 0; z0 < n; z0 += 16) {
        float t[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) t[j] = z0 + j < n ? p[(size_t)(z0 + j) * stride] : 0.f;
#pragma unroll
        for (int j = 0; j < 16; ++j)
            if (z0 + j < n) s = z0 + j == 0 ? t[0] : s + t[j];
    }
    return s;
}
}  // namespace train

// A CTA updates 32 x 8 weights (the transposed copy leaves through shared
// memory in 64-byte rows) or, the last four CTAs, one layer's biases.  Five
// CTAs per SM take the 644 in one wave; with the four that unbounded registers
// allow a second wave held 36 of them (10.8 us, now 6.5).  The parameters too
// are read behind the wait: the step before wrote them, and only a kernel that
// has waited itself is promised to see what an earlier one of the chain wrote.
__global__ void __launch_bounds__(256, 5) train_update_kernel(const UpdateParams P)
{
    using namespace train;
    __shared__ bf16 tile[8][34];
    launch_dependents();
    int b = (int)blockIdx.x;
    const int tid = threadIdx.x;
#pragma unroll 1
    for (int l = 0; l < 4; ++l) {
        const UpdateLayer& L = P.layer[l];
        const int tn = L.n / 8, count = (L.k / 32) * tn;
        if (b < count) {
            const int r = (b / tn) * 32 + (tid >> 3), c = (b % tn) * 8 + (tid & 7);
            const size_t i = (size_t)r * L.n + c, mn = (size_t)L.k * L.n;
            dependency_wait();
            const Moments o{L.w[i], L.mw[i], L.vw[i]};
            const float g = ordered_sum(L.part + i, mn, L.splits);
            L.gw[i] = g;
            const bf16 h = __float2bfloat16(adamw(P, o, L.w, L.mw, L.vw, i, g, P.wd));
            L.w16[i] = h;
            tile[tid & 7][tid >> 3] = h;
            __syncthreads();
            L.wt16[(size_t)((b % tn) * 8 + (tid >> 5)) * L.k + (b / tn) * 32 + (tid & 31)] = tile[tid >> 5][tid & 31];
            return;
        }
        b -= count;
    }
    dependency_wait();
    const UpdateLayer& L = P.layer[b];
    for (int c = tid; c < L.n; c += 256) {
        const Moments o{L.b[c], L.mb[c], L.vb[c]};
        const float g = 0.f + ordered_sum(L.col + c, L.n, L.slabs);   // from +0, as the general kernel
        L.gb[c] = g;
        adamw(P, o, L.b, L.mb, L.vb, c, g, 0.0f);
    }
}

cudaError_t launch_train_step(const RowsParams& R, const GradsParams& G, const UpdateParams& U, bool keep,
                              cudaStream_t s)
{
    const void* rows = keep ? (const void*)train_rows_kernel<true> : (const void*)train_rows_kernel<false>;
    cudaError_t e = cudaFuncSetAttribute(rows, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)train::kRowsSmem);
    if (e != cudaSuccess) return e;
    int grads = 256, updates = 4;   // loss blocks; bias blocks
    for (const GradLayer& L : G.layer) grads += (L.k / 64) * (L.n / 64) * L.splits + (L.n / 32) * L.slabs;
    for (const UpdateLayer& L : U.layer) updates += (L.k / 32) * (L.n / 8);
    // chained from step to step: the first kernel too reads nothing before its wait
    void* ar[] = {const_cast<RowsParams*>(&R)};
    void* ag[] = {const_cast<GradsParams*>(&G)};
    void* au[] = {const_cast<UpdateParams*>(&U)};
    if ((e = launch_chained(rows, R.batch / train::kRows, train::kThreads, train::kRowsSmem, s, ar))) return e;
    if ((e = launch_chained((const void*)train_grads_kernel, grads, train::kGradThreads, 0, s, ag))) return e;
    return launch_chained((const void*)train_update_kernel, updates, 256, 0, s, au);
}

}  // namespace sfh
