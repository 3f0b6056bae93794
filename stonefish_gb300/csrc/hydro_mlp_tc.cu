// hydro_mlp_tc.cu -- fused inference of the wrench surrogate on the 5th-
// generation tensor cores: a CTA takes blocks of 128 states through all four
// layers (16 -> 256 -> 256 -> 256 -> 16) with the activations and the
// accumulators in tensor memory.
//
//   * persistent: a CTA per SM loops over pairs of 128-state blocks, both in
//     flight: while one block's epilogue runs, the tensor pipe works for the
//     other.  One block alone leaves the MUFU (one tanh per activation) idle
//     while its MMAs, their commits and waits run, a quarter of the time;
//   * each block has 128 accumulator columns and 128 columns of tensor
//     memory with its activations, two BF16 to a column, as the A operand:
//     an MMA then reads only its weights from shared memory (with the
//     activations there too, an M = 128, N = 256, K = 16 instruction caused 24
//     KB of shared-memory traffic, 190 cycles' worth for 128 of arithmetic);
//   * a layer runs as two halves of N = 128 columns.  The first half's
//     results wait in registers, since the activations they replace are still
//     the second half's operand, and both halves are written after it;
//   * weights are K-major BF16 in the 128-byte-swizzled canonical layout
//     (8-row x 128-byte atoms, 16-byte chunk c of row r stored at chunk
//     c ^ (r % 8)), packed once into that image in global memory
//     (pack_sw128_kernel).  The second layer's 128 KB and the last layer's
//     stay in shared memory; the first and third layers' stream through five
//     16 KB slots (64 columns of K by half the rows, contiguous in the
//     image) by 1-D bulk copies that a warp of its own keeps ahead, each
//     used for both blocks;
//   * one lane of a warp issues tcgen05.mma (FP32 accumulate);
//   * eight epilogue warps per block read its accumulator with tcgen05.ld
//     (warp w reads TMEM lanes 32 (w % 4) .. +31), add the bias, apply SiLU,
//     round to BF16 and write the next A operand with tcgen05.st;
//   * four more warps write the output rows (FP32 rows of 16, bias added) and
//     the next pair's features, loaded, normalised and rounded ahead.
//
// Bound: MUFU (2,048 cycles per block and hidden layer) and the tensor pipe
// (2,112), each with its hand-over: half a layer takes 1,450 cycles of either.
// 65,536 states: 36.8 us with one block in flight and its activations in
// shared memory, 28 us now (26.1 in a graph: 686 TFLOP/s, 35% of the measured
// 1,954).  With no more blocks than CTAs a CTA takes one, its halves in an
// accumulator each: 16,384 states 10.5 -> 9.8 us in a graph.
//
// Every mbarrier wait is bounded (%globaltimer); a timeout sets *err, the
// CTA stops issuing work, waits (bounded) for its tensor-core work and its
// copies to retire, frees its tensor memory and returns.
#include <algorithm>
#include <atomic>
#include <cstdint>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "hydro_chain.cuh"
#include "hydro_internal.h"

namespace sfh {

typedef __nv_bfloat16 bf16;

namespace tc {

constexpr int kRows = 128;      // states per CTA = UMMA M
constexpr int kHid = 256;
constexpr int kIn = 16;         // features = layer-0 K
constexpr int kOut = 16;        // output columns (6 used)
constexpr int kEpiWarps = 16;                   // epilogue warps
constexpr int kThreads = (kEpiWarps + 6) * 32;  // + MMA warp + weight-copy warp + four in/out warps
constexpr uint32_t kTmemCols = 512;

// shared-memory image (offsets from a 1024-byte-aligned base)
constexpr uint32_t kSlots = 5;
constexpr uint32_t kOffW1 = 0;                       // second layer: 256 x 256 bf16, 4 K-blocks of 32 KB
constexpr uint32_t kOffRing = kOffW1 + 4 * 32768;    // 128 weight rows x 64 columns of K per slot
constexpr uint32_t kOffW3 = kOffRing + kSlots * 16384;   // 16 x 256 bf16, 4 K-blocks of 2 KB
constexpr uint32_t kOffBias = kOffW3 + 4 * 2048;     // 3 x 256 + 16 floats
constexpr int kNormOff = 3 * kHid + kOut;            // feature means and inverse deviations
constexpr uint32_t kOffBar = kOffBias + (kNormOff + 2 * kIn) * 4;
constexpr uint32_t kBarRoom = 32 * 8;
constexpr uint32_t kOffTmem = kOffBar + kBarRoom;
constexpr uint32_t kSmemBytes = kOffTmem + 16 + 1024; // + alignment slack
static_assert(kSmemBytes <= 227 * 1024, "one CTA per SM");

// tensor memory columns of block t: accumulator, A operand
constexpr uint32_t kColD = 0, kColA = 256;      // + 128 t

// mbarriers (byte offsets from kOffBar; [2]: one per block in flight)
enum : uint32_t {
    kBarFull = 0,                         // [kSlots] a weight slot has arrived
    kBarFree = kBarFull + 8 * kSlots,     // [kSlots] the MMAs that read a slot have retired
    kBarD = kBarFree + 8 * kSlots,        // [2] half a hidden layer is in the accumulator
    kBarOut = kBarD + 16,                 // [2] the output layer is
    kBarDrained = kBarOut + 16,           // [2] the first half has been read from the accumulator
    kBarAct = kBarDrained + 16,           // [2] the second half too, and the next A operand is written
    kBarIn = kBarAct + 16,                // [2] the output has been read, the next features are written
    kBarW1 = kBarIn + 16,                 // [4] a K-block of the second layer's weights
    kBarFixed = kBarW1 + 32,              // the last layer's weights; at the end the last MMAs
    kBarEnd = kBarFixed + 8
};
static_assert(kBarEnd <= kBarRoom, "mbarrier room");

// global weight image (bytes)
constexpr uint32_t kImgW0 = 0;                       // 256 x 64 (K 16 used) = 32 KB
constexpr uint32_t kImgW1 = kImgW0 + 32768;
constexpr uint32_t kImgW2 = kImgW1 + 131072;
constexpr uint32_t kImgW3 = kImgW2 + 131072;         // 16 x 256 = 8 KB
constexpr uint32_t kImgBytes = kImgW3 + 8192;

__device__ __forceinline__ uint32_t sw128_offset(uint32_t rows, uint32_t r, uint32_t k)
{
    // byte offset of element (r, k) of a [rows x K] bf16 operand
    const uint32_t blk = k >> 6, kk = k & 63;
    return blk * rows * 128u + r * 128u + ((((kk >> 3) ^ (r & 7u)) & 7u) << 4) + ((kk & 7u) << 1);
}

__device__ __forceinline__ uint32_t smem_u32(const void* p)
{
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// tcgen05 shared-memory matrix descriptor: K-major, 128-byte swizzle,
// 8-row groups 1024 bytes apart (SBO), descriptor version 1.
__device__ __forceinline__ uint64_t sw128_desc(uint32_t saddr)
{
    uint64_t d = (uint64_t)((saddr & 0x3FFFFu) >> 4);
    d |= (uint64_t)1u << 16;                 // leading byte offset (unused by swizzled K-major)
    d |= (uint64_t)(1024u >> 4) << 32;       // stride byte offset
    d |= (uint64_t)1u << 46;                 // version
    d |= (uint64_t)2u << 61;                 // SWIZZLE_128B
    return d;
}

// instruction descriptor, kind::f16: BF16 A and B, FP32 D, both K-major
__host__ __device__ constexpr uint32_t idesc_bf16(uint32_t M, uint32_t N)
{
    return (1u << 4) | (1u << 7) | (1u << 10) | ((N >> 3) << 17) | ((M >> 4) << 24);
}

__device__ __forceinline__ uint64_t globaltimer()
{
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
                 : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}

// Bounded wait: gives up after limit_ns.  A try suspends the thread in
// hardware until the phase completes or a system-dependent time passes;
// sleeping between tries instead woke up to 1,700 cycles late.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, uint64_t limit_ns)
{
    if (mbar_try(bar, parity)) return true;
    const uint64_t t0 = globaltimer();
    for (;;) {
        for (int i = 0; i < 16; ++i)
            if (mbar_try(bar, parity)) return true;
        if (globaltimer() - t0 > limit_ns) return false;
    }
}

__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 :: "r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}

__device__ __forceinline__ void expect_tx(uint32_t bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" :: "r"(bar), "r"(bytes) : "memory");
}

// D[tmem_d] (+)= A[tmem_a] B[desc b]
__device__ __forceinline__ void mma(uint32_t tmem_d, uint32_t tmem_a, uint64_t b, uint32_t idesc, uint32_t acc)
{
    asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
                 " tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}\n"
                 :: "r"(tmem_d), "r"(tmem_a), "l"(b), "r"(idesc), "r"(acc) : "memory");
}

// One lane of a converged warp, in a form that the compiler knows to be a
// single one: behind a plain lane test every tcgen05.mma moved its operands
// to uniform registers by a loop over the active lanes and took 160 to 200
// cycles to issue, more than its 66 (N = 128) to execute.
__device__ __forceinline__ bool elect_one()
{
    uint32_t p;
    asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(p));
    return p != 0;
}

__device__ __forceinline__ void mma_commit(uint32_t bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                 :: "r"(bar) : "memory");
}

__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16])
{
    uint32_t r[16];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 "
                 "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
                   "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
                   "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32])
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                 "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
                 "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n"
                 "tcgen05.wait::ld.sync.aligned;"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
                   "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
                   "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]),
                   "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
                   "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
                 : "r"(taddr) : "memory");
}

__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16])
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
                 "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};\n"
                 "tcgen05.wait::st.sync.aligned;"
                 :: "r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]),
                    "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]),
                    "r"(r[15]) : "memory");
}

__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&r)[8])
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};\n"
                 "tcgen05.wait::st.sync.aligned;"
                 :: "r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                 : "memory");
}

__device__ __forceinline__ uint32_t pack2(float a, float b)
{
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" :: "r"(bar) : "memory");
}

// 32 accumulator columns col .. of this warp's rows: bias, then SiLU(z) =
// z sigmoid(z) = u + u tanh(u) with u = z / 2, two columns at a time with
// the packed FP32 instructions (each half rounds as the scalar operation
// would); one hardware tanh (tanh.approx.f32, relative error about 2^-11) per
// value, so the absolute error is at most |z| 2^-12, below the BF16 rounding
// that follows.
__device__ __forceinline__ void silu32(const uint32_t (&z)[32], const float* bias, uint32_t (&w)[16])
{
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const float2 b2 = *reinterpret_cast<const float2*>(bias + 2 * i);
        const float2 z2 = __fadd2_rn(make_float2(__uint_as_float(z[2 * i]), __uint_as_float(z[2 * i + 1])), b2);
        const float2 u2 = __fmul2_rn(z2, make_float2(0.5f, 0.5f));
        float t0, t1;
        asm("tanh.approx.f32 %0, %1;" : "=f"(t0) : "f"(u2.x));
        asm("tanh.approx.f32 %0, %1;" : "=f"(t1) : "f"(u2.y));
        const float2 s2 = __ffma2_rn(u2, make_float2(t0, t1), u2);
        w[i] = pack2(s2.x, s2.y);
    }
}

}  // namespace tc

// One network's parameters and output.
struct MlpNet {
    const float* fmean;
    const float* fistd;
    const unsigned char* wimg;
    const float* b[4];
    float* out;
};

struct MlpParams {
    const float* feats;
    uint32_t n;
    uint32_t n_nets;
    MlpNet net[2];
    unsigned* err;
};

// CTA c works for network c % n_nets on the groups of `both` 128-state
// blocks c / n_nets, + gridDim.x / n_nets, ...  (the grid is a multiple of
// n_nets).
template <uint32_t both>
__global__ void __launch_bounds__(tc::kThreads, 1) mlp_tc_kernel(const __grid_constant__ MlpParams P)
{
    using namespace tc;
    extern __shared__ unsigned char smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    unsigned char* base = smem_raw + (((raw + 1023u) & ~1023u) - raw);
    const uint32_t sb = smem_u32(base), bars = sb + kOffBar;
    float* bias = reinterpret_cast<float*>(base + kOffBias);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(base + kOffTmem);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const MlpNet& N = P.net[blockIdx.x % P.n_nets];
    const uint32_t n_blocks = (P.n + kRows - 1) / kRows;
    const uint32_t n_groups = (n_blocks + both - 1) / both;
    const uint32_t first = blockIdx.x / P.n_nets, stride = gridDim.x / P.n_nets;
    const uint64_t kLimit = 1000000000ull;   // 1 s per wait

    // Before the CTA's first barrier, each role starts what takes longest: the
    // weight copies, the feature loads, the tensor-memory allocation.
    uint32_t copied = 0;   // weight slots filled (the copy warp's elected lane)
    float raw_in[kIn];     // the first block's features (in/out warps, one block)
    if (warp == kEpiWarps + 1) {
        if (elect_one()) {
            for (uint32_t b = 0; b < kBarEnd; b += 8) {
                const uint32_t count = b >= kBarDrained && b < kBarIn ? 8u : b >= kBarIn && b < kBarW1 ? 4u : 1u;
                asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(bars + b), "r"(count) : "memory");
            }
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
            for (; copied < 2; ++copied) {
                expect_tx(bars + kBarFull + 8u * copied, 16384u);
                bulk_load(sb + kOffRing + 16384u * copied, N.wimg + kImgW0 + 16384u * copied, 16384u,
                          bars + kBarFull + 8u * copied);
            }
            for (uint32_t g = 0; g < 4; ++g) {
                expect_tx(bars + kBarW1 + 8u * g, 32768u);
                bulk_load(sb + kOffW1 + 32768u * g, N.wimg + kImgW1 + 32768u * g, 32768u, bars + kBarW1 + 8u * g);
            }
            expect_tx(bars + kBarFixed, 8192u);
            bulk_load(sb + kOffW3, N.wimg + kImgW3, 8192u, bars + kBarFixed);
        }
        __syncwarp();
    } else if (warp >= kEpiWarps + 2) {
        dependency_wait();   // the only warps that touch what an earlier kernel of the call writes
        if (both == 1u) {
            const uint32_t gr = first * (uint32_t)kRows + 32u * (uint32_t)(warp & 3) + (uint32_t)lane;
#pragma unroll
            for (int k = 0; k < kIn; ++k) raw_in[k] = gr < P.n ? P.feats[(size_t)gr * kIn + k] : 0.f;
        }
    } else {
        if (warp == 0) {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                         :: "r"(smem_u32(tmem_slot)), "r"(kTmemCols) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        }
        for (int i = tid; i < kHid; i += (kEpiWarps + 1) * 32) {
            bias[i] = N.b[0][i];
            bias[kHid + i] = N.b[1][i];
            bias[2 * kHid + i] = N.b[2][i];
        }
        if (tid < kOut) bias[3 * kHid + tid] = N.b[3][tid];
        if (tid < kIn) {
            bias[kNormOff + tid] = N.fmean[tid];
            bias[kNormOff + kIn + tid] = N.fistd[tid];
        }
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = *tmem_slot;

    bool ok = true;
    if (warp >= kEpiWarps + 2) {
        // ---- in/out warps: warp with quadrant q holds rows 32 q .. +31
        const uint32_t lanes = (32u * (uint32_t)(warp & 3)) << 16, row = 32u * (uint32_t)(warp & 3) + (uint32_t)lane;
        uint32_t x[both][8];
        auto normalise = [&](uint32_t t, uint32_t group, const float (&v)[kIn]) {
            const bool in = (both * group + t) * (uint32_t)kRows + row < P.n;
            const float* mean = bias + kNormOff;
            const float* istd = mean + kIn;
#pragma unroll
            for (int k = 0; k < 8; ++k)
                x[t][k] = in ? pack2((v[2 * k] - mean[2 * k]) * istd[2 * k],
                                     (v[2 * k + 1] - mean[2 * k + 1]) * istd[2 * k + 1]) : 0u;
        };
        auto load_in = [&](uint32_t t, uint32_t group) {
            const uint32_t gr = (both * group + t) * (uint32_t)kRows + row;
            float v[kIn];
#pragma unroll
            for (int k = 0; k < kIn; ++k) v[k] = gr < P.n ? P.feats[(size_t)gr * kIn + k] : 0.f;
            normalise(t, group, v);
        };
        auto store_in = [&](uint32_t t) {
            tmem_st8(tmem + kColA + 128u * t + lanes, x[t]);
            fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bars + kBarIn + 8u * t);
        };
#pragma unroll
        for (uint32_t t = 0; t < both; ++t) {
            if (both == 1u) normalise(t, first, raw_in);
            else load_in(t, first);
            store_in(t);
        }
        uint32_t k = 0;
#pragma unroll 1
        for (uint32_t group = first; group < n_groups && ok; group += stride, ++k) {
            const bool more = group + stride < n_groups;
#pragma unroll
            for (uint32_t t = 0; t < both; ++t)
                if (more) load_in(t, group + stride);
#pragma unroll
            for (uint32_t t = 0; t < both; ++t) {
                const uint32_t blk = both * group + t;
                if (blk >= n_blocks || !ok) break;
                ok = mbar_wait(bars + kBarOut + 8u * t, k & 1u, kLimit);
                if (!ok) break;
                fence_after();
                float v[16];
                tmem_ld16(tmem + kColD + 128u * t + lanes, v);
                if (more) store_in(t);
                const uint32_t gr = blk * (uint32_t)kRows + row;
                if (gr < P.n) {
                    float4* o = reinterpret_cast<float4*>(N.out + (size_t)gr * kOut);
                    const float* bb = bias + 3 * kHid;
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        o[i] = make_float4(v[4 * i] + bb[4 * i], v[4 * i + 1] + bb[4 * i + 1],
                                           v[4 * i + 2] + bb[4 * i + 2], v[4 * i + 3] + bb[4 * i + 3]);
                }
            }
        }
        if (!ok && lane == 0) atomicOr(P.err, 1u);
    } else if (warp == kEpiWarps + 1) {
        // ---- weight copies, in the order the MMA warp uses them
        if (elect_one()) {
            uint32_t use = copied;
            auto copy = [&](const unsigned char* src) {
                const uint32_t s = use % kSlots;
                if (ok && use >= kSlots) ok = mbar_wait(bars + kBarFree + 8u * s, (use / kSlots - 1u) & 1u, kLimit);
                if (!ok) return;
                expect_tx(bars + kBarFull + 8u * s, 16384u);
                bulk_load(sb + kOffRing + 16384u * s, src, 16384u, bars + kBarFull + 8u * s);
                ++use;
            };
#pragma unroll 1
            for (uint32_t group = first; group < n_groups && ok; group += stride) {
                if (group != first) {
                    copy(N.wimg + kImgW0);
                    copy(N.wimg + kImgW0 + 16384u);
                }
#pragma unroll 1
                for (uint32_t i = 0; i < 8; ++i)   // half i / 4, K-block i % 4
                    copy(N.wimg + kImgW2 + 32768u * (i & 3u) + 16384u * (i >> 2));
            }
            // every copy has landed before the CTA may end (bounded)
            for (uint32_t u = use > kSlots ? use - kSlots : 0u; u < use; ++u)
                if (!mbar_wait(bars + kBarFull + 8u * (u % kSlots), (u / kSlots) & 1u, kLimit)) ok = false;
            if (!ok) atomicOr(P.err, 1u);
        }
        __syncwarp();
    } else if (warp == kEpiWarps) {
        // ---- MMA warp: one lane issues every MMA
        if (elect_one()) {
            const uint32_t id_half = idesc_bf16(128, 128), id_out = idesc_bf16(128, kOut);
            const uint64_t ring = sw128_desc(sb + kOffRing), w1 = sw128_desc(sb + kOffW1), w3 = sw128_desc(sb + kOffW3);
            uint32_t use = 0, k = 0;
            bool fixed = false;
#pragma unroll 1
            for (uint32_t group = first; group < n_groups && ok; group += stride, ++k) {
                if (both == 1u) {
                    // One block: its halves have an accumulator each.  The next
                    // layer's first half starts on the first half of K while the
                    // epilogue is at the second.
                    ok = mbar_wait(bars + kBarIn, k & 1u, kLimit);
#pragma unroll 1
                    for (uint32_t h = 0; h < 2 && ok; ++h, ++use) {   // K = 16
                        const uint32_t s = use % kSlots;
                        ok = mbar_wait(bars + kBarFull + 8u * s, (use / kSlots) & 1u, kLimit);
                        if (!ok) break;
                        fence_after();
                        mma(tmem + kColD + 128u * h, tmem + kColA, ring + 1024u * s, id_half, 0u);
                        mma_commit(bars + kBarD + 8u * h);
                        mma_commit(bars + kBarFree + 8u * s);
                    }
#pragma unroll 1
                    for (uint32_t l = 1; l < 3 && ok; ++l) {
                        if (l == 1 && !fixed)
                            for (uint32_t g = 0; g < 4 && ok; ++g) ok = mbar_wait(bars + kBarW1 + 8u * g, 0u, kLimit);
#pragma unroll 1
                        for (uint32_t q = 0; q < 4 && ok; ++q) {   // half q / 2 over half q % 2 of K
                            const uint32_t h = q >> 1, g = 2u * (q & 1u);
                            const uint32_t d = tmem + kColD + 128u * h, a = tmem + kColA + 32u * g;
                            uint64_t w[2] = {w1 + 2048u * g + 1024u * h, w1 + 2048u * (g + 1u) + 1024u * h};
                            if (q < 2) ok = mbar_wait(bars + kBarAct + 8u * q, (3u * k + l - 1u) & 1u, kLimit);
                            if (l == 2)
#pragma unroll
                                for (uint32_t e = 0; e < 2; ++e) {
                                    const uint32_t s = (use + e) % kSlots;
                                    w[e] = ring + 1024u * s;
                                    ok = ok && mbar_wait(bars + kBarFull + 8u * s, ((use + e) / kSlots) & 1u, kLimit);
                                }
                            if (!ok) break;
                            fence_after();
#pragma unroll
                            for (uint32_t j = 0; j < 8; ++j)
                                mma(d, a + 8u * j, w[j >> 2] + 2u * (j & 3u), id_half, (g | j) ? 1u : 0u);
                            if (q & 1u) mma_commit(bars + kBarD + 8u * h);
                            if (l == 2)
                                for (uint32_t e = 0; e < 2; ++e, ++use) mma_commit(bars + kBarFree + 8u * (use % kSlots));
                        }
                    }
                    if (ok && !fixed) {
                        ok = mbar_wait(bars + kBarFixed, 0u, kLimit);
                        fixed = ok;
                    }
                    for (uint32_t h = 0; h < 2 && ok; ++h)
                        ok = mbar_wait(bars + kBarAct + 8u * h, (3u * k + 2u) & 1u, kLimit);
                    if (!ok) break;
                    fence_after();
#pragma unroll
                    for (uint32_t i = 0; i < 16; ++i)
                        mma(tmem + kColD, tmem + kColA + 8u * i, w3 + 128u * (i >> 2) + 2u * (i & 3u), id_out, i ? 1u : 0u);
                    mma_commit(bars + kBarOut);
                    continue;
                }
                const uint32_t nt = min(2u, n_blocks - 2u * group);
                // first layer, K = 16
#pragma unroll 1
                for (uint32_t h = 0; h < 2 && ok; ++h, ++use) {
                    const uint32_t s = use % kSlots;
                    ok = mbar_wait(bars + kBarFull + 8u * s, (use / kSlots) & 1u, kLimit);
#pragma unroll 1
                    for (uint32_t t = 0; t < nt && ok; ++t) {
                        ok = h == 0 ? mbar_wait(bars + kBarIn + 8u * t, k & 1u, kLimit)
                                    : mbar_wait(bars + kBarDrained + 8u * t, (3u * k) & 1u, kLimit);
                        if (!ok) break;
                        fence_after();
                        mma(tmem + kColD + 128u * t, tmem + kColA + 128u * t, ring + 1024u * s, id_half, 0u);
                        mma_commit(bars + kBarD + 8u * t);
                    }
                    mma_commit(bars + kBarFree + 8u * s);
                }
#pragma unroll 1
                for (uint32_t lh = 2; lh < 6 && ok; ++lh) {   // layer lh / 2, half lh % 2
                    const uint32_t l = lh >> 1, h = lh & 1u;
#pragma unroll 1
                    for (uint32_t t = 0; t < nt && ok; ++t) {
                        // block t's operand is written and its accumulator free
                        ok = h == 0 ? mbar_wait(bars + kBarAct + 8u * t, (3u * k + l - 1u) & 1u, kLimit)
                                    : mbar_wait(bars + kBarDrained + 8u * t, (3u * k + l) & 1u, kLimit);
                        if (!ok) break;
                        fence_after();
                        const uint32_t d = tmem + kColD + 128u * t, a = tmem + kColA + 128u * t;
#pragma unroll 1
                        for (uint32_t g = 0; g < 4; ++g) {
                            const uint32_t s = (use + g) % kSlots;
                            uint64_t w = w1 + 2048u * g + 1024u * h;   // descriptors count 16 bytes
                            if (l == 1 && !fixed) {   // the first group's second layer
                                ok = mbar_wait(bars + kBarW1 + 8u * g, 0u, kLimit);
                                if (!ok) break;
                            }
                            if (l == 2) {
                                w = ring + 1024u * s;
                                if (t == 0) ok = mbar_wait(bars + kBarFull + 8u * s, ((use + g) / kSlots) & 1u, kLimit);
                                if (!ok) break;
                            }
#pragma unroll
                            for (uint32_t j = 0; j < 4; ++j)
                                mma(d, a + 32u * g + 8u * j, w + 2u * j, id_half, (g | j) ? 1u : 0u);
                            if (l == 2 && t + 1u == nt) mma_commit(bars + kBarFree + 8u * s);
                        }
                        if (!ok) break;
                        mma_commit(bars + kBarD + 8u * t);
                    }
                    if (l == 2) use += 4u;
                }
                if (ok && !fixed) {
                    ok = mbar_wait(bars + kBarFixed, 0u, kLimit);
                    fixed = ok;
                }
                // output layer, N = 16
#pragma unroll 1
                for (uint32_t t = 0; t < nt && ok; ++t) {
                    ok = mbar_wait(bars + kBarAct + 8u * t, (3u * k + 2u) & 1u, kLimit);
                    if (!ok) break;
                    fence_after();
#pragma unroll
                    for (uint32_t i = 0; i < 16; ++i)
                        mma(tmem + kColD + 128u * t, tmem + kColA + 128u * t + 8u * i, w3 + 128u * (i >> 2) + 2u * (i & 3u),
                            id_out, i ? 1u : 0u);
                    mma_commit(bars + kBarOut + 8u * t);
                }
            }
            if (!ok) atomicOr(P.err, 1u);
            // issued tensor-core work retires before the tensor memory is
            // freed (bounded): one more commit, on the barrier whose only
            // phase so far was the last layer's weights', after the copies
            // that were not waited for
            if (!fixed) {
                for (uint32_t g = 0; g < 4; ++g) mbar_wait(bars + kBarW1 + 8u * g, 0u, kLimit);
                mbar_wait(bars + kBarFixed, 0u, kLimit);
            }
            mma_commit(bars + kBarFixed);
            if (!mbar_wait(bars + kBarFixed, 1u, kLimit)) atomicOr(P.err, 1u);
        }
        __syncwarp();
    } else {
        // ---- epilogue warps: block t = warp / 8, columns 64 sub .. +63 of each half
        const uint32_t t = (uint32_t)warp >> 3, sub = ((uint32_t)warp >> 2) & 1u;
        const uint32_t lanes = (32u * (uint32_t)(warp & 3)) << 16;
        const uint32_t d = tmem + kColD + 128u * t + lanes + 64u * sub, a = tmem + kColA + 128u * t + lanes + 32u * sub;
        uint32_t k = 0;
        if (both == 1u) {
            // one block: warps 0..7 take its first half, 8..15 its second
            const uint32_t a1 = tmem + kColA + lanes + 64u * t + 32u * sub;
#pragma unroll 1
            for (uint32_t blk = first; blk < n_blocks && ok; blk += stride, ++k) {
#pragma unroll 1
                for (uint32_t l = 0; l < 3; ++l) {
                    const float* b = bias + l * kHid + 128u * t + 64u * sub;
                    const uint32_t par = (3u * k + l) & 1u;
                    uint32_t z[32], w0[16], w1[16];
                    ok = mbar_wait(bars + kBarD + 8u * t, par, kLimit);
                    if (!ok) break;
                    fence_after();
                    tmem_ld32(d, z);
                    silu32(z, b, w0);
                    tmem_ld32(d + 32u, z);
                    silu32(z, b + 32, w1);
                    if (t == 0u) ok = mbar_wait(bars + kBarD + 8u, par, kLimit);   // the A operand is free now
                    if (!ok) break;
                    fence_after();
                    tmem_st16(a1, w0);
                    tmem_st16(a1 + 16u, w1);
                    fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(bars + kBarAct + 8u * t);
                }
            }
        }
#pragma unroll 1
        for (uint32_t group = first; both == 2u && 2u * group + t < n_blocks && ok; group += stride, ++k) {
#pragma unroll 1
            for (uint32_t l = 0; l < 3; ++l) {
                const float* b = bias + l * kHid + 64u * sub;
                uint32_t z[32], w0[16], w1[16];
                ok = mbar_wait(bars + kBarD + 8u * t, 0u, kLimit);   // six phases a group: halves alternate
                if (!ok) break;
                fence_after();
                tmem_ld32(d, z);
                silu32(z, b, w0);
                tmem_ld32(d + 32u, z);
                fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(bars + kBarDrained + 8u * t);
                silu32(z, b + 32, w1);
                ok = mbar_wait(bars + kBarD + 8u * t, 1u, kLimit);   // the A operand is free now
                if (!ok) break;
                fence_after();
                tmem_st16(a, w0);
                tmem_st16(a + 16u, w1);
                tmem_ld32(d, z);
                silu32(z, b + 128, w0);
                tmem_ld32(d + 32u, z);
                tmem_st16(a + 64u, w0);
                silu32(z, b + 160, w1);
                tmem_st16(a + 80u, w1);
                fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(bars + kBarAct + 8u * t);
            }
        }
        if (!ok && lane == 0) atomicOr(P.err, 1u);
    }
    fence_before();
    __syncthreads();
    if (warp == 0) {
        fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(kTmemCols) : "memory");
    }
}

// dst = 128-byte-swizzled K-major image of src[rows][K] (row stride ld),
// K padded with zeros to kpad (a multiple of 64); one thread per 16 bytes.
__global__ void pack_sw128_kernel(const bf16* __restrict__ src, int rows, int K, int ld, int kpad,
                                  unsigned char* __restrict__ dst)
{
    const uint32_t chunks = (uint32_t)rows * (uint32_t)(kpad / 8);
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= chunks) return;
    const uint32_t r = i / (uint32_t)(kpad / 8), k0 = (i % (uint32_t)(kpad / 8)) * 8u;
    uint16_t v[8];
    const uint16_t* s = reinterpret_cast<const uint16_t*>(src);
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = (k0 + j < (uint32_t)K) ? s[(size_t)r * ld + k0 + j] : (uint16_t)0;
    uint4 w;
    w.x = v[0] | ((uint32_t)v[1] << 16);
    w.y = v[2] | ((uint32_t)v[3] << 16);
    w.z = v[4] | ((uint32_t)v[5] << 16);
    w.w = v[6] | ((uint32_t)v[7] << 16);
    *reinterpret_cast<uint4*>(dst + tc::sw128_offset((uint32_t)rows, r, k0)) = w;
}

cudaError_t launch_pack_sw128(const void* src, int rows, int K, int ld, int kpad, void* dst, cudaStream_t s)
{
    if (rows <= 0 || K <= 0 || kpad % 64 || K > kpad || ld < K) return cudaErrorInvalidValue;
    const uint32_t chunks = (uint32_t)rows * (uint32_t)(kpad / 8);
    pack_sw128_kernel<<<(chunks + 255) / 256, 256, 0, s>>>(static_cast<const bf16*>(src), rows, K, ld, kpad,
                                                           static_cast<unsigned char*>(dst));
    return cudaGetLastError();
}

size_t mlp_tc_image_bytes() { return tc::kImgBytes; }

// The kernel's shared-memory attribute and the SM count, once per device
// (first 16): host calls that would otherwise precede every launch.
static cudaError_t mlp_sms(int* sms)
{
    constexpr int kDevCache = 16;
    static std::atomic<int> known[kDevCache];
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < kDevCache && (*sms = known[dev].load(std::memory_order_acquire)) > 0) return cudaSuccess;
    e = cudaFuncSetAttribute(mlp_tc_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tc::kSmemBytes);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(mlp_tc_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tc::kSmemBytes);
    if (e != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
    if (dev < kDevCache) known[dev].store(*sms, std::memory_order_release);
    return cudaSuccess;
}

// chained: behind the kernel that writes the features, in the same call.  The
// kernel itself does not trigger early: its CTAs fill their SMs, so that what
// follows would be placed on the few that have none (16,384 states, 128 CTAs:
// a rollout step 83 -> 88 us).
static cudaError_t launch_mlp(const MlpParams& P, cudaStream_t s, bool chained)
{
    int sms = 1;
    const cudaError_t e = mlp_sms(&sms);
    if (e != cudaSuccess) return e;
    // one CTA per SM; two blocks in flight where there are more than CTAs
    const uint32_t blocks = (P.n + tc::kRows - 1) / tc::kRows;
    const uint32_t per_net = std::max(1u, (uint32_t)sms / P.n_nets);
    void* args[] = {const_cast<MlpParams*>(&P)};
    if (blocks > per_net)
        return launch_chained((const void*)mlp_tc_kernel<2>, std::min((blocks + 1) / 2, per_net) * P.n_nets,
                              tc::kThreads, tc::kSmemBytes, s, args, chained);
    return launch_chained((const void*)mlp_tc_kernel<1>, blocks * P.n_nets, tc::kThreads, tc::kSmemBytes, s, args,
                          chained);
}

cudaError_t launch_mlp_tc(const float* feats, uint32_t n, const float* fmean, const float* fistd,
                          const void* wimg, const float* b0, const float* b1, const float* b2, const float* b3,
                          float* out, unsigned* err, cudaStream_t s)
{
    if (n == 0) return cudaSuccess;
    MlpParams P{feats, n, 1u, {}, err};
    P.net[0] = MlpNet{fmean, fistd, static_cast<const unsigned char*>(wimg), {b0, b1, b2, b3}, out};
    return launch_mlp(P, s, false);
}

cudaError_t launch_mlp_nets(const float* feats, uint32_t n, const PredictNet* nets, int n_nets, unsigned* err,
                            cudaStream_t s)
{
    if (n == 0) return cudaSuccess;
    MlpParams P{feats, n, (uint32_t)n_nets, {}, err};
    for (int k = 0; k < n_nets; ++k) {
        const PredictNet& N = nets[k];
        P.net[k] = MlpNet{N.fmean, N.fistd, static_cast<const unsigned char*>(N.image), {N.b[0], N.b[1], N.b[2], N.b[3]},
                          N.z};
    }
    return launch_mlp(P, s, true);
}

}  // namespace sfh
