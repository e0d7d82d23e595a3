// Prefill GEMM: fused NVFP4 dequantisation + tcgen05 GEMM on pairs of SMs.
//
//   C[M,N] = bf16( A[M,K] * W[N,K]^T (+ residual) ),  W = e2m1(code) * ue4m3(scale) / global_scale
//
// The weights are the M side of the MMA and are expanded straight into tensor memory; the tokens are the N side.  A
// cluster of two CTAs works on one tile of 256 weight rows x T tokens (tcgen05.mma.cta_group::2: M = 256, N = T, K = 16):
// each CTA expands 128 of the rows into its own tensor memory and stages T/2 of the tokens in its own shared memory, and
// the tensor cores of both read the two halves.  Where the shape allows, a work item is two row tiles on the same tokens
// (512 x T: one accumulator each, every staged token block used twice).
//   warp 0      TMA: raw weight stages (128 rows x 256 k: 16 KB codes, 2 KB scales) of this CTA, barriers of this CTA.
//   warp 2      TMA: token blocks (T/2 x 64 k, FP16, 128-byte swizzle); both CTAs' blocks complete on the leader's barrier.
//   warps 8-15  dequantise: thread = weight row = TMEM lane; every other unit each group, cvt.rn.f16x2.e2m1x2 + one f16x2 multiply by
//               the block scale (exact), tcgen05.st into a ring of A units; arrive on the leader's barrier.
//   warps 1, 3  of the leader CTA issue the MMAs, one row tile or every other unit each; commits free the A units and token stages, in
//               both CTAs.
//   warps 4-7, 16-19  epilogue: thread = weight row, registers = tokens: a warp stores 32 consecutive outputs of one token.
//
// What bounds it and why this form.  With both operands in shared memory (128 tokens x 256 rows per CTA, a dequantised block
// for one or two token tiles) the shared memory was the bound: per 128 x 256 x 64 block the MMA reads 96 B/clk, the
// dequantised block's stores 32-64, TMA and raw weights 50-70, of 128 B/clk.  From tensor memory the weights cost no
// shared-memory bandwidth, and a pair of SMs stages each token once: 60-80 B/clk.  T is any multiple of 32, so 149 tokens are one
// tile of 160 instead of two of 128.  Then the hand-overs were the bound: a wait that finds its phase complete costs a warp 60-130
// clocks, a commit 75, and a group of dequantising warps spent 800 clocks on 64 k of every unit, 250 of them on arithmetic.  Now a
// group takes whole units in turn (128 k: one wait, one arrival), where tensor memory leaves only two of those (T = 160, 192; FINE)
// units of 64 k, and commits reach both CTAs' barriers themselves (a warp that passed them on came 200 clocks later).  Issuers at
// T = 128 / 160 / 192: 100 / 100 / 120 clocks an MMA -> 75 / 81 / 110.  What bounds it now is the issue of the MMAs for T <= 128, the way
// around the A ring at T = 192, draining the accumulators (5-8 thousand clocks an item), and the power cap for long runs.
// Measured, before whole units in turn -> now, pre-pass included, weights from memory, calls back to back in short bursts on one box:
// 34816 x 5120 at 100 / 149 / 256 / 512 / 1111 / 2048 tokens 50.2 -> 45.2, 54.6 -> 49.8, 90.5 -> 80.8, 151 -> 146, 282 -> 267, 497 -> 476 us;
// 5120 x 17408 with a residual at 149 / 256 / 1111 40.3 -> 37.5, 59.7 -> 54.2, 165 -> 146; BF16 5120 x 5120 at 100 / 512 20.3 -> 19.2,
// 37.4 -> 32.6, 34816 x 5120 at 4096 1107 -> 1054, with a residual 1247 -> 1123.
//
// Operands are FP16 because the hardware E2M1 conversion produces FP16 and every e2m1 x ue4m3 product is exact in FP16
// (kind::f16 takes both operands in ONE 16-bit format).  A pre-pass turns the BF16 activations into FP16 with an exact
// per-token power-of-two scale in the handle workspace.
//
// Work items left over after whole waves may be split along k (pair_plan.h): partial tiles in FP32 with a flag per part, every
// participant then sums its own slice of the tile in a fixed order (deterministic).
//
// DENSE: the weight is BF16 [N,K] and the activations are the caller's BF16 rows; the weight blocks (128 rows x 64 k)
// come by TMA as the shared-memory A operand and nothing is dequantised.
//
// Every mbarrier wait is bounded: a wait that runs out records its code in the handle's status word and the kernel winds
// down (both CTAs reach the closing cluster barrier, TMEM is always freed).
#include <cuda.h>
#include <cmath>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "nvfp4_format.cuh"
#include "nvfp4_internal.h"
#include "pair_plan.h"
#include "ptx.cuh"
#include "umma.cuh"

namespace nvfp4 {
namespace {

using namespace pair;
using namespace umma;

constexpr int kThreads = 640;
constexpr int kGroupWarps = 4, kEpiWarps = 4;  // two dequantising groups of four warps (one per TMEM lane quarter)
constexpr int kMaxT = 256;                     // columns a partial slot has room for
constexpr int kSlotFloats = TR * kMaxT;        // one FP32 partial: [token][row]

struct PairParams : Plan {
    const __nv_bfloat16* residual;
    __nv_bfloat16* C;
    const float* unscale;      // per token: 1 / activation scale (null: BF16 weights)
    unsigned int* status;
    float* partials;           // [grid][2][kSlotFloats]
    unsigned int* flags;       // [grid][2], the launch's tag once that partial is stored
    uint32_t idesc;
    float inv_gs;
    float out_mul;             // what the epilogue multiplies the sums by besides the token factor: 2^8 / gs, or 1 / wshift
    float wshift;              // WROUND: the power of two that keeps the rounded weights in FP16's normal range
    int swiglu_out;            // weight rows interleaved in slabs of 16 (8 gate, 8 up): C is [M, N/2] = bf16(silu(gate) * up)
    int out_f32;               // C is FP32 [M,N]: the scaled sums unrounded, no residual
};

enum Mode { kExact = 0, kRounded = 1, kDense = 2 };

// Position in a ring of buffers and the phase its barriers are in.
struct Ring {
    int i, n;
    uint32_t phase;
    __device__ __forceinline__ explicit Ring(int size) : i(0), n(size), phase(0) {}
    __device__ __forceinline__ void advance(int by) {          // by <= n
        i += by;
        if (i >= n) { i -= n; phase ^= 1u; }
    }
};

// ---------------------------------------------------------------- tcgen05, CTA pairs
// The MMAs of a unit on one accumulator, which the first clears when `accumulate` is 0, from one elected lane of a converged warp: eight
// (128 k, B in two blocks `step` 16-byte units apart) or the four of one block (64 k).  A from tensor memory (8 columns per MMA) or from
// shared memory (two blocks 16 KB apart, or one).  Election and address arithmetic sit inside one asm block: the issuing warp
// shares its scheduler and instruction cache with the dequantising warps, and every instruction of its loop counts.
__device__ __forceinline__ void mma8_ts(uint32_t d, uint32_t a, uint64_t b, uint32_t step, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, q, t;\n\t.reg .b32 a1, a2, a3, a4, a5, a6, a7;\n\t.reg .b64 s, b1, b2, b3, b4, b5, b6, b7;\n\t"
        "setp.ne.b32 p, %4, 0;\n\tsetp.eq.u32 t, 0, 0;\n\tcvt.u64.u32 s, %5;\n\t"
        "add.u32 a1, %1, 8;\n\tadd.u32 a2, %1, 16;\n\tadd.u32 a3, %1, 24;\n\tadd.u32 a4, %1, 32;\n\t"
        "add.u32 a5, %1, 40;\n\tadd.u32 a6, %1, 48;\n\tadd.u32 a7, %1, 56;\n\t"
        "add.u64 b1, %2, 2;\n\tadd.u64 b2, %2, 4;\n\tadd.u64 b3, %2, 6;\n\tadd.u64 b4, %2, s;\n\t"
        "add.u64 b5, b4, 2;\n\tadd.u64 b6, b4, 4;\n\tadd.u64 b7, b4, 6;\n\t"
        "elect.sync _|q, 0xffffffff;\n\t"
        "@q tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t"
        "@q tcgen05.mma.cta_group::2.kind::f16 [%0], [a1], b1, %3, t;\n\t"
        "@q tcgen05.mma.cta_group::2.kind::f16 [%0], [a2], b2, %3, t;\n\t"
        "@q tcgen05.mma.cta_group::2.kind::f16 [%0], [a3], b3, %3, t;\n\t"
        "@q tcgen05.mma.cta_group::2.kind::f16 [%0], [a4], b4, %3, t;\n\t"
        "@q tcgen05.mma.cta_group::2.kind::f16 [%0], [a5], b5, %3, t;\n\t"
        "@q tcgen05.mma.cta_group::2.kind::f16 [%0], [a6], b6, %3, t;\n\t"
        "@q tcgen05.mma.cta_group::2.kind::f16 [%0], [a7], b7, %3, t;\n\t}"
        ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(accumulate), "r"(step)
        : "memory");
}
__device__ __forceinline__ void mma4_ts(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, q, t;\n\t.reg .b32 a1, a2, a3;\n\t.reg .b64 b1, b2, b3;\n\t"
        "setp.ne.b32 p, %4, 0;\n\tsetp.eq.u32 t, 0, 0;\n\t"
        "add.u32 a1, %1, 8;\n\tadd.u32 a2, %1, 16;\n\tadd.u32 a3, %1, 24;\n\t"
        "add.u64 b1, %2, 2;\n\tadd.u64 b2, %2, 4;\n\tadd.u64 b3, %2, 6;\n\t"
        "elect.sync _|q, 0xffffffff;\n\t"
        "@q tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t"
        "@q tcgen05.mma.cta_group::2.kind::f16 [%0], [a1], b1, %3, t;\n\t"
        "@q tcgen05.mma.cta_group::2.kind::f16 [%0], [a2], b2, %3, t;\n\t"
        "@q tcgen05.mma.cta_group::2.kind::f16 [%0], [a3], b3, %3, t;\n\t}"
        ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void mma8_ss(uint32_t d, uint64_t a, uint64_t b, uint32_t step, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, q, t;\n\t.reg .b64 s, a1, a2, a3, a4, a5, a6, a7, b1, b2, b3, b4, b5, b6, b7;\n\t"
        "setp.ne.b32 p, %4, 0;\n\tsetp.eq.u32 t, 0, 0;\n\tcvt.u64.u32 s, %5;\n\t"
        "add.u64 a1, %1, 2;\n\tadd.u64 a2, %1, 4;\n\tadd.u64 a3, %1, 6;\n\tadd.u64 a4, %1, 1024;\n\t"
        "add.u64 a5, a4, 2;\n\tadd.u64 a6, a4, 4;\n\tadd.u64 a7, a4, 6;\n\t"
        "add.u64 b1, %2, 2;\n\tadd.u64 b2, %2, 4;\n\tadd.u64 b3, %2, 6;\n\tadd.u64 b4, %2, s;\n\t"
        "add.u64 b5, b4, 2;\n\tadd.u64 b6, b4, 4;\n\tadd.u64 b7, b4, 6;\n\t"
        "elect.sync _|q, 0xffffffff;\n\t"
        "@q tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t"
        "@q tcgen05.mma.cta_group::2.kind::f16 [%0], a1, b1, %3, t;\n\t"
        "@q tcgen05.mma.cta_group::2.kind::f16 [%0], a2, b2, %3, t;\n\t"
        "@q tcgen05.mma.cta_group::2.kind::f16 [%0], a3, b3, %3, t;\n\t"
        "@q tcgen05.mma.cta_group::2.kind::f16 [%0], a4, b4, %3, t;\n\t"
        "@q tcgen05.mma.cta_group::2.kind::f16 [%0], a5, b5, %3, t;\n\t"
        "@q tcgen05.mma.cta_group::2.kind::f16 [%0], a6, b6, %3, t;\n\t"
        "@q tcgen05.mma.cta_group::2.kind::f16 [%0], a7, b7, %3, t;\n\t}"
        ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate), "r"(step)
        : "memory");
}
__device__ __forceinline__ void mma4_ss(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, q, t;\n\t.reg .b64 a1, a2, a3, b1, b2, b3;\n\t"
        "setp.ne.b32 p, %4, 0;\n\tsetp.eq.u32 t, 0, 0;\n\t"
        "add.u64 a1, %1, 2;\n\tadd.u64 a2, %1, 4;\n\tadd.u64 a3, %1, 6;\n\t"
        "add.u64 b1, %2, 2;\n\tadd.u64 b2, %2, 4;\n\tadd.u64 b3, %2, 6;\n\t"
        "elect.sync _|q, 0xffffffff;\n\t"
        "@q tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t"
        "@q tcgen05.mma.cta_group::2.kind::f16 [%0], a1, b1, %3, t;\n\t"
        "@q tcgen05.mma.cta_group::2.kind::f16 [%0], a2, b2, %3, t;\n\t"
        "@q tcgen05.mma.cta_group::2.kind::f16 [%0], a3, b3, %3, t;\n\t}"
        ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
        : "memory");
}
// Arrives on the leader's barrier at this shared-memory address once all MMAs issued so far have completed, in both CTAs
// (converged warp).
__device__ __forceinline__ void commit_leader(uint32_t bar) {
    asm volatile(
        "{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\t"
        "@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(bar) : "memory");
}
// ... and on the same barrier of the other CTA, `other` bytes on in the cluster's shared memory.
__device__ __forceinline__ void commit_pair(uint32_t bar, uint32_t other) {
    asm volatile(
        "{\n\t.reg .pred q;\n\t.reg .b32 r;\n\tadd.u32 r, %0, %1;\n\telect.sync _|q, 0xffffffff;\n\t"
        "@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t"
        "@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [r];\n\t}" ::"r"(bar), "r"(other) : "memory");
}
// The leader's barrier has completed a phase: complete the same one of the other CTA.  For the token stages, whose ring is deep; a
// commit of the issuers' own costs them 70 clocks more.
__device__ __forceinline__ void relay(uint64_t* bar) {
    tc_fence_after();
    tc_fence_before();
    ptx::mbar_arrive_cluster(ptx::mapa_shared(ptx::smem_u32(bar), 1));
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
        "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
          "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// For whole, converged warps (.sync.aligned): lanes that come from a wait, or from rows beyond the weight, one by one are brought together by
// a __syncwarp() or a vote first.
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// ---------------------------------------------------------------- outputs
__device__ __forceinline__ float token_factor(const PairParams& p, int m) { return p.unscale ? p.unscale[m] * p.out_mul : 1.0f; }
__device__ __forceinline__ float silu_pair(float gate, float up) {     // both already scaled; rounded as separate kernels would store them
    return silu(__bfloat162float(__float2bfloat16_rn(gate))) * __bfloat162float(__float2bfloat16_rn(up));
}
__device__ __forceinline__ void store4(__nv_bfloat16* dst, float a, float b, float c, float d) {
    const __nv_bfloat162 lo = __floats2bfloat162_rn(a, b), hi = __floats2bfloat162_rn(c, d);
    *reinterpret_cast<uint2*>(dst) = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
}

// SPLIT: what the plan left to split by k.  An instantiation each, because the registers run out (96 a thread): with the code of
// parts and reduction in one kernel every call paid for its spills, 0.5-1 us (149 x 5120 x 17408 35.7 -> 34.4 us, BF16 100 x 5120 x 5120
// 19.1 -> 17.9), and whole items had none left to ask for the residual a chunk ahead (2048 x 5120 x 5120 with a residual 92 -> 83.4).
// Split tiles behind whole waves have it all, hence one for calls with a residual (which have neither SwiGLU nor FP32 outputs) and one for
// those without: in one, the residual was waited for element by element (2048 x 17408 x 5120 with one 385 us).
enum Split { kWhole = 0, kAllSplit = 1, kTailSplit = 2, kTailSplitRes = 3 };

// Every participant calls this once its own parts are stored: it waits (bounded) for the parts of the others -- the CTAs of
// the same rank in their pairs, which hold the same 128 rows -- and sums its own 1/P of the tile in pair order.
template <int SPLIT>
__device__ __forceinline__ void reduce_split(const PairParams& p, unsigned int epoch, int tile, int kstages, int t, int nthreads,
                                             volatile int* s_abort) {
    int first, last;
    participants(p, kstages, gridDim.x >> 1, blockIdx.x >> 1, tile, first, last);
    const int rank = blockIdx.x & 1;
    {
        const long long t0 = clock64();
        for (int c = first + (t & 31); c <= last; c += 32) {
            const unsigned int* f = &p.flags[(2 * c + rank) * 2 + (c == first ? 1 : 0)];
            while (ptx::ld_acquire_gpu(f) != epoch) {
                if (*s_abort) break;
                if (clock64() - t0 > ptx::kWaitBudgetClocks) {
                    *s_abort = 1;
                    atomicCAS(p.status, 0u, 0x480u);
                    break;
                }
            }
        }
        __syncwarp();
        if (*s_abort) return;
    }
    int rg, mt;
    Work::place(p, p.dp_items + tile / p.R, rg, mt);
    const int n0 = (rg * p.R + tile % p.R) * 2 * TR + rank * TR, m0 = mt * p.T;
    const int tokens = min(p.T, p.M - m0);
    const int P = last - first + 1, me = (int)(blockIdx.x >> 1) - first;
    const int total = tokens * (TR / 4);         // chunks of four rows
    const int e0 = (int)((long long)me * total / P), e1 = (int)((long long)(me + 1) * total / P);
    const float4* parts = reinterpret_cast<const float4*>(p.partials);
    const float4* head = parts + ((size_t)(2 * first + rank) * 2 + 1) * (kSlotFloats / 4);
    const bool has_residual = SPLIT == kTailSplitRes || (SPLIT != kTailSplit && p.residual);
    const int shift = SPLIT != kTailSplitRes && p.swiglu_out ? 2 : 0;      // an up chunk lies two chunks behind its gate chunk
    constexpr int U = 4;                         // loads of four chunks in flight: the reduction is L2 round trips
    for (int b = e0 + t; b < e1; b += U * nthreads) {
        float4 s[U], g[U];
        for (int pass = 0; pass < (shift ? 2 : 1); ++pass) {
#pragma unroll
            for (int i = 0; i < U; ++i) {
                const int e = b + i * nthreads;
                if (pass) g[i] = s[i];
                if (e < e1 && !(shift && (e & 2))) s[i] = __ldcg(head + e + pass * shift);
            }
            for (int c = first + 1; c <= last; ++c) {
                const float4* src = parts + (size_t)(2 * c + rank) * 2 * (kSlotFloats / 4) + pass * shift;
                float4 x[U];
#pragma unroll
                for (int i = 0; i < U; ++i) {
                    const int e = b + i * nthreads;
                    x[i] = e < e1 && !(shift && (e & 2)) ? __ldcg(src + e) : make_float4(0.f, 0.f, 0.f, 0.f);
                }
#pragma unroll
                for (int i = 0; i < U; ++i) { s[i].x += x[i].x; s[i].y += x[i].y; s[i].z += x[i].z; s[i].w += x[i].w; }
            }
        }
        float factor[U];                         // before the stores, behind which the loads would wait for one another
#pragma unroll
        for (int i = 0; i < U; ++i) factor[i] = b + i * nthreads < e1 ? token_factor(p, m0 + (b + i * nthreads) / (TR / 4)) : 0.0f;
#pragma unroll
        for (int i = 0; i < U; ++i) {
            const int e = b + i * nthreads;
            const int m = m0 + e / (TR / 4), n = n0 + e % (TR / 4) * 4;
            if (e >= e1 || n >= p.N) continue;   // N % 8 == 0: a chunk is inside or outside
            const float mul = factor[i];
            const float v[4] = {s[i].x * mul, s[i].y * mul, s[i].z * mul, s[i].w * mul};
            if (shift) {
                if (e & 2) continue;
                const float gate[4] = {g[i].x * mul, g[i].y * mul, g[i].z * mul, g[i].w * mul};
                store4(p.C + (size_t)m * (p.N / 2) + 8 * (n >> 4) + (n & 7), silu_pair(gate[0], v[0]), silu_pair(gate[1], v[1]),
                       silu_pair(gate[2], v[2]), silu_pair(gate[3], v[3]));
                continue;
            }
            const size_t o = (size_t)m * p.N + n;
            if (SPLIT != kTailSplitRes && p.out_f32) {
                *reinterpret_cast<float4*>(reinterpret_cast<float*>(p.C) + o) = make_float4(v[0], v[1], v[2], v[3]);
                continue;
            }
            float r[4] = {0.f, 0.f, 0.f, 0.f};
            if (has_residual) {
                const uint2 rr = *reinterpret_cast<const uint2*>(p.residual + o);
                r[0] = bf16_bits_to_float(rr.x & 0xFFFFu);
                r[1] = bf16_bits_to_float(rr.x >> 16);
                r[2] = bf16_bits_to_float(rr.y & 0xFFFFu);
                r[3] = bf16_bits_to_float(rr.y >> 16);
            }
            store4(p.C + o, v[0] + r[0], v[1] + r[1], v[2] + r[2], v[3] + r[3]);
        }
    }
}

template <int MODE, bool FINE, int SPLIT>
__global__ void __launch_bounds__(kThreads, 1)
prefill_pair_kernel(const __grid_constant__ CUtensorMap tm_act, const __grid_constant__ CUtensorMap tm_w,
                    const __grid_constant__ CUtensorMap tm_scale, const PairParams p) {
    constexpr bool kTail = SPLIT == kTailSplit || SPLIT == kTailSplitRes;
    const bool has_residual = SPLIT == kTailSplitRes || (SPLIT != kTailSplit && p.residual);
    const bool swiglu_out = SPLIT != kTailSplitRes && p.swiglu_out, out_f32 = SPLIT != kTailSplitRes && p.out_f32;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = smem_raw + ((1024u - (ptx::smem_u32(smem_raw) & 1023u)) & 1023u);
    const int xbytes = p.T / 2 * (XK * 2);                           // this CTA's T/2 tokens x 128 k, two blocks of 64 k
    unsigned char* s_x = smem;
    unsigned char* s_w = s_x + p.x_stages * xbytes;                  // raw weight stages, or (DENSE) the ring of A blocks
    uint64_t* bars = reinterpret_cast<uint64_t*>(s_w + (MODE == kDense ? p.units * kDenseUnitBytes : p.w_stages * kWStageBytes));
    uint64_t* afull = bars;                        // [kRingMax]    leader's, both CTAs' dequantisers (or TMA) arrive
    uint64_t* aempty = afull + kRingMax;          // [kRingMax]    each CTA its own, by commit
    uint64_t* xfull = aempty + kRingMax;          // [kMaxX]       leader's
    uint64_t* xempty = xfull + kMaxX;              // [kMaxX]       each CTA its own, by commit (!FINE: the other's by relay)
    uint64_t* wfull = xempty + kMaxX;              // [kMaxW]       each CTA its own
    uint64_t* wempty = wfull + kMaxW;              // [kMaxW]       each CTA its own
    uint64_t* tfull = wempty + kMaxW;              // [kMaxAccs]    each CTA its own, by commit
    uint64_t* tempty = tfull + kMaxAccs;           // [kMaxAccs]    leader's
    float* s_factor = reinterpret_cast<float*>(tempty + kMaxAccs);   // [kMaxT]
    uint32_t* s_tmem = reinterpret_cast<uint32_t*>(s_factor + kMaxT);
    volatile int* s_abort = reinterpret_cast<volatile int*>(s_tmem + 1);
    volatile unsigned int* s_epoch = reinterpret_cast<volatile unsigned int*>(s_tmem + 2);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int rank = (int)ptx::cluster_ctarank();
    const int kstages = p.K / WK;
    const int spare = spare_units(p, MODE == kDense), ring = ring_units(p, MODE == kDense);
    constexpr uint32_t kRingCols = FINE ? kUnitCols / 2 : kUnitCols;
    constexpr int kUnitK = FINE ? BK : XK, kLoadBytes = FINE ? kDenseBlockBytes : kDenseUnitBytes;      // of a unit (the latter: BF16, a CTA's)

    if (tid == 0) {
        for (int i = 0; i < kRingMax; ++i) { ptx::mbar_init(&afull[i], MODE == kDense ? 1 : 2 * kGroupWarps); ptx::mbar_init(&aempty[i], 1); }
        for (int i = 0; i < kMaxX; ++i) { ptx::mbar_init(&xfull[i], 1); ptx::mbar_init(&xempty[i], FINE || rank == 0 ? 2 : 1); }
        for (int i = 0; i < kMaxW; ++i) { ptx::mbar_init(&wfull[i], 1); ptx::mbar_init(&wempty[i], 2 * kGroupWarps); }
        for (int i = 0; i < kMaxAccs; ++i) { ptx::mbar_init(&tfull[i], 1); ptx::mbar_init(&tempty[i], 4 * kEpiWarps); }
        *s_abort = 0;
        ptx::fence_mbar_init();
    }
    if (warp == 1) {   // all 512 columns in both CTAs: accumulators from column 0, the A ring behind them
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(ptx::smem_u32(s_tmem)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    ptx::cluster_sync();                   // both CTAs' barriers exist before anyone arrives on the other's
    tc_fence_after();
    const uint32_t tmem_base = *s_tmem, a_col0 = tmem_base + (uint32_t)(p.a_col0 - spare * (kUnitCols / 2));
    ptx::griddep_launch_dependents();      // the next kernel in the stream may start its own prologue

    Work work(p, kstages, gridDim.x >> 1, blockIdx.x >> 1);
    Item it;
    if (warp == 0 || (MODE == kDense && warp == 8)) {
        // ------------------------------------------------------------------ weight stream
        ptx::prefetch_tensormap(&tm_w);
        const uint64_t pol = ptx::policy_evict_first();
        int s = 0;
        uint32_t ph = 0;
        if (MODE == kDense) {
            // Two warps, every other unit each, as the issuers: one warp's turn (wait, expectation, copy) takes as long as the MMAs.
            const int me = warp >> 3;
            const uint32_t full0 = ptx::mapa_shared(ptx::smem_u32(afull), 0);
            s = me;
            ptx::griddep_wait();           // a BF16 weight may come from the kernel right before; there is no pre-pass to stream behind
            while (work.next(p, it)) {
                const int row = ((it.rt + (it.rows == 2 ? me : 0)) * 2 + rank) * TR, step = it.rows == 2 ? kUnitK : 2 * kUnitK;
                for (int k = it.ks0 * WK + (it.rows == 2 ? 0 : me * kUnitK); k < it.ks1 * WK; k += step) {
                    const bool ok = ptx::mbar_wait(&aempty[s], ph ^ 1u, s_abort, p.status, 0x410u + s);
                    if (ptx::elect_one() && ok) {
                        if (rank == 0) ptx::mbar_arrive_expect_tx(&afull[s], 2 * kLoadBytes);
                        ptx::tma_load_2d_pair(s_w + s * kLoadBytes, &tm_w, full0 + s * 8, k, row, pol);
                        if (!FINE) ptx::tma_load_2d_pair(s_w + s * kLoadBytes + kDenseBlockBytes, &tm_w, full0 + s * 8, k + BK, row, pol);
                    }
                    s += 2;
                    if (s >= ring) { s = me; ph ^= 1u; }
                }
            }
            for (int i = 0; i < ring; i += 2) {      // nothing of the leader's may still be on its way to this CTA's barriers at the end
                ptx::mbar_wait(&aempty[s], ph ^ 1u, s_abort, p.status, 0x41Fu);
                s += 2;
                if (s >= ring) { s = me; ph ^= 1u; }
            }
        } else {
            ptx::prefetch_tensormap(&tm_scale);
            // Weights follow the stream: they may come from the kernel in front of the call.  (Not waiting here, the ring filled
            // beside the pre-pass: 34816 x 5120 with 65 tokens, calls back to back, 43.3 against 43.7 us.  Letting the pre-pass start
            // this kernel only after its own wait keeps that and costs the prologue: 44.9 us.)
            ptx::griddep_wait();
            while (work.next(p, it)) {
                for (int ks = it.ks0; ks < it.ks1; ++ks) {
                    for (int r = 0; r < it.rows; ++r) {
                        const bool ok = ptx::mbar_wait(&wempty[s], ph ^ 1u, s_abort, p.status, 0x410u + s);
                        if (ptx::elect_one() && ok) {
                            const int row = ((it.rt + r) * 2 + rank) * TR;
                            ptx::mbar_arrive_expect_tx(&wfull[s], kWStageBytes);
                            ptx::tma_load_2d(s_w + s * kWPackedBytes, &tm_w, &wfull[s], ks * (WK / 2), row, pol);
                            ptx::tma_load_2d(s_w + p.w_stages * kWPackedBytes + s * kWScaleBytes, &tm_scale, &wfull[s], ks * (WK / 16), row, pol);
                        }
                        if (++s == p.w_stages) { s = 0; ph ^= 1u; }
                    }
                }
            }
        }
    } else if (warp == 2) {
        // ------------------------------------------------------------------ token stream
        ptx::prefetch_tensormap(&tm_act);
        ptx::griddep_wait();               // the activations are the preceding kernel's output
        const uint64_t pol = ptx::policy_evict_last();
        int s = 0, turn = 0;
        uint32_t ph = 0;
        while (work.next(p, it)) {
            for (int k = it.ks0 * WK; k < it.ks1 * WK; k += XK) {
                const bool ok = ptx::mbar_wait(&xempty[s], ph ^ 1u, s_abort, p.status, 0x400u + s);
                const bool pass = !FINE && rank == 0 && turn++ >= p.x_stages;      // the first round finds fresh barriers
                if (ptx::elect_one() && ok) {
                    if (pass) relay(&xempty[s]);
                    if (rank == 0) ptx::mbar_arrive_expect_tx(&xfull[s], 2u * (uint32_t)xbytes);
                    const uint32_t bar = ptx::mapa_shared(ptx::smem_u32(&xfull[s]), 0);
                    const int m = it.mt * p.T + rank * (p.T / 2);
                    ptx::tma_load_2d_pair(s_x + s * xbytes, &tm_act, bar, k, m, pol);
                    ptx::tma_load_2d_pair(s_x + s * xbytes + xbytes / 2, &tm_act, bar, k + BK, m, pol);
                }
                if (++s == p.x_stages) { s = 0; ph ^= 1u; }
            }
        }
        for (int i = 0; i < p.x_stages; ++i) {       // as above
            const bool ok = ptx::mbar_wait(&xempty[s], ph ^ 1u, s_abort, p.status, 0x40Eu);
            const bool pass = !FINE && rank == 0 && turn++ >= p.x_stages;
            if (ptx::elect_one() && ok && pass) relay(&xempty[s]);
            if (++s == p.x_stages) { s = 0; ph ^= 1u; }
        }
    } else if (warp == 1 || warp == 3) {
        // ------------------------------------------------------------------ MMA issuers (leader only): one warp per row tile
        if (rank == 0) {
            const int me = warp >> 1;
            // The issue rate is the bound to watch for T <= 128.  Measured alone, a warp takes 60 clocks an MMA whatever T is, ~75 a
            // commit and up to ~130 for a wait that finds its phase complete; hence two warps, 128 k (eight MMAs) a turn, one look
            // at all barriers of a turn, and waits only where that look came too early.
            // Two row tiles: each warp its own, on the same token stage.  One: the warps take its units in turn, each on an
            // accumulator of its own, which the epilogue adds.  Either way the warps take every other unit, and an item takes two
            // accumulators.
            // With accumulators of 160 and 192 columns tensor memory is left for two units of 128 k, and a unit's way around -- commit,
            // dequantisers, stores, arrival -- takes longer than the other's eight MMAs: 1111 tokens ran at 120 clocks an MMA of 96.
            // There a unit and a turn are 64 k: 81 clocks at T = 160 (of 80).
            // A parity wait cannot tell a phase from the one two before it, so whoever waits on a barrier must have seen
            // each of its phases: every warp waits for every token stage, and a stage is free when both have said so; the
            // numbers of units and accumulators are even, so a warp always meets the same ones.
            Ring x(p.x_stages), u(ring), t(p.accs);
            u.advance(me);
            t.advance(me);
            bool ok = true;
            const uint32_t x0 = ptx::smem_u32(s_x), xhalf = (uint32_t)xbytes / 2;
            const uint32_t aempty0 = ptx::smem_u32(aempty), xempty0 = ptx::smem_u32(xempty), tfull0 = ptx::smem_u32(tfull);
            const uint32_t other = ptx::mapa_shared(aempty0, 1) - aempty0;
            while (ok && work.next(p, it)) {
                const bool one = it.rows == 1;
                const bool pairwise = one && !FINE;            // two token stages a turn, one of them this warp's
                const int turns = (it.ks1 - it.ks0) * (FINE ? 4 : 2) / (one ? 2 : 1);
                const uint32_t d = tmem_base + (uint32_t)(t.i * p.T);
                ok = ptx::mbar_wait(&tempty[t.i], t.phase ^ 1u, s_abort, p.status, 0x440u + t.i);
                for (int turn = 0; turn < turns; ++turn) {
                    const bool second = FINE && !one && (turn & 1);       // the other block of the last turn's token stage
                    Ring y = x;                                           // pairwise: the stage behind x
                    if (!FINE) y.advance(1);
                    bool ready = ptx::mbar_test_wait(&afull[u.i], u.phase);
                    if (!second) ready &= ptx::mbar_test_wait(&xfull[x.i], x.phase);
                    if (pairwise) ready &= ptx::mbar_test_wait(&xfull[y.i], y.phase);
                    if (!ready) {
                        if (!second) ok = ok && ptx::mbar_wait(&xfull[x.i], x.phase, s_abort, p.status, 0x420u + x.i);
                        if (pairwise) ok = ok && ptx::mbar_wait(&xfull[y.i], y.phase, s_abort, p.status, 0x420u + y.i);
                        ok = ok && ptx::mbar_wait(&afull[u.i], u.phase, s_abort, p.status, 0x430u + u.i);
                    }
                    // One decision for the warp: where a wait runs out in some lanes only, those would leave and the others
                    // stay for ever in the elections of the MMAs and commits below.
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) break;
                    tc_fence_after();
                    const uint32_t xstage = x0 + (uint32_t)(pairwise && me ? y.i : x.i) * xbytes;
                    const uint64_t xdesc = umma_desc_sw128(xstage + (second || (FINE && one && me) ? xhalf : 0u));
                    const uint64_t wdesc = umma_desc_sw128(ptx::smem_u32(s_w) + (uint32_t)u.i * kLoadBytes);
                    if (MODE == kDense && FINE) mma4_ss(d, wdesc, xdesc, p.idesc, (uint32_t)turn);
                    else if (MODE == kDense) mma8_ss(d, wdesc, xdesc, xhalf >> 4, p.idesc, (uint32_t)turn);
                    else if (FINE) mma4_ts(d, a_col0 + (uint32_t)u.i * kRingCols, xdesc, p.idesc, (uint32_t)turn);
                    else mma8_ts(d, a_col0 + (uint32_t)u.i * kRingCols, xdesc, xhalf >> 4, p.idesc, (uint32_t)turn);
                    commit_pair(aempty0 + (uint32_t)u.i * 8, other);
                    u.advance(2);
                    if (FINE) {
                        if (one || second) {
                            commit_pair(xempty0 + (uint32_t)x.i * 8, other);
                            x.advance(1);
                        }
                    } else {
                        commit_leader(xempty0 + (uint32_t)x.i * 8);
                        if (pairwise) commit_leader(xempty0 + (uint32_t)y.i * 8);
                        x.advance(pairwise ? 2 : 1);
                    }
                }
                if (ok) commit_pair(tfull0 + (uint32_t)t.i * 8, other);
                t.advance(2);
            }
        }
    } else if (warp >= 8 && warp < 16) {
        if (MODE != kDense) {
        // ------------------------------------------------------------------ dequantise into TMEM
        // Two groups of four warps fill the units in turn, the order the MMAs take them in: two row tiles, one each; one, every other
        // unit.
        const int quarter = warp & 3;                     // TMEM lanes 32*quarter .. +31 (= warp id % 4)
        const int group = (warp - 8) >> 2;
        const int row = quarter * 32 + lane;
        const int sw7 = row & 7;
        int sw = 0, su = group;
        uint32_t pw = 0, pu = 0;
        const uint32_t full0 = ptx::mapa_shared(ptx::smem_u32(afull), 0);
        const uint32_t a_base = a_col0 + ((uint32_t)(quarter * 32) << 16);
        while (work.next(p, it)) {
            const bool two = it.rows == 2;
            for (int ks = it.ks0; ks < it.ks1; ++ks) {
                // every warp waits for every stage, see the issuers
                const int first = sw;
                int st = sw;
                ptx::mbar_wait(&wfull[sw], pw, s_abort, p.status, 0x450u + sw);
                if (two) {
                    if (++sw == p.w_stages) { sw = 0; pw ^= 1u; }
                    ptx::mbar_wait(&wfull[sw], pw, s_abort, p.status, 0x450u + sw);
                    if (group) st = sw;
                }
                const unsigned char* wp = s_w + st * kWPackedBytes + row * 128;
                const unsigned char* ws = s_w + p.w_stages * kWPackedBytes + st * kWScaleBytes + row * 16;
                // this group's 64-k blocks of the stage: two row tiles, all; one, every other unit's
                const int j0 = two ? 0 : (FINE ? group : 2 * group), step = !two && FINE ? 2 : 1, count = two ? 4 : 2;
                for (int i = 0; i < count; ++i) {
                    const int j = j0 + i * step;
                    const bool opens = FINE || !(i & 1), closes = FINE || (i & 1);
                    const uint4 q0 = *reinterpret_cast<const uint4*>(wp + (((2 * j) ^ sw7) << 4));
                    const uint4 q1 = *reinterpret_cast<const uint4*>(wp + (((2 * j + 1) ^ sw7) << 4));
                    const uint32_t scw = mask_scale_bytes(*reinterpret_cast<const uint32_t*>(ws + 4 * j));
                    const bool ready = !opens || ptx::mbar_test_wait(&aempty[su], pu ^ 1u);
                    const uint32_t q[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
                    uint32_t o[2][16];
                    uint32_t one = 0u, more = 0u;          // kRounded: what a block's 1.0 comes to, and twice what 1.5 has over it
#pragma unroll
                    for (int c = 0; c < 8; ++c) {          // 8 consecutive k = one 32-bit word of codes
                        uint32_t e[4];
                        ptx::cvt_e2m1x8_to_f16x2(q[c], e);
                        if (MODE == kRounded) {
                            // The bits of the reference's dequantisation: FP32 block scale times 1/gs, FP32 product with the code's
                            // value, one rounding to BF16; then a power of two into FP16 (exact).  A code is p or 1.5 p, p a power
                            // of two, which commutes with the roundings, so a block takes two of them, and an element is
                            // p * one + (code - p) * more, exact in FP16 (one and 1.5's value have eight bits each).  One rounding
                            // an element bound the kernel: 34816 x 5120 at 256 / 2048 tokens 164 / 832 us, 125 / 644 so.
                            if (!(c & 1)) {
                                const float bs = ue4m3_to_float((scw >> (8 * (c >> 1))) & 0xFFu) * p.inv_gs;
                                const float2 b = __bfloat1622float2(__floats2bfloat162_rn(bs, 1.5f * bs));
                                const float x = b.x * p.wshift, y = 2.0f * (b.y - b.x) * p.wshift;
                                one = ptx::pack_f16x2(x, x);
                                more = ptx::pack_f16x2(y, y);
                            }
#pragma unroll
                            for (int i = 0; i < 4; ++i) {
                                const uint32_t pow2 = e[i] & 0xFDFFFDFFu;           // without FP16's top mantissa bit, set in 1.5, 3 and 6
                                o[c >> 2][(c & 3) * 4 + i] = ptx::fma_f16x2(ptx::sub_f16x2(e[i], pow2), more, ptx::mul_f16x2(pow2, one));
                            }
                        } else {
                            const uint32_t S = scale_byte_to_f16x2(scw, c >> 1);     // scale / 2^8, undone in the epilogue
#pragma unroll
                            for (int i = 0; i < 4; ++i) o[c >> 2][(c & 3) * 4 + i] = ptx::mul_f16x2(e[i], S);
                        }
                    }
                    // The stores want one warp: lanes that saw the unit free and lanes that waited for it meet here.  (A vote in front of the
                    // wait instead: 149 tokens of an MLP 5120 x 17408 101.8 us, so 100.5; in the few-token kernel the vote is ahead.)
                    if (!ready) ptx::mbar_wait(&aempty[su], pu ^ 1u, s_abort, p.status, 0x460u + su);
                    __syncwarp();
                    if (opens) tc_fence_after();
                    const uint32_t a_addr = a_base + (uint32_t)su * kRingCols + (opens ? 0u : (uint32_t)(kUnitCols / 2));
                    tmem_st16(a_addr, o[0]);
                    tmem_st16(a_addr + 16, o[1]);
                    if (closes) {
                        tmem_wait_st();
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) ptx::mbar_arrive_cluster(full0 + su * 8);
                        su += 2;
                        if (su >= ring) { su = group; pu ^= 1u; }
                    }
                }
                if (lane == 0) {
                    ptx::mbar_arrive(&wempty[first]);
                    if (two) ptx::mbar_arrive(&wempty[sw]);
                }
                if (++sw == p.w_stages) { sw = 0; pw ^= 1u; }
            }
        }
        for (int i = 0; i < ring; i += 2) {          // as above
            ptx::mbar_wait(&aempty[su], pu ^ 1u, s_abort, p.status, 0x46Fu);
            su += 2;
            if (su >= ring) { su = group; pu ^= 1u; }
        }
        }
    } else {
        // ------------------------------------------------------------------ epilogue: thread = weight row
        // Two groups of four warps.  Two row tiles: one each.  One: half of the tokens each, adding the two accumulators.
        const int eg = warp >> 4;                         // warps 4-7: 0, warps 16-19: 1
        const int ew = warp & 3;                          // TMEM lanes 32*ew .. +31 (= warp id % 4)
        const int te = ew * 32 + lane, tt = eg * kEpiWarps * 32 + te;
        Ring t(p.accs);
        int pend[2] = {-1, -1};
        int m_seen = -1;
        ptx::griddep_wait();                              // C, the residual and the scratch belong to earlier kernels until now
        if (tt == 0) *s_epoch = ptx::take_launch_epoch(p.status);
        ptx::named_barrier_sync(1, 2 * kEpiWarps * 32);
        const unsigned int epoch = *s_epoch;
        bool more = work.next(p, it);
        while (more) {
            const int m0 = it.mt * p.T, tokens = min(p.T, p.M - m0);
            if (m0 != m_seen) {                           // this tile's token factors, zero beyond M
                m_seen = m0;
                ptx::named_barrier_sync(1, 2 * kEpiWarps * 32);
                for (int i = tt; i < p.T; i += 2 * kEpiWarps * 32) s_factor[i] = i < tokens ? token_factor(p, m0 + i) : 0.0f;
                ptx::named_barrier_sync(1, 2 * kEpiWarps * 32);
            }
            const float* factor = s_factor;
            const bool complete = SPLIT == kWhole || (kTail && it.ks0 == 0 && it.ks1 == kstages);      // all split: no part is a whole tile
            const int which = it.ks0 == 0 ? 1 : 0;        // head of a tile (span end) or tail (span start)
            const bool two = it.rows == 2;
            // Both groups wait for and free both accumulators (accs is even: a pair never wraps).
            const int begin = two ? 0 : eg * (p.T / 2), end = two ? tokens : min(tokens, (eg + 1) * (p.T / 2));
            const int n = ((it.rt + (two ? eg : 0)) * 2 + rank) * TR + te;
            if (has_residual && complete && n - lane < p.N) {    // its way from memory goes behind the MMAs: 64 bytes a token and warp into L2
                const __nv_bfloat16* src = p.residual + (size_t)m0 * p.N;
                for (int i = 2 * begin + lane; i < 2 * end; i += 32)
                    ptx::prefetch_l2(src + (size_t)(i >> 1) * p.N + min(n - lane + 16 * (i & 1), p.N - 1));
            }
            // the residual of sixteen tokens, all in flight together (it may be C itself): asked for a chunk ahead, the first before the wait
            unsigned short res[16];
            auto ask = [&](int c0) {
                const unsigned short* src = reinterpret_cast<const unsigned short*>(p.residual) + (size_t)(m0 + c0) * p.N + n;
#pragma unroll
                for (int i = 0; i < 16; ++i) res[i] = c0 + i < end ? src[(size_t)i * p.N] : (unsigned short)0;
            };
            if (SPLIT != kAllSplit && has_residual && complete && n < p.N) ask(begin);
            for (int i = t.i; i < t.i + 2; ++i) ptx::mbar_wait(&tfull[i], t.phase, s_abort, p.status, 0x470u + i);
            __syncwarp();
            tc_fence_after();
            {
                const uint32_t t_addr = tmem_base + ((uint32_t)(ew * 32) << 16) + (uint32_t)((t.i + (two ? eg : 0)) * p.T);
                float* slot = p.partials + ((size_t)blockIdx.x * 2 + which) * kSlotFloats + te;
                // The sums of sixteen tokens; called by the whole warp (lanes beyond the weight left the last chunk early).
                auto sums = [&](int c0, uint32_t (&v)[16]) {
                    __syncwarp();
                    tmem_ld16(t_addr + c0, v);
                    if (two) return;
                    uint32_t w[16];
                    tmem_ld16(t_addr + p.T + c0, w);
#pragma unroll
                    for (int i = 0; i < 16; ++i) v[i] = __float_as_uint(__uint_as_float(v[i]) + __uint_as_float(w[i]));
                };
                // A loop each for parts and for whole tiles: registers again.
                for (int c0 = begin; SPLIT != kWhole && !complete && c0 < end; c0 += 16) {
                    uint32_t v[16];
                    sums(c0, v);
                    const int cnt = min(16, end - c0);
#pragma unroll
                    for (int i = 0; i < 16; ++i)           // [token][row]: a warp stores 128 contiguous bytes
                        if (i < cnt) __stcg(slot + (c0 + i) * TR, __uint_as_float(v[i]));
                }
                for (int c0 = begin; SPLIT != kAllSplit && complete && c0 < end; c0 += 16) {
                    uint32_t v[16];
                    sums(c0, v);
                    const int cnt = min(16, end - c0);
                    float f[16];
#pragma unroll
                    for (int i = 0; i < 16; i += 4) {
                        const float4 k4 = *reinterpret_cast<const float4*>(factor + c0 + i);
                        f[i] = __uint_as_float(v[i]) * k4.x;
                        f[i + 1] = __uint_as_float(v[i + 1]) * k4.y;
                        f[i + 2] = __uint_as_float(v[i + 2]) * k4.z;
                        f[i + 3] = __uint_as_float(v[i + 3]) * k4.w;
                    }
                    if (swiglu_out) {
                        // A gate lane and its up lane (eight rows on) hold both halves of sixteen outputs: the gate lane finishes
                        // the first eight tokens, the up lane the others, one exchange and one SiLU each.
                        const int late = n & 8;
                        __nv_bfloat16* dst = p.C + (size_t)(m0 + c0 + late) * (p.N / 2) + 8 * (n >> 4) + (n & 7);
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            const float other = __shfl_xor_sync(0xffffffffu, late ? f[i] : f[i + 8], 8);
                            const float y = silu_pair(late ? other : f[i], late ? f[i + 8] : other);
                            if (late + i < cnt && n < p.N) dst[(size_t)i * (p.N / 2)] = __float2bfloat16_rn(y);
                        }
                        continue;
                    }
                    if (n >= p.N) continue;
                    const size_t o = (size_t)(m0 + c0) * p.N + n;
                    if (out_f32) {
                        float* dst = reinterpret_cast<float*>(p.C) + o;
#pragma unroll
                        for (int i = 0; i < 16; ++i) if (i < cnt) dst[(size_t)i * p.N] = f[i];
                        continue;
                    }
                    if (has_residual) {
#pragma unroll
                        for (int i = 0; i < 16; ++i) f[i] += bf16_bits_to_float(res[i]);
                        if (c0 + 16 < end) ask(c0 + 16);
                    }
                    __nv_bfloat16* dst = p.C + o;
                    if (cnt == 16) {
#pragma unroll
                        for (int i = 0; i < 16; ++i, dst += p.N) *dst = __float2bfloat16_rn(f[i]);
                    } else {
#pragma unroll
                        for (int i = 0; i < 16; ++i, dst += p.N) if (i < cnt) *dst = __float2bfloat16_rn(f[i]);
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) {                               // sixteen arrivals free an accumulator: eight warps of two CTAs
                    ptx::mbar_arrive_cluster(ptx::mapa_shared(ptx::smem_u32(&tempty[t.i]), 0));
                    ptx::mbar_arrive_cluster(ptx::mapa_shared(ptx::smem_u32(&tempty[t.i + 1]), 0));
                }
            }
            t.advance(2);
            if (!complete) {
                __threadfence();
                ptx::named_barrier_sync(1, 2 * kEpiWarps * 32);       // all rows and tokens stored before the flag goes up
                if (tt == 0) ptx::st_release_gpu(&p.flags[blockIdx.x * 2 + which], epoch);
                pend[which] = it.sk;
            }
            more = work.next(p, it);
            // Whole items follow the split ones: these warps reduce the split tiles they stored now, behind the MMAs
            // of the next items.  (With no whole items all warps do it at the end.)
            if (kTail && (pend[0] >= 0 || pend[1] >= 0) && (!more || it.sk < 0)) {
#pragma unroll
                for (int w = 0; w < 2; ++w) {
                    if (pend[w] >= 0) reduce_split<SPLIT>(p, epoch, pend[w], kstages, tt, 2 * kEpiWarps * 32, s_abort);
                    pend[w] = -1;
                }
            }
        }
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (*s_abort) {                        // a wait ran out: nobody issues any more; give what is in flight time to land
        for (int i = 0; i < 200; ++i) __nanosleep(1000);
    }
    ptx::cluster_sync();                   // neither CTA leaves, or frees its tensor memory, while the other may still reach it
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512) : "memory");
    }
    if (SPLIT == kAllSplit) {
        // Every tile was split and nothing else is left to do: all 20 warps reduce.
        ptx::griddep_wait();
        const unsigned int epoch = *s_epoch;
        const int pairs = gridDim.x >> 1, id = blockIdx.x >> 1;
        const long long units = (long long)p.sk_tiles * kstages;
        const long long u0 = (long long)id * units / pairs, u1 = (long long)(id + 1) * units / pairs;
        if (u0 < u1) {
            const int t0 = (int)(u0 / kstages), t1 = (int)((u1 - 1) / kstages);
            if (u0 % kstages != 0 || u1 - u0 < kstages) reduce_split<SPLIT>(p, epoch, t0, kstages, tid, kThreads, s_abort);
            if (t1 != t0 && u1 - (long long)t1 * kstages < kstages) reduce_split<SPLIT>(p, epoch, t1, kstages, tid, kThreads, s_abort);
        }
    }
}

size_t act_bytes(int M, int K) { return ((size_t)M * K * 2 + 255) / 256 * 256; }

constexpr size_t kPartialBytes = (size_t)kSlotFloats * 4;
constexpr int kMaxPrefillGrid = 160;
constexpr size_t kStreamKBytes = 4096 + 2 * kMaxPrefillGrid * kPartialBytes;

// The tile plan of one launch and what follows from it; returns the grid, and the dynamic shared memory in *smem.
int plan_pair(PairParams& p, const nvfp4_device_info& dev, bool dense, int* smem) {
    int pairs = (dev.sm_count < kMaxPrefillGrid ? dev.sm_count : kMaxPrefillGrid) / 2;
    if (dev.max_pairs > 0 && dev.max_pairs < pairs) pairs = dev.max_pairs;
    pairs = make_plan(p, pairs, dev.prefill_stream_k != 0, dense, smem);
    p.idesc = (1u << 4) | ((uint32_t)(p.T >> 3) << 17) | ((uint32_t)(2 * TR >> 4) << 24);
    if (dense) p.idesc |= (1u << 7) | (1u << 10);         // A and B formats: BF16 instead of FP16
    return 2 * pairs;
}

template <int MODE, bool FINE, int SPLIT>
cudaError_t launch_as(const PairParams& p, int grid, int smem, const CUtensorMap& tma, const CUtensorMap& tmw, const CUtensorMap& tms,
                   cudaStream_t s) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = 2;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    return cudaLaunchKernelEx(&cfg, prefill_pair_kernel<MODE, FINE, SPLIT>, tma, tmw, tms, p);
}

template <int MODE, bool FINE>
cudaError_t launch_split(const PairParams& p, int grid, int smem, const CUtensorMap& tma, const CUtensorMap& tmw, const CUtensorMap& tms,
                   cudaStream_t s) {
    if (p.sk_tiles == 0) return launch_as<MODE, FINE, kWhole>(p, grid, smem, tma, tmw, tms, s);
    if (p.dp_items == 0) {
        if constexpr (MODE == kDense && !FINE) return cudaErrorInvalidValue;      // two row tiles an item: never split all over
        else return launch_as<MODE, FINE, kAllSplit>(p, grid, smem, tma, tmw, tms, s);
    }
    return p.residual ? launch_as<MODE, FINE, kTailSplitRes>(p, grid, smem, tma, tmw, tms, s)
                      : launch_as<MODE, FINE, kTailSplit>(p, grid, smem, tma, tmw, tms, s);
}

template <int MODE>
cudaError_t launch(const PairParams& p, int grid, int smem, const CUtensorMap& tma, const CUtensorMap& tmw, const CUtensorMap& tms,
                   cudaStream_t s) {
    return fine_units(p, MODE == kDense) ? launch_split<MODE, true>(p, grid, smem, tma, tmw, tms, s)
                                         : launch_split<MODE, false>(p, grid, smem, tma, tmw, tms, s);
}

template <int MODE, bool FINE>
cudaError_t configure() {
    cudaError_t e = configure_large_smem(prefill_pair_kernel<MODE, FINE, kWhole>, kSmemMax);
    if constexpr (MODE != kDense || FINE)
        if (e == cudaSuccess) e = configure_large_smem(prefill_pair_kernel<MODE, FINE, kAllSplit>, kSmemMax);
    if (e == cudaSuccess) e = configure_large_smem(prefill_pair_kernel<MODE, FINE, kTailSplit>, kSmemMax);
    if (e == cudaSuccess) e = configure_large_smem(prefill_pair_kernel<MODE, FINE, kTailSplitRes>, kSmemMax);
    return e;
}

}  // namespace

bool prefill_umma_supported(const LinearArgs& a) {
    if (a.M < 1 || (a.K % WK) != 0 || (a.N % 8) != 0) return false;
    if (a.swiglu_out && ((a.N % 32) != 0 || a.residual)) return false;
    if (a.out_f32 && (a.swiglu_out || a.residual)) return false;
    if ((reinterpret_cast<uintptr_t>(a.packed) & 15u) || (reinterpret_cast<uintptr_t>(a.scale) & 15u)) return false;
    return true;
}

size_t prefill_umma_reserved_bytes() { return kStreamKBytes; }

// Stream-K flags and partial tiles (fixed place, so a flag word only ever holds launch tags),
// then the FP16 copy of the activations and one FP32 per token.  What a launch writes, whatever M is: options send
// calls of 16 tokens and fewer here too.
size_t prefill_umma_scratch_bytes(int M, int /*N*/, int K) {
    return kStreamKBytes + act_bytes(M, K) + ((size_t)M * 4 + 255) / 256 * 256;
}

cudaError_t configure_prefill_umma(nvfp4_device_info& dev) {
    cudaError_t e = configure<kExact, false>();
    if (e == cudaSuccess) e = configure<kExact, true>();
    if (e == cudaSuccess) e = configure<kRounded, false>();
    if (e == cudaSuccess) e = configure<kRounded, true>();
    if (e == cudaSuccess) e = configure<kDense, false>();
    if (e == cudaSuccess) e = configure<kDense, true>();
    if (e != cudaSuccess) return e;
    // The split tiles need every pair resident at once: no more pairs than the device can place.
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(2 * (dev.sm_count / 2));
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = kSmemMax;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int clusters = 0;
    e = cudaOccupancyMaxActiveClusters(&clusters, prefill_pair_kernel<kExact, true, kAllSplit>, &cfg);
    if (e != cudaSuccess) return e;
    if (clusters < 1) return cudaErrorLaunchOutOfResources;
    dev.max_pairs = clusters;
    return cudaSuccess;
}

// scratch: [0, 256) status word (shared with the GEMV kernel); from `offset` the stream-K flags
// (4 KB) and partial tiles, then the FP16 activations and the per-token factors.
cudaError_t launch_prefill_umma(const LinearArgs& a, nvfp4_device_info& dev, void* scratch, size_t scratch_bytes,
                                size_t offset, int* launches, cudaStream_t s) {
    const size_t need = prefill_umma_scratch_bytes(a.M, a.N, a.K);
    if (offset + need > scratch_bytes) return cudaErrorMemoryAllocation;
    char* sk = static_cast<char*>(scratch) + offset;
    char* base = sk + kStreamKBytes;
    __half* ah = reinterpret_cast<__half*>(base);
    float* unscale = reinterpret_cast<float*>(base + act_bytes(a.M, a.K));
    PairParams p{};
    p.M = a.M; p.N = a.N; p.K = a.K;
    int smem = 0;
    const int grid = plan_pair(p, dev, false, &smem);
    CUtensorMap tma, tmp, tms;
    if (!make_map_cached(dev.maps, &tma, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, ah, (uint64_t)a.K, (uint64_t)a.M, BK, p.T / 2,
                  CU_TENSOR_MAP_SWIZZLE_128B) ||
        !make_map_cached(dev.maps, &tmp, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, a.packed, (uint64_t)a.K / 2, (uint64_t)a.N, 128, TR,
                  CU_TENSOR_MAP_SWIZZLE_128B) ||
        !make_map_cached(dev.maps, &tms, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, a.scale, (uint64_t)a.K / 16, (uint64_t)a.N, 16, TR,
                  CU_TENSOR_MAP_SWIZZLE_NONE))
        return cudaErrorInvalidValue;
    cudaError_t e = launch_act_to_f16(a.A, a.M, a.K, ah, unscale, dev.sm_count, s);
    if (e != cudaSuccess) return e;
    p.residual = static_cast<const __nv_bfloat16*>(a.residual);
    p.C = static_cast<__nv_bfloat16*>(a.C);
    p.unscale = unscale;
    p.status = static_cast<unsigned int*>(scratch);
    p.inv_gs = a.inv_gs;
    p.out_mul = kBlockScaleUnfold * a.inv_gs;
    p.swiglu_out = a.swiglu_out ? 1 : 0;
    p.out_f32 = a.out_f32 ? 1 : 0;
    p.flags = reinterpret_cast<unsigned int*>(sk);
    p.partials = reinterpret_cast<float*>(sk + 4096);
    if (a.round_weights) {
        // largest weight 6 * 448 / gs -> just under 2^15 (FP16's largest binade); the smallest, 0.5 * 2^-9 / gs, then sits at 2^-7
        int ex = 0;
        std::frexp(2688.0f * a.inv_gs, &ex);                 // 2688 / gs = f * 2^ex, f in [0.5, 1)
        p.wshift = std::ldexp(1.0f, 15 - ex);
        p.out_mul = std::ldexp(1.0f, ex - 15);
        e = launch<kRounded>(p, grid, smem, tma, tmp, tms, s);
    } else {
        e = launch<kExact>(p, grid, smem, tma, tmp, tms, s);
    }
    if (launches) *launches = 2;
    return e;
}

bool dense_umma_supported(const DenseArgs& a) {
    if (a.M < 1 || (a.K % WK) != 0 || (a.N % 8) != 0) return false;
    return (reinterpret_cast<uintptr_t>(a.W) & 15u) == 0;
}

size_t dense_umma_scratch_bytes() { return kStreamKBytes; }

// The same kernel on a BF16 weight [N,K] and the caller's BF16 activations: no pre-pass.  scratch as above.
cudaError_t launch_dense_umma(const DenseArgs& a, nvfp4_device_info& dev, void* scratch, size_t scratch_bytes, size_t offset,
                              int* launches, cudaStream_t s) {
    if (offset + kStreamKBytes > scratch_bytes) return cudaErrorMemoryAllocation;
    char* sk = static_cast<char*>(scratch) + offset;
    PairParams p{};
    p.M = a.M; p.N = a.N; p.K = a.K;
    int smem = 0;
    const int grid = plan_pair(p, dev, true, &smem);
    CUtensorMap tma, tmw;
    if (!make_map_cached(dev.maps, &tma, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, a.A, (uint64_t)a.K, (uint64_t)a.M, BK, p.T / 2,
                  CU_TENSOR_MAP_SWIZZLE_128B) ||
        !make_map_cached(dev.maps, &tmw, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, a.W, (uint64_t)a.K, (uint64_t)a.N, BK, TR,
                  CU_TENSOR_MAP_SWIZZLE_128B))
        return cudaErrorInvalidValue;
    p.residual = static_cast<const __nv_bfloat16*>(a.residual);
    p.C = static_cast<__nv_bfloat16*>(a.C);
    p.status = static_cast<unsigned int*>(scratch);
    p.flags = reinterpret_cast<unsigned int*>(sk);
    p.partials = reinterpret_cast<float*>(sk + 4096);
    const cudaError_t e = launch<kDense>(p, grid, smem, tma, tmw, tmw, s);
    if (launches) *launches = 1;
    return e;
}

cudaError_t configure_kernels(nvfp4_device_info& dev) {
    cudaError_t e = configure_decode_mma();
    if (e == cudaSuccess) e = configure_prefill_umma(dev);
    if (e == cudaSuccess) e = configure_skinny_umma();
    if (e == cudaSuccess) e = configure_decode_wide();
    if (e == cudaSuccess) e = configure_dense_gemv();
    if (e == cudaSuccess) e = configure_decode_fp4();
    if (e == cudaSuccess) e = configure_decode_fp4_stream();
    return e;
}

}  // namespace nvfp4
