// Last step of the NVFP4 tensor-core GEMVs' epilogue (decode_fp4.cu, decode_fp4_stream.cu): a thread holds
// the finished FP32 sums of one weight row for every token and stores them.
#pragma once
#include <cuda_bf16.h>

#include "nvfp4_format.cuh"
#include "ptx.cuh"

namespace nvfp4 {

struct Fp4Out {
    const __nv_bfloat16* residual;
    __nv_bfloat16* C;
    float inv_gs;
    int M, N;
    int out_f32;        // unrounded FP32 sums, no residual
    int swiglu_out;     // weight rows interleaved in slabs of 16 (8 gate rows, their 8 up rows): C is [M, N/2] = bf16(silu(gate) * up)
};

// The residual of a row, asked for before the row's sums are there: at the end of a call it would be a trip to L2 or memory more
// (5120 x 17408 at 8 / 16 tokens 17.7 -> 16.2, 21.5 -> 19.1 us, with the token factors in shared memory for the same reason).  No
// other thread's element is read: the residual may be C itself.
template <int KTOK>
__device__ __forceinline__ void fp4_ask_residual(unsigned short (&res)[KTOK], const Fp4Out& o, int tile, int te) {
    const int n = tile * 128 + te;
#pragma unroll
    for (int m = 0; m < KTOK; ++m)
        if (m < o.M && n < o.N) res[m] = reinterpret_cast<const unsigned short*>(o.residual)[(size_t)m * o.N + n];
}

// te: the thread's row within the 128-row tile (= its tensor-memory lane); res: as fp4_ask_residual left it (not read without a
// residual).  Called by whole warps.  The output's form is decided once, not per token (sixteen tokens took 1.3 us so).
template <int KTOK>
__device__ __forceinline__ void fp4_store_rows(const float (&v)[KTOK], const unsigned short (&res)[KTOK], const Fp4Out& o, int tile, int te) {
    const int n = tile * 128 + te, M = o.M;
    const float inv_gs = o.inv_gs;
    if (o.swiglu_out) {
        // A gate row and its up row sit 8 lanes apart in one warp.  The projection's outputs are rounded to BF16 as
        // the separate kernels would store them, then silu(gate) * up with one more rounding (the reference's
        // SwiGLU, src/engine/light_ops.cu:186-187).  Of two tokens the gate lane finishes the first, the up lane the second.
        const int late = (te >> 3) & 1;
        const size_t stride = (size_t)(o.N / 2);
        __nv_bfloat16* dst = o.C + tile * 64 + (te >> 4) * 8 + (te & 7) + (late ? stride : 0);
#pragma unroll
        for (int m = 0; m < KTOK; m += 2) {
            if (m >= M) break;
            const float a = __bfloat162float(__float2bfloat16_rn(v[m] * inv_gs));
            const float b = m + 1 < KTOK ? __bfloat162float(__float2bfloat16_rn(v[m + 1 < KTOK ? m + 1 : m] * inv_gs)) : 0.0f;
            const float other = __shfl_xor_sync(0xffffffffu, late ? a : b, 8);
            const float y = silu(late ? other : a) * (late ? b : other);
            if (m + late < M && n < o.N) *dst = __float2bfloat16_rn(y);
            dst += 2 * stride;
        }
        return;
    }
    if (n >= o.N) return;
    if (o.out_f32) {
        float* dst = reinterpret_cast<float*>(o.C) + n;
#pragma unroll
        for (int m = 0; m < KTOK; ++m, dst += o.N) if (m < M) *dst = v[m] * inv_gs;
        return;
    }
    __nv_bfloat16* dst = o.C + n;
    if (o.residual) {
#pragma unroll
        for (int m = 0; m < KTOK; ++m, dst += o.N) if (m < M) *dst = __float2bfloat16_rn(v[m] * inv_gs + bf16_bits_to_float(res[m]));
    } else {
#pragma unroll
        for (int m = 0; m < KTOK; ++m, dst += o.N) if (m < M) *dst = __float2bfloat16_rn(v[m] * inv_gs);
    }
}

// FP32 partial sums on their way from one CTA to another: three tokens of a row and the launch's tag in sixteen bytes, which travel
// as one access ([CTA][group of three tokens][128 rows] x {value, value, value, tag}).  A word without a token holds the tag too
// and is compared as well: where the reader ignored it, the load came apart (sixteen tokens, the last alone in its group:
// now and then a new tag beside an old value).
constexpr int kQuadTokens = 3;
__host__ __device__ constexpr int quads_of(int tokens) { return (tokens + kQuadTokens - 1) / kQuadTokens; }

template <int KTOK>
__device__ __forceinline__ void fp4_publish(const float (&v)[KTOK], unsigned char* slot, int M, int te, unsigned int tag) {
#pragma unroll
    for (int g = 0; g < quads_of(KTOK); ++g) {
        if (g * kQuadTokens >= M) break;
        uint32_t w[kQuadTokens];
#pragma unroll
        for (int i = 0; i < kQuadTokens; ++i) {
            const int m = g * kQuadTokens + i;
            w[i] = m < KTOK ? __float_as_uint(v[m < KTOK ? m : 0]) : tag;
        }
        ptx::st_relaxed_b128(slot + (g * 128 + te) * 16, w[0], w[1], w[2], tag);
    }
}

// Requests GN groups of three tokens of CN CTAs together (one trip to L2), asks again until all carry this launch's tag,
// then adds them to v in CTA order per token.  Bounded; false after the budget.
template <int KTOK, int CN, int GN>
__device__ __forceinline__ bool fp4_gather_block(float (&v)[KTOK], const unsigned char* pairs, size_t slot_bytes, int first, int last,
                                                 int groups, int te, unsigned int tag, volatile int* abort_flag,
                                                 unsigned int* status, unsigned int code) {
    const long long t0 = clock64();
    for (int c0 = first; c0 <= last; c0 += CN) {
        while (true) {
            uint4 x[CN][GN];
            bool ready = true;
#pragma unroll
            for (int ci = 0; ci < CN; ++ci)
#pragma unroll
                for (int g = 0; g < GN; ++g) {
                    x[ci][g] = make_uint4(0u, tag, tag, tag);
                    if (g < groups && c0 + ci <= last) x[ci][g] = ptx::ld_relaxed_b128(pairs + (size_t)(c0 + ci) * slot_bytes + (g * 128 + te) * 16);
                }
#pragma unroll
            for (int ci = 0; ci < CN; ++ci)
#pragma unroll
                for (int g = 0; g < GN; ++g) {
                    ready &= x[ci][g].w == tag;
                    if (g * kQuadTokens + 1 >= KTOK) ready &= x[ci][g].y == tag;
                    if (g * kQuadTokens + 2 >= KTOK) ready &= x[ci][g].z == tag;
                }
            if (ready) {
#pragma unroll
                for (int ci = 0; ci < CN; ++ci)
#pragma unroll
                    for (int g = 0; g < GN; ++g) {
                        const uint32_t w[3] = {x[ci][g].x, x[ci][g].y, x[ci][g].z};
#pragma unroll
                        for (int i = 0; i < kQuadTokens; ++i)
                            if (g * kQuadTokens + i < KTOK && c0 + ci <= last) v[g * kQuadTokens + i] += __uint_as_float(w[i]);
                    }
                break;
            }
            if (*abort_flag || clock64() - t0 > ptx::kWaitBudgetClocks) {
                *abort_flag = 1;
                atomicCAS(status, 0u, code);
                return false;
            }
        }
    }
    return true;
}

// Adds to v the FP32 partial sums the CTAs first .. last published for this row tile (slot_bytes per CTA), in CTA order per
// token (a fixed summation order).  Each trip to L2 costs the owner ~0.7 us at the end of its call, so as many accesses travel
// together as the registers hold: up to 3 / 6 / 9 tokens four of one group / eight of two / six of three, in the sixteen-token kernel above
// six tokens twelve of six.  {value, tag} pairs before, sixteen accesses a trip and four trips for two contributors of sixteen
// tokens: 7168 x 5120 at 16 tokens 12.7 -> 10.0 us, 5120 x 17408 18.9 -> 16.4 (with the stores above), 5120 x 6144 at 12 12.0 -> 10.1;
// two decode layers of sixteen tokens 159.5 -> 140.4, of four 120.8 -> 118.3.
template <int KTOK>
__device__ __forceinline__ bool fp4_gather(float (&v)[KTOK], const unsigned char* pairs, size_t slot_bytes, int first, int last,
                                           int M, int te, unsigned int tag, volatile int* abort_flag, unsigned int* status,
                                           unsigned int code) {
    constexpr int G = quads_of(KTOK);
    const int groups = quads_of(M);
    if (G == 1 || groups == 1) return fp4_gather_block<KTOK, 4, 1>(v, pairs, slot_bytes, first, last, groups, te, tag, abort_flag, status, code);
    if (G == 2 || groups == 2) return fp4_gather_block<KTOK, 4, 2>(v, pairs, slot_bytes, first, last, groups, te, tag, abort_flag, status, code);
    return fp4_gather_block<KTOK, 2, G>(v, pairs, slot_bytes, first, last, groups, te, tag, abort_flag, status, code);
}

}  // namespace nvfp4
