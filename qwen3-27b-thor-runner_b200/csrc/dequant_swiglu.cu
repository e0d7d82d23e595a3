// Whole-matrix dequantisation, SwiGLU and RMSNorm: the small bandwidth kernels beside
// the linear layer.
#include "nvfp4_format.cuh"
#include "nvfp4_internal.h"
#include "ptx.cuh"

namespace nvfp4 {
namespace {

// out[n,k] = bf16( e2m1 * (ue4m3 * inv_gs) ), bit-exact to the reference's
// fp4_dequant_kernel (src/engine/dense_gemm_fp4_sm110.cu:444-467): the block
// scale is multiplied by inv_gs in FP32 first, then by the table value, then
// rounded once.  One thread per scale block: 8 packed bytes in, 32 bytes out.
__global__ void __launch_bounds__(256)
dequant_bf16_kernel(const uint8_t* __restrict__ packed, const uint8_t* __restrict__ scale,
                    __nv_bfloat16* __restrict__ out, float inv_gs, long long total_groups) {
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x; g < total_groups; g += stride) {
        const float gs = ue4m3_to_float(scale[g]) * inv_gs;
        const uint2 pk = *reinterpret_cast<const uint2*>(packed + g * 8);
        uint32_t o[8];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const __nv_bfloat16 lo0 = __float2bfloat16_rn(e2m1_lut((pk.x >> (8 * j)) & 0xFu) * gs);
            const __nv_bfloat16 hi0 = __float2bfloat16_rn(e2m1_lut((pk.x >> (8 * j + 4)) & 0xFu) * gs);
            const __nv_bfloat16 lo1 = __float2bfloat16_rn(e2m1_lut((pk.y >> (8 * j)) & 0xFu) * gs);
            const __nv_bfloat16 hi1 = __float2bfloat16_rn(e2m1_lut((pk.y >> (8 * j + 4)) & 0xFu) * gs);
            o[j] = (uint32_t)__bfloat16_as_ushort(lo0) | ((uint32_t)__bfloat16_as_ushort(hi0) << 16);
            o[4 + j] = (uint32_t)__bfloat16_as_ushort(lo1) | ((uint32_t)__bfloat16_as_ushort(hi1) << 16);
        }
        uint4* dst = reinterpret_cast<uint4*>(out + g * 16);
        dst[0] = make_uint4(o[0], o[1], o[2], o[3]);
        dst[1] = make_uint4(o[4], o[5], o[6], o[7]);
    }
}

// silu(x) = x / (1 + exp(-x)) in FP32, product rounded once to BF16
// (src/engine/light_ops.cu:168-199 and :1542-1577).  gate and up rows are
// row_stride_in elements apart (I for separate tensors, 2I for the merged layout).  interleaved:
// the input row holds slabs of 16 columns, 8 gate values followed by their 8 up values (the
// output of a linear on row-interleaved gate/up weights); gate points at column 0, up at column 8.
// Few tokens: bound by the launch, so it starts while the kernel before it finishes and lets the one behind it start its
// prologue (a few-token linear: its weight stream).  With the norm below: an MLP of 5120 x 17408 on 40 tokens 69.8 -> 64.9 us,
// two decode layers of 4 tokens 132.8 -> 131.0 (replayed from a graph, where plain launches follow each other faster).
// One vector of eight outputs a thread and step: two in flight took 53 registers instead of 34, and so half as many threads on an SM
// (149 x 17408 4.3 us, with two 5.2; 1024 x 5120 7.4 and 8.9; 8192 x 17408 166 and 167).

__global__ void __launch_bounds__(256)
swiglu_kernel(const __nv_bfloat16* gate, const __nv_bfloat16* up,
              __nv_bfloat16* out, long long row_stride_in, long long row_stride_out, int M, int I,
              int interleaved) {
    ptx::griddep_launch_dependents();
    ptx::griddep_wait();                       // gate and up are the output of the kernel before this one
    const int vec_per_row = I >> 3;
    const long long total = (long long)M * vec_per_row;
    const long long stride = (long long)gridDim.x * blockDim.x;
    long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (v < total) {
        const unsigned vec = (unsigned)vec_per_row;
        int m = total <= 0xffffffffLL ? (int)((unsigned)v / vec) : (int)(v / vec_per_row);
        int c = (int)(v - (long long)m * vec_per_row);
        auto one = [&]() {
            const size_t from = (size_t)m * row_stride_in + (interleaved ? 16 : 8) * c;
            const uint4 g4 = *reinterpret_cast<const uint4*>(gate + from), u4 = *reinterpret_cast<const uint4*>(up + from);
            *reinterpret_cast<uint4*>(out + (size_t)m * row_stride_out + c * 8) = swiglu_bf16x8(g4, u4);
        };
        one();
        if ((v += stride) < total) {
            // row and column carried along instead of divided out each time (the grid is small: 32 bits hold the stride)
            const int dm = (int)((unsigned)stride / vec), dc = (int)((unsigned)stride - (unsigned)dm * vec);
            do {
                m += dm;
                c += dc;
                if (c >= vec_per_row) { c -= vec_per_row; ++m; }
                one();
            } while ((v += stride) < total);
        }
    }
    // I % 8 tail columns, scalar.
    const int tail0 = vec_per_row * 8;
    if (tail0 < I) {
        const long long ttotal = (long long)M * (I - tail0);
        for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < ttotal; t += stride) {
            const int m = (int)(t / (I - tail0)), c = tail0 + (int)(t % (I - tail0));
            const float g = __bfloat162float(gate[(size_t)m * row_stride_in + c]);
            const float u = __bfloat162float(up[(size_t)m * row_stride_in + c]);
            out[(size_t)m * row_stride_out + c] = __float2bfloat16_rn(silu(g) * u);
        }
    }
}

// Launch with programmatic stream serialization: the kernel's prologue may run while the kernel before it finishes.
template <class... P, class... A>
cudaError_t launch_behind(void (*kernel)(P...), int grid, int threads, cudaStream_t s, A... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(threads);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

int grid_for(long long work_items, int block) {
    long long blocks = (work_items + block - 1) / block;
    const long long cap = 148LL * 16;   // a few waves of 148 SMs; kernels grid-stride beyond it
    if (blocks > cap) blocks = cap;
    if (blocks < 1) blocks = 1;
    return (int)blocks;
}

}  // namespace

cudaError_t launch_dequant_bf16(const uint8_t* packed, const uint8_t* scale, float inv_gs, int N, int K,
                                void* out, cudaStream_t s) {
    const long long groups = (long long)N * (K >> 4);
    dequant_bf16_kernel<<<grid_for(groups, 256), 256, 0, s>>>(packed, scale, static_cast<__nv_bfloat16*>(out),
                                                            inv_gs, groups);
    return cudaGetLastError();
}

namespace {

// How many block-scale bytes of a weight are 0x7F or 0xFF: 480 to the reference's decoder
// (src/engine/dense_gemm_fp4_sm110.cu:30-41), NaN to the tensor core's FP8 E4M3.  16 bytes per load where the
// pointer allows it, byte by byte for the rest.
__global__ void __launch_bounds__(256)
count_nan_scales_kernel(const uint8_t* __restrict__ scale, long long bytes, unsigned long long* count) {
    const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x, nthr = (long long)gridDim.x * blockDim.x;
    const long long vecs = (reinterpret_cast<uintptr_t>(scale) & 15u) == 0 ? bytes >> 4 : 0;
    unsigned int n = 0;
    for (long long i = tid; i < vecs; i += nthr) {
        const uint4 x = __ldg(reinterpret_cast<const uint4*>(scale) + i);
        n += (__popc(__vcmpeq4(x.x | 0x80808080u, 0xFFFFFFFFu)) + __popc(__vcmpeq4(x.y | 0x80808080u, 0xFFFFFFFFu)) +
              __popc(__vcmpeq4(x.z | 0x80808080u, 0xFFFFFFFFu)) + __popc(__vcmpeq4(x.w | 0x80808080u, 0xFFFFFFFFu))) >> 3;
    }
    for (long long i = (vecs << 4) + tid; i < bytes; i += nthr) n += (scale[i] & 0x7Fu) == 0x7Fu;
    n = __reduce_add_sync(0xffffffffu, n);
    if ((threadIdx.x & 31) == 0 && n) atomicAdd(count, (unsigned long long)n);
}

}  // namespace

cudaError_t launch_count_nan_scales(const uint8_t* scale, long long bytes, unsigned long long* count, cudaStream_t s) {
    count_nan_scales_kernel<<<grid_for((bytes + 15) >> 4, 256), 256, 0, s>>>(scale, bytes, count);
    return cudaGetLastError();
}

namespace {

// RMSNorm with the centred weight, one CTA per token:
//   out = bf16( (x * rsqrt(mean(x^2) + eps)) * (1 + w) ), FP32 throughout
// (rmsnorm_kernel, src/engine/light_ops.cu:65-106).  BIAS: the row is x + bias first, kept
// unrounded for the norm, and bf16(x + bias) goes back to x (fused_add_rmsnorm_kernel, :270-318).
// 16-byte chunks; a thread keeps up to kNormCache chunks in registers between the two passes, as the BF16 they
// came as, and reads the row again beyond that.  1/sqrtf and a true division, not the fast-math forms.
// Bound by latency: a launch, one trip to memory, two barriers.  So all loads (without a bias the weight's too) go out before the
// first use, the kernel starts while the one before it finishes and lets the one behind it do the same; for that a CTA has to
// fit beside a persistent GEMV's (128 registers x 384 threads), hence at most 64 registers, at 20 (8 with a bias) bytes of spills.
constexpr int kNormThreads = 256;
constexpr int kNormCache = 4, kNormBiasCache = 3;   // x 256 threads x 8 elements: 8192 (6144 with a bias) columns from registers

template <bool BIAS>
__global__ void __launch_bounds__(kNormThreads, 4)
rmsnorm_kernel(__nv_bfloat16* out, __nv_bfloat16* x, const __nv_bfloat16* bias, const __nv_bfloat16* weight, float eps, int K) {
    __shared__ float s_part[kNormThreads / 32];
    constexpr int kHeld = BIAS ? kNormBiasCache : kNormCache;
    const int tid = threadIdx.x;
    const size_t row = (size_t)blockIdx.x * K;
    const int chunks = K >> 3;
    ptx::griddep_launch_dependents();
    ptx::griddep_wait();                      // x (and bias) are the output of the kernel before this one
    auto load_x = [&](int c) { return *reinterpret_cast<const uint4*>(x + row + (size_t)c * 8); };
    auto load_b = [&](int c) { return *reinterpret_cast<const uint4*>(bias + row + (size_t)c * 8); };
    auto load_w = [&](int c) { return *reinterpret_cast<const uint4*>(weight + (size_t)c * 8); };
    auto values = [&](const uint4& a, const uint4& b, float (&v)[8]) {
        const uint32_t aw[4] = {a.x, a.y, a.z, a.w}, bw[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            v[2 * i] = __uint_as_float(aw[i] << 16);
            v[2 * i + 1] = __uint_as_float(aw[i] & 0xFFFF0000u);
            if (BIAS) {
                v[2 * i] += __uint_as_float(bw[i] << 16);
                v[2 * i + 1] += __uint_as_float(bw[i] & 0xFFFF0000u);
            }
        }
    };
    uint4 xs[kHeld], bs[BIAS ? kHeld : 1], ws[kHeld];
#pragma unroll
    for (int j = 0; j < kHeld; ++j) {
        const int c = tid + j * kNormThreads;
        xs[j] = c < chunks ? load_x(c) : make_uint4(0u, 0u, 0u, 0u);
        if (BIAS) bs[j] = c < chunks ? load_b(c) : make_uint4(0u, 0u, 0u, 0u);
    }
    if (!BIAS) {
#pragma unroll
        for (int j = 0; j < kHeld; ++j)
            if (tid + j * kNormThreads < chunks) ws[j] = load_w(tid + j * kNormThreads);
    }
    float ss = 0.0f;
#pragma unroll
    for (int j = 0; j < kHeld; ++j) {            // chunks beyond the row are zeros
        float v[8];
        values(xs[j], bs[BIAS ? j : 0], v);
#pragma unroll
        for (int i = 0; i < 8; ++i) ss = fmaf(v[i], v[i], ss);
    }
    for (int c = tid + kHeld * kNormThreads; c < chunks; c += kNormThreads) {
        float v[8];
        values(load_x(c), BIAS ? load_b(c) : make_uint4(0u, 0u, 0u, 0u), v);
#pragma unroll
        for (int i = 0; i < 8; ++i) ss = fmaf(v[i], v[i], ss);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if ((tid & 31) == 0) s_part[tid >> 5] = ss;
    if (BIAS) {                                  // here the registers have room; behind the first store a load would wait for the one before
#pragma unroll
        for (int j = 0; j < kHeld; ++j)
            if (tid + j * kNormThreads < chunks) ws[j] = load_w(tid + j * kNormThreads);
    }
    __syncthreads();
    float t = 0.0f;
#pragma unroll
    for (int i = 0; i < kNormThreads / 32; ++i) t += s_part[i];      // the same sum in every thread
    const float inv = 1.0f / sqrtf(t / (float)K + eps);
    auto store = [&](int c, const float (&v)[8], const uint4& w4) {
        const uint32_t ww[4] = {w4.x, w4.y, w4.z, w4.w};
        uint32_t o[4], r[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float w0 = 1.0f + __uint_as_float(ww[i] << 16), w1 = 1.0f + __uint_as_float(ww[i] & 0xFFFF0000u);
            const __nv_bfloat162 y = __floats2bfloat162_rn(v[2 * i] * inv * w0, v[2 * i + 1] * inv * w1);
            o[i] = *reinterpret_cast<const uint32_t*>(&y);
            const __nv_bfloat162 q = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
            r[i] = *reinterpret_cast<const uint32_t*>(&q);
        }
        if (BIAS) *reinterpret_cast<uint4*>(x + row + (size_t)c * 8) = make_uint4(r[0], r[1], r[2], r[3]);
        *reinterpret_cast<uint4*>(out + row + (size_t)c * 8) = make_uint4(o[0], o[1], o[2], o[3]);
    };
    // the uncached tail first: with a bias its x is still the old value only until it is stored
    for (int c = tid + kHeld * kNormThreads; c < chunks; c += kNormThreads) {
        float v[8];
        values(load_x(c), BIAS ? load_b(c) : make_uint4(0u, 0u, 0u, 0u), v);
        store(c, v, load_w(c));
    }
#pragma unroll
    for (int j = 0; j < kHeld; ++j) {
        const int c = tid + j * kNormThreads;
        float v[8];
        values(xs[j], bs[BIAS ? j : 0], v);
        if (c < chunks) store(c, v, ws[j]);
    }
}

}  // namespace

cudaError_t launch_rmsnorm(void* out, void* x, const void* bias, const void* weight, float eps, int M, int K,
                           cudaStream_t s) {
    __nv_bfloat16 *o = static_cast<__nv_bfloat16*>(out), *xb = static_cast<__nv_bfloat16*>(x);
    const __nv_bfloat16 *b = static_cast<const __nv_bfloat16*>(bias), *w = static_cast<const __nv_bfloat16*>(weight);
    return b ? launch_behind(rmsnorm_kernel<true>, M, kNormThreads, s, o, xb, b, w, eps, K)
             : launch_behind(rmsnorm_kernel<false>, M, kNormThreads, s, o, xb, b, w, eps, K);
}

cudaError_t launch_swiglu(const void* gate, const void* up, long long row_stride_in, int M, int I,
                          void* out, long long row_stride_out, cudaStream_t s, bool interleaved) {
    const long long vecs = (long long)M * ((I + 7) >> 3);
    return launch_behind(swiglu_kernel, grid_for(vecs, 256), 256, s, static_cast<const __nv_bfloat16*>(gate),
                         static_cast<const __nv_bfloat16*>(up), static_cast<__nv_bfloat16*>(out), row_stride_in, row_stride_out, M,
                         I, interleaved ? 1 : 0);
}

}  // namespace nvfp4
