// Activation pre-pass of the tcgen05 kernels: BF16 -> FP16 with an exact per-token power-of-two
// scale (largest magnitude of the token -> [2^14, 2^15)), so BF16's wider exponent range costs
// nothing; the GEMM epilogue multiplies by the inverse factor in FP32.  The tensor core takes
// both operands in one 16-bit format, and the hardware E2M1 conversion produces FP16 weights.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "nvfp4_internal.h"
#include "ptx.cuh"

namespace nvfp4 {
namespace {

constexpr int kHeld = 4;       // 16-byte vectors a thread keeps between the two steps

// One CTA per token.  Latency-bound: the row is read once (all loads of a thread in flight together) and stays in registers
// between the row maximum and the conversion; rows beyond kHeld x blockDim vectors are read again for the rest.
__global__ void __launch_bounds__(1024)
act_to_f16_kernel(const __nv_bfloat16* A, __half* out, float* unscale, int K) {
    __shared__ unsigned int s_max;
    const int m = blockIdx.x, nv = K / 8;
    const uint4* src = reinterpret_cast<const uint4*>(A + (size_t)m * K);
    uint4* dst = reinterpret_cast<uint4*>(out + (size_t)m * K);
    if (threadIdx.x == 0) s_max = 0u;
    ptx::griddep_launch_dependents();      // the GEMM behind this kernel may set itself up (few tokens: start streaming weights)
    ptx::griddep_wait();                   // A is the output of the kernel before this one: plain loads, see ptx::griddep_wait
    __syncthreads();
    unsigned int amax = 0;
    auto largest = [&](const uint4& x) {
        const uint32_t v[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
        for (int q = 0; q < 4; ++q) amax = max(amax, max(v[q] & 0x7FFFu, (v[q] >> 16) & 0x7FFFu));
    };
    uint4 held[kHeld];
#pragma unroll
    for (int j = 0; j < kHeld; ++j) {
        const int i = threadIdx.x + j * blockDim.x;
        held[j] = i < nv ? src[i] : make_uint4(0u, 0u, 0u, 0u);
    }
#pragma unroll
    for (int j = 0; j < kHeld; ++j) largest(held[j]);
    for (int i = threadIdx.x + kHeld * blockDim.x; i < nv; i += blockDim.x) largest(src[i]);
    amax = __reduce_max_sync(0xffffffffu, amax);
    if ((threadIdx.x & 31) == 0 && amax) atomicMax(&s_max, amax);
    __syncthreads();
    int se = 268 - (int)(s_max >> 7);      // scale = 2^(141 - biased exponent): largest -> exponent 14
    se = se < 1 ? 1 : (se > 254 ? 254 : se);
    const float sc = __uint_as_float((uint32_t)se << 23);
    if (threadIdx.x == 0) unscale[m] = __uint_as_float((uint32_t)(254 - se) << 23);
    auto convert = [&](const uint4& x, int i) {
        const uint32_t v[4] = {x.x, x.y, x.z, x.w};
        uint32_t y[4];
#pragma unroll
        for (int q = 0; q < 4; ++q)
            y[q] = ptx::pack_f16x2(__uint_as_float(v[q] << 16) * sc, __uint_as_float(v[q] & 0xFFFF0000u) * sc);
        dst[i] = make_uint4(y[0], y[1], y[2], y[3]);
    };
#pragma unroll
    for (int j = 0; j < kHeld; ++j) {
        const int i = threadIdx.x + j * blockDim.x;
        if (i < nv) convert(held[j], i);
    }
    for (int i = threadIdx.x + kHeld * blockDim.x; i < nv; i += blockDim.x) convert(src[i], i);
}

}  // namespace

cudaError_t launch_act_to_f16(const void* A, int M, int K, void* out_f16, float* unscale, int sm_count, cudaStream_t s) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(M);
    // as many threads as hold the row in kHeld vectors each; few tokens: half as many vectors (latency, SMs to spare)
    const int per = M <= sm_count ? kHeld / 2 : kHeld;
    int threads = ((K / 8 + per - 1) / per + 31) / 32 * 32;
    cfg.blockDim = dim3(threads < 64 ? 64 : (threads > 1024 ? 1024 : threads));
    cfg.dynamicSmemBytes = 0;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, act_to_f16_kernel, static_cast<const __nv_bfloat16*>(A), static_cast<__half*>(out_f16),
                              unscale, K);
}

}  // namespace nvfp4
