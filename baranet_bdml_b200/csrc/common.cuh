// Shared helpers of the attention module: status/error plumbing and small
// device utilities.  Everything here is internal; the public surface is
// include/bn_attn.h.
#pragma once

#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <stdint.h>

#include "bn_attn.h"
#include "launch.cuh"

namespace bn {

// Records `code` and a printf-style message for bn_last_error(); returns code.
int fail(int code, const char* fmt, ...);

// BN_OK when the current device is compute capability 10.x, else BN_ERR_ARCH.
int require_sm100();

// Converts a pending launch error into BN_ERR_CUDA.
int launch_status(const char* what);

inline cudaStream_t as_stream(bn_stream_t s) { return reinterpret_cast<cudaStream_t>(s); }

inline int ceil_div(int a, int b) { return (a + b - 1) / b; }

// SMs of the current device
inline int sm_count() {
    static thread_local int known_dev = -1, sms = 148;
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev != known_dev && cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess) known_dev = dev;
    return sms;
}

// Lets `kernel` be launched with this much dynamic shared memory.  The limit belongs to the kernel, in all threads: it is set to the
// same number for every call, or a call of fewer bytes would take it from under another thread's.  `most`: that number, for kernels
// whose own arrays leave no room for 200 KB (227 KB are all there is); `own`: the bytes of those arrays, which count towards the 48 KB
// that need no asking.
constexpr size_t SMEM_MOST = 200 * 1024;
template <typename K>
inline int allow_smem(K kernel, size_t bytes, const char* what, size_t most = SMEM_MOST, size_t own = 0) {
    if (bytes + own <= 48 * 1024) return BN_OK;
    if (bytes > most) return fail(BN_ERR_UNSUPPORTED, "%s: %zu bytes of shared memory", what, bytes);
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
    return e == cudaSuccess ? BN_OK : fail(BN_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
}

// Byte offsets inside the scratch buffer of bn_attn_prefill_bf16 (cos/sin table, per-tile key norms, rotated K) and
// its size: the fused q/k/v projection writes the last two itself.
inline void prefill_bf16_workspace_layout(int B, int S, int Hkv, size_t* table, size_t* kmax2, size_t* krot, size_t* total) {
    auto up = [](size_t x) { return (x + 255) / 256 * 256; };
    *table = 256;                                                        // after the header (error word)
    *kmax2 = *table + up((size_t)S * 32 * sizeof(float2));               // [B][Hkv][key tiles of 128] largest |k|^2
    *krot = *kmax2 + up((size_t)B * Hkv * ((S + 127) / 128) * sizeof(float));
    *total = *krot + up((size_t)B * S * Hkv * 64 * sizeof(__nv_bfloat16));
}

// The times of bn_mm_f32 and of bn_linear_f32_stream in us, roughly (mm_f32.cu, mm_stream_f32.cu)
float mm_f32_estimate(int M, int N, int K);
float mm_stream_estimate(int M, int N, int K);

// The RoPE frequency of pair i, with the reference's exact arithmetic
// (src/ops/op_rope.cuh:82): fp32 exponent, fp32 pow, reciprocal taken in
// double, rounded to fp32.
__device__ __forceinline__ float rope_inv_freq(int pair, int head_dim, float theta) {
    return (float)(1.0 / powf(theta, (float)(2 * pair) / head_dim));
}

}  // namespace bn
