// Arithmetic that the strict f32 kernels share (strict.cu, strict_step.cu): the reference's operations one by one.  Only for
// files compiled with --fmad=false.
#pragma once

#include "common.cuh"

namespace tb {

__device__ __forceinline__ float strict_expf(float x) { return (float)exp((double)x); }
__device__ __forceinline__ float strict_logf(float x) { return (float)log((double)x); }

// nn::sigmoid op by op (src/nn/activations.rs:5-14).
__device__ __forceinline__ float strict_sigmoid(float x) {
    float negative = (-x > 0.0f) ? 1.0f : 0.0f;
    float nonnegative = 1.0f - negative;
    float magnitude = x * (1.0f - negative * 2.0f);
    float z = strict_expf(-magnitude);
    float denominator = z + 1.0f;
    float a = (nonnegative != 0.0f) ? (1.0f / denominator) : 0.0f;
    float b = (negative != 0.0f) ? (z / denominator) : 0.0f;
    return a + b;
}

// nn::gelu op by op (src/nn/activations.rs:29-47).
__device__ __forceinline__ float strict_gelu(float x) {
    float negative = (-x > 0.0f) ? 1.0f : 0.0f;
    float nonnegative = 1.0f - negative;
    float magnitude = (x * (1.0f - negative * 2.0f)) * 0.70710678118654752440f;
    float t = 1.0f / (magnitude * 0.3275911f + 1.0f);
    float polynomial =
        ((((t * 1.0614054f - 1.4531521f) * t + 1.4214138f) * t - 0.28449672f) * t + 0.2548296f) * t;
    float tail = (polynomial * strict_expf(-(magnitude * magnitude))) * 0.5f;
    float a = (nonnegative != 0.0f) ? (1.0f - tail) : 0.0f;
    float b = (negative != 0.0f) ? tail : 0.0f;
    return x * (a + b);
}

// tanh form of gelu in f32 with the full-precision tanh.
__device__ __forceinline__ float strict_gelu_tanh(float x) {
    return 0.5f * x * (1.0f + tanhf(0.79788456080286536f * (x + 0.044715f * (x * x * x))));
}

// What follows the sum of an output: bias, activation, layer scale, residual, rounding, and the row it is stored in.
__device__ __forceinline__ void strict_finish(const GemmEpilogue& ep, float sum, uint32_t row, uint32_t col, void* out, uint32_t ldc) {
    float v = sum;
    if (ep.bias) v = v + ep.bias[col];
    if (ep.activation == ACT_RELU) v = fmaxf(v, 0.0f);
    else if (ep.activation == ACT_GELU) v = strict_gelu(v);
    else if (ep.activation == ACT_GELU_TANH) v = strict_gelu_tanh(v);
    if (ep.scale) v = v * ep.scale[col];
    if (ep.residual) v = ep.residual[(size_t)row * ep.ldr + col] + v;
    if (ep.round_bf16) v = round_to_bf16(v);
    size_t orow = row;
    if (ep.rows_per_session) {
        uint32_t off = ep.d_row_offset ? *ep.d_row_offset : ep.row_offset;
        orow = (size_t)(row / ep.rows_per_session) * ep.out_session_rows + off + row % ep.rows_per_session;
    }
    if (ep.out_dtype == TNSR_B200_BF16)
        reinterpret_cast<bf16*>(out)[orow * ldc + col] = __float2bfloat16_rn(v);
    else
        reinterpret_cast<float*>(out)[orow * ldc + col] = v;
}

template <typename KV>
__device__ __forceinline__ float kv_load(const KV* p, size_t i);
template <>
__device__ __forceinline__ float kv_load<float>(const float* p, size_t i) { return p[i]; }
template <>
__device__ __forceinline__ float kv_load<bf16>(const bf16* p, size_t i) { return __bfloat162float(p[i]); }

}  // namespace tb
