// What the GEMM engines share behind the accumulator: the parameters of an epilogue and its scalar forms, one element at a time.
#pragma once

#include "common.cuh"

namespace tb {

struct EpiParams {
    GemmEpilogue ep;
    GemmQkvTargets qkv;
    GemmSegments seg;
    void* out;
    uint32_t ldc;
    uint32_t m, n;  // n = columns of the accumulator (packed width for SWIGLU)
};

// ---- epilogue: scalar forms ---------------------------------------------------
__device__ __forceinline__ size_t map_out_row(const GemmEpilogue& ep, uint32_t row) {
    if (!ep.rows_per_session) return row;
    uint32_t off = ep.d_row_offset ? *ep.d_row_offset : ep.row_offset;
    return (size_t)(row / ep.rows_per_session) * ep.out_session_rows + off + row % ep.rows_per_session;
}

__device__ __forceinline__ void store_plain(const EpiParams& P, uint32_t row, uint32_t col, float acc) {
    float v = acc;
    if (P.ep.bias) v += P.ep.bias[col];
    v = apply_activation(v, P.ep.activation);
    size_t orow = map_out_row(P.ep, row);
    if (P.ep.out_dtype == TNSR_B200_BF16) {
        reinterpret_cast<bf16*>(P.out)[orow * P.ldc + col] = __float2bfloat16_rn(v);
    } else {
        if (P.ep.scale) v *= P.ep.scale[col];
        if (P.ep.residual) v += P.ep.residual[(size_t)row * P.ep.ldr + col];
        reinterpret_cast<float*>(P.out)[orow * P.ldc + col] = v;
    }
}

__device__ __forceinline__ void store_qkv(const EpiParams& P, uint32_t row, uint32_t col, float acc) {
    float v = acc;
    if (P.ep.bias) v += P.ep.bias[col];
    const uint32_t d = P.qkv.d, which = col / d, c = col % d;
    if (which == 0) {
        P.qkv.q[(size_t)row * d + c] = __float2bfloat16_rn(v);
    } else {
        const uint32_t session = row / P.qkv.chunk;
        uint32_t pos = P.qkv.d_position ? P.qkv.d_position[session * P.qkv.position_stride] : P.qkv.position;
        size_t crow = kv_row(P.qkv.paging, session, pos + row % P.qkv.chunk, P.qkv.capacity);
        (which == 1 ? P.qkv.k_cache : P.qkv.v_cache)[crow * d + c] = __float2bfloat16_rn(v);
    }
}

// Range of column `col` (GEMM_SEGMENTS).
__device__ __forceinline__ uint32_t segment_of(const EpiParams& P, uint32_t col) {
    uint32_t i = 0;
    if (P.seg.count > 1 && col >= P.seg.s[1].col0) i = 1;
    if (P.seg.count > 2 && col >= P.seg.s[2].col0) i = 2;
    return i;
}

__device__ __forceinline__ void store_segment(const EpiParams& P, uint32_t row, uint32_t col, float acc) {
    const GemmSegment& g = P.seg.s[segment_of(P, col)];
    const float v = apply_activation(P.ep.bias ? acc + P.ep.bias[col] : acc, g.activation);
    const size_t o = (size_t)row * g.ld + (col - g.col0);
    if (g.out_dtype == TNSR_B200_BF16) reinterpret_cast<bf16*>(g.out)[o] = __float2bfloat16_rn(v);
    else reinterpret_cast<float*>(g.out)[o] = v;
}

// g, u: accumulators of packed columns pc and pc + 16; output column oc.
__device__ __forceinline__ void store_swiglu(const EpiParams& P, uint32_t row, uint32_t pc, uint32_t oc,
                                             float g, float u) {
    if (P.ep.bias) {
        g += P.ep.bias[pc];
        u += P.ep.bias[pc + 16];
    }
    reinterpret_cast<bf16*>(P.out)[(size_t)row * P.ldc + oc] = __float2bfloat16_rn(fast_silu(g) * u);
}

// Few rows, any epilogue but GEMM_ARGMAX: operands straight into registers (gemm_few.cu).
bool gemm_few_pays(const bf16* a, const bf16* w, uint32_t m, uint32_t n, uint32_t k);
int launch_gemm_few(const bf16* a, const bf16* w, const EpiParams& epi, uint32_t k, GemmMode mode, cudaStream_t stream);

}  // namespace tb
