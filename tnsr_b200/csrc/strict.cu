// Strict f32 kernels: the arithmetic of tnsr's CPU executor, operation by
// operation, for sessions created with weight_dtype = F32.
//
// This file is compiled with --fmad=false so that no multiply is fused into a
// following add: the reference rounds every product before adding it
// (src/lib.rs:1202-1208) and its own GPU decoder forces the same with
// MatMulPrecision::StrictF32 (src/nn/kv_cache/cuda.rs:480-486).  Reductions run
// in increasing index order from a zero start.  exp/ln go through the f64
// routines and are rounded once to f32, which is the nearest-f32 result the
// host libm delivers in all but rare last-bit cases.
#include <algorithm>

#include "strict.cuh"

namespace tb {

// ---------------------------------------------------------------------------
// GEMM: a block of 256 threads owns a TM x TN tile of the output, a thread RM x RN of its elements (a sixteenth of each), K is walked in
// order through 32-deep shared tiles.  An output is one chain of rounded products and rounded sums; the RM * RN chains of a
// thread are independent of each other and hide each other's latency.  Two columns go through one packed instruction whose halves
// round as the scalar ones do: mul.rn.f32x2, then fma.rn.f32x2 with a factor of one that only the launch knows, because the
// assembler joins a packed product and a packed sum into one operation with one rounding.  The rows' values are stored twice side
// by side so that a pair of them is loaded and not made.  The next tile's global loads are in flight while a tile is worked on.
// ---------------------------------------------------------------------------
constexpr uint32_t SK = 32;
constexpr size_t SMOST = 200 * 1024;      // dynamic shared memory of a block of the kernels here, at the most

__device__ __forceinline__ uint64_t mul_f32x2(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
// sum + p, as p * one + sum
__device__ __forceinline__ uint64_t add_f32x2(uint64_t sum, uint64_t p, uint64_t one) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(p), "l"(one), "l"(sum));
    return d;
}

// Four values src[0 .. 3] along a row of `limit` values from `at` on; zeros past the end or for a row that is not there.
__device__ __forceinline__ float4 strict_load4(const float* row, uint32_t at, uint32_t limit, bool live, bool vec) {
    if (vec) return live && at < limit ? *reinterpret_cast<const float4*>(row + at) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    float4 v;
    v.x = live && at < limit ? row[at] : 0.0f;
    v.y = live && at + 1 < limit ? row[at + 1] : 0.0f;
    v.z = live && at + 2 < limit ? row[at + 2] : 0.0f;
    v.w = live && at + 3 < limit ? row[at + 3] : 0.0f;
    return v;
}

// Products of one left-hand side with up to three matrices of one shape, blockIdx.z = which: the query, key and value projections of a narrow model
// are 182 tiles each at 48 x 121 rows, a block on most SMs and two on a few, 68 us one behind the other and 40 us together.
struct StrictSets {
    const float* b[3];
    void* out[3];
    GemmEpilogue ep[3];
};

template <int TM, int TN, bool BT>
__global__ void __launch_bounds__(256)
gemm_strict_tile_kernel(const float* __restrict__ a, const __grid_constant__ StrictSets sets, uint32_t ldc, uint32_t m,
                        uint32_t k, uint32_t n, bool vec_a, bool vec_b, float one) {
    const float* __restrict__ b = sets.b[blockIdx.z];
    constexpr uint32_t RM = TM / 16, RN = TN / 16, LA = TM * SK / 4 / 256, LB = TN * SK / 4 / 256;      // LA, LB: float4 loads per thread (1 or 2)
    __shared__ __align__(16) float as[SK][2 * TM];                // every value twice
    __shared__ __align__(16) float bs[SK][TN];
    const uint32_t tid = threadIdx.x, tx = tid % 16, ty = tid / 16, row0 = blockIdx.y * TM, col0 = blockIdx.x * TN;
    float4 ra[LA], rb[LB];
    auto fetch = [&](uint32_t k0) {
#pragma unroll
        for (uint32_t i = 0; i < LA; ++i) {
            const uint32_t e = tid + i * 256, r = e % TM, q = e / TM;    // along k: lanes on different rows, so that stores do not collide
            ra[i] = strict_load4(a + (size_t)(row0 + r) * k, k0 + 4 * q, k, row0 + r < m, vec_a);
        }
#pragma unroll
        for (uint32_t i = 0; i < LB; ++i) {
            const uint32_t e = tid + i * 256;
            if (BT) {
                const uint32_t r = e % TN, q = e / TN;
                rb[i] = strict_load4(b + (size_t)(col0 + r) * k, k0 + 4 * q, k, col0 + r < n, vec_b);
            } else {
                const uint32_t p = e / (TN / 4), c = e % (TN / 4);
                rb[i] = strict_load4(b + (size_t)(k0 + p) * n, col0 + 4 * c, n, k0 + p < k, vec_b);
            }
        }
    };
    uint64_t acc[RM][RN / 2];
#pragma unroll
    for (uint32_t i = 0; i < RM; ++i)
#pragma unroll
        for (uint32_t j = 0; j < RN / 2; ++j) acc[i][j] = 0;
    const uint64_t one2 = (uint64_t)__float_as_uint(one) << 32 | __float_as_uint(one);
    fetch(0);
    for (uint32_t k0 = 0; k0 < k; k0 += SK) {
        __syncthreads();
#pragma unroll
        for (uint32_t i = 0; i < LA; ++i) {
            const uint32_t e = tid + i * 256, r = e % TM, q = e / TM;
            const float va[4] = {ra[i].x, ra[i].y, ra[i].z, ra[i].w};
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j) *reinterpret_cast<float2*>(&as[4 * q + j][2 * r]) = make_float2(va[j], va[j]);
        }
#pragma unroll
        for (uint32_t i = 0; i < LB; ++i) {
            const uint32_t e = tid + i * 256, r = e % TN, q = e / TN;
            const float vb[4] = {rb[i].x, rb[i].y, rb[i].z, rb[i].w};
            if (!BT) *reinterpret_cast<float4*>(&bs[e / (TN / 4)][4 * (e % (TN / 4))]) = rb[i];
#pragma unroll
            for (uint32_t j = 0; BT && j < 4; ++j) bs[4 * q + j][r] = vb[j];
        }
        __syncthreads();
        if (k0 + SK < k) fetch(k0 + SK);
        auto step = [&](uint32_t p) {
            uint64_t av[RM], bv[RN / 2];
            const ulonglong2* ap = reinterpret_cast<const ulonglong2*>(&as[p][2 * RM * ty]);
#pragma unroll
            for (uint32_t i = 0; i < RM / 2; ++i) { const ulonglong2 v = ap[i]; av[2 * i] = v.x; av[2 * i + 1] = v.y; }
            if (RN == 2) {
                bv[0] = *reinterpret_cast<const uint64_t*>(&bs[p][2 * tx]);
            } else {
                const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(&bs[p][RN * tx]);
                bv[0] = v.x;
                bv[RN / 2 - 1] = v.y;
            }
#pragma unroll
            for (uint32_t i = 0; i < RM; ++i)
#pragma unroll
                for (uint32_t j = 0; j < RN / 2; ++j) acc[i][j] = add_f32x2(acc[i][j], mul_f32x2(av[i], bv[j]), one2);
        };
        if (k - k0 >= SK) {
#pragma unroll 8
            for (uint32_t p = 0; p < SK; ++p) step(p);
        } else {
            for (uint32_t p = 0; p < k - k0; ++p) step(p);     // never a product past the end: it would be a rounded sum more
        }
    }
#pragma unroll
    for (uint32_t i = 0; i < RM; ++i)
#pragma unroll
        for (uint32_t j = 0; j < RN; ++j) {
            const uint32_t row = row0 + RM * ty + i, col = col0 + RN * tx + j;
            const uint32_t bits = (uint32_t)(acc[i][j / 2] >> (j % 2 ? 32 : 0));
            if (row < m && col < n) strict_finish(sets.ep[blockIdx.z], __uint_as_float(bits), row, col, sets.out[blockIdx.z], ldc);
        }
}

template <int TM, int TN>
static void launch_strict_tile(const float* a, const StrictSets& sets, uint32_t count, uint32_t ldc, uint32_t m, uint32_t k, uint32_t n, bool b_transposed,
                               cudaStream_t stream) {
    const bool vec_a = k % 4 == 0 && reinterpret_cast<uintptr_t>(a) % 16 == 0;
    bool vec_b = (b_transposed ? k : n) % 4 == 0;
    for (uint32_t i = 0; i < count; ++i) vec_b = vec_b && reinterpret_cast<uintptr_t>(sets.b[i]) % 16 == 0;
    const dim3 grid(ceil_div(n, (uint32_t)TN), ceil_div(m, (uint32_t)TM), count);
    if (b_transposed) gemm_strict_tile_kernel<TM, TN, true><<<grid, 256, 0, stream>>>(a, sets, ldc, m, k, n, vec_a, vec_b, 1.0f);
    else gemm_strict_tile_kernel<TM, TN, false><<<grid, 256, 0, stream>>>(a, sets, ldc, m, k, n, vec_a, vec_b, 1.0f);
}

// Few rows (decode steps, short prefills): one block per (row, 32 output columns).  The sum of an output is
// still ONE sequential chain in increasing k -- that is the reference's arithmetic -- but the terms are
// independent of the chain, so all 512 threads first form the rounded products a[row,p] * b[p,col] side by
// side into shared memory (every global load of the block is in flight at once), and then one lane per column
// walks its K products in order.  Same values, same order of additions as gemm_strict_tile_kernel.
constexpr int SR_COLS = 32, SR_THREADS = 512;

template <bool BT>
__global__ void __launch_bounds__(SR_THREADS)
gemm_strict_rows_kernel(const float* __restrict__ a, const __grid_constant__ StrictSets sets, uint32_t ldc, uint32_t m, uint32_t k, uint32_t n) {
    const float* __restrict__ b = sets.b[blockIdx.z];
    extern __shared__ float prod[];   // [k][SR_COLS]
    const uint32_t row = blockIdx.y, col0 = blockIdx.x * SR_COLS;
    const float* ar = a + (size_t)row * k;
    if (BT) {
        // b is [n, k]: lanes run along p so that a warp reads one contiguous piece of a b row
        for (uint32_t e = threadIdx.x; e < k * SR_COLS; e += SR_THREADS) {
            const uint32_t c = e / k, p = e % k, col = col0 + c;
            prod[p * SR_COLS + c] = col < n ? ar[p] * b[(size_t)col * k + p] : 0.0f;
        }
    } else {
        for (uint32_t e = threadIdx.x; e < k * SR_COLS; e += SR_THREADS) {
            const uint32_t p = e / SR_COLS, c = e % SR_COLS, col = col0 + c;
            prod[e] = col < n ? ar[p] * b[(size_t)p * n + col] : 0.0f;
        }
    }
    __syncthreads();
    const uint32_t col = col0 + threadIdx.x;
    if (threadIdx.x >= SR_COLS || col >= n) return;
    float sum = 0.0f;
#pragma unroll 8
    for (uint32_t p = 0; p < k; ++p) sum = sum + prod[p * SR_COLS + threadIdx.x];
    strict_finish(sets.ep[blockIdx.z], sum, row, col, sets.out[blockIdx.z], ldc);
}

static int launch_gemm_strict_sets(const float* a, const StrictSets& sets, uint32_t count, uint32_t ldc, uint32_t m, uint32_t k, uint32_t n,
                                   bool b_transposed, cudaStream_t stream) {
    if (m == 0 || n == 0) return TNSR_B200_OK;
    const size_t rows_smem = (size_t)k * SR_COLS * sizeof(float);
    if (m <= 64 && k > 0 && rows_smem <= SMOST) {
        if (rows_smem > 48 * 1024) {
            const int rc = b_transposed ? allow_shared<gemm_strict_rows_kernel<true>>(SMOST, "gemm_strict_rows attribute")
                                        : allow_shared<gemm_strict_rows_kernel<false>>(SMOST, "gemm_strict_rows attribute");
            if (rc) return rc;
        }
        dim3 grid(ceil_div(n, SR_COLS), m, count);
        if (b_transposed)
            gemm_strict_rows_kernel<true><<<grid, SR_THREADS, rows_smem, stream>>>(a, sets, ldc, m, k, n);
        else
            gemm_strict_rows_kernel<false><<<grid, SR_THREADS, rows_smem, stream>>>(a, sets, ldc, m, k, n);
        count_launch();
        return check_launch("gemm_strict_rows");
    }
    if (ceil_div(m, 16u) > 65535u) {
        set_thread_error("strict GEMM: too many rows for one launch");
        return TNSR_B200_ERR_UNSUPPORTED;
    }
    // A block is latency first: what a tile costs is its first wave and, less, every further one of an SM.  us at k = 512 by blocks per SM
    // (1, 2, 3, 4): 64 x 64 tiles 37, 63, 90, 117; 32 x 64 22, 39, 57, 74; 32 x 32 17, 29, 41, 52.  (64 x 64 wherever there was one for every SM, else
    // 32 x 32, the rule before: 5808 x 512 x 128 63 us, 56 here; 2000 x 512 x 128 29 / 25; 700 x 768 x 768 77 / 53; 5808 x 128 x 96 23 / 18.)
    auto cost = [&](uint32_t tm, uint32_t tn, uint32_t first, uint32_t wave) {
        return first + wave * ceil_div64((uint64_t)ceil_div(m, tm) * ceil_div(n, tn) * count, 148u);
    };
    const uint64_t c64 = cost(64, 64, 110, 262), c48 = cost(32, 64, 42, 175), c32 = cost(32, 32, 46, 119);
    if (c64 <= std::min(c48, c32)) launch_strict_tile<64, 64>(a, sets, count, ldc, m, k, n, b_transposed, stream);
    else if (c48 <= c32) launch_strict_tile<32, 64>(a, sets, count, ldc, m, k, n, b_transposed, stream);
    else launch_strict_tile<32, 32>(a, sets, count, ldc, m, k, n, b_transposed, stream);
    count_launch();
    return check_launch("gemm_strict");
}

int launch_gemm_strict(const float* a, const float* b, void* out, uint32_t ldc, uint32_t m, uint32_t k,
                       uint32_t n, bool b_transposed, const GemmEpilogue& ep, cudaStream_t stream) {
    StrictSets sets = {};
    sets.b[0] = b;
    sets.out[0] = out;
    sets.ep[0] = ep;
    return launch_gemm_strict_sets(a, sets, 1, ldc, m, k, n, b_transposed, stream);
}

int launch_gemm_strict_three(const float* a, const float* const* b, void* const* out, uint32_t ldc, uint32_t m, uint32_t k, uint32_t n,
                             const GemmEpilogue* ep, cudaStream_t stream) {
    StrictSets sets;
    for (uint32_t i = 0; i < 3; ++i) {
        sets.b[i] = b[i];
        sets.out[i] = out[i];
        sets.ep[i] = ep[i];
    }
    return launch_gemm_strict_sets(a, sets, 3, ldc, m, k, n, false, stream);
}

// ---------------------------------------------------------------------------
// LayerNorm (src/nn.rs:199-212 on the interpreter's Mean reduction,
// src/lib.rs:1752-1754): mean = sum of x/n in order; var = sum of (c*c)/n in
// order; inv = exp(ln(var + eps) * -0.5); y = ((c * inv) * w) + b.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(128)
layernorm_strict_kernel(const float* __restrict__ x, const float* __restrict__ w, const float* __restrict__ b,
                        float* __restrict__ y, uint32_t width, float eps) {
    // The two sums are sequential chains in index order (the reference's arithmetic); their terms -- x/n and
    // (x - mean)^2/n -- do not depend on the chain, so all threads form them side by side and one thread adds them up.
    extern __shared__ float row[];     // [width] values, then [width] terms
    float* term = row + width;
    __shared__ float stats[2];
    const float* xr = x + (size_t)blockIdx.x * width;
    const float nf = (float)width;
    for (uint32_t c = threadIdx.x; c < width; c += blockDim.x) {
        const float v = xr[c];
        row[c] = v;
        term[c] = v / nf;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        float mean = 0.0f;
#pragma unroll 8
        for (uint32_t c = 0; c < width; ++c) mean = mean + term[c];
        stats[0] = mean;
    }
    __syncthreads();
    {
        const float mean0 = stats[0];
        for (uint32_t c = threadIdx.x; c < width; c += blockDim.x) {
            float d = row[c] - mean0;
            float sq = d * d;
            term[c] = sq / nf;
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        float var = 0.0f;
#pragma unroll 8
        for (uint32_t c = 0; c < width; ++c) var = var + term[c];
        stats[1] = strict_expf(strict_logf(var + eps) * -0.5f);
    }
    __syncthreads();
    const float mean = stats[0], inv = stats[1];
    float* yr = y + (size_t)blockIdx.x * width;
    for (uint32_t c = threadIdx.x; c < width; c += blockDim.x) {
        float d = row[c] - mean;
        yr[c] = ((d * inv) * w[c]) + b[c];
    }
}

// Many rows: a block owns 32 of them, all threads form the terms of all rows, and the 32 lanes of one warp then walk a row's
// chain each -- 32 chains in the time of one.
constexpr uint32_t LR = 32;
__global__ void __launch_bounds__(256)
layernorm_strict_rows_kernel(const float* __restrict__ x, const float* __restrict__ w, const float* __restrict__ b, float* __restrict__ y,
                             uint32_t rows, uint32_t width, float eps) {
    extern __shared__ float smem[];    // [LR][width + 1] values, then as many terms
    __shared__ float stats[2][LR];
    const uint32_t pitch = width | 1, row0 = blockIdx.x * LR, n = min(LR, rows - row0), lane = threadIdx.x % 32, warp = threadIdx.x / 32;
    float* term = smem + LR * pitch;
    const float nf = (float)width;
    for (uint32_t r = warp; r < n; r += 8)
        for (uint32_t c = lane; c < width; c += 32) {
            const float v = x[(size_t)(row0 + r) * width + c];
            smem[r * pitch + c] = v;
            term[r * pitch + c] = v / nf;
        }
    __syncthreads();
    if (threadIdx.x < n) {
        float mean = 0.0f;
#pragma unroll 8
        for (uint32_t c = 0; c < width; ++c) mean = mean + term[threadIdx.x * pitch + c];
        stats[0][threadIdx.x] = mean;
    }
    __syncthreads();
    for (uint32_t r = warp; r < n; r += 8) {
        const float mean = stats[0][r];
        for (uint32_t c = lane; c < width; c += 32) {
            const float d = smem[r * pitch + c] - mean;
            const float sq = d * d;
            term[r * pitch + c] = sq / nf;
        }
    }
    __syncthreads();
    if (threadIdx.x < n) {
        float var = 0.0f;
#pragma unroll 8
        for (uint32_t c = 0; c < width; ++c) var = var + term[threadIdx.x * pitch + c];
        stats[1][threadIdx.x] = strict_expf(strict_logf(var + eps) * -0.5f);
    }
    __syncthreads();
    for (uint32_t r = warp; r < n; r += 8) {
        const float mean = stats[0][r], inv = stats[1][r];
        for (uint32_t c = lane; c < width; c += 32) {
            const float d = smem[r * pitch + c] - mean;
            y[(size_t)(row0 + r) * width + c] = ((d * inv) * w[c]) + b[c];
        }
    }
}

// From this many rows on blocks of 32 give every SM more than a row's chain at a time.
constexpr uint32_t LR_MIN_ROWS = 1024;
constexpr size_t LR_SMEM = 100 * 1024;     // two blocks per SM at least

int launch_layernorm_strict(const float* x, const float* w, const float* b, float* out, uint32_t rows,
                            uint32_t width, float eps, cudaStream_t stream) {
    if (rows == 0) return TNSR_B200_OK;
    const size_t rows_smem = 2 * (size_t)LR * (width | 1) * sizeof(float);
    int rc;
    if (rows >= LR_MIN_ROWS && rows_smem <= LR_SMEM) {
        if (rows_smem > 48 * 1024 && (rc = allow_shared<layernorm_strict_rows_kernel>(LR_SMEM, "layernorm_strict_rows attribute"))) return rc;
        layernorm_strict_rows_kernel<<<ceil_div(rows, LR), 256, rows_smem, stream>>>(x, w, b, out, rows, width, eps);
        count_launch();
        return check_launch("layernorm_strict_rows");
    }
    size_t smem = 2 * (size_t)width * sizeof(float);
    if (smem > SMOST) {
        set_thread_error("strict LayerNorm: row does not fit shared memory");
        return TNSR_B200_ERR_UNSUPPORTED;
    }
    if (smem > 48 * 1024 && (rc = allow_shared<layernorm_strict_kernel>(SMOST, "layernorm_strict attribute"))) return rc;
    layernorm_strict_kernel<<<rows, 128, smem, stream>>>(x, w, b, out, width, eps);
    count_launch();
    return check_launch("layernorm_strict");
}

// ---------------------------------------------------------------------------
// Elementwise silu(gate) * up in the reference's op order.
// ---------------------------------------------------------------------------
__global__ void swiglu_strict_kernel(const float* __restrict__ gate, const float* __restrict__ up,
                                     float* __restrict__ out, size_t n) {
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        float g = gate[i];
        out[i] = (g * strict_sigmoid(g)) * up[i];
    }
}

int launch_swiglu_strict(const float* gate, const float* up, float* out, size_t n, cudaStream_t stream) {
    if (n == 0) return TNSR_B200_OK;
    swiglu_strict_kernel<<<(unsigned)ceil_div64(n, 256), 256, 0, stream>>>(gate, up, out, n);
    count_launch();
    return check_launch("swiglu_strict");
}

// ---------------------------------------------------------------------------
// Attention over the live prefix in the order of the decode graph
// (src/nn/kv_cache/graph.rs:82-107, src/nn.rs:158-161): score_j = (q . k_j) *
// scale + 0; m = max_j; e_j = exp(score_j - m); S = e_0 + e_1 + ... in order;
// p_j = e_j / S; out_c = sum_j p_j * v[j, c] in order.  The new rows are already
// in the cache, so every key is read from it.  One block per (session, head,
// query).
// ---------------------------------------------------------------------------
template <typename KV>
__global__ void __launch_bounds__(128)
attention_strict_kernel(const float* __restrict__ q, const KV* __restrict__ kc, const KV* __restrict__ vc,
                        float* __restrict__ out, uint32_t chunk, uint32_t position,
                        const uint32_t* __restrict__ d_position, uint32_t capacity, uint32_t heads,
                        uint32_t hd, float scale, int round_bf16) {
    extern __shared__ float smem[];
    __shared__ float red[128];
    const uint32_t t = blockIdx.x % chunk;
    const uint32_t h = (blockIdx.x / chunk) % heads;
    const uint32_t s = blockIdx.x / (chunk * heads);
    const uint32_t d = heads * hd;
    const uint32_t past = d_position ? *d_position : position;
    uint32_t total = past + t + 1;
    if (total > capacity) total = capacity;  // guarded by the host; never read past the cache
    float* qs = smem;            // [hd]
    float* sc = smem + hd;       // [total]
    const float* qr = q + ((size_t)s * chunk + t) * d + (size_t)h * hd;
    for (uint32_t c = threadIdx.x; c < hd; c += blockDim.x) qs[c] = qr[c];
    __syncthreads();
    const KV* kb = kc + (size_t)s * capacity * d + (size_t)h * hd;
    const KV* vb = vc + (size_t)s * capacity * d + (size_t)h * hd;
    float mx = -INFINITY;
    for (uint32_t j = threadIdx.x; j < total; j += blockDim.x) {
        float sum = 0.0f;
        for (uint32_t c = 0; c < hd; ++c) sum = sum + qs[c] * kv_load<KV>(kb, (size_t)j * d + c);
        float v = sum * scale;
        v = v + 0.0f;  // the mask term of visible keys
        sc[j] = v;
        mx = fmaxf(mx, v);
    }
    red[threadIdx.x] = mx;
    __syncthreads();
    for (uint32_t w = blockDim.x / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w) red[threadIdx.x] = fmaxf(red[threadIdx.x], red[threadIdx.x + w]);
        __syncthreads();
    }
    mx = red[0];
    __syncthreads();
    for (uint32_t j = threadIdx.x; j < total; j += blockDim.x) sc[j] = strict_expf(sc[j] - mx);
    __syncthreads();
    if (threadIdx.x == 0) {
        float sum = 0.0f;
        for (uint32_t j = 0; j < total; ++j) sum = sum + sc[j];
        red[0] = sum;
    }
    __syncthreads();
    const float denom = red[0];
    __syncthreads();
    for (uint32_t j = threadIdx.x; j < total; j += blockDim.x) sc[j] = sc[j] / denom;
    __syncthreads();
    float* orow = out + ((size_t)s * chunk + t) * d + (size_t)h * hd;
    for (uint32_t c = threadIdx.x; c < hd; c += blockDim.x) {
        float acc = 0.0f;
        for (uint32_t j = 0; j < total; ++j) acc = acc + sc[j] * kv_load<KV>(vb, (size_t)j * d + c);
        orow[c] = round_bf16 ? round_to_bf16(acc) : acc;
    }
}

// Chunks of new rows: a block owns QT queries of one (session, head).  The keys pass through shared memory 64 at a time, once for
// the scores and once (the values) for the outputs; every (query, key) and (query, column) is a chain of its own in the reference's
// order, with HP = head width padded to 32, 64 or 128 deciding how outputs spread over threads: a thread's NI outputs share their
// column, so a value is loaded once for all of them.  The sums over the keys of a row are walked by one lane per query.
constexpr uint32_t AT_KEYS = 64;

template <typename KV, int HP, int QT>
__global__ void __launch_bounds__(256)
attention_strict_tile_kernel(const float* __restrict__ q, const KV* __restrict__ kc, const KV* __restrict__ vc, float* __restrict__ out,
                             uint32_t chunk, uint32_t position, const uint32_t* __restrict__ d_position, uint32_t capacity, uint32_t heads,
                             uint32_t hd, float scale, int round_bf16, uint32_t pitch) {
    constexpr uint32_t NI = QT * HP / 256, QG = QT / 4;       // outputs of a thread; queries of a thread's scores
    extern __shared__ __align__(16) float smem[];
    float* qs = smem;                            // [QT][HP]
    float* kv = qs + QT * HP;                    // [AT_KEYS][HP + 1]
    float* sc = kv + AT_KEYS * (HP + 1);         // [QT][pitch]
    __shared__ float denom[QT];
    const uint32_t tid = threadIdx.x, lane = tid % 32, warp = tid / 32;
    // queries with the most keys first
    const uint32_t t0 = (gridDim.x - 1 - blockIdx.x) * QT, h = blockIdx.y, s = blockIdx.z, n = min((uint32_t)QT, chunk - t0), d = heads * hd;
    const uint32_t past = d_position ? *d_position : position;
    const uint32_t total = min(past + t0 + n, capacity);     // keys of the last query; never past the cache
    auto keys_of = [&](uint32_t i) { return min(past + t0 + min(i, n - 1) + 1, capacity); };
    const float* qr = q + ((size_t)s * chunk + t0) * d + (size_t)h * hd;
    for (uint32_t i = tid; i < QT * HP; i += 256) {
        const uint32_t r = i / HP, c = i % HP;
        qs[i] = r < n && c < hd ? qr[(size_t)r * d + c] : 0.0f;
    }
    const KV* kb = kc + (size_t)s * capacity * d + (size_t)h * hd;
    const KV* vb = vc + (size_t)s * capacity * d + (size_t)h * hd;
    auto stage = [&](const KV* base, uint32_t j0) {
        for (uint32_t i = tid; i < AT_KEYS * HP; i += 256) {
            const uint32_t r = i / HP, c = i % HP;
            if (c < hd) kv[r * (HP + 1) + c] = j0 + r < total ? kv_load<KV>(base, (size_t)(j0 + r) * d + c) : 0.0f;
        }
    };
    {
        const uint32_t key = tid % AT_KEYS, q0 = (tid / AT_KEYS) * QG;
        for (uint32_t j0 = 0; j0 < total; j0 += AT_KEYS) {
            __syncthreads();
            stage(kb, j0);
            __syncthreads();
            float sum[QG];
#pragma unroll
            for (uint32_t i = 0; i < QG; ++i) sum[i] = 0.0f;
            uint32_t c = 0;
            for (; c + 4 <= hd; c += 4) {
                float kr[4];
#pragma unroll
                for (uint32_t e = 0; e < 4; ++e) kr[e] = kv[key * (HP + 1) + c + e];
#pragma unroll
                for (uint32_t i = 0; i < QG; ++i) {
                    const float4 v = *reinterpret_cast<const float4*>(qs + (q0 + i) * HP + c);
                    sum[i] = sum[i] + v.x * kr[0];
                    sum[i] = sum[i] + v.y * kr[1];
                    sum[i] = sum[i] + v.z * kr[2];
                    sum[i] = sum[i] + v.w * kr[3];
                }
            }
            for (; c < hd; ++c)
#pragma unroll
                for (uint32_t i = 0; i < QG; ++i) sum[i] = sum[i] + qs[(q0 + i) * HP + c] * kv[key * (HP + 1) + c];
            if (j0 + key < total)
#pragma unroll
                for (uint32_t i = 0; i < QG; ++i) {
                    float v = sum[i] * scale;
                    v = v + 0.0f;  // the mask term of visible keys
                    sc[(q0 + i) * pitch + j0 + key] = v;
                }
        }
    }
    __syncthreads();
    for (uint32_t i = warp; i < n; i += 8) {
        const uint32_t keys = keys_of(i);
        float mx = -INFINITY;
        for (uint32_t j = lane; j < keys; j += 32) mx = fmaxf(mx, sc[i * pitch + j]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        for (uint32_t j = lane; j < keys; j += 32) sc[i * pitch + j] = strict_expf(sc[i * pitch + j] - mx);
    }
    __syncthreads();
    if (tid < n) {
        const uint32_t keys = keys_of(tid);
        const float* row = sc + tid * pitch;
        float sum = 0.0f;
        uint32_t j = 0;
        for (; j + 4 <= keys; j += 4) {
            const float4 v = *reinterpret_cast<const float4*>(row + j);
            sum = sum + v.x;
            sum = sum + v.y;
            sum = sum + v.z;
            sum = sum + v.w;
        }
        for (; j < keys; ++j) sum = sum + row[j];
        denom[tid] = sum;
    }
    __syncthreads();
    for (uint32_t i = warp; i < n; i += 8) {
        const uint32_t keys = keys_of(i);
        for (uint32_t j = lane; j < keys; j += 32) sc[i * pitch + j] = sc[i * pitch + j] / denom[i];
    }
    float acc[NI];
    uint32_t keys[NI];
#pragma unroll
    for (uint32_t i = 0; i < NI; ++i) {
        acc[i] = 0.0f;
        keys[i] = keys_of(tid / HP + i * (256 / HP));
    }
    const uint32_t col = tid % HP, qi = tid / HP;
    const uint32_t least = keys_of(0);           // every query of the block sees these
    for (uint32_t j0 = 0; j0 < total; j0 += AT_KEYS) {
        __syncthreads();
        stage(vb, j0);
        __syncthreads();
        const uint32_t end = min(AT_KEYS, total - j0);
        uint32_t j = 0;
        for (; j + 4 <= end && j0 + j + 4 <= least; j += 4) {
            float v[4];
#pragma unroll
            for (uint32_t e = 0; e < 4; ++e) v[e] = kv[(j + e) * (HP + 1) + col];
#pragma unroll
            for (uint32_t i = 0; i < NI; ++i) {
                const float4 p = *reinterpret_cast<const float4*>(sc + (qi + i * (256 / HP)) * pitch + j0 + j);
                acc[i] = acc[i] + p.x * v[0];
                acc[i] = acc[i] + p.y * v[1];
                acc[i] = acc[i] + p.z * v[2];
                acc[i] = acc[i] + p.w * v[3];
            }
        }
        for (; j < end; ++j) {
            const float v = kv[j * (HP + 1) + col];
#pragma unroll
            for (uint32_t i = 0; i < NI; ++i)
                if (j0 + j < keys[i]) acc[i] = acc[i] + sc[(qi + i * (256 / HP)) * pitch + j0 + j] * v;
        }
    }
    if (col >= hd) return;
#pragma unroll
    for (uint32_t i = 0; i < NI; ++i) {
        const uint32_t r = qi + i * (256 / HP);
        if (r < n) out[((size_t)s * chunk + t0 + r) * d + (size_t)h * hd + col] = round_bf16 ? round_to_bf16(acc[i]) : acc[i];
    }
}

// Shared memory of a block, or 0 if the scores of its queries do not fit.
template <int HP, int QT>
static size_t strict_tile_smem(uint32_t longest, uint32_t* pitch) {
    *pitch = (longest + 3) / 4 * 4 + 4;          // 16-byte rows that do not all start in the same bank
    const size_t bytes = ((size_t)QT * HP + AT_KEYS * (HP + 1) + (size_t)QT * *pitch) * sizeof(float);
    return bytes <= SMOST ? bytes : 0;
}

template <typename KV, int HP, int QT>
static bool launch_strict_tile_attention(const float* q, const void* kc, const void* vc, float* out, uint32_t sessions, uint32_t chunk, uint32_t position,
                                         const uint32_t* d_position, uint32_t capacity, uint32_t heads, uint32_t hd, float scale, int round_bf16,
                                         cudaStream_t stream) {
    uint32_t pitch;
    const size_t smem = strict_tile_smem<HP, QT>(d_position ? capacity : std::min(capacity, position + chunk), &pitch);
    if (!smem) return false;
    if (smem > 48 * 1024 && allow_shared<attention_strict_tile_kernel<KV, HP, QT>>(SMOST, "attention_strict_tile attribute")) return false;
    attention_strict_tile_kernel<KV, HP, QT><<<dim3(ceil_div(chunk, (uint32_t)QT), heads, sessions), 256, smem, stream>>>(
        q, (const KV*)kc, (const KV*)vc, out, chunk, position, d_position, capacity, heads, hd, scale, round_bf16, pitch);
    return true;
}

// Queries of a block of the tiled kernel, or 0: the kernel above, with a block per query.  A tile reads every key once for its queries, but its
// block walks all their chains: it pays when there are more queries than the GPU takes side by side, the more so the wider the head (below 32
// columns most of a block's lanes idle).  Long rows of scores leave room for a block or two per SM: the tiles then run in waves, which
// have to be full (16 sessions of 4 x 32, 17 ids, 4049 keys: 3889 / 5451 us), and below 32 columns they lose at any number.  32
// queries instead of 8 need shared memory for their scores and a chunk that fills them.  Measured on B200 over 2862 chunks (widths 8 to
// 128, 1 to 64 sessions, 2 to 256 ids, up to 4096 keys): none more than 6 % slower than the other kernel.  Four layers, us per block and query /
// in tiles of 8 / of 32:
//     heads x width, sessions x ids, keys
//     4 x 32    1 x   2  1024     452 /   582 /   660        4 x 32    16 x 64   1024    2885 /  969 /  975
//     4 x 32    8 x  16  1024     764 /   705 /   812        4 x 32    32 x 64    320    1908 /  853 /  771
//     8 x 8    64 x   8  1024    1277 /   933 /  2869        8 x 8     16 x 64   4096    8655 / 14925 / 14929
//     4 x 64    8 x  64  1024    2869 /  1611 /  1916        6 x 16    32 x 16   1024    1671 /  968 /  1648
static uint32_t strict_tile_queries(uint64_t units, uint32_t chunk, uint32_t hd, uint32_t longest) {
    if (chunk < 2 || hd > 128) return 0;
    const uint64_t queries = units * chunk;
    if (hd >= 32 ? queries < (chunk >= 8 ? 1024 : 1536) : chunk < 8 || longest > 2048 || queries < (hd >= 16 ? 1536 : 2048)) return 0;
    if (longest > 2048 && queries < 962 * ceil_div64(units * ceil_div(chunk, 8u), 148)) return 0;      // of a wave's 148 x 8
    return chunk >= 32 && queries >= 8192 && longest <= 640 ? 32 : 8;
}

template <typename KV, int HP>
static bool launch_strict_tile_width(uint32_t tile, const float* q, const void* kc, const void* vc, float* out, uint32_t sessions, uint32_t chunk,
                                     uint32_t position, const uint32_t* d_position, uint32_t capacity, uint32_t heads, uint32_t hd, float scale,
                                     int round_bf16, cudaStream_t stream) {
    if (tile == 32 &&
        launch_strict_tile_attention<KV, HP, 32>(q, kc, vc, out, sessions, chunk, position, d_position, capacity, heads, hd, scale, round_bf16, stream))
        return true;
    return launch_strict_tile_attention<KV, HP, 8>(q, kc, vc, out, sessions, chunk, position, d_position, capacity, heads, hd, scale, round_bf16, stream);
}

template <typename KV>
static bool launch_strict_tile_any(const float* q, const void* kc, const void* vc, float* out, uint32_t sessions, uint32_t chunk, uint32_t position,
                                   const uint32_t* d_position, uint32_t capacity, uint32_t heads, uint32_t hd, float scale, int round_bf16,
                                   cudaStream_t stream) {
    const uint32_t longest = d_position ? capacity : std::min(capacity, position + chunk);
    const uint32_t tile = strict_tile_queries((uint64_t)sessions * heads, chunk, hd, longest);
    if (!tile || heads > 65535u || sessions > 65535u) return false;
    if (hd <= 32) return launch_strict_tile_width<KV, 32>(tile, q, kc, vc, out, sessions, chunk, position, d_position, capacity, heads, hd, scale, round_bf16, stream);
    if (hd <= 64) return launch_strict_tile_width<KV, 64>(tile, q, kc, vc, out, sessions, chunk, position, d_position, capacity, heads, hd, scale, round_bf16, stream);
    return launch_strict_tile_width<KV, 128>(tile, q, kc, vc, out, sessions, chunk, position, d_position, capacity, heads, hd, scale, round_bf16, stream);
}

int launch_attention_strict(const float* q, const void* k_cache, const void* v_cache, float* out,
                            uint32_t sessions, uint32_t chunk, uint32_t position,
                            const uint32_t* d_position, uint32_t capacity, uint32_t heads,
                            uint32_t head_dim, int kv_dtype, int round_bf16, cudaStream_t stream) {
    if (sessions == 0 || chunk == 0) return TNSR_B200_OK;
    // (width as f32 / heads as f32).sqrt().recip()  -- src/nn/kv_cache/graph.rs:105
    const float scale = 1.0f / sqrtf((float)(heads * head_dim) / (float)heads);
    size_t smem = ((size_t)head_dim + capacity) * sizeof(float);
    if (smem > SMOST) {
        set_thread_error("strict attention: context does not fit shared memory");
        return TNSR_B200_ERR_UNSUPPORTED;
    }
    uint64_t blocks = (uint64_t)sessions * heads * chunk;
    if (blocks > 0x7fffffffull) {
        set_thread_error("strict attention: too many queries for one launch");
        return TNSR_B200_ERR_UNSUPPORTED;
    }
    if (kv_dtype == TNSR_B200_BF16
            ? launch_strict_tile_any<bf16>(q, k_cache, v_cache, out, sessions, chunk, position, d_position, capacity, heads, head_dim, scale, round_bf16, stream)
            : launch_strict_tile_any<float>(q, k_cache, v_cache, out, sessions, chunk, position, d_position, capacity, heads, head_dim, scale, round_bf16, stream)) {
        count_launch();
        return check_launch("attention_strict_tile");
    }
    int rc;
    if (kv_dtype == TNSR_B200_BF16) {
        if (smem > 48 * 1024 && (rc = allow_shared<attention_strict_kernel<bf16>>(SMOST, "attention_strict attribute"))) return rc;
        attention_strict_kernel<bf16><<<(unsigned)blocks, 128, smem, stream>>>(
            q, (const bf16*)k_cache, (const bf16*)v_cache, out, chunk, position, d_position, capacity, heads,
            head_dim, scale, round_bf16);
    } else {
        if (smem > 48 * 1024 && (rc = allow_shared<attention_strict_kernel<float>>(SMOST, "attention_strict attribute"))) return rc;
        attention_strict_kernel<float><<<(unsigned)blocks, 128, smem, stream>>>(
            q, (const float*)k_cache, (const float*)v_cache, out, chunk, position, d_position, capacity, heads,
            head_dim, scale, round_bf16);
    }
    count_launch();
    return check_launch("attention_strict");
}

}  // namespace tb
