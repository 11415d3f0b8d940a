// A whole step of a small f32 session in one launch: embedding, every layer, final LayerNorm and output head.
//
// A step of the character model (4 layers of 128 columns) is 38 short kernels one behind the other, each about 3 us of launch, of one
// or two dependent trips to L2 and of one chain of additions (the reference's order allows no other: 128 to 512 sums of 4 cycles).
// Here a cluster of 16 CTAs takes whole sessions through the step: a layer is five phases (LayerNorm and q/k/v, attention, output
// projection, LayerNorm and first feed-forward matrix, second matrix), every CTA owns a sixteenth of a phase's output columns and
// stores them into the shared memory of all sixteen, and the phases meet at the cluster's hardware barrier (180 cycles; through global
// memory the stores took 1100 cycles to be visible and the loads 1500 to come back).  The weights of a CTA's next columns are on
// their way while it waits there.  Sessions do not depend on each other, so clusters never wait for one another.
//
// Arithmetic is strict.cu's, operation by operation: all threads form the rounded products of an output side by side in shared
// memory, one lane per output adds them up in order.  What is left is chains: sums, and the f64 exp and log of a LayerNorm and of the
// scores -- and instructions: straight-line code that runs once per phase does not stay in the nearest instruction cache, so a layer's phases are
// rounds of one loop and the sums are a function.  (All phases inlined 84 us a step on the device, so 63; inlined, with loads further ahead, 115.)
// One step of one session at 4 x 128 columns and 60 keys, ids in to logits out, B200: 197 us in 38 launches, 105 us here; 48 sessions 246 and 140 us.
#include <algorithm>

#include "strict.cuh"

namespace tb {

namespace {

constexpr uint32_t SS_CTAS = 16, SS_THREADS = 512, SS_WARPS = SS_THREADS / 32;
constexpr uint32_t SS_COLS = 32;            // columns a CTA works on at a time: one lane each
constexpr uint32_t SS_MAX_D = 256;
constexpr uint32_t SS_SMEM = 200 * 1024;
constexpr uint32_t SS_VALUES = 8192;        // weight x value products of a head in shared memory at a time

struct SsParams {
    StrictStepArgs a;
    uint32_t sessions_per_cluster;
    float part;                          // 1 / d, if that is exact
};

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }

// Stores v where `local` lies, in the shared memory of every CTA of the cluster.
__device__ __forceinline__ void store_to_all(float* local, float v) {
    const uint32_t at = (uint32_t)__cvta_generic_to_shared(local);
#pragma unroll
    for (uint32_t peer = 0; peer < SS_CTAS; ++peer) {
        uint32_t remote;
        asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(at), "r"(peer));
        asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(remote), "f"(v) : "memory");
    }
}

// The matrix of a phase: [k, n] row-major; q, k and v are three of `width` columns each side by side.
struct Matrix {
    const float *w0, *w1, *w2;
    uint32_t k, n, width;
    __device__ __forceinline__ const float* column(uint32_t j) const { return j < width ? w0 + j : j < 2 * width ? w1 + (j - width) : w2 + (j - 2 * width); }
};

// A CTA's share of a phase: columns [col0, col0 + cols) of n, at most SS_COLS of them at a time; in shared memory there is room for
// 1 << log2_pad of them, each with its k products in order (row pitch k + 4: 16-byte accesses of neighbouring lanes do not collide).
struct Share {
    uint32_t col0, cols, log2_pad;
};
__device__ __forceinline__ uint32_t per_cta(uint32_t n) { return (n + SS_CTAS - 1) / SS_CTAS; }
__device__ __forceinline__ Share share_of(uint32_t n, uint32_t rank, uint32_t round) {
    const uint32_t per = per_cta(n), first = rank * per + round * SS_COLS, end = min(n, (rank + 1) * per), room = min(per, SS_COLS);
    return {first, first < end ? min(SS_COLS, end - first) : 0u, room <= 1 ? 0u : 32u - __clz(room - 1)};
}

// Four weights of one column, one below the other.
__device__ __forceinline__ float4 weights4(const float* w, uint32_t ld) { return make_float4(__ldg(w), __ldg(w + ld), __ldg(w + 2 * (size_t)ld), __ldg(w + 3 * (size_t)ld)); }

// Thread t forms the products of column t % pad, four rows of the matrix at a time, groups of four dealt over the threads.  The first
// two groups are asked for before the phase's barrier.
__device__ __forceinline__ void ask_weights(const Matrix& m, const Share& s, float4 (&ahead)[2]) {
    const uint32_t c = threadIdx.x & ((1u << s.log2_pad) - 1), g = threadIdx.x >> s.log2_pad, groups = SS_THREADS >> s.log2_pad;
    if (c >= s.cols) return;
    const float* w = m.column(s.col0 + c);
#pragma unroll
    for (uint32_t i = 0; i < 2; ++i)
        if (4 * (g + i * groups) < m.k) ahead[i] = weights4(w + (size_t)4 * (g + i * groups) * m.width, m.width);
}
__device__ __forceinline__ void form_products(const Matrix& m, const Share& s, const float4 (&ahead)[2], bool use_ahead, const float* xs, float* prod,
                                              uint32_t rows) {
    const uint32_t c = threadIdx.x & ((1u << s.log2_pad) - 1), g = threadIdx.x >> s.log2_pad, groups = SS_THREADS >> s.log2_pad, k = m.k;
    if (c >= s.cols) return;
    const float* w = m.column(s.col0 + c);
    float* mine = prod + c * (k + 4);
    const uint32_t row_pitch = (k + 4) << s.log2_pad;
    auto put = [&](uint32_t p, const float4& v) {
        for (uint32_t r = 0; r < rows; ++r) {
            const float4 x = *reinterpret_cast<const float4*>(xs + r * k + p);
            *reinterpret_cast<float4*>(mine + r * row_pitch + p) = make_float4(x.x * v.x, x.y * v.y, x.z * v.z, x.w * v.w);
        }
    };
    uint32_t p = 4 * g;
    if (use_ahead) {
#pragma unroll
        for (uint32_t i = 0; i < 2; ++i, p += 4 * groups)
            if (p < k) put(p, ahead[i]);
    }
    for (; p < k; p += 4 * groups) put(p, weights4(w + (size_t)p * m.width, m.width));
}

// sum of terms[0 .. n) in order from a zero start, n a multiple of 4, terms 16-byte aligned in shared memory: eight values on their way while
// eight are added.
__device__ __noinline__ float add_up(uint32_t terms, uint32_t n) {
    auto quad = [](uint32_t at) {
        float4 v;
        asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(at) : "memory");
        return v;
    };
    float sum = 0.0f;
    auto add = [&](const float4& v) {
        sum = sum + v.x;
        sum = sum + v.y;
        sum = sum + v.z;
        sum = sum + v.w;
    };
    const uint32_t end = terms + 4 * n;
    uint32_t at = terms;
    if (at + 32 <= end) {
        float4 u0 = quad(at), u1 = quad(at + 16);
        at += 32;
#pragma unroll 1
        for (; at + 64 <= end; at += 64) {
            const float4 v0 = quad(at), v1 = quad(at + 16);
            add(u0);
            add(u1);
            u0 = quad(at + 32);
            u1 = quad(at + 48);
            add(v0);
            add(v1);
        }
        add(u0);
        add(u1);
    }
#pragma unroll 1
    for (; at < end; at += 16) add(quad(at));
    return sum;
}
// acc + the n values at `at`, `at` + stride bytes, ... in shared memory, in order, eight on their way while eight are added: behind thousands of keys
// these sums are half of a step.  (Eight loaded and then added, as rows of more than 128 columns have it, whose registers are full: 16 sessions x
// 6 heads of 16 x 4096 keys 788 us a step, 721 so.)
__device__ __noinline__ float add_column(uint32_t at, uint32_t stride, uint32_t n, float acc) {
    float u[8], v[8];
    auto load = [&](float (&x)[8]) {
#pragma unroll
        for (uint32_t i = 0; i < 8; ++i, at += stride) asm volatile("ld.shared.f32 %0, [%1];" : "=f"(x[i]) : "r"(at) : "memory");
    };
    auto add = [&](const float (&x)[8]) {
#pragma unroll
        for (uint32_t i = 0; i < 8; ++i) acc = acc + x[i];
    };
    if (n >= 8) {
        load(u);
#pragma unroll 1
        for (n -= 8; n >= 16; n -= 16) {
            load(v);
            add(u);
            load(u);
            add(v);
        }
        if (n >= 8) load(v);
        add(u);
        if (n >= 8) add(v), n -= 8;
    }
#pragma unroll
    for (uint32_t i = 0; i < 7; ++i, at += stride)
        if (i < n) asm volatile("ld.shared.f32 %0, [%1];" : "=f"(u[i]) : "r"(at) : "memory");
#pragma unroll
    for (uint32_t i = 0; i < 7; ++i)
        if (i < n) acc = acc + u[i];
    return acc;
}
__device__ __forceinline__ float add_up(const float* terms, uint32_t n) { return add_up((uint32_t)__cvta_generic_to_shared(terms), n); }

// Scale and shift of a LayerNorm, asked for before the phase's barrier: a warp per row, lane l holds columns l, l + 32, ...
template <uint32_t V>
__device__ __forceinline__ void ask_norm(const float* __restrict__ w, const float* __restrict__ b, uint32_t rows, uint32_t d, float (&wv)[V], float (&bv)[V]) {
    if (threadIdx.x / 32 >= rows) return;
#pragma unroll
    for (uint32_t i = 0; i < V; ++i) {
        const uint32_t c = threadIdx.x % 32 + 32 * i;
        if (c < d) wv[i] = __ldg(w + c), bv[i] = __ldg(b + c);
    }
}
// LayerNorm of row r (x + r * stride) by warp r, in strict.cu's order, into xs; `term`: d floats per row.  With a width of 2^n a term is divided
// by multiplying with `part` = 2^-n (0: another width): the same value, rounded once.
template <uint32_t V>
__device__ __forceinline__ void norm_rows(float* xs, float* term, const float* x, uint32_t stride, const float (&wv)[V], const float (&bv)[V],
                                          uint32_t rows, uint32_t d, float eps, float part) {
    const uint32_t warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    if (warp >= rows) return;
    const float nf = (float)d;
    const bool whole = part != 0.0f;
    float v[V], t[V], mean = 0.0f, inv = 0.0f;
    float* mine = term + warp * d;
#pragma unroll
    for (uint32_t i = 0; i < V; ++i)
        if (lane + 32 * i < d) t[i] = v[i] = x[warp * stride + lane + 32 * i];
#pragma unroll 1
    for (uint32_t pass = 0; pass < 2; ++pass) {      // mean, variance
#pragma unroll
        for (uint32_t i = 0; i < V; ++i)
            if (lane + 32 * i < d) mine[lane + 32 * i] = whole ? t[i] * part : t[i] / nf;
        __syncwarp();
        const float sum = __shfl_sync(0xffffffffu, lane == 0 ? add_up(mine, d) : 0.0f, 0);
        __syncwarp();
        if (pass) {
            inv = strict_expf(strict_logf(sum + eps) * -0.5f);
            break;
        }
        mean = sum;
#pragma unroll
        for (uint32_t i = 0; i < V; ++i) {
            const float c = v[i] - mean;
            t[i] = c * c;
        }
    }
#pragma unroll
    for (uint32_t i = 0; i < V; ++i)
        if (lane + 32 * i < d) {
            const float c = v[i] - mean;
            xs[warp * d + lane + 32 * i] = ((c * inv) * wv[i]) + bv[i];
        }
}

__device__ __forceinline__ float4 load_kv4(const float* p) { return __ldcg(reinterpret_cast<const float4*>(p)); }
__device__ __forceinline__ float4 load_kv4(const bf16* p) {
    const uint2 v = __ldcg(reinterpret_cast<const uint2*>(p));
    return make_float4(__uint_as_float(v.x << 16), __uint_as_float(v.x & 0xffff0000u), __uint_as_float(v.y << 16), __uint_as_float(v.y & 0xffff0000u));
}

// Attention of one (row, head) by the whole CTA, in the order of attention_strict_kernel: thread c < head width returns output c.
// `scratch`: scores, then products.
template <typename KV, bool AHEAD>
__device__ __forceinline__ float attend(const StrictStepArgs& a, const KV* kb, const KV* vb, const float* qs, uint32_t total, float* scratch) {
    __shared__ float red[SS_WARPS + 1];
    const uint32_t tid = threadIdx.x, lane = tid % 32, warp = tid / 32, hd = a.d / a.heads, quads = hd / 4, d = a.d;
    float* sc = scratch;
    float* prod = sc + (total + 3) / 4 * 4;
    const uint32_t tile = SS_VALUES / hd;            // keys whose products fit
    // the first values are asked for before anything else
    float4 early[2];
#pragma unroll
    for (uint32_t i = 0; i < 2; ++i) {
        const uint32_t e = tid + i * SS_THREADS;
        if (e < min(total, tile) * quads) early[i] = load_kv4(vb + (size_t)(e / quads) * d + 4 * (e % quads));
    }
    float mx = -INFINITY;
    for (uint32_t j = tid; j < total; j += SS_THREADS) {
        float sum = 0.0f;
        const KV* row = kb + (size_t)j * d;
#pragma unroll 4
        for (uint32_t c = 0; c < hd; c += 4) {
            const float4 k = load_kv4(row + c), v = *reinterpret_cast<const float4*>(qs + c);
            sum = sum + v.x * k.x;
            sum = sum + v.y * k.y;
            sum = sum + v.z * k.z;
            sum = sum + v.w * k.w;
        }
        float v = sum * a.scale;
        v = v + 0.0f;  // the mask term of visible keys
        sc[j] = v;
        mx = fmaxf(mx, v);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if (lane == 0) red[warp] = mx;
    __syncthreads();
    mx = red[0];
#pragma unroll
    for (uint32_t w = 1; w < SS_WARPS; ++w) mx = fmaxf(mx, red[w]);
    for (uint32_t j = tid; j < total; j += SS_THREADS) sc[j] = strict_expf(sc[j] - mx);
    __syncthreads();
    if (tid == 0) {
        float sum = add_up(sc, total & ~3u);
        for (uint32_t j = total & ~3u; j < total; ++j) sum = sum + sc[j];
        red[SS_WARPS] = sum;
    }
    __syncthreads();
    const float denom = red[SS_WARPS];
    for (uint32_t j = tid; j < total; j += SS_THREADS) sc[j] = sc[j] / denom;
    __syncthreads();
    float acc = 0.0f;
    for (uint32_t j0 = 0; j0 < total; j0 += tile) {
        const uint32_t keys = min(tile, total - j0);
        if (j0) __syncthreads();
        auto put = [&](uint32_t e, const float4& v) {
            const float p = sc[j0 + e / quads];
            reinterpret_cast<float4*>(prod)[e] = make_float4(p * v.x, p * v.y, p * v.z, p * v.w);
        };
        uint32_t e = tid;
        if (j0 == 0) {
#pragma unroll
            for (uint32_t i = 0; i < 2; ++i, e += SS_THREADS)
                if (e < keys * quads) put(e, early[i]);
        }
        for (; e < keys * quads; e += SS_THREADS) put(e, load_kv4(vb + (size_t)(j0 + e / quads) * d + 4 * (e % quads)));
        __syncthreads();
        if (tid < hd) {
            if (AHEAD) {
                acc = add_column((uint32_t)__cvta_generic_to_shared(prod + tid), 4 * hd, keys, acc);
            } else {
                const float* p = prod + tid;
#pragma unroll 8
                for (uint32_t j = 0; j < keys; ++j, p += hd) acc = acc + *p;
            }
        }
    }
    __syncthreads();
    return a.round_bf16 ? round_to_bf16(acc) : acc;
}

// Shared floats of one row: residual, queries, attention output, normalised row, its terms, hidden row.
__host__ __device__ __forceinline__ uint32_t floats_per_row(uint32_t d, uint32_t f) { return 5 * d + f; }

// V: columns of a row that a lane of a LayerNorm holds; with 4 there are registers left for values on their way in attention.
template <typename KV, uint32_t V>
__global__ void __launch_bounds__(SS_THREADS, 1)
strict_step_kernel(const __grid_constant__ SsParams P) {
    extern __shared__ __align__(16) float smem[];
    const StrictStepArgs& a = P.a;
    const uint32_t rank = blockIdx.x % SS_CTAS, cluster = blockIdx.x / SS_CTAS, tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
    const uint32_t s0 = cluster * P.sessions_per_cluster, ns = min(P.sessions_per_cluster, a.sessions - s0);
    const uint32_t row0 = s0 * a.chunk, rows = ns * a.chunk, d = a.d, f = a.f, hd = d / a.heads;
    float* h = smem;                         // [rows][d] each
    float* q = h + rows * d;
    float* att = q + rows * d;
    float* xs = att + rows * d;
    float* term = xs + rows * d;
    float* ff = term + rows * d;             // [rows][f]
    float* prod = ff + rows * f;
    float4 ahead[2];
    for (uint32_t r = 0; r < rows; ++r) {    // every CTA keeps the residual rows
        const uint32_t id = a.ids[row0 + r], position = a.position + r % a.chunk;
        if (id >= a.vocab && tid == 0 && rank == 0) atomicCAS(a.d_status, DEV_OK, DEV_TOKEN_RANGE);
        for (uint32_t c = tid; c < d; c += SS_THREADS) h[r * d + c] = id < a.vocab ? a.tok[(size_t)id * d + c] + a.pos[(size_t)position * d + c] : 0.0f;
    }
    __syncthreads();
    cluster_arrive();
    // A layer is four products, each of rows of k values (a LayerNorm of h, or what the phase before left) and the CTA's columns of a matrix;
    // attention follows the first one.  The round behind the last layer ends with the rows of the output head.
    enum : uint32_t { QKV = 0, OUT = 1, UP = 2, DOWN = 3 };
    const uint32_t products = 4 * a.num_layers, wanted = a.last_only ? ns : rows;
    auto matrix = [&](uint32_t step) {
        const StrictStepLayer& L = P.a.layers[step / 4];
        switch (step % 4) {
            case QKV: return Matrix{L.wq, L.wk, L.wv, d, 3 * d, d};
            case OUT: return Matrix{L.wo, nullptr, nullptr, d, d, d};
            case UP: return Matrix{L.w_in, nullptr, nullptr, d, f, f};
            default: return Matrix{L.w_out, nullptr, nullptr, f, d, d};
        }
    };
#pragma unroll 1
    for (uint32_t step = 0;; ++step) {
        const uint32_t kind = step % 4;
        const bool head = step == products;
        const StrictStepLayer& L = P.a.layers[head ? 0 : step / 4];
        const Matrix m = matrix(head ? 0 : step);
        const float* bias_of = kind == OUT ? L.bo : kind == UP ? L.b_in : L.b_out;
        float wv[V], bv[V];
        if (!head) ask_weights(m, share_of(m.n, rank, 0), ahead);
        if (head) ask_norm(a.fnw, a.fnb, wanted, d, wv, bv);
        else if (kind == QKV || kind == UP) ask_norm(kind == QKV ? L.ln1w : L.ln2w, kind == QKV ? L.ln1b : L.ln2b, rows, d, wv, bv);
        float bias = 0.0f;
        auto ask_bias = [&](const Share& s) {
            if (warp >= rows || lane >= s.cols) return;
            const uint32_t col = s.col0 + lane;
            bias = kind != QKV ? __ldg(bias_of + col) : __ldg(col < d ? L.bq + col : col < 2 * d ? L.bk + (col - d) : L.bv + (col - 2 * d));
        };
        if (!head) ask_bias(share_of(m.n, rank, 0));
        cluster_wait();
        if (head && !a.logits) break;
        if (head) norm_rows(xs, term, a.last_only ? h + (a.chunk - 1) * d : h, a.last_only ? a.chunk * d : d, wv, bv, wanted, d, a.eps, P.part);
        else if (kind == QKV || kind == UP) norm_rows(xs, term, h, d, wv, bv, rows, d, a.eps, P.part);
        if (head) break;
        const float* x = kind == OUT ? att : kind == DOWN ? ff : xs;
        const uint32_t rounds = (per_cta(m.n) + SS_COLS - 1) / SS_COLS;
#pragma unroll 1
        for (uint32_t round = 0; round < rounds; ++round) {
            const Share s = share_of(m.n, rank, round);
            if (round) ask_bias(s);
            __syncthreads();
            form_products(m, s, ahead, round == 0, x, prod, rows);
            __syncthreads();
            if (warp >= rows || lane >= s.cols) continue;
            const uint32_t r = warp, col = s.col0 + lane;
            const float sum = add_up(prod + (((warp << s.log2_pad) + lane) * (m.k + 4)), m.k);
            float v = sum + bias;
            float* to = h + r * d + col;
            if (kind == QKV) {
                const uint32_t part = col < d ? 0 : col < 2 * d ? 1 : 2, c = col - part * d;
                if (a.round_bf16) v = round_to_bf16(v);
                to = q + r * d + c;
                if (part != 0) {
                    KV* cache = reinterpret_cast<KV*>(part == 1 ? L.kcache : L.vcache);
                    const size_t at = ((size_t)(s0 + r / a.chunk) * a.capacity + a.position + r % a.chunk) * d + c;
                    if constexpr (sizeof(KV) == 2) cache[at] = __float2bfloat16_rn(v);
                    else cache[at] = v;
                    continue;
                }
            } else if (kind == UP) {
                v = a.activation == ACT_GELU ? strict_gelu(v) : fmaxf(v, 0.0f);
                to = ff + r * f + col;
            } else {
                v = *to + v;
            }
            store_to_all(to, v);
        }
        cluster_arrive();
        if (kind != QKV) continue;
        const KV* kcache = reinterpret_cast<const KV*>(L.kcache);
        const KV* vcache = reinterpret_cast<const KV*>(L.vcache);
        cluster_wait();
#pragma unroll 1
        for (uint32_t i = rank; i < rows * a.heads; i += SS_CTAS) {
            const uint32_t r = i / a.heads, head_at = r * d + i % a.heads * hd;
            const size_t base = (size_t)(s0 + r / a.chunk) * a.capacity * d + (size_t)(i % a.heads) * hd;
            const float v = attend<KV, V == 4>(a, kcache + base, vcache + base, q + head_at, min(a.position + r % a.chunk + 1, a.capacity), prod);
            if (tid < hd) store_to_all(att + head_at + tid, v);
        }
        cluster_arrive();
    }
    if (!a.logits) {                        // a large vocabulary: the head is a launch of its own
        for (uint32_t i = rank * SS_THREADS + tid; i < rows * d; i += SS_CTAS * SS_THREADS) a.h[(size_t)row0 * d + i] = h[i];
        return;
    }
    // the tied head: rows of the token table [vocab, d], so lanes run along d; every row, or the last one of each session
    const uint32_t per = per_cta(a.vocab), col0 = rank * per, cols = col0 < a.vocab ? min(per, a.vocab - col0) : 0u;
    for (uint32_t c0 = 0; c0 < cols; c0 += SS_COLS) {
        const uint32_t nc = min(SS_COLS, cols - c0);
        __syncthreads();
        for (uint32_t c = warp; c < nc; c += SS_WARPS)
            for (uint32_t p = 4 * lane; p < d; p += 128) {
                const float* w = a.tok + (size_t)(col0 + c0 + c) * d + p;
                const float4 v = make_float4(__ldg(w), __ldg(w + 1), __ldg(w + 2), __ldg(w + 3));
                for (uint32_t r = 0; r < wanted; ++r) {
                    const float4 x = *reinterpret_cast<const float4*>(xs + r * d + p);
                    *reinterpret_cast<float4*>(prod + (r * SS_COLS + c) * (d + 4) + p) = make_float4(x.x * v.x, x.y * v.y, x.z * v.z, x.w * v.w);
                }
            }
        __syncthreads();
        if (warp < wanted && lane < nc)
            a.logits[(size_t)((a.last_only ? s0 : row0) + warp) * a.vocab + col0 + c0 + lane] = add_up(prod + (warp * SS_COLS + lane) * (d + 4), d);
    }
}

// Rows that fit a cluster's shared memory: their values, their products in the widest phase, and a head's scores and products.
uint32_t rows_that_fit(const StrictStepArgs& a) {
    auto room = [](uint32_t n) {
        const uint32_t per = std::min(ceil_div(n, SS_CTAS), SS_COLS);
        uint32_t p = 1;
        while (p < per) p *= 2;
        return p;
    };
    const uint32_t products = std::max({(a.d + 4) * room(3 * a.d), (a.d + 4) * room(a.f), (a.f + 4) * room(a.d), (a.d + 4) * SS_COLS});
    const uint32_t floats = SS_SMEM / 4, head = a.capacity + 4 + SS_VALUES, each = floats_per_row(a.d, a.f);
    if (head + each > floats) return 0;
    return std::min({SS_WARPS, floats / (each + products), (floats - head) / each});
}

template <typename KV, uint32_t V>
int clusters_at_once_kind() {
    static std::atomic<int> known[64];      // per device: clusters of 16 CTAs that run side by side, -1: none, 0: not asked yet
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
    int n = known[dev].load(std::memory_order_acquire);
    if (n == 0) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(SS_CTAS);
        cfg.blockDim = dim3(SS_THREADS);
        cfg.dynamicSmemBytes = SS_SMEM;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = SS_CTAS;
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        const bool fits = cudaFuncSetAttribute(strict_step_kernel<KV, V>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SS_SMEM) == cudaSuccess &&
                          cudaFuncSetAttribute(strict_step_kernel<KV, V>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
                          cudaOccupancyMaxActiveClusters(&n, strict_step_kernel<KV, V>, &cfg) == cudaSuccess && n > 0;
        if (!fits) cudaGetLastError();
        n = fits ? n : -1;
        known[dev].store(n, std::memory_order_release);
    }
    return std::max(0, n);
}

template <typename KV>
int clusters_at_once(uint32_t d) { return d <= 128 ? clusters_at_once_kind<KV, 4>() : clusters_at_once_kind<KV, SS_MAX_D / 32>(); }

}  // namespace

// Most rows that one cluster takes through a step: a warp each.  Up to there it is the faster form at every size measured (4 x 128: 8 rows 152
// against 298 us, 4 x 256: 2 rows 170 against 370 us); what ends it earlier is shared memory (rows_that_fit).
constexpr uint32_t SS_MAX_ROWS = 16;
// A cluster reads every weight through 16 SMs: beyond this many bytes of one layer the launches of strict.cu, which use all SMs, are faster.
constexpr uint64_t SS_MAX_LAYER_BYTES = 4u << 20;

// Attention is a (row, head) per CTA at a time, where the launches of strict.cu give every query an SM's share: a longer chunk of few sessions
// with more than four of them per CTA loses once the keys take longer than the launches (8 heads of 8, one session, 16 ids, four layers, us here /
// there: 128 keys 223 / 228, 272 keys 270 / 257, 1024 keys 508 / 362, 4096 keys 1515 / 815; 8 ids, 1024 keys 296 / 360).
constexpr uint32_t SS_MAX_QUERIES = 4 * SS_CTAS, SS_MANY_KEYS = 128;

bool strict_step_supported(const StrictStepArgs& a, bool kv_bf16) {
    if (!a.num_layers || a.num_layers > SS_MAX_LAYERS || a.d > SS_MAX_D || a.d % 4 || a.f % 4 || a.d % a.heads || (a.d / a.heads) % 4) return false;
    if ((4ull * a.d * a.d + 2ull * a.d * a.f) * 4 > SS_MAX_LAYER_BYTES || a.capacity > 16384) return false;
    const int at_once = kv_bf16 ? clusters_at_once<bf16>(a.d) : clusters_at_once<float>(a.d);
    if (at_once <= 0) return false;
    const uint64_t rows = (uint64_t)ceil_div(a.sessions, (uint32_t)at_once) * a.chunk;
    if (a.chunk >= 8 && rows * a.heads > SS_MAX_QUERIES && a.position + a.chunk > SS_MANY_KEYS) return false;
    return rows <= std::min(SS_MAX_ROWS, rows_that_fit(a));
}

// Largest vocabulary whose output head is part of the launch.
bool strict_step_has_head(uint32_t vocab) { return vocab <= 2048; }

template <typename KV>
static int launch_strict_step_kind(const StrictStepArgs& a, cudaStream_t stream) {
    SsParams P;
    P.a = a;
    const int at_once = std::max(1, clusters_at_once<KV>(a.d));
    P.part = (a.d & (a.d - 1)) == 0 ? 1.0f / (float)a.d : 0.0f;
    P.sessions_per_cluster = ceil_div(a.sessions, (uint32_t)at_once);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ceil_div(a.sessions, P.sessions_per_cluster) * SS_CTAS);
    cfg.blockDim = dim3(SS_THREADS);
    cfg.dynamicSmemBytes = SS_SMEM;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = SS_CTAS;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (a.d <= 128) cudaLaunchKernelEx(&cfg, strict_step_kernel<KV, 4>, P);
    else cudaLaunchKernelEx(&cfg, strict_step_kernel<KV, SS_MAX_D / 32>, P);
    count_launch();
    return check_launch("strict_step");
}

int launch_strict_step(const StrictStepArgs& a, bool kv_bf16, cudaStream_t stream) {
    return kv_bf16 ? launch_strict_step_kind<bf16>(a, stream) : launch_strict_step_kind<float>(a, stream);
}

}  // namespace tb
