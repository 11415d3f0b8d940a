// bf16 GEMM for few activation rows, every epilogue of a decode step: out[m, n] = epilogue(a[m, :] . w[n, :]).
//
// A projection of a single-token step is a few MB of weights against a few dozen rows: neither the tensor cores nor HBM are what it
// waits for, but the chain of latencies behind the previous kernel -- tensor-map fetch, a ring of TMA copies (one SM takes in 128
// padded rows at about 70 GB/s), TMEM and the epilogue's transposes came to 7 to 22 us a launch.  Here nothing is staged: a thread's
// weights are 32-byte loads straight into registers (whole 128-byte lines per row), asked for before the previous kernel has ended
// (they do not depend on it), the activation rows follow the same way from L2, and warp-level products consume both where they land.
// The order of k inside a block of 64 is free as long as both operands agree, so lane t of a row takes k = 16t .. 16t + 15 and feeds
// four m16n8k16 products.
//
//  * a CTA owns 16 MT rows x 8 NT columns at a time, its eight warps divide K; partial tiles are added in warp order through shared
//    memory.  With more column tiles than CTAs the next tile's weights are on their way while this one is added up and written;
//  * K may be divided over a cluster of CTAs (ck): each takes in 1 / ck of the rows' and the weights' bytes, the partial tiles meet
//    through distributed shared memory, added in rank order.
// How K is divided depends on n and k only, so within this engine the bits of an element do not depend on how many rows share the call.
#include <algorithm>
#include <atomic>

#include "feed_forward.cuh"
#include "gemm_epilogue.cuh"

namespace tb {

namespace {

constexpr uint32_t FW_THREADS = 256, FW_WARPS = FW_THREADS / 32, FW_BLOCK = 64;

struct FewParams {
    const bf16* a;         // [m, k]
    const bf16* w;         // [n, k]
    EpiParams epi;
    uint32_t k;
    uint32_t ck;           // CTAs of a cluster, each with its range of k
    uint32_t tiles;        // column tiles
    int mode;
};

struct Words { uint32_t x[8]; };

__device__ __forceinline__ Words fw_zero() { return {{0u, 0u, 0u, 0u, 0u, 0u, 0u, 0u}}; }
// Weights and rows alike may be what a kernel wrote before which this grid was resident already: no form of load that takes them for constant
// (.nc, __ldg), here or in the other kernels of a product.
__device__ __forceinline__ Words fw_load_weights(const bf16* p) {
    Words v;
    asm volatile("ld.global.L1::no_allocate.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(v.x[0]), "=r"(v.x[1]), "=r"(v.x[2]), "=r"(v.x[3]), "=r"(v.x[4]), "=r"(v.x[5]), "=r"(v.x[6]), "=r"(v.x[7]) : "l"(p));
    return v;
}
__device__ __forceinline__ Words fw_load_rows(const bf16* p) {
    Words v;
    asm volatile("ld.global.L1::no_allocate.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(v.x[0]), "=r"(v.x[1]), "=r"(v.x[2]), "=r"(v.x[3]), "=r"(v.x[4]), "=r"(v.x[5]), "=r"(v.x[6]), "=r"(v.x[7]) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void fw_mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ float fw_load_peer(const float* local, uint32_t rank) {
    const uint32_t at = (uint32_t)__cvta_generic_to_shared(local);
    uint32_t remote;
    float v;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(at), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(remote) : "memory");
    return v;
}
__device__ __forceinline__ void fw_cluster_sync() { asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory"); }

// MT: 16-row tiles, NT: 8-column tiles of a CTA, S: k blocks whose weights a warp has in registers at a time.
template <int MT, int NT, int S>
__global__ void __launch_bounds__(FW_THREADS, MT == 1 ? 2 : 1)
gemm_few_kernel(const __grid_constant__ FewParams P) {
    constexpr uint32_t ROWS = 16 * MT, COLS = 8 * NT, TILE = ROWS * COLS;
    constexpr int AHEAD = MT == 1 ? 2 : 1;                      // k blocks whose rows are asked for at a time
    constexpr int MINE = (TILE + FW_THREADS - 1) / FW_THREADS;
    extern __shared__ __align__(16) float fw_smem[];            // [8 warps][TILE]; then this CTA's sums over warp 0's
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    const uint32_t rank = blockIdx.x % P.ck, row0 = blockIdx.y * ROWS;
    const uint32_t m = P.epi.m, n = P.epi.n, k = P.k, tile_step = gridDim.x / P.ck;
    const bool swiglu = P.mode == GEMM_SWIGLU;
    const uint32_t blocks = (k + FW_BLOCK - 1) / FW_BLOCK, slices = P.ck * FW_WARPS;
    const uint32_t per = (blocks + slices - 1) / slices, b0 = min(blocks, (rank * FW_WARPS + warp) * per), b1 = min(blocks, b0 + per);
    // first column of a tile and the distance of its 8-column parts: side by side, or (packed gate / up, NT = 2) a gate part and its up part
    const uint32_t col_step = swiglu && NT == 2 ? 16 : 8;
    auto first_col = [&](uint32_t tile) { return swiglu && NT == 2 ? (tile >> 1) * 32 + (tile & 1) * 8 : tile * COLS; };

    Words w[NT][S];
    auto load_w = [&](int s, uint32_t tile, uint32_t b) {
        const uint32_t col = first_col(tile) + g;
        const bool ok = tile < P.tiles && b < b1 && b * FW_BLOCK + 16 * t < k;
        const bf16* p = P.w + (size_t)col * k + b * FW_BLOCK + 16 * t;
#pragma unroll
        for (int j = 0; j < NT; ++j) w[j][s] = ok && col + j * col_step < n ? fw_load_weights(p + (size_t)j * col_step * k) : fw_zero();
    };
    uint32_t tile = blockIdx.x / P.ck;
    // A thread finishes elements tid, tid + 256, ... of the (ck = 1) tile, all of one column: its bias and scale
    const uint32_t threads = FW_THREADS * P.ck, tid = rank * FW_THREADS + threadIdx.x;
    const uint32_t my_cols = swiglu ? COLS / 2 : COLS, my_col = tid % my_cols;
    float bias = 0.0f, bias_up = 0.0f, scale = 1.0f;
    auto load_col = [&](uint32_t col) {
        if (col >= n) return;
        if (P.epi.ep.bias) {
            bias = P.epi.ep.bias[col];
            if (swiglu) bias_up = P.epi.ep.bias[col + 16];
        }
        if (P.mode == GEMM_PLAIN && P.epi.ep.scale) scale = P.epi.ep.scale[col];
    };
    if (P.epi.ep.wait_first) {
        // L2 may have what is at the weights' places now: whoever still writes them does so there (1 x 4096 x 4096 back to back 11.5 us without,
        // 10.4 with; 1 x 4096 x 1024 4.4 / 3.7)
#pragma unroll
        for (int s = 0; s < S; ++s) {
            const uint32_t c = first_col(tile) + g, b = b0 + s;
#pragma unroll
            for (int j = 0; j < NT; ++j)
                if (tile < P.tiles && b < b1 && b * FW_BLOCK + 16 * t < k && c + j * col_step < n)
                    asm volatile("prefetch.global.L2 [%0];" ::"l"(P.w + (size_t)(c + j * col_step) * k + b * FW_BLOCK + 16 * t));
        }
        pdl_wait();
    }
#pragma unroll
    for (int s = 0; s < S; ++s) load_w(s, tile, b0 + s);
    load_col(first_col(tile) + my_col);

    pdl_wait();
    pdl_trigger();
    const bf16* ap = P.a + (size_t)(row0 + g) * k + 16 * t;       // rows g, g + 8, g + 16 ... of the tile
    for (bool first = true; tile < P.tiles; tile += tile_step, first = false) {
        const uint32_t col0 = first_col(tile), col = col0 + my_col;
        if (!first) load_col(col);
        // what the end of the tile reads from memory per element: the residual, or the row of the cache
        uint32_t early[MINE];
#pragma unroll
        for (int i = 0; i < MINE; ++i) {
            const uint32_t e = tid + i * threads, row = row0 + e / COLS;
            early[i] = 0u;
            if (e >= TILE || row >= m || col >= n) continue;
            if (P.mode == GEMM_PLAIN && P.epi.ep.residual) early[i] = __float_as_uint(__ldcg(P.epi.ep.residual + (size_t)row * P.epi.ep.ldr + col));
            if (P.mode == GEMM_QKV && col >= P.epi.qkv.d) {
                const GemmQkvTargets& q = P.epi.qkv;
                const uint32_t session = row / q.chunk, at = q.d_position ? q.d_position[session * q.position_stride] : q.position;
                early[i] = (uint32_t)kv_row(q.paging, session, at + row % q.chunk, q.capacity);
            }
        }
        float acc[MT][NT][4];
#pragma unroll
        for (int i = 0; i < MT; ++i)
#pragma unroll
            for (int j = 0; j < NT; ++j) acc[i][j][0] = acc[i][j][1] = acc[i][j][2] = acc[i][j][3] = 0.0f;
        for (uint32_t b = b0; b < b1; b += S) {
            const bool more = b + S < b1;
#pragma unroll
            for (int s0 = 0; s0 < S; s0 += AHEAD) {
                Words a[AHEAD][2 * MT];
#pragma unroll
                for (int s = 0; s < AHEAD; ++s) {
                    const uint32_t at = (b + s0 + s) * FW_BLOCK;
                    const bool ok = b + s0 + s < b1 && at + 16 * t < k;
#pragma unroll
                    for (int i = 0; i < 2 * MT; ++i) a[s][i] = ok && row0 + 8 * i + g < m ? fw_load_rows(ap + (size_t)i * 8 * k + at) : fw_zero();
                }
#pragma unroll
                for (int s = 0; s < AHEAD; ++s) {
                    if (b + s0 + s < b1) {
#pragma unroll
                        for (int q = 0; q < 4; ++q)
#pragma unroll
                            for (int j = 0; j < NT; ++j)
#pragma unroll
                                for (int i = 0; i < MT; ++i)
                                    fw_mma(acc[i][j], a[s][2 * i].x[2 * q], a[s][2 * i + 1].x[2 * q], a[s][2 * i].x[2 * q + 1], a[s][2 * i + 1].x[2 * q + 1],
                                           w[j][s0 + s].x[2 * q], w[j][s0 + s].x[2 * q + 1]);
                    }
                    // the place is free: the same block of the next round, or of the next tile
                    if (more) load_w(s0 + s, tile, b + S + s0 + s);
                    else load_w(s0 + s, tile + tile_step, b0 + s0 + s);
                }
            }
        }
        float* mine = fw_smem + warp * TILE;
#pragma unroll
        for (int i = 0; i < MT; ++i)
#pragma unroll
            for (int j = 0; j < NT; ++j) {
                *reinterpret_cast<float2*>(mine + (16 * i + g) * COLS + 8 * j + 2 * t) = make_float2(acc[i][j][0], acc[i][j][1]);
                *reinterpret_cast<float2*>(mine + (16 * i + g + 8) * COLS + 8 * j + 2 * t) = make_float2(acc[i][j][2], acc[i][j][3]);
            }
        __syncthreads();
        auto sum_of = [&](uint32_t e) {
            float v = fw_smem[e];
#pragma unroll
            for (uint32_t i = 1; i < FW_WARPS; ++i) v += fw_smem[i * TILE + e];
            return v;
        };
        if (P.ck > 1) {
            for (uint32_t e = threadIdx.x; e < TILE; e += FW_THREADS) fw_smem[e] = sum_of(e);     // a thread reads and writes its own elements
            fw_cluster_sync();
        }
        auto total = [&](uint32_t e) {
            if (P.ck == 1) return sum_of(e);
            float v = fw_load_peer(fw_smem + e, 0);
            for (uint32_t r = 1; r < P.ck; ++r) v += fw_load_peer(fw_smem + e, r);
            return v;
        };
        if (swiglu) {
            constexpr uint32_t HALF = COLS / 2;      // gate columns of the tile, then their up columns
#pragma unroll
            for (int i = 0; i < (MINE + 1) / 2; ++i) {
                const uint32_t e = tid + i * threads, r = e / HALF, c = e % HALF, row = row0 + r;
                if (e >= ROWS * HALF || row >= m || col >= n) continue;
                const float gate = total(r * COLS + c) + bias, up = total(r * COLS + HALF + c) + bias_up;
                reinterpret_cast<bf16*>(P.epi.out)[(size_t)row * P.epi.ldc + (col / 32 * 16 + col % 32)] = __float2bfloat16_rn(fast_silu(gate) * up);
            }
        } else {
#pragma unroll
            for (int i = 0; i < MINE; ++i) {
                const uint32_t e = tid + i * threads, row = row0 + e / COLS;
                if (e >= TILE || row >= m || col >= n) continue;
                float v = total(e);
                if (P.mode == GEMM_QKV) {
                    const GemmQkvTargets& q = P.epi.qkv;
                    const uint32_t part = col / q.d, c = col - part * q.d;
                    const size_t at = part == 0 ? row : early[i];
                    (part == 0 ? q.q : part == 1 ? q.k_cache : q.v_cache)[at * q.d + c] = __float2bfloat16_rn(v + bias);
                } else if (P.mode == GEMM_SEGMENTS) {
                    const GemmSegment& s = P.epi.seg.s[segment_of(P.epi, col)];
                    v = apply_activation(v + bias, s.activation);
                    const size_t o = (size_t)row * s.ld + (col - s.col0);
                    if (s.out_dtype == TNSR_B200_BF16) reinterpret_cast<bf16*>(s.out)[o] = __float2bfloat16_rn(v);
                    else reinterpret_cast<float*>(s.out)[o] = v;
                } else {
                    const GemmEpilogue& ep = P.epi.ep;
                    v = apply_activation(v + bias, ep.activation);
                    const size_t o = map_out_row(ep, row) * P.epi.ldc + col;
                    if (ep.out_dtype == TNSR_B200_BF16) {
                        reinterpret_cast<bf16*>(P.epi.out)[o] = __float2bfloat16_rn(v);
                    } else {
                        if (ep.scale) v *= scale;
                        if (ep.residual) v += __uint_as_float(early[i]);
                        reinterpret_cast<float*>(P.epi.out)[o] = v;
                    }
                }
            }
        }
        if (P.ck > 1) fw_cluster_sync();       // peers may still read this CTA's sums
        else if (tile + tile_step < P.tiles) __syncthreads();
    }
}

template <int MT, int NT, int S>
int launch_shape(FewParams P, cudaStream_t stream) {
    constexpr uint32_t bytes = FW_WARPS * 16 * MT * 8 * NT * 4;
    static std::atomic<int> per_sm[64] = {};            // CTAs that fit an SM, 0: not asked yet
    int dev = 0;
    cudaGetDevice(&dev);
    dev = dev < 0 || dev >= 64 ? 63 : dev;
    int resident = per_sm[dev].load(std::memory_order_relaxed);
    if (!resident) {
        prefer_max_shared_carveout(reinterpret_cast<const void*>(gemm_few_kernel<MT, NT, S>));
        if (bytes > 48 * 1024 && cudaFuncSetAttribute(gemm_few_kernel<MT, NT, S>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) != cudaSuccess)
            return check_launch("gemm_few attribute");
        int sms = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&resident, gemm_few_kernel<MT, NT, S>, FW_THREADS, bytes) != cudaSuccess ||
            cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || resident < 1)
            return check_launch("gemm_few occupancy");
        resident *= sms;
        per_sm[dev].store(resident, std::memory_order_relaxed);
    }
    P.tiles = ceil_div(P.epi.n, 8u * NT);
    const uint32_t row_tiles = ceil_div(P.epi.m, 16u * MT);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(std::min(P.tiles, std::max(1u, (uint32_t)resident / (row_tiles * P.ck))) * P.ck, row_tiles);
    cfg.blockDim = dim3(FW_THREADS);
    cfg.dynamicSmemBytes = bytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    uint32_t count = 0;
    if (t_pdl) {
        attr[count].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[count++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (P.ck > 1) {
        attr[count].id = cudaLaunchAttributeClusterDimension;
        attr[count].val.clusterDim.x = P.ck;
        attr[count].val.clusterDim.y = 1;
        attr[count++].val.clusterDim.z = 1;
    }
    cfg.attrs = attr;
    cfg.numAttrs = count;
    cudaLaunchKernelEx(&cfg, gemm_few_kernel<MT, NT, S>, P);
    count_launch();
    return check_launch("gemm_few");
}

template <int NT, int S>
int launch_rows(const FewParams& P, cudaStream_t stream) {
    const uint32_t m = P.epi.m;
    if (m <= 16) return launch_shape<1, NT, S>(P, stream);
    if (m <= 32) return launch_shape<2, NT, S>(P, stream);
    if (m <= 48) return launch_shape<3, NT, S>(P, stream);
    return launch_shape<4, NT, S>(P, stream);
}

}  // namespace

// Whether this engine is the faster one.  Measured on B200 as chains of 48 dependent launches over 420 MB of weights, us per launch here /
// in the tcgen05 engine (at most 16 rows and 4 M weights: the streaming engine), by rows:
//     n x k            1           24          48          64          128
//     768 x 768     1.8 / 7.0   2.6 / 7.0   3.6 / 7.1   4.0 / 7.1   5.3 / 7.2
//     768 x 2048    3.1 / 12.5  4.6 / 12.5  5.4 / 12.5  6.1 / 12.5  10.1 / 12.6   (split-K of that engine: about 7 and a fold)
//     768 x 4608    7.5 / 22.4  8.0 / 22.4  9.4 / 22.4  10.9 / 22.5 16.1 / 22.6
//     2304 x 768    2.0 / 7.4   3.3 / 7.0   4.3 / 7.1   5.4 / 7.1   9.4 / 7.3
//     4096 x 768    2.8 / 8.8   5.5 / 8.4   7.0 / 8.0   8.0 / 7.5   14.3 / 6.7
//     4096 x 4096   9.8 / 12.6  16.2 / 20.1 20.0 / 20.3 21.7 / 20.4 39 / 20.6
//     32000 x 768   17.3 / 26.1 31 / 18.1   51 / 18.2   62 / 19.1   118 / 17.3
// Every column tile takes in all rows, so what ends it is rows x columns: from 17 rows on a wave of the widest tiles (32 columns, 16 past 32
// rows) has to hold the matrix, unless a long k makes up for it; past 64 rows only a matrix that is small altogether gains.  What that
// leaves to the tcgen05 engine, us here / there, and two that stay:
//     32 rows: 6144 x 512  10.4 / 8.6     6144 x 2048  19.6 / 15.5    16384 x 1024  22.3 / 14.0    32000 x 512  31.5 / 14.4
//     24 rows: 8192 x 256   8.2 / 7.4;    8192 x 1024  12.2 / 14.1 stays, and 6144 x 768 10.9 / 10.3 in a session, where the weights are
//              on their way before the previous kernel ends (Bolonex, 24 sessions: a request 7.65 ms with, 7.84 ms without)
//     64 rows: 3072 x 512   8.8 / 6.6     4096 x 512    9.3 / 7.3;    2304 x 512     5.7 / 6.5  stays
// At most 16 rows gain at nearly any size against the streaming engine: 8 and 16 rows of 32000 x 768 19.9 / 27.7 and 20.6 / 31.0, of
// 8192 x 8192 40.6 / 53.2 and 45.5 / 44.4, of 28672 x 4096 70.6 / 86.1 and 76.6 / 92.2 (launch_gemm_impl has the exception).  The 768 x 768
// projection of 128 rows gains alone, but not inside a step of two ranges of sessions: its CTAs do not fit beside the other range's attention.
bool gemm_few_pays(const bf16* a, const bf16* w, uint32_t m, uint32_t n, uint32_t k) {
    if (m == 0 || m > 128 || n == 0 || k % 16 != 0 || k == 0) return false;
    if (reinterpret_cast<uintptr_t>(a) % 32 != 0 || reinterpret_cast<uintptr_t>(w) % 32 != 0) return false;
    const uint64_t weights = (uint64_t)n * k;
    if (m <= 16) return true;
    if (m <= 32) return weights <= (17ull << 20) && (n <= 32 * 148 || (m < 32 && n <= 8192 && k >= 768));
    if (m <= 64 && n <= 1024) return true;
    if (m <= 48 && weights <= (3ull << 20)) return n <= 16 * 148 || k >= 768;
    if (m <= 64 && weights <= (2ull << 20)) return n <= 16 * 148;
    return weights <= (300u << 10);
}

int launch_gemm_few(const bf16* a, const bf16* w, const EpiParams& epi, uint32_t k, GemmMode mode, cudaStream_t stream) {
    FewParams P;
    P.a = a; P.w = w; P.epi = epi; P.k = k; P.mode = mode; P.tiles = 0;
    const uint32_t m = epi.m, n = epi.n;
    // a narrow matrix with a long k (an output or down projection) has fewer column tiles than SMs: two CTAs share its k
    P.ck = k > 1024 && n <= 1024 ? 2 : 1;
    // up to 16 rows 16 columns per CTA were the fastest throughout; with more rows as few CTAs as still make a wave
    uint32_t nt = 2;
    if (m > 16) {
        const uint32_t row_tiles = ceil_div(m, 64u);
        nt = mode == GEMM_SWIGLU ? 2 : 1;
        while (nt < 4 && ceil_div(n, 8 * nt) * P.ck * row_tiles > 148) nt *= 2;
    }
    const uint32_t per = ceil_div(ceil_div(k, FW_BLOCK), P.ck * FW_WARPS);
    if (nt == 4) return launch_rows<4, 2>(P, stream);
    if (nt == 2) return per <= 2 ? launch_rows<2, 2>(P, stream) : launch_rows<2, 4>(P, stream);
    return per <= 2 ? launch_rows<1, 2>(P, stream) : launch_rows<1, 4>(P, stream);
}

// ---- grouped products of few rows -------------------------------------------------------------
// The experts of a step: groups of a few rows each, which ones only the device knows.  Block (x, y) = 16 columns of the y-th 16-row tile of
// the groups in turn; it finds its group from the offsets, a trip that the weights have to wait for, and then works as above.
namespace {

struct GroupedFewParams {
    const bf16* a;             // [rows, k], group after group
    const bf16* w;             // [groups, n, k]
    void* out;                 // [rows, n]
    const uint32_t* offsets;   // [groups + 1]
    uint32_t groups, rows, n, k;
    int activation, out_dtype;
};

__global__ void __launch_bounds__(FW_THREADS, 2)
gemm_grouped_few_kernel(GroupedFewParams P) {
    constexpr uint32_t COLS = 16, TILE = 16 * COLS;
    constexpr int NT = 2, S = 2;             // k blocks whose operands a warp has in registers at a time
    __shared__ float sums[FW_WARPS * TILE];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3, col0 = blockIdx.x * COLS;
    pdl_wait();
    pdl_trigger();
    // the group of this block's tile: lanes count the tiles of 32 groups at a time.  A group list that does not fit the rows is cut to
    // them, as in gemm_grouped.cu.
    uint32_t group = 0, row0 = 0, row1 = 0, before = 0;
    bool found = false;
    for (uint32_t e0 = 0; e0 < P.groups && !found; e0 += 32) {
        const uint32_t e = e0 + lane;
        const uint32_t first = e < P.groups ? min(P.rows, __ldcg(P.offsets + e)) : 0u, last = e < P.groups ? min(P.rows, __ldcg(P.offsets + e + 1)) : 0u;
        const uint32_t tiles = last > first ? (last - first + 15) / 16 : 0u;
        uint32_t upto = tiles;
#pragma unroll
        for (uint32_t o = 1; o < 32; o <<= 1) {
            const uint32_t u = __shfl_up_sync(0xffffffffu, upto, o);
            if (lane >= o) upto += u;
        }
        const uint32_t hit = __ballot_sync(0xffffffffu, blockIdx.y < before + upto);
        if (hit) {
            const uint32_t at = __ffs(hit) - 1;
            group = e0 + at;
            const uint32_t tile = blockIdx.y - before - __shfl_sync(0xffffffffu, upto - tiles, at);
            row0 = __shfl_sync(0xffffffffu, first, at) + tile * 16;
            row1 = __shfl_sync(0xffffffffu, last, at);
            found = true;
        }
        before += __shfl_sync(0xffffffffu, upto, 31);
    }
    if (!found) return;           // the same for the whole block
    const uint32_t blocks = (P.k + FW_BLOCK - 1) / FW_BLOCK, per = (blocks + FW_WARPS - 1) / FW_WARPS;
    const uint32_t b0 = min(blocks, warp * per), b1 = min(blocks, b0 + per);
    const bf16* wp = P.w + ((size_t)group * P.n + col0 + g) * P.k + 16 * t;
    const bf16* ap = P.a + (size_t)(row0 + g) * P.k + 16 * t;
    float acc[NT][4] = {};
    for (uint32_t b = b0; b < b1; b += S) {
        Words w[NT][S], a[2][S];
#pragma unroll
        for (int s = 0; s < S; ++s) {
            const uint32_t at = (b + s) * FW_BLOCK;
            const bool ok = b + s < b1 && at + 16 * t < P.k;
#pragma unroll
            for (int j = 0; j < NT; ++j) w[j][s] = ok && col0 + 8 * j + g < P.n ? fw_load_weights(wp + (size_t)j * 8 * P.k + at) : fw_zero();
#pragma unroll
            for (int i = 0; i < 2; ++i) a[i][s] = ok && row0 + 8 * i + g < row1 ? fw_load_rows(ap + (size_t)i * 8 * P.k + at) : fw_zero();
        }
#pragma unroll
        for (int s = 0; s < S; ++s)
#pragma unroll
            for (int q = 0; q < 4; ++q)
#pragma unroll
                for (int j = 0; j < NT; ++j)
                    fw_mma(acc[j], a[0][s].x[2 * q], a[1][s].x[2 * q], a[0][s].x[2 * q + 1], a[1][s].x[2 * q + 1], w[j][s].x[2 * q], w[j][s].x[2 * q + 1]);
    }
    float* mine = sums + warp * TILE;
#pragma unroll
    for (int j = 0; j < NT; ++j) {
        *reinterpret_cast<float2*>(mine + g * COLS + 8 * j + 2 * t) = make_float2(acc[j][0], acc[j][1]);
        *reinterpret_cast<float2*>(mine + (g + 8) * COLS + 8 * j + 2 * t) = make_float2(acc[j][2], acc[j][3]);
    }
    __syncthreads();
    const uint32_t row = row0 + threadIdx.x / COLS, col = col0 + threadIdx.x % COLS;
    if (row >= row1 || col >= P.n) return;
    float v = sums[threadIdx.x];
#pragma unroll
    for (uint32_t i = 1; i < FW_WARPS; ++i) v += sums[i * TILE + threadIdx.x];
    if (P.activation == ACT_RELU_SQUARED) {
        v = fmaxf(v, 0.0f);
        v *= v;
    } else {
        v = apply_activation(v, P.activation);
    }
    if (P.out_dtype == TNSR_B200_BF16) reinterpret_cast<bf16*>(P.out)[(size_t)row * P.n + col] = __float2bfloat16_rn(v);
    else reinterpret_cast<float*>(P.out)[(size_t)row * P.n + col] = v;
}

}  // namespace

// Blocks of the launch: a column of them per 16 columns, in it one per 16-row tile that the groups can have (every group may end in a ragged one).
static uint32_t grouped_few_tiles(const GroupedGemm& g) { return g.rows / 16 + std::min(g.groups, g.rows); }

// Which groups have rows only the device knows, so there are blocks for the most tiles there can be, and each group's weights are read once per
// tile of it.  Three blocks per SM are the line (two run at a time).  Measured on B200 as chains of launches, us here / in the tcgen05 kernel:
//     groups, rows, n x k       blocks    rows even      all in one group
//      4,  96,  256 x 2048       160     4.1 / 12.3      4.1 / 12.3
//     16,   4,  768 x 768        192     4.1 /  7.0      3.5 /  7.2
//     16,   8,  768 x 768        384     5.9 /  7.5      4.1 /  7.4
//      4,  32, 1024 x 4096       384    12.2 / 21.1      7.1 / 20.2
//     16,  32,  768 x 768        864     9.4 /  8.7      6.3 /  7.2
//      8, 128, 3072 x 768       3072    22.2 / 12.8     17.8 / 10.9
//     64, 128, 3072 x 768      13824     159 / 52        178 / 12
// Of 1892 products (1 to 64 groups, 1 to 128 rows, 128 to 3072 columns, rows spread evenly, half of them in one group, all of them) 1167 are
// within the line, 1164 of these more than 5 % faster here and none slower; past it the share of slower ones grows.
bool gemm_grouped_few_pays(const GroupedGemm& g) {
    if (!g.offsets || g.rows > 128 || g.k % 16 != 0 || reinterpret_cast<uintptr_t>(g.a) % 32 != 0 || reinterpret_cast<uintptr_t>(g.w) % 32 != 0) return false;
    return (uint64_t)ceil_div(g.n, 16u) * grouped_few_tiles(g) <= 3 * 148;
}

int launch_gemm_grouped_few(const GroupedGemm& g, cudaStream_t stream) {
    GroupedFewParams P;
    P.a = (const bf16*)g.a; P.w = (const bf16*)g.w; P.out = g.out; P.offsets = g.offsets; P.groups = g.groups; P.rows = g.rows; P.n = g.n; P.k = g.k;
    P.activation = g.activation; P.out_dtype = g.out_dtype;
    const dim3 grid(ceil_div(g.n, 16u), grouped_few_tiles(g));
    launch_kernel(gemm_grouped_few_kernel, grid, dim3(FW_THREADS), 0, stream, P);
    count_launch();
    return check_launch("gemm_grouped_few");
}

}  // namespace tb
