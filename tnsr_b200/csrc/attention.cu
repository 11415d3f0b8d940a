// KV-cache attention on bf16 caches.
//
//  * decode_attention_*: one query per (session, head) scanned over the live
//    prefix only, split over the key axis so that every SM streams a contiguous
//    slab of K and V rows (all heads) through a shared-memory ring filled by
//    bulk async copies (cp.async.bulk, mbarrier completion); f32 online softmax;
//    partials (max, sum, numerator) are merged inside the same kernel by whichever
//    warp stores the last partial of a (session, head) pair.  This is
//    the job of the reference's AttentionScan / MergeScan pair
//    (src/nn/kv_cache/attention.rs:31-239, :242-393; fixed 16/32 partitions,
//    src/nn/kv_cache/cuda.rs:31-32,110-116) with two differences: the split is
//    by fixed key-slab size chosen from the total live length, so ragged
//    per-session lengths balance across SMs, and K/V are read as whole cache
//    rows (all heads at once) so HBM sees only long contiguous bursts.
//  * attention_generic: any head width and chunk, one warp per query/head.
//
// HBM traffic per decode step is the live K and V rows once: 4 * d bytes per
// live key per session (d = heads * head_dim) plus q / out / partials.
#include <algorithm>

#include "common.cuh"

namespace tb {

thread_local KernelTimer* t_attention_timer = nullptr;
thread_local bool t_pdl = false;

__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float warp_sum_f(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// ===========================================================================
// Generic kernel (bf16): one warp per (session, head, query); lane c owns dims
// c, c+32, ...; keys walked in order with a running max / sum / numerator.
// ===========================================================================
constexpr int GEN_MAX_SLOTS = 8;  // head_dim <= 256

__global__ void __launch_bounds__(128)
attention_generic_kernel(const bf16* q, const bf16* kc, const bf16* vc,
                         bf16* __restrict__ out, uint32_t total_queries, uint32_t chunk, uint32_t position,
                         const uint32_t* d_position, uint32_t capacity, uint32_t heads, uint32_t hd,
                         float scale_log2, KvPaging paging) {
    pdl_wait();
    pdl_trigger();
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t idx = blockIdx.x * 4 + (threadIdx.x >> 5);
    if (idx >= total_queries) return;
    const uint32_t t = idx % chunk, h = (idx / chunk) % heads, s = idx / (chunk * heads);
    const uint32_t d = heads * hd;
    const uint32_t past = d_position ? *d_position : position;
    uint32_t total = past + t + 1;
    if (total > capacity) total = capacity;
    float qv[GEN_MAX_SLOTS], acc[GEN_MAX_SLOTS];
    const bf16* qr = q + ((size_t)s * chunk + t) * d + (size_t)h * hd;
#pragma unroll
    for (int i = 0; i < GEN_MAX_SLOTS; ++i) {
        uint32_t c = lane + 32 * i;
        qv[i] = c < hd ? __bfloat162float(qr[c]) * scale_log2 : 0.0f;
        acc[i] = 0.0f;
    }
    const bf16* kb = kc + (size_t)h * hd;
    const bf16* vb = vc + (size_t)h * hd;
    float m = -INFINITY, l = 0.0f;
    for (uint32_t j0 = 0; j0 < total; ++j0) {
        const size_t j = kv_row(paging, s, j0, capacity);
        float part = 0.0f;
#pragma unroll
        for (int i = 0; i < GEN_MAX_SLOTS; ++i) {
            uint32_t c = lane + 32 * i;
            if (c < hd) part = fmaf(qv[i], __bfloat162float(kb[(size_t)j * d + c]), part);
        }
        const float sc = warp_sum_f(part);
        const float m_new = fmaxf(m, sc);
        const float m_safe = (m_new == -INFINITY) ? 0.0f : m_new;
        const float corr = ex2(m - m_safe), p = ex2(sc - m_safe);
        l = l * corr + p;
#pragma unroll
        for (int i = 0; i < GEN_MAX_SLOTS; ++i) {
            uint32_t c = lane + 32 * i;
            if (c < hd) acc[i] = acc[i] * corr + p * __bfloat162float(vb[(size_t)j * d + c]);
        }
        m = m_new;
    }
    bf16* orow = out + ((size_t)s * chunk + t) * d + (size_t)h * hd;
#pragma unroll
    for (int i = 0; i < GEN_MAX_SLOTS; ++i) {
        uint32_t c = lane + 32 * i;
        if (c < hd) orow[c] = __float2bfloat16_rn(acc[i] / l);
    }
}

int launch_attention_generic(const bf16* q, const bf16* k_cache, const bf16* v_cache, bf16* out,
                             uint32_t sessions, uint32_t chunk, uint32_t position,
                             const uint32_t* d_position, uint32_t capacity, uint32_t heads,
                             uint32_t head_dim, cudaStream_t stream, const KvPaging* paging) {
    if (sessions == 0 || chunk == 0) return TNSR_B200_OK;
    if (head_dim > 32 * GEN_MAX_SLOTS) {
        set_thread_error("attention: head_dim above 256 is outside the bf16 kernels");
        return TNSR_B200_ERR_UNSUPPORTED;
    }
    uint64_t total = (uint64_t)sessions * heads * chunk;
    if (total > 0x7fffffffull) return TNSR_B200_ERR_UNSUPPORTED;
    const float scale_log2 = (1.0f / sqrtf((float)head_dim)) * 1.4426950408889634f;
    launch_kernel(attention_generic_kernel, dim3((unsigned)ceil_div64(total, 4)), dim3(128), 0, stream, q, k_cache, v_cache, out,
                  (uint32_t)total, chunk, position, d_position, capacity, heads, head_dim, scale_log2, paging ? *paging : KvPaging());
    count_launch();
    return check_launch("attention_generic");
}

// ===========================================================================
// Split-KV decode attention
// ===========================================================================
constexpr uint32_t DA_KS = 16;             // keys per ring stage (8 in the lean form, see launch_decode_attention_ex)
constexpr uint32_t DA_MAX_STAGES = 8;
constexpr uint32_t DA_SMEM_BUDGET = 200 * 1024;
// Lean form: half the shared memory, so that a CTA of another kernel (the projections of the other half of the batch)
// fits on the same SM while this one streams K/V.
constexpr uint32_t DA_KS_LEAN = 8;
constexpr uint32_t DA_SMEM_BUDGET_LEAN = 106 * 1024;
constexpr uint32_t DA_MAX_CTAS = 256;      // upper bound on the grid (one CTA per SM)

// A work item: keys [key0, key0 + nkeys) of one session, all heads.  `slot` is the index of its
// partial result, or DA_DIRECT when the item covers the whole session and writes the output row itself.
constexpr uint32_t DA_DIRECT = 0xffffffffu;
struct DaItem {
    uint32_t session, key0, nkeys, slot;
    uint32_t n_parts, first_slot;  // pieces of the session and the slot of its first piece (for the merge)
    uint32_t pad[2];
};

// Work is split by position in the concatenation of all sessions' live keys, counted in stages of
// DA_KS keys: CTA c owns stages [c * quota, (c + 1) * quota).  Every CTA therefore streams the same
// amount of K/V (+-1 stage) whatever the per-session lengths are, a session is cut only where a CTA
// boundary falls inside it, and there are at most batch + grid items.
//
// Workspace layout (all offsets 256-byte aligned):
//   header    : uint32 total_stages, quota, n_items
//   first     : uint32 [batch]          first partial slot of each session
//   count     : uint32 [batch]          number of pieces of each session (0 for an empty session)
//   done      : uint32 [batch * heads]  partials stored so far per (session, head); zero between launches
//   sstart    : uint32 [batch + 1]      first global stage of each session
//   cta_begin : uint32 [DA_MAX_CTAS + 1] first item of each CTA
//   items     : DaItem [batch + DA_MAX_CTAS]   (32 bytes each)
//   partial   : float  [batch + DA_MAX_CTAS][heads][head_dim + 2]   (numerator, then max, then sum)
struct DaLayout {
    uint64_t first, count, done, sstart, cta_begin, items, partial, bytes;
    uint32_t max_items;
};

static uint64_t align256(uint64_t x) { return (x + 255) & ~255ull; }

static DaLayout da_layout(uint32_t batch, uint32_t heads, uint32_t head_dim) {
    DaLayout L;
    const uint64_t per_item = (uint64_t)heads * (head_dim + 2) * 4;
    L.max_items = batch + DA_MAX_CTAS;
    L.first = 256;
    L.count = align256(L.first + 4ull * batch);
    L.done = align256(L.count + 4ull * batch);
    L.sstart = align256(L.done + 4ull * batch * heads);
    L.cta_begin = align256(L.sstart + 4ull * (batch + 1));
    L.items = align256(L.cta_begin + 4ull * (DA_MAX_CTAS + 1));
    L.partial = align256(L.items + sizeof(DaItem) * (uint64_t)L.max_items);
    L.bytes = L.partial + per_item * L.max_items;
    return L;
}

uint64_t decode_attention_workspace_bytes(uint32_t batch, uint32_t capacity, uint32_t heads, uint32_t head_dim) {
    (void)capacity;  // the scratch depends on the number of sessions, not on how long they may grow
    return da_layout(batch, heads, head_dim).bytes;
}

bool decode_attention_supported(uint32_t heads, uint32_t head_dim) {
    if (!(head_dim == 32 || head_dim == 64 || head_dim == 128)) return false;
    if (heads == 0 || heads > 32) return false;
    uint64_t stage = 2ull * DA_KS * heads * head_dim * 2 + (uint64_t)heads * head_dim * 2;
    return stage * 2 <= DA_SMEM_BUDGET;  // at least a double buffer
}

// ---- plan: one block ---------------------------------------------------------------
// Session b has lengths[b] + extra keys; lengths == nullptr means (d_position ? *d_position : 0) + extra for all.
__global__ void __launch_bounds__(1024)
da_plan_kernel(const uint32_t* lengths, const uint32_t* d_position, uint32_t extra,
               uint32_t batch, uint32_t heads, uint32_t capacity, uint32_t grid, uint32_t ks, uint32_t* __restrict__ header,
               uint32_t* __restrict__ first, uint32_t* __restrict__ count, uint32_t* __restrict__ done,
               uint32_t* __restrict__ sstart, uint32_t* __restrict__ cta_begin, DaItem* __restrict__ items,
               int* __restrict__ d_status) {
    __shared__ uint32_t s_carry, s_warp_tot[32], s_quota, s_total;
    pdl_wait();
    pdl_trigger();
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    auto len_of = [&](uint32_t b) -> uint32_t {
        uint32_t L = (lengths ? lengths[b] : (d_position ? *d_position : 0u)) + extra;
        if (L > capacity) {
            if (d_status) atomicCAS(d_status, DEV_OK, DEV_BAD_LENGTH);
            L = capacity;
        }
        return L;
    };
    // block-wide exclusive scan of f(b) over the sessions, 1024 at a time; returns the total
    auto scan = [&](auto f, uint32_t* out_excl) -> uint32_t {
        if (tid == 0) s_carry = 0;
        __syncthreads();
        for (uint32_t base = 0; base < batch; base += blockDim.x) {
            const uint32_t b = base + tid;
            const uint32_t v = b < batch ? f(b) : 0;
            uint32_t incl = v;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= (uint32_t)o) incl += t;
            }
            if (lane == 31) s_warp_tot[warp] = incl;
            __syncthreads();
            uint32_t before = s_carry;
            for (uint32_t w = 0; w < warp; ++w) before += s_warp_tot[w];
            if (b < batch) out_excl[b] = before + incl - v;
            __syncthreads();
            if (tid == blockDim.x - 1) s_carry = before + incl;
            __syncthreads();
        }
        return s_carry;
    };
    // the merge counters must be zero when the attention kernel starts
    for (uint32_t i = tid; i < batch * heads; i += blockDim.x) done[i] = 0;
    // 1. global stage offsets of the sessions
    const uint32_t total = scan([&](uint32_t b) { return (len_of(b) + ks - 1) / ks; }, sstart);
    if (tid == 0) {
        sstart[batch] = total;
        const uint32_t ctas = total < grid ? (total ? total : 1) : grid;
        // two stages at least: with one per CTA a session of 1000 keys is 63 pieces, whose merge costs more than the second stage (one
        // session's attention, 12 heads: 21.1 -> 19.2 us with the plan)
        s_quota = max(2u, (total + ctas - 1) / ctas);
        s_total = total;
    }
    __syncthreads();
    const uint32_t quota = s_quota;
    // 2. pieces per session = CTAs its stage range touches; slots by exclusive scan
    auto pieces = [&](uint32_t b) -> uint32_t {
        const uint32_t s0 = sstart[b], n = (len_of(b) + ks - 1) / ks;
        return n ? (s0 + n - 1) / quota - s0 / quota + 1 : 0;
    };
    const uint32_t n_items = scan(pieces, first);
    // 3. items, one thread per session
    for (uint32_t b = tid; b < batch; b += blockDim.x) {
        const uint32_t L = len_of(b), s0 = sstart[b], n = (L + ks - 1) / ks;
        const uint32_t c = pieces(b), f = first[b];
        count[b] = c;
        const uint32_t cta0 = s0 / quota;
        for (uint32_t j = 0; j < c; ++j) {
            const uint32_t lo = max(s0, (cta0 + j) * quota), hi = min(s0 + n, (cta0 + j + 1) * quota);
            DaItem it;
            it.session = b;
            it.key0 = (lo - s0) * ks;
            it.nkeys = min(L, (hi - s0) * ks) - it.key0;
            it.slot = c == 1 ? DA_DIRECT : f + j;
            it.n_parts = c;
            it.first_slot = f;
            it.pad[0] = it.pad[1] = 0;
            items[f + j] = it;
        }
    }
    __syncthreads();
    // 4. first item of every CTA: the piece that contains global stage c * quota
    for (uint32_t c = tid; c <= grid; c += blockDim.x) {
        const uint32_t g = c * quota;
        uint32_t begin = n_items;
        if (g < s_total) {
            uint32_t lo = 0, hi = batch;  // last session with sstart <= g and at least one stage
            while (hi - lo > 1) {
                const uint32_t mid = (lo + hi) / 2;
                if (sstart[mid] <= g) lo = mid; else hi = mid;
            }
            begin = first[lo] + (g / quota - sstart[lo] / quota);
        }
        cta_begin[c] = begin;
    }
    if (tid == 0) {
        header[0] = s_total;
        header[1] = quota;
        header[2] = n_items;
    }
}

// ---- main kernel ------------------------------------------------------------------
__device__ __forceinline__ uint32_t da_smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void da_mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(da_smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void da_mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(da_smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void da_mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(da_smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool da_mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(da_smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ uint64_t da_timer_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ bool da_mbar_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag, uint64_t limit_ns) {
    if (da_mbar_try_wait(bar, parity)) return true;
    const uint64_t start = da_timer_ns();
    for (uint32_t it = 1;; ++it) {
        if (da_mbar_try_wait(bar, parity)) return true;
        if ((it & 63u) == 0) {
            if (*abort_flag) return false;
            if (da_timer_ns() - start > limit_ns) {
                *abort_flag = 1;
                return false;
            }
        }
    }
}
// Plain (untiled) bulk copy global -> this CTA's shared memory; 16-byte aligned, size % 16 == 0.
__device__ __forceinline__ void da_bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(da_smem_u32(dst)), "l"(src), "r"(bytes), "r"(da_smem_u32(bar))
                 : "memory");
}

// The same copy for data that is read exactly once (K/V rows): evict-first in L2, so that a long scan does not push out
// what other kernels keep there.
__device__ __forceinline__ void da_bulk_load_once(void* dst, const void* src, uint32_t bytes, uint64_t* bar, uint64_t policy) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;"
                 ::"r"(da_smem_u32(dst)), "l"(src), "r"(bytes), "r"(da_smem_u32(bar)), "l"(policy)
                 : "memory");
}

struct DaStageMeta {
    uint32_t slot;        // partial slot of the item, or DA_DIRECT
    uint32_t nk;          // valid keys in this stage (1..DA_KS)
    uint32_t flags;       // bit 0: first stage of the item, bit 1: last stage
    uint32_t session;
    uint32_t n_parts;     // pieces of this session (for the merge)
    uint32_t first_slot;  // partial slot of the session's first piece
    uint32_t pad[2];
};

struct DaParams {
    const bf16* q;
    const bf16* kc;
    const bf16* vc;
    const uint32_t* first;
    const uint32_t* count;
    uint32_t* done;
    const uint32_t* cta_begin;
    const DaItem* items;
    float* partial;
    bf16* out;
    uint32_t batch, capacity, heads;
    uint32_t stages;
    float scale_log2;
    int* d_status;
    uint64_t wait_limit_ns;   // bound of every mbarrier wait (tnsr_b200_set_wait_limit_ns)
    KvPaging paging;          // page pools instead of per-session slabs (page_rows is a multiple of the stage size)
    uint32_t early;           // the item list is older than the previous kernel, which wrote no key but every session's last
};

// HD: head width; LPK = HD / 8 lanes share one (key, head) row slice, each lane
// owning 8 consecutive dims (one 16-byte shared-memory load); KPW = 32 / LPK keys
// are processed side by side in a warp.  HPW: heads per consumer warp.
template <int HD, int HPW, int KS>
__global__ void __launch_bounds__(576, 1)
decode_attention_kernel(DaParams P) {
    constexpr uint32_t LPK = HD / 8, KPW = 32 / LPK, ITERS = KS / KPW;
    static_assert(KS % KPW == 0, "stage must hold whole key groups");
    extern __shared__ __align__(128) uint8_t smem[];
    const uint32_t d = P.heads * HD, row_bytes = d * 2;
    const uint32_t k_bytes = KS * row_bytes;
    const uint32_t stage_bytes = 2 * k_bytes + row_bytes;  // K slab, V slab, q row
    uint8_t* ring = smem;
    uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + (size_t)P.stages * stage_bytes);
    uint64_t* empty_bar = full_bar + DA_MAX_STAGES;
    DaStageMeta* meta = reinterpret_cast<DaStageMeta*>(empty_bar + DA_MAX_STAGES);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(meta + DA_MAX_STAGES);

    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t consumers = (blockDim.x >> 5) - 1;  // last warp is the producer
    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < P.stages; ++s) { da_mbar_init(full_bar + s, 1); da_mbar_init(empty_bar + s, consumers); }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    const bool early = KS != DA_KS_LEAN && P.early;
    if (!(early && warp == consumers)) {
        pdl_wait();
        pdl_trigger();
    }
    const uint32_t item_begin = __ldcg(P.cta_begin + blockIdx.x), item_end = __ldcg(P.cta_begin + blockIdx.x + 1);

    if (warp == consumers) {
        // ---------------- producer ----------------
        if (lane == 0) {
            uint32_t stage = 0, phase = 0;
            bool ok = true;
            uint64_t once;
            asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(once));
            // item records and the per-session piece counts are fetched one item ahead, so their latency
            // hides behind the copies of the current item
            auto item_at = [&](uint32_t i) {
                const uint4 a = __ldcg(reinterpret_cast<const uint4*>(P.items + i)), b = __ldcg(reinterpret_cast<const uint4*>(P.items + i) + 1);
                return DaItem{a.x, a.y, a.z, a.w, b.x, b.y, {0u, 0u}};
            };
            // stage s of item `it` into the ring, with the session's query row, which the item's first stage carries, unless that is still
            // being written (`ahead`: the previous kernel may be running)
            auto fill = [&](const DaItem& it, uint32_t s, uint32_t n_stages, bool ahead) {
                const uint32_t nk = min((uint32_t)KS, it.nkeys - s * KS);
                uint8_t* sk = ring + (size_t)stage * stage_bytes;
                DaStageMeta mt;
                mt.slot = it.slot;
                mt.nk = nk;
                mt.flags = (s == 0 ? 1u : 0u) | (s + 1 == n_stages ? 2u : 0u);
                mt.session = it.session;
                mt.n_parts = it.n_parts;
                mt.first_slot = it.first_slot;
                meta[stage] = mt;
                const uint32_t bytes = nk * row_bytes;
                da_mbar_expect_tx(full_bar + stage, 2 * bytes + (s == 0 ? row_bytes : 0));
                // a stage never straddles pages: key0 and the page size are multiples of the stage size
                const uint32_t key = it.key0 + s * KS;
                const size_t base = (ahead ? kv_row_l2(P.paging, it.session, key, P.capacity) : kv_row(P.paging, it.session, key, P.capacity)) * d;
                da_bulk_load_once(sk, P.kc + base, bytes, full_bar + stage, once);
                da_bulk_load_once(sk + k_bytes, P.vc + base, bytes, full_bar + stage, once);
                if (s == 0 && !ahead) da_bulk_load(sk + 2 * k_bytes, P.q + (size_t)it.session * d, row_bytes, full_bar + stage);
            };
            DaItem it = {}, nxt = {};
            if (item_begin < item_end) it = nxt = item_at(item_begin);
            uint32_t item = item_begin, s = 0;
            if (early) {
                // The previous kernel writes the queries and every session's last key; the keys before it are whole steps old.  Up to a ring
                // of them is asked for now, the query rows follow once that kernel has ended (12 layers, us per step without / with: one
                // session at 1000 341 / 332, 48 at 1000 700 / 692, 64 at 512 652 / 640).
                uint32_t filled = 0, waiting = 0;
                while (item < item_end && filled < P.stages) {
                    const uint32_t n_stages = (it.nkeys + KS - 1) / KS;
                    if (s + 1 == n_stages && (it.slot == DA_DIRECT || it.slot + 1 == it.first_slot + it.n_parts)) break;
                    stage = filled;
                    fill(it, s, n_stages, true);
                    if (s == 0) waiting |= 1u << filled;
                    ++filled;
                    if (++s == n_stages) {
                        s = 0;
                        if (++item < item_end) it = item_at(item);
                    }
                }
                nxt = it;
                pdl_wait();
                for (uint32_t i = 0; i < filled; ++i)
                    if (waiting >> i & 1u)
                        da_bulk_load(ring + (size_t)i * stage_bytes + 2 * k_bytes, P.q + (size_t)meta[i].session * d, row_bytes, full_bar + i);
                stage = filled == P.stages ? 0 : filled;
                phase = filled == P.stages ? 1 : 0;
            }
            for (; ok && item < item_end; ++item, s = 0) {
                it = nxt;
                if (item + 1 < item_end) nxt = item_at(item + 1);
                const uint32_t n_stages = (it.nkeys + KS - 1) / KS;
                for (; s < n_stages; ++s) {
                    if (!da_mbar_wait(empty_bar + stage, phase ^ 1, abort_flag, P.wait_limit_ns)) { ok = false; break; }
                    fill(it, s, n_stages, false);
                    if (++stage == P.stages) { stage = 0; phase ^= 1; }
                }
            }
        }
        if (early) {
            pdl_wait();
            pdl_trigger();
        }
    } else {
        // ---------------- consumers ----------------
        const uint32_t grp = lane / LPK;       // which of the KPW parallel keys
        const uint32_t sub = lane % LPK;       // which 8-dim slice of the head
        float qf[HPW][8], acc[HPW][8], m[HPW], l[HPW];
        uint32_t stage = 0, phase = 0;
        bool ok = true;
        for (uint32_t item = item_begin; ok && item < item_end; ++item) {
            for (;;) {
                if (!da_mbar_wait(full_bar + stage, phase, abort_flag, P.wait_limit_ns)) { ok = false; break; }
                const DaStageMeta mt = meta[stage];
                const uint8_t* sk = ring + (size_t)stage * stage_bytes;
                const uint8_t* sv = sk + k_bytes;
                if (mt.flags & 1u) {
                    const uint8_t* sq = sk + 2 * k_bytes;
#pragma unroll
                    for (int hh = 0; hh < HPW; ++hh) {
                        const uint32_t h = warp + hh * consumers;
                        m[hh] = -INFINITY;
                        l[hh] = 0.0f;
#pragma unroll
                        for (int e = 0; e < 8; ++e) acc[hh][e] = 0.0f;
                        if (h < P.heads) {
                            const uint4 qq = *reinterpret_cast<const uint4*>(sq + ((size_t)h * HD + sub * 8) * 2);
                            const uint32_t w[4] = {qq.x, qq.y, qq.z, qq.w};
#pragma unroll
                            for (int e = 0; e < 4; ++e) {
                                float2 f = bf16x2_to_f32(w[e]);
                                qf[hh][2 * e] = f.x * P.scale_log2;
                                qf[hh][2 * e + 1] = f.y * P.scale_log2;
                            }
                        }
                    }
                }
#pragma unroll
                for (int hh = 0; hh < HPW; ++hh) {
                    const uint32_t h = warp + hh * consumers;
                    if (h >= P.heads) continue;
                    const uint32_t col = (h * HD + sub * 8) * 2;
                    float sc[ITERS];
#pragma unroll
                    for (uint32_t itr = 0; itr < ITERS; ++itr) {
                        const uint32_t key = itr * KPW + grp;
                        const uint4 kk = *reinterpret_cast<const uint4*>(sk + (size_t)key * row_bytes + col);
                        const uint32_t w[4] = {kk.x, kk.y, kk.z, kk.w};
                        float part = 0.0f;
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            float2 f = bf16x2_to_f32(w[e]);
                            part = fmaf(qf[hh][2 * e], f.x, part);
                            part = fmaf(qf[hh][2 * e + 1], f.y, part);
                        }
#pragma unroll
                        for (uint32_t o = LPK / 2; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
                        sc[itr] = key < mt.nk ? part : -INFINITY;
                    }
                    float m_new = m[hh];
#pragma unroll
                    for (uint32_t itr = 0; itr < ITERS; ++itr) m_new = fmaxf(m_new, sc[itr]);
                    const float m_safe = (m_new == -INFINITY) ? 0.0f : m_new;
                    const float corr = ex2(m[hh] - m_safe);
                    m[hh] = m_new;
                    float lsum = l[hh] * corr;
#pragma unroll
                    for (int e = 0; e < 8; ++e) acc[hh][e] *= corr;
#pragma unroll
                    for (uint32_t itr = 0; itr < ITERS; ++itr) {
                        const uint32_t key = itr * KPW + grp;
                        const float p = ex2(sc[itr] - m_safe);  // 0 for masked keys
                        lsum += p;
                        if (key < mt.nk) {
                            const uint4 vv = *reinterpret_cast<const uint4*>(sv + (size_t)key * row_bytes + col);
                            const uint32_t w[4] = {vv.x, vv.y, vv.z, vv.w};
#pragma unroll
                            for (int e = 0; e < 4; ++e) {
                                float2 f = bf16x2_to_f32(w[e]);
                                acc[hh][2 * e] = fmaf(p, f.x, acc[hh][2 * e]);
                                acc[hh][2 * e + 1] = fmaf(p, f.y, acc[hh][2 * e + 1]);
                            }
                        }
                    }
                    l[hh] = lsum;
                }
                // the stage's shared memory is no longer needed: hand it back before any finishing work
                __syncwarp();
                if (lane == 0) da_mbar_arrive(empty_bar + stage);
                if (++stage == P.stages) { stage = 0; phase ^= 1; }
                const bool last = (mt.flags & 2u) != 0;
                if (!last) continue;
                // ---- end of the item: fold the KPW side-by-side key groups, then store or merge ----
#pragma unroll
                for (int hh = 0; hh < HPW; ++hh) {
                    const uint32_t h = warp + hh * consumers;
                    if (h >= P.heads) continue;
                    float mm = m[hh];
#pragma unroll
                    for (uint32_t o = LPK; o < 32; o <<= 1) mm = fmaxf(mm, __shfl_xor_sync(0xffffffffu, mm, o));
                    const float m_safe = (mm == -INFINITY) ? 0.0f : mm;
                    const float f = ex2(m[hh] - m_safe);
                    float ll = l[hh] * f;
                    float a[8];
#pragma unroll
                    for (int e = 0; e < 8; ++e) a[e] = acc[hh][e] * f;
#pragma unroll
                    for (uint32_t o = LPK; o < 32; o <<= 1) {
                        ll += __shfl_xor_sync(0xffffffffu, ll, o);
#pragma unroll
                        for (int e = 0; e < 8; ++e) a[e] += __shfl_xor_sync(0xffffffffu, a[e], o);
                    }
                    if (mt.slot == DA_DIRECT) {
                        // the item is the whole session: normalise and write the output row
                        if (grp == 0) {
                            const float inv = 1.0f / ll;
                            bf16* o = P.out + (size_t)mt.session * d + (size_t)h * HD + sub * 8;
                            *reinterpret_cast<uint4*>(o) = make_uint4(pack_bf16x2(a[0] * inv, a[1] * inv), pack_bf16x2(a[2] * inv, a[3] * inv),
                                                                      pack_bf16x2(a[4] * inv, a[5] * inv), pack_bf16x2(a[6] * inv, a[7] * inv));
                        }
                        continue;
                    }
                    if (grp == 0) {
                        float* dst = P.partial + ((size_t)mt.slot * P.heads + h) * (HD + 2);
                        // (HD + 2) floats per head keeps 8-byte alignment only: store as float2
#pragma unroll
                        for (int e = 0; e < 4; ++e)
                            *reinterpret_cast<float2*>(dst + sub * 8 + 2 * e) = make_float2(a[2 * e], a[2 * e + 1]);
                        if (sub == 0) *reinterpret_cast<float2*>(dst + HD) = make_float2(mm, ll);
                        __threadfence();
                    }
                    __syncwarp();
                    // whoever stores the last partial of (session, head) merges them
                    const uint32_t n_parts = mt.n_parts;
                    uint32_t seen = 0;
                    if (lane == 0) seen = atomicAdd(P.done + (size_t)mt.session * P.heads + h, 1u);
                    seen = __shfl_sync(0xffffffffu, seen, 0);
                    if (seen + 1 == n_parts) {
                        __threadfence();
                        constexpr int DPL = HD / 32;  // output dims per lane
                        const float* base = P.partial + ((size_t)mt.first_slot * P.heads + h) * (HD + 2);
                        const size_t step = (size_t)P.heads * (HD + 2);
                        // Sums go in a fixed order of the pieces, f32.
                        float o[DPL], mx = -INFINITY, lt = 0.0f;
#pragma unroll
                        for (int e = 0; e < DPL; ++e) o[e] = 0.0f;
                        constexpr uint32_t FEW = 4;
                        if (n_parts <= FEW) {
                            // the usual case of a full GPU (a session cut in two to four pieces): every value of every piece is
                            // requested before the first is used, one L2 round trip
                            float pm[FEW], pl[FEW], pn[FEW][DPL];
#pragma unroll
                            for (uint32_t i = 0; i < FEW; ++i) {
                                const float* pp = base + i * step;
                                const bool have = i < n_parts;
                                pm[i] = have ? __ldcg(pp + HD) : -INFINITY;
                                pl[i] = have ? __ldcg(pp + HD + 1) : 0.0f;
#pragma unroll
                                for (int e = 0; e < DPL; ++e) pn[i][e] = have ? __ldcg(pp + lane * DPL + e) : 0.0f;
                            }
#pragma unroll
                            for (uint32_t i = 0; i < FEW; ++i) mx = fmaxf(mx, pm[i]);
                            const float ms = (mx == -INFINITY) ? 0.0f : mx;
#pragma unroll
                            for (uint32_t i = 0; i < FEW; ++i) {
                                if (i < n_parts) {
                                    const float w = ex2(pm[i] - ms);
                                    lt = fmaf(pl[i], w, lt);
#pragma unroll
                                    for (int e = 0; e < DPL; ++e) o[e] = fmaf(pn[i][e], w, o[e]);
                                }
                            }
                        } else if (KS == DA_KS_LEAN) {
                            // a range of a large batch: sessions in more pieces are rare, and the code below makes the scan itself 3 %
                            // slower here (256 sessions 1.23 -> 1.27 ms per step)
                            for (uint32_t i = 0; i < n_parts; ++i) mx = fmaxf(mx, __ldcg(base + i * step + HD));
                            const float ms = (mx == -INFINITY) ? 0.0f : mx;
                            for (uint32_t i = 0; i < n_parts; ++i) {
                                const float* pp = base + i * step;
                                const float w = ex2(__ldcg(pp + HD) - ms);
                                lt = fmaf(__ldcg(pp + HD + 1), w, lt);
#pragma unroll
                                for (int e = 0; e < DPL; ++e) o[e] = fmaf(__ldcg(pp + lane * DPL + e), w, o[e]);
                            }
                        } else {
                            // Few sessions on many SMs: lane i holds maximum and sum of pieces i, i + 32, ...; the numerators are asked for up
                            // to eight pieces at a time, so a merge costs a few trips to L2 however the session was cut (one session
                            // of 1000 keys is 32 pieces; a piece after the other took most of a launch: a step of 12 layers 448 ->
                            // 409 us).
                            constexpr uint32_t LOTS = DA_MAX_CTAS / 32, TOGETHER = HD == 128 ? 4 : 8;
                            float pm[LOTS], pl[LOTS];
#pragma unroll
                            for (uint32_t r = 0; r < LOTS; ++r) {
                                const bool have = r * 32 + lane < n_parts;
                                const float* pp = base + (size_t)(r * 32 + lane) * step;
                                const float2 v = have ? __ldcg(reinterpret_cast<const float2*>(pp + HD)) : make_float2(-INFINITY, 0.0f);
                                pm[r] = v.x;
                                pl[r] = v.y;
                                mx = fmaxf(mx, v.x);
                            }
#pragma unroll
                            for (uint32_t x = 16; x > 0; x >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, x));
                            const float ms = (mx == -INFINITY) ? 0.0f : mx;
#pragma unroll
                            for (uint32_t r = 0; r < LOTS; ++r) {
                                pm[r] = ex2(pm[r] - ms);           // the piece's weight
                                lt = fmaf(pl[r], pm[r], lt);
                            }
#pragma unroll
                            for (uint32_t x = 16; x > 0; x >>= 1) lt += __shfl_xor_sync(0xffffffffu, lt, x);
#pragma unroll
                            for (uint32_t r = 0; r < LOTS; ++r) {
                                if (r * 32 >= n_parts) continue;   // warp-uniform
#pragma unroll
                                for (uint32_t i0 = 0; i0 < 32; i0 += TOGETHER) {
                                    if (r * 32 + i0 >= n_parts) continue;
                                    float pn[TOGETHER][DPL];
#pragma unroll
                                    for (uint32_t i = 0; i < TOGETHER; ++i)
#pragma unroll
                                        for (int e = 0; e < DPL; ++e)
                                            pn[i][e] = r * 32 + i0 + i < n_parts ? __ldcg(base + (size_t)(r * 32 + i0 + i) * step + lane * DPL + e) : 0.0f;
#pragma unroll
                                    for (uint32_t i = 0; i < TOGETHER; ++i) {
                                        const float w = __shfl_sync(0xffffffffu, pm[r], i0 + i);
#pragma unroll
                                        for (int e = 0; e < DPL; ++e) o[e] = fmaf(pn[i][e], w, o[e]);
                                    }
                                }
                            }
                        }
                        const float inv = 1.0f / lt;
                        bf16* orow = P.out + (size_t)mt.session * d + (size_t)h * HD + lane * DPL;
#pragma unroll
                        for (int e = 0; e < DPL; ++e) orow[e] = __float2bfloat16_rn(o[e] * inv);
                        if (lane == 0) P.done[(size_t)mt.session * P.heads + h] = 0;
                    }
                }
                break;
            }
        }
        // sessions without any live key own no item: their output row is zero
        for (uint32_t b = blockIdx.x * consumers + warp; b < P.batch; b += gridDim.x * consumers) {
            if (P.count[b] != 0) continue;
            for (uint32_t c = lane * 8; c < d; c += 32 * 8)
                *reinterpret_cast<uint4*>(P.out + (size_t)b * d + c) = make_uint4(0u, 0u, 0u, 0u);
        }
    }
    __syncthreads();
    if (*abort_flag) {
        const uint64_t start = da_timer_ns();
        while (da_timer_ns() - start < 200000ull) __nanosleep(1000);
        if (threadIdx.x == 0 && P.d_status) atomicCAS(P.d_status, DEV_OK, DEV_TIMEOUT);
        __syncthreads();
    }
}

// ===========================================================================
// Few keys in all: one launch, no plan, no workspace
// ===========================================================================
// With a few MB of keys the kernel above is a chain of latencies: work list, ring, partial results to L2, counters, merge (12 us for one
// session of 1000 keys x 12 heads, whose 3 MB are 0.5 us of HBM).  Here a cluster of CTAs shares one (session, head): rank r takes an even share
// of its keys, 16 bytes per lane straight into registers, 32 KB of keys (256, 128 or 64 of them) per CTA and pass, the next pass on its way while
// one is summed up.
// All keys but a session's newest are older than the previous kernel (the QKV product): their first pass is asked for before it ends.
// Partial (maximum, sum, numerator) go to rank 0 through distributed shared memory, which adds them in rank order.
constexpr uint32_t DS_THREADS = 256, DS_WARPS = DS_THREADS / 32;
constexpr int DS_U = 4;                      // keys of a lane group per pass
constexpr uint32_t DS_PAGES = 1536;          // pages that a CTA's share of keys may touch (ds_pays)

struct DsParams {
    const bf16* q;
    const bf16* kc;
    const bf16* vc;
    const uint32_t* lengths;
    const uint32_t* d_position;
    bf16* out;
    uint32_t extra, capacity, heads, ck;     // ck: CTAs of a cluster
    float scale_log2;
    int* d_status;
    KvPaging paging;
    uint32_t early;                          // the previous kernel writes no key but every session's newest
    uint32_t page_inverse;                   // 2^32 / page_rows rounded up: finds the page of every key, as capacity * page_rows <= 2^32
};

__device__ __forceinline__ uint4 ds_load(const bf16* p) {
    uint4 v;
    asm volatile("ld.global.cg.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void ds_cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void ds_cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }

template <int HD>
__global__ void __launch_bounds__(DS_THREADS, 3)
decode_attention_short_kernel(const __grid_constant__ DsParams P) {
    constexpr uint32_t LPK = HD / 8, KPW = 32 / LPK, PASS = DS_WARPS * KPW;   // lanes per key, keys of a warp and of the CTA side by side
    constexpr uint32_t PART = HD + 2;
    __shared__ float warp_part[DS_WARPS][PART], cta_part[8][PART];           // numerator, maximum, sum
    __shared__ uint32_t page_row[DS_PAGES];                                  // first rows of the pages of this CTA's keys
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, grp = lane / LPK, sub = lane % LPK;
    const uint32_t rank = blockIdx.x % P.ck, unit = blockIdx.x / P.ck, h = unit % P.heads, session = unit / P.heads, d = P.heads * HD;
    if (P.ck > 1) ds_cluster_arrive();
    if (!P.early) pdl_wait();
    uint32_t L = (P.lengths ? __ldcg(P.lengths + session) : (P.d_position ? __ldcg(P.d_position) : 0u)) + P.extra;
    if (L > P.capacity) {
        if (threadIdx.x == 0 && P.d_status) atomicCAS(P.d_status, DEV_OK, DEV_BAD_LENGTH);
        L = P.capacity;
    }
    // an even share, but half a pass at least: how many CTAs a short session is given does not show in its bits
    const uint32_t share = max((L + P.ck - 1) / P.ck, DS_U * PASS / 2), k0 = min(L, rank * share), k1 = min(L, k0 + share);
    const uint32_t mine = k0 + warp * KPW + grp;        // this lane group's keys: mine, mine + PASS, ...
    const size_t col = (size_t)h * HD + sub * 8;
    uint4 kx[DS_U], vx[DS_U];
    const uint4 none = make_uint4(0u, 0u, 0u, 0u);
    // The pages of the share are looked up once, all side by side: a look-up per key and pass is a chain of its own (a step of 20 sessions x 12 heads
    // of 64 at 575 keys, 4 layers, 168 us so, 156 from here; the streaming kernel 143).  Rows fit 32 bits: 2^32 of the narrowest are 256 GB.
    auto page_of = [&](uint32_t key) { return __umulhi(key, P.page_inverse); };
    const uint32_t first_page = P.paging.table ? page_of(k0) : 0u;
    if (P.paging.table) {
        const uint32_t pages = k1 > k0 ? page_of(k1 - 1) - first_page + 1 : 0u;
        const uint32_t* table = P.paging.table + (size_t)session * P.paging.pages_per_session + first_page;
        for (uint32_t i = threadIdx.x; i < pages; i += DS_THREADS) page_row[i] = __ldcg(table + i) * P.paging.page_rows;
        __syncthreads();
    }
    auto row_of = [&](uint32_t key) -> uint32_t {
        if (!P.paging.table) return session * P.capacity + key;
        const uint32_t page = page_of(key);
        return page_row[page - first_page] + (key - page * P.paging.page_rows);
    };
    auto at = [&](uint32_t row) { return (size_t)row * d + col; };
    constexpr uint32_t NO_ROW = ~0u;
    const uint32_t ahead = P.early ? L - 1 : k1;        // keys below it may be read now (a session of a step has one at least)
#pragma unroll
    for (int u = 0; u < DS_U; ++u) {
        const uint32_t key = mine + u * PASS;
        kx[u] = vx[u] = none;
        if (key < k1 && key < ahead) {
            const size_t o = at(row_of(key));
            kx[u] = ds_load(P.kc + o);
            vx[u] = ds_load(P.vc + o);
        }
    }
    if (P.early) pdl_wait();
    pdl_trigger();
    const uint4 qq = ds_load(P.q + (size_t)session * d + col);
    if (P.early && k1 == L) {
#pragma unroll
        for (int u = 0; u < DS_U; ++u) {
            if (mine + u * PASS != L - 1) continue;
            const size_t o = at(row_of(L - 1));
            kx[u] = ds_load(P.kc + o);
            vx[u] = ds_load(P.vc + o);
        }
    }
    float qf[8], acc[8], m = -INFINITY, l = 0.0f;
    {
        const uint32_t w[4] = {qq.x, qq.y, qq.z, qq.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float2 f = bf16x2_to_f32(w[e]);
            qf[2 * e] = f.x * P.scale_log2;
            qf[2 * e + 1] = f.y * P.scale_log2;
            acc[2 * e] = acc[2 * e + 1] = 0.0f;
        }
    }
    for (uint32_t base = 0; k0 + base < k1; base += DS_U * PASS) {
        float sc[DS_U];
        float m_new = m;
        uint32_t row[DS_U];                      // of the next pass
#pragma unroll
        for (int u = 0; u < DS_U; ++u) {
            const uint32_t key = mine + base + (DS_U + u) * PASS;
            row[u] = key < k1 ? row_of(key) : NO_ROW;
        }
#pragma unroll
        for (int u = 0; u < DS_U; ++u) {
            const uint32_t w[4] = {kx[u].x, kx[u].y, kx[u].z, kx[u].w};
            float part = 0.0f;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float2 f = bf16x2_to_f32(w[e]);
                part = fmaf(qf[2 * e], f.x, part);
                part = fmaf(qf[2 * e + 1], f.y, part);
            }
#pragma unroll
            for (uint32_t o = LPK / 2; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
            sc[u] = mine + base + u * PASS < k1 ? part : -INFINITY;
            m_new = fmaxf(m_new, sc[u]);
        }
#pragma unroll
        for (int u = 0; u < DS_U; ++u) kx[u] = row[u] != NO_ROW ? ds_load(P.kc + at(row[u])) : none;
        const float m_safe = m_new == -INFINITY ? 0.0f : m_new, corr = ex2(m - m_safe);
        m = m_new;
        l *= corr;
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[e] *= corr;
#pragma unroll
        for (int u = 0; u < DS_U; ++u) {
            const float p = ex2(sc[u] - m_safe);        // 0 for keys past the range
            l += p;
            const uint32_t w[4] = {vx[u].x, vx[u].y, vx[u].z, vx[u].w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float2 f = bf16x2_to_f32(w[e]);
                acc[2 * e] = fmaf(p, f.x, acc[2 * e]);
                acc[2 * e + 1] = fmaf(p, f.y, acc[2 * e + 1]);
            }
            vx[u] = row[u] != NO_ROW ? ds_load(P.vc + at(row[u])) : none;
        }
    }
    // lane groups of the warp, warps of the CTA, CTAs of the cluster
    float mm = m;
#pragma unroll
    for (uint32_t o = LPK; o < 32; o <<= 1) mm = fmaxf(mm, __shfl_xor_sync(0xffffffffu, mm, o));
    const float f = ex2(m - (mm == -INFINITY ? 0.0f : mm));
    l *= f;
#pragma unroll
    for (int e = 0; e < 8; ++e) acc[e] *= f;
#pragma unroll
    for (uint32_t o = LPK; o < 32; o <<= 1) {
        l += __shfl_xor_sync(0xffffffffu, l, o);
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[e] += __shfl_xor_sync(0xffffffffu, acc[e], o);
    }
    if (grp == 0) {
#pragma unroll
        for (int e = 0; e < 8; ++e) warp_part[warp][sub * 8 + e] = acc[e];
        if (sub == 0) { warp_part[warp][HD] = mm; warp_part[warp][HD + 1] = l; }
    }
    __syncthreads();
    if (threadIdx.x >= HD && P.ck == 1) return;
    // sums `parts` partials of dimension c: (numerator, maximum, sum)
    auto join = [&](const float (*part)[PART], uint32_t parts, uint32_t c) {
        float top = -INFINITY, num = 0.0f, sum = 0.0f;
        for (uint32_t i = 0; i < parts; ++i) top = fmaxf(top, part[i][HD]);
        const float safe = top == -INFINITY ? 0.0f : top;
        for (uint32_t i = 0; i < parts; ++i) {
            const float w = ex2(part[i][HD] - safe);
            num = fmaf(part[i][c], w, num);
            sum = fmaf(part[i][HD + 1], w, sum);
        }
        return make_float3(num, top, sum);
    };
    const uint32_t c = threadIdx.x;
    float3 all = make_float3(0.0f, -INFINITY, 0.0f);
    if (c < HD) all = join(warp_part, DS_WARPS, c);
    if (P.ck > 1) {
        ds_cluster_wait();                       // rank 0 is there
        if (c < HD) {
            uint32_t to;
            const uint32_t from = (uint32_t)__cvta_generic_to_shared(&cta_part[rank][0]);
            asm("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(to) : "r"(from));
            asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(to + 4 * c), "f"(all.x) : "memory");
            if (c == 0) {
                asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(to + 4 * HD), "f"(all.y) : "memory");
                asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(to + 4 * HD + 4), "f"(all.z) : "memory");
            }
        }
        ds_cluster_arrive();
        ds_cluster_wait();
        if (rank != 0 || c >= HD) return;
        all = join(cta_part, P.ck, c);
    }
    // a session without keys: zeros
    P.out[(size_t)session * d + h * HD + c] = __float2bfloat16_rn(L ? all.x / all.z : 0.0f);
}

static int da_sm_count() {
    static int n = 0;
    if (!n) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        if (n <= 0) n = 148;
    }
    return n;
}

// Clusters of `ck` CTAs that run side by side (they do not cross a GPC: 444, 222, 142, 104, 82, 71, 56, 48 of 1 to 8 on a B200, not 444 / ck).
template <int HD>
static uint32_t ds_clusters_at_once(uint32_t ck) {
    static std::atomic<int> known[64][9];          // 0: not asked yet
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
    int n = known[dev][ck].load(std::memory_order_relaxed);
    if (n == 0) {
        prefer_max_shared_carveout(reinterpret_cast<const void*>(decode_attention_short_kernel<HD>));
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(ck);
        cfg.blockDim = dim3(DS_THREADS);
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = ck;
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        if (cudaOccupancyMaxActiveClusters(&n, decode_attention_short_kernel<HD>, &cfg) != cudaSuccess) cudaGetLastError();
        if (n <= 0) n = -1;
        known[dev][ck].store(n, std::memory_order_relaxed);
    }
    return n > 0 ? (uint32_t)n : 0u;
}
// CTAs per (session, head): the largest cluster, portable ones, of which all run at once.  (One too large is a second wave: a step of 12 sessions x
// 12 heads at 1215 keys 156 us in clusters of three, 138 in clusters of two.)
template <int HD>
static uint32_t ds_cluster(uint32_t units) {
    uint32_t ck = 8;
    while (ck > 1 && units > ds_clusters_at_once<HD>(ck)) --ck;
    return ck;
}

// Whether the launch above is the faster one: `longest` keys that a session can have, `chained` in a session's step (no plan to save there, as
// that is made once for all layers).  Its CTAs are not balanced by length and their many short streams stop at 4 TB/s, so what ends it is keys x
// heads in all.  us with the streaming kernel / here, B200, operator, sessions x heads of 64 x capacity, lengths anywhere:
//       1 x 12 x 64     13.8 / 6.2     16 x 12 x 1000  20.7 / 15.9    1 x 16 x 4096   28.5 / 11.6    64 x 16 x 300   22.3 / 18.4
//       1 x 12 x 1000   17.1 / 7.3     32 x 12 x 1000  23.6 / 22.2    4 x 12 x 4096   25.7 / 15.4    16 x 16 x 4096  34.9 / 49.3
//       16 x 12 x 300   18.3 / 9.4     48 x 12 x 900   25.7 / 24.5    8 x 12 x 2048   23.2 / 15.0    64 x 16 x 1000  34.8 / 39.3
// so 400 K (at that line 0.82 of the streaming kernel's time on average and 0.98 at most, heads of 32 0.77 and 0.99).  Heads of 128 have twice the bytes:
// 0.87 on average at 300 K, 0.97 at 400 K; chains of more than 20 passes lose there (4 x 4 x 12496 39.1 / 42.1), but with few rows (1 x 4 x 12496 38.7 / 30.7).
// In a step, measured over 1328 handles of 4 layers, heads of 32, 64 and 128, contiguous and in pages, at their last key and at a third of it: 180 K keys x
// heads; two waves at most (48 x 24 heads of 32 at 21 keys 1.08 times as long); and no chain of more than 12 passes (four where a CTA has a session's
// head alone and few are there to hide it), unless the rows are few, where the streaming kernel is a chain itself.  At the last key / at a third of
// it, time here over time there: 0.87 / 0.83 on average inside these lines, 1.06 at worst; past them
//       sessions x heads x capacity   20 x 12 x 64, 576: 1.07 / 0.92 (4.5 passes, alone)      2 x 4 x 128, 7488: 1.07 / 0.72 (14.6 passes)
//       64 x 12 x 32, 448 (344 K): 1.09 / 0.95                                                 1 x 8 x 128, 7488: 0.75 / 0.68 (14.6 passes, few rows: taken)
static bool ds_pays(uint32_t batch, uint32_t heads, uint32_t ck, uint32_t longest, uint32_t head_dim, bool chained) {
    const uint64_t units = (uint64_t)batch * heads, keys = units * longest, rows = (uint64_t)batch * longest;
    const uint32_t pass = 8192 / head_dim, passes = ceil_div(ceil_div(longest, ck), pass);
    if (!chained) return head_dim <= 64 ? keys <= 400000u : keys <= 300000u && (passes <= 20u || rows <= 16384u);
    return keys <= 180000u && units <= 888u && (ck == 1 ? passes <= 4u : passes <= 12u || rows <= 8192u);
}

// Launches an attention kernel, between two events of the handle's record while one is kept: the same kernel either way.
template <typename Launch>
static int launch_timed(cudaStream_t stream, const char* name, Launch&& launch) {
    KernelTimer* timer = t_attention_timer;
    size_t at = 0;
    if (timer) {
        while (timer->used + 2 > timer->events.size()) {
            cudaEvent_t e;
            if (cudaEventCreate(&e) != cudaSuccess) return check_launch("decode_attention event");
            timer->events.push_back(e);
        }
        at = timer->used;
        timer->used += 2;
        cudaEventRecord(timer->events[at], stream);
    }
    launch();
    if (timer) cudaEventRecord(timer->events[at + 1], stream);
    count_launch();
    return check_launch(name);
}

template <int HD>
static int launch_ds(const DsParams& P, uint32_t units, cudaStream_t stream) {
    return launch_timed(stream, "decode_attention_short", [&] {
        launch_kernel_clusters(decode_attention_short_kernel<HD>, dim3(units * P.ck), dim3(DS_THREADS), 0, P.ck, stream, P);
    });
}

template <int HD, int HPW, int KS>
static int launch_da_t(const DaParams& P, uint32_t threads, size_t smem, uint32_t grid, cudaStream_t stream) {
    static size_t configured[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || configured[dev] < smem) {
        if (cudaFuncSetAttribute(decode_attention_kernel<HD, HPW, KS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
            return check_launch("decode_attention attribute");
        if (dev >= 0 && dev < 64) configured[dev] = smem;
    }
    return launch_timed(stream, "decode_attention", [&] { launch_kernel(decode_attention_kernel<HD, HPW, KS>, dim3(grid), dim3(threads), smem, stream, P); });
}

// lengths may be nullptr: then every session holds (d_position ? *d_position : 0) + extra keys.
int launch_decode_attention_ex(const bf16* q, const bf16* k_cache, const bf16* v_cache, const uint32_t* d_lengths,
                               const uint32_t* d_position, uint32_t extra, bf16* out, void* workspace,
                               uint64_t workspace_bytes, uint32_t batch, uint32_t capacity, uint32_t heads,
                               uint32_t head_dim, bool plan, int* d_status, cudaStream_t stream, bool lean,
                               const KvPaging* paging) {
    if (batch == 0) return TNSR_B200_OK;
    if (!decode_attention_supported(heads, head_dim)) {
        set_thread_error("decode attention: head_dim must be 32, 64 or 128 and heads <= 32");
        return TNSR_B200_ERR_UNSUPPORTED;
    }
    if ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k_cache) | reinterpret_cast<uintptr_t>(v_cache) |
         reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(workspace)) % 16) {
        set_thread_error("decode attention: pointers must be 16-byte aligned");
        return TNSR_B200_ERR_INVALID_ARGUMENT;
    }
    const DaLayout L = da_layout(batch, heads, head_dim);
    if (L.bytes > workspace_bytes) {
        set_thread_error("decode attention: workspace too small");
        return TNSR_B200_ERR_INVALID_ARGUMENT;
    }
    if (paging && paging->table && (paging->page_rows == 0 || paging->page_rows % DA_KS != 0)) {
        set_thread_error("decode attention: the page size must be a multiple of 16 rows");
        return TNSR_B200_ERR_INVALID_ARGUMENT;
    }
    const uint32_t units = batch * heads;
    const uint32_t ck = head_dim == 32 ? ds_cluster<32>(units) : head_dim == 64 ? ds_cluster<64>(units) : ds_cluster<128>(units);
    const bool paged = paging && paging->table;
    const bool addressed = !paged || ((uint64_t)capacity * paging->page_rows <= 1ull << 32 && ceil_div(capacity, ck) / paging->page_rows + 2 <= DS_PAGES);
    // a step's newest key comes on top of the lengths
    if (!lean && addressed && ds_pays(batch, heads, ck, capacity, head_dim, extra > 0)) {
        DsParams S;
        S.q = q; S.kc = k_cache; S.vc = v_cache; S.out = out;
        S.lengths = d_lengths; S.d_position = d_position; S.extra = extra;
        S.capacity = capacity; S.heads = heads; S.ck = ck;
        S.scale_log2 = (1.0f / sqrtf((float)head_dim)) * 1.4426950408889634f;
        S.d_status = d_status;
        if (paged) S.paging = *paging;
        S.page_inverse = paged ? (uint32_t)(((1ull << 32) + paging->page_rows - 1) / paging->page_rows) : 0u;
        S.early = t_pdl && extra > 0;
        return head_dim == 32 ? launch_ds<32>(S, units, stream) : head_dim == 64 ? launch_ds<64>(S, units, stream) : launch_ds<128>(S, units, stream);
    }
    uint8_t* ws = reinterpret_cast<uint8_t*>(workspace);
    uint32_t* header = reinterpret_cast<uint32_t*>(ws);
    uint32_t* first = reinterpret_cast<uint32_t*>(ws + L.first);
    uint32_t* count = reinterpret_cast<uint32_t*>(ws + L.count);
    uint32_t* done = reinterpret_cast<uint32_t*>(ws + L.done);
    uint32_t* sstart = reinterpret_cast<uint32_t*>(ws + L.sstart);
    uint32_t* cta_begin = reinterpret_cast<uint32_t*>(ws + L.cta_begin);
    DaItem* items = reinterpret_cast<DaItem*>(ws + L.items);
    float* partial = reinterpret_cast<float*>(ws + L.partial);
    uint32_t grid = (uint32_t)da_sm_count();
    if (grid > DA_MAX_CTAS) grid = DA_MAX_CTAS;
    // keys per ring stage: 8 in the lean form if two such stages (the least a ring needs) fit its budget
    const uint32_t d = heads * head_dim, row_bytes = d * 2;
    if (lean && 2 * (2 * DA_KS_LEAN * row_bytes + row_bytes) > DA_SMEM_BUDGET_LEAN) lean = false;
    const uint32_t ks = lean ? DA_KS_LEAN : DA_KS;
    if (!d_lengths) {
        // Every session has the same length (the decoder's own steps).  If the grid divides the batch, or the batch
        // divides the grid, the equal key ranges of the CTAs line up with the sessions: whole sessions per CTA (no
        // partial results, no merge) or an even split of every session.  That is worth more than the SMs left idle:
        // 256 sessions on 128 CTAs take 81 us per launch against 86 us on 148 (measured), as long as at least three
        // quarters of the SMs stay in use.
        uint32_t aligned = 0;
        if (batch >= grid) {
            for (uint32_t g = grid; g >= 1 && 4 * g >= 3 * grid; --g)
                if (batch % g == 0) { aligned = g; break; }
        } else if (batch > 0) {
            aligned = batch * (grid / batch);
            if (4 * aligned < 3 * grid) aligned = 0;
        }
        if (aligned) grid = aligned;
    }
    if (plan) {
        launch_kernel(da_plan_kernel, dim3(1), dim3(1024), 0, stream, d_lengths, d_position, extra, batch, heads, capacity, grid,
                      ks, header, first, count, done, sstart, cta_begin, items, d_status);
        count_launch();
        int rc = check_launch("decode_attention plan");
        if (rc) return rc;
    }
    const uint32_t stage_bytes = 2 * ks * row_bytes + row_bytes;
    uint32_t stages = (lean ? DA_SMEM_BUDGET_LEAN : DA_SMEM_BUDGET) / stage_bytes;
    if (stages > DA_MAX_STAGES) stages = DA_MAX_STAGES;
    const size_t smem = (size_t)stages * stage_bytes + 2 * DA_MAX_STAGES * 8 + DA_MAX_STAGES * sizeof(DaStageMeta) + 16;
    const uint32_t hpw = heads > 16 ? 2 : 1;
    const uint32_t consumers = ceil_div(heads, hpw);
    DaParams P;
    P.q = q; P.kc = k_cache; P.vc = v_cache;
    P.first = first; P.count = count; P.done = done; P.cta_begin = cta_begin; P.items = items; P.partial = partial;
    P.out = out;
    P.batch = batch; P.capacity = capacity; P.heads = heads; P.stages = stages;
    P.scale_log2 = (1.0f / sqrtf((float)head_dim)) * 1.4426950408889634f;
    P.d_status = d_status;
    P.wait_limit_ns = g_wait_limit_ns.load(std::memory_order_relaxed);
    P.early = !plan && t_pdl;
    if (paging && paging->table) P.paging = *paging;
    const uint32_t threads = (consumers + 1) * 32;
    if (lean) {
        if (hpw == 1) {
            return head_dim == 32 ? launch_da_t<32, 1, DA_KS_LEAN>(P, threads, smem, grid, stream)
                 : head_dim == 64 ? launch_da_t<64, 1, DA_KS_LEAN>(P, threads, smem, grid, stream)
                                  : launch_da_t<128, 1, DA_KS_LEAN>(P, threads, smem, grid, stream);
        }
        return head_dim == 32 ? launch_da_t<32, 2, DA_KS_LEAN>(P, threads, smem, grid, stream)
             : head_dim == 64 ? launch_da_t<64, 2, DA_KS_LEAN>(P, threads, smem, grid, stream)
                              : launch_da_t<128, 2, DA_KS_LEAN>(P, threads, smem, grid, stream);
    }
    if (hpw == 1) {
        return head_dim == 32 ? launch_da_t<32, 1, DA_KS>(P, threads, smem, grid, stream)
             : head_dim == 64 ? launch_da_t<64, 1, DA_KS>(P, threads, smem, grid, stream)
                              : launch_da_t<128, 1, DA_KS>(P, threads, smem, grid, stream);
    }
    return head_dim == 32 ? launch_da_t<32, 2, DA_KS>(P, threads, smem, grid, stream)
         : head_dim == 64 ? launch_da_t<64, 2, DA_KS>(P, threads, smem, grid, stream)
                          : launch_da_t<128, 2, DA_KS>(P, threads, smem, grid, stream);
}

int launch_decode_attention(const bf16* q, const bf16* k_cache, const bf16* v_cache, const uint32_t* d_lengths,
                            bf16* out, void* workspace, uint64_t workspace_bytes, uint32_t batch,
                            uint32_t capacity, uint32_t heads, uint32_t head_dim, int* d_status,
                            cudaStream_t stream) {
    return launch_decode_attention_ex(q, k_cache, v_cache, d_lengths, nullptr, 0, out, workspace, workspace_bytes, batch,
                                      capacity, heads, head_dim, true, d_status, stream, false);
}

}  // namespace tb
