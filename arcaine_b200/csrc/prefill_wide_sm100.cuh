// GQA flash-attention prefill kernel for sm_100a, head dim 256: a pair of CTAs works on 256 query rows together.
//
// What bounds head dim 256.  One key block of 128 keys costs a 128-row tile 2048 clk of the tensor pipe (16 MMAs of
// 64 clk for S = Q K^T, 8 of 128 clk for O += P V) and 1024 clk of the ex2 unit; Q, one K and one V tile are 64 KB
// each, so a CTA on its own has room for one stage of each and pulls 128 KB per block through L2: 64 bytes per clk
// and SM at the tensor rate, more than L2 delivers to 148 SMs (the one-tile kernel takes 3700 clk per block).  The
// MMAs of a CTA pair (cta_group::2, M = 256) take half of B from either CTA: each CTA loads 64 of the block's keys
// for K and 128 of V's 256 columns — half the traffic, 32 KB stages, two of each.
//
// The pair's two tiles are the same 128 tokens of two query heads of one KV group (even group), else 256
// consecutive tokens of one head.  Tensor memory per CTA: two score buffers of 128 columns, O 256 columns.  S(j+1)
// is computed while the softmax warps work on S(j), so the tensor pipe only waits when a softmax takes longer than
// 2048 clk.
//
// Warp roles of each CTA (320 threads): 0-3 softmax (one row per thread), 4-7 epilogue, 8 TMA producer
// (its CTA's Q tile and halves of K and V), 9 MMA issuer (leader CTA only).  Full barriers live in the leader, which
// expects the bytes of both CTAs; empty and score barriers are committed to both (commit with multicast — the loads
// themselves use none).  The softmax and epilogue warps of both CTAs arrive on the leader's barriers.
//
// Masks, lazy rescaling, bounded waits and the status word are as in prefill_pair_sm100.cuh; P is written over the scores.
#pragma once
#include <type_traits>

#include "decode_sm100.cuh"
#include "prefill_pair_sm100.cuh"

namespace arc {

struct WideCfg {
    static constexpr int HD = 256;
    static constexpr int BM = 128;  // rows per CTA
    static constexpr int BN = 128;  // keys per block
    static constexpr int Q_BYTES = BM * HD * 2;
    static constexpr int Q_CHUNK = 128 * 128;      // 128 rows x 64 columns
    static constexpr int K_BYTES = BN / 2 * HD * 2;  // this CTA's 64 keys
    static constexpr int K_CHUNK = 64 * 128;       // 64 keys x 64 columns
    static constexpr int V_BYTES = BN * HD / 2 * 2;  // this CTA's 128 columns
    static constexpr int V_CHUNK = 128 * 128;      // 128 keys x 64 columns
    static constexpr int STAGES = 2;               // of K and of V
    static constexpr int COL_S = 0;                // + 128 * buffer
    static constexpr int COL_O = 256;
    // first[4] q_empty, {k,v}_{full,empty}[2], s_full[2], p_half[buffer][half], o_full o_empty fin[4], gate[epilogue warp][2], next_full next_empty, gate[softmax warp][2]
    static constexpr int NUM_BARS = 5 + 8 + 2 + 4 + 2 + 4 + 8 + 2 + 8;
    // Arrivals that complete a phase of barrier i: the eight softmax or epilogue warps of both CTAs, the four of one, or one thread.
    __device__ static constexpr int arrivals(int i) {
        return (i >= 15 && i < 19) || i == 20 ? 8 : (i >= 21 && i < 25) || i == 33 || i == 34 ? 4 : 1;  // p_half, o_empty; fin, next_full, next_empty
    }
    static constexpr int SMEM_BYTES = Q_BYTES + STAGES * (K_BYTES + V_BYTES) + STAGE_BYTES + NUM_BARS * 8 + 16 + 4 * 128 * 4 + 2 * 32 + 128 * 4;
    static_assert(SMEM_BYTES <= 232448, "more shared memory than a CTA can have");
    static constexpr int MOST_FOLDED = 4;  // parts of a split unit that fold themselves as one cluster
    static constexpr int EPILOGUE_WARP = 4, PRODUCER_WARP = 8, ISSUER_WARP = 9;
    static constexpr int THREADS = 320;
};

// One unit of the pair: this CTA's tile, and the key blocks [lo, hi) the pair walks (the union over both tiles).
struct WideWork {
    int q0, h, b, kvh, lo, hi;
    int part;  // of the key range
};

// ---------------------------------------------------------------------------
// Additive masks.  Read element by element from every row, head and block, the (seq, kv_len) f32 buffer made an
// attention of 1000 queries over 1300 keys take 180 us, of which the attention itself is 20.  In practice a mask is 0
// where a key is visible and -inf where it is not, and the same for all heads: one pass over the buffer turns it into a
// bit per key and a class per 32 rows x 128 keys.  The attention then skips key blocks nobody sees, tests nothing in
// those everybody sees and selects by bits in the others; only where other values occur does it read the mask itself.
// ---------------------------------------------------------------------------
constexpr uint32_t MASK_SEEN = 1;     // some key is not hidden
constexpr uint32_t MASK_HIDDEN = 2;   // some key is hidden or past the end
constexpr uint32_t MASK_VALUES = 4;   // some value is neither 0 nor hides its key

// A mask value hides its key where the softmax's log2 domain holds no number for it: -inf, and the type's lowest values
// with it, as in the kernels that add the mask to the scaled score.  (-2^128 / log2(e); the product itself cost the scan
// 0.6 us of a buffer of 1000 x 1300.)
__device__ __forceinline__ bool mask_hides(float value) { return value < -2.3586e38f; }

// Block = 32 rows x 128 keys, warp = 2 rows, a lane four consecutive keys of each, 16 bytes at once where all rows allow it.  Bound by
// its own latency (of 2.4 us 1.6 were those of one block), much of it instructions fetched cold, so there are few of them.  (us, the two
// calls of a masked layer: 64 queries 10.6 -> 10.1, 200 over 216 keys 12.1 -> 11.6, 2000 41.5 -> 40.4, 2048 over 4048 55.2 -> 54.3.)
__global__ void __launch_bounds__(512) mask_scan_kernel(const float* mask, int seq, int kv_len, int blocks, uint32_t* cls, uint32_t* bits) {
    __shared__ uint32_t s_class;
    if (threadIdx.x == 0) s_class = 0u;
    __syncthreads();
    grid_dependency_wait();
    grid_launch_dependents();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int j = blockIdx.x, r0 = blockIdx.y * 32 + warp * 2, key = j * 128 + lane * 4;
    const bool quads = ((reinterpret_cast<uintptr_t>(mask) & 15u) | (kv_len & 3)) == 0;
    float4 v[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        v[i] = make_float4(-CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F);
        const float* src = mask + (long long)(r0 + i) * kv_len + key;
        if (r0 + i >= seq) continue;
        if (quads) {
            if (key < kv_len) v[i] = *reinterpret_cast<const float4*>(src);
        } else {
            if (key < kv_len) v[i].x = src[0];
            if (key + 1 < kv_len) v[i].y = src[1];
            if (key + 2 < kv_len) v[i].z = src[2];
            if (key + 3 < kv_len) v[i].w = src[3];
        }
    }
    uint32_t c8 = 0;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const float e[4] = {v[i].x, v[i].y, v[i].z, v[i].w};
        uint32_t w = 0;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            w |= e[c] == 0.f ? 1u << c : 0u;
            if (r0 + i < seq) c8 |= mask_hides(e[c]) ? MASK_HIDDEN : e[c] != 0.f ? MASK_SEEN | MASK_VALUES : MASK_SEEN;
        }
        w <<= 4 * (lane & 7);  // eight lanes make a word of 32 keys
        w |= __shfl_xor_sync(0xffffffffu, w, 1);
        w |= __shfl_xor_sync(0xffffffffu, w, 2);
        w |= __shfl_xor_sync(0xffffffffu, w, 4);
        const int row = r0 + i;
        if ((lane & 7) == 0) bits[(((long long)(row >> 7) * blocks + j) * 128 + (row & 127)) * 4 + (lane >> 3)] = w;
    }
    c8 = __reduce_or_sync(0xffffffffu, c8);
    if (lane == 0) atomicOr(&s_class, c8);
    __syncthreads();
    if (threadIdx.x == 0) {
        const int row = blockIdx.y * 32;
        reinterpret_cast<uint8_t*>(cls + (long long)(row >> 7) * blocks + j)[(row >> 5) & 3] = static_cast<uint8_t>(s_class);
    }
}

// Key blocks [lo, hi) between the first and the last one somebody in the row tiles [t0, t1) sees.  Whole warps.
__device__ __forceinline__ void masked_blocks(const PrefillParams& p, int t0, int t1, int& lo, int& hi) {
    const int lane = threadIdx.x & 31;
    lo = hi = 0;
    for (int j0 = 0; j0 < p.mask_blocks; j0 += 32) {
        uint32_t c = 0;
        if (j0 + lane < p.mask_blocks)
            for (int t = t0; t < t1; ++t) c |= p.mask_class[(long long)t * p.mask_blocks + j0 + lane];
        const uint32_t seen = __ballot_sync(0xffffffffu, (c & (MASK_SEEN * 0x01010101u)) != 0);
        if (!seen) continue;
        if (hi == 0) lo = j0 + __ffs(seen) - 1;
        hi = j0 + 32 - __clz(seen);
    }
}

// One chunk of 32 keys: hidden scores become -inf.
__device__ __forceinline__ void select_chunk(uint32_t (&v)[32], uint32_t bits) {
#pragma unroll
    for (int e = 0; e < 32; ++e) v[e] = (bits >> e) & 1u ? v[e] : 0xff800000u;
}

// A block with values: score * scale + mask in the log2 domain, as the softmax goes on to use it (with a scale of one),
// back into tensor memory.  (Not mask / scale beside the raw score: where the mask is large, the product with the scale is
// then off by more than an exponent holds.)  A thread is a row, so a load touches 32 lines whatever its width: four values
// a load where all rows are 16-byte aligned (6400 clk a block of 128 rows against 17600).
__device__ __forceinline__ void add_mask_values(uint32_t tS, const float* mask, int row, int rows, int key0, int kv_len, float sl) {
    const float* mask_row = mask + (long long)row * kv_len;
    const bool quads = ((reinterpret_cast<uintptr_t>(mask) & 15u) | (kv_len & 3)) == 0;
#pragma unroll 1
    for (int c = 0; c < 128; c += 32) {
        const int n = row < rows ? kv_len - key0 - c : 0;  // keys of the chunk that there are
        const float* src = mask_row + key0 + c;
        float m[32];
        if (quads) {
#pragma unroll
            for (int e = 0; e < 32; e += 4) {
                const float4 f = e < n ? *reinterpret_cast<const float4*>(src + e) : make_float4(-CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F);
                m[e] = f.x, m[e + 1] = f.y, m[e + 2] = f.z, m[e + 3] = f.w;
            }
        } else {
#pragma unroll
            for (int e = 0; e < 32; ++e) m[e] = e < n ? src[e] : -CUDART_INF_F;
        }
        uint32_t v[32];
        tmem_ld32(tS + c, v);
        tmem_wait_ld();
#pragma unroll
        for (int e = 0; e < 32; ++e) v[e] = __float_as_uint(__uint_as_float(v[e]) * sl + m[e] * 1.4426950408889634f);
        tmem_st32(tS + c, v);
    }
    tmem_wait_st();
}

template <bool VISION>
__device__ __forceinline__ void wide_blocks(const PrefillParams& p, int q_first, int q_last, int& lo, int& hi) {
    const int off = p.kv_len - p.seq;
    lo = 0;
    hi = (p.kv_len + WideCfg::BN - 1) / WideCfg::BN;
    if (p.mask_type == 3) {
        q_last = min(q_last, p.seq - 1);
        // (the span ends are monotone in the row, so the last row decides)
        const int last_key = VISION ? vision_end(p, q_last + off) - 1 : min(p.kv_len - 1, q_last + off);
        hi = last_key >= 0 ? last_key / WideCfg::BN + 1 : 0;
        if (p.window > 0 && p.window != 0x7fffffff) lo = max(0, q_first + off - p.window + 1) / WideCfg::BN;
    }
    if (hi < lo) hi = lo;
}

// Position of a CTA pair in the list of units.  Plain order: token tiles fastest, then heads, then sequences (pairs that
// run side by side share K and V in L2).  long_first (causal, with a window or not, more units than pairs,
// whose keys and values stay in L2): the units with most key blocks first, all heads of a token tile together, and every second wave in
// reverse order, so that the sums of a pair's units are about equal.
// few > 0: the first `few` pairs share the longest units [0, few_end) in that way and the others the rest, of which they take
// one more each.
template <bool ONE>  // one unit a pair: the walk ends behind it
struct WideCursor {
    int w, i;
    __device__ __forceinline__ explicit WideCursor(const PrefillParams& p) : i(-1) { advance(p); }
    __device__ __forceinline__ void advance(const PrefillParams& p) {
        if constexpr (ONE) {
            w = ++i == 0 ? (int)(blockIdx.x >> 1) : 0x7fffffff;
            return;
        }
        const int place = (int)(blockIdx.x >> 1);
        const bool rest = place >= p.few;  // (few is 0 where nothing is divided in this way)
        const int base = rest ? p.few_end : 0, first = rest ? place - p.few : place;
        const int step = rest ? (int)(gridDim.x >> 1) - p.few : p.few;
        ++i;
        w = base + i * step + (p.long_first && (i & 1) ? step - 1 - first : first);
    }
};

// The unit at the cursor, without its key blocks: nothing here depends on memory.
template <bool SPLIT, bool ONE>
__device__ __forceinline__ WideWork wide_place(const PrefillParams& p, const WideCursor<ONE>& cur, int rank) {
    WideWork t;
    int qt;
    t.part = SPLIT ? cur.w % p.num_splits : 0;
    if (!SPLIT && p.long_first) {
        const int per = p.cur_heads * p.batch, rest = cur.w % per;
        qt = p.q_tiles - 1 - cur.w / per;
        t.h = rest % p.cur_heads;
        t.b = rest / p.cur_heads;
    } else {
        const int w = SPLIT ? cur.w / p.num_splits : cur.w;
        const int rest = w / p.q_tiles;
        qt = w % p.q_tiles;
        t.h = rest % p.cur_heads;
        t.b = rest / p.cur_heads;
    }
    if (p.head_pair) {
        t.h = t.h * 2 + rank;
        t.q0 = qt * WideCfg::BM;
    } else {
        t.q0 = (qt * 2 + rank) * WideCfg::BM;
    }
    t.kvh = p.group_shift >= 0 ? (t.h >> p.group_shift) : t.h / p.group;
    return t;
}

template <bool MASKED, bool SPLIT, bool VISION>
__device__ __forceinline__ void wide_find_blocks(const PrefillParams& p, int rank, WideWork& t) {
    const int rows = p.head_pair ? WideCfg::BM : 2 * WideCfg::BM;  // tokens of the unit
    const int q0 = p.head_pair ? t.q0 : t.q0 - rank * WideCfg::BM;
    if constexpr (MASKED) masked_blocks(p, q0 >> 7, min(q0 + rows, p.seq + 127) >> 7, t.lo, t.hi);
    else wide_blocks<VISION>(p, q0, q0 + rows - 1, t.lo, t.hi);
    if (SPLIT) {
        const int lo = t.lo, n = t.hi - t.lo;
        t.lo = lo + n * t.part / p.num_splits;
        t.hi = lo + n * (t.part + 1) / p.num_splits;
    }
}

// MASKED: with an additive mask, as mask_scan_kernel has read it.  (With SPLIT: few queries over a long cache.  16 of 8 heads
// over 32768 keys take 299 us as whole units and 59 in parts; 64 over 4096 keys 45 and 18.)
// SPLIT: a unit is one of num_splits parts of the key blocks, one unit per pair, for calls whose tiles would leave most
// pairs idle.  The part's normalised rows go to the partial records as f32 with their log-sum-exp.  SPLIT 2: two to four
// parts are the pairs of one cluster; each CTA stores only the columns the other parts' CTAs finish, and after a cluster
// barrier finishes its own columns.  SPLIT 1: more parts are folded by sdpa_uniform_merge_kernel.  The values pass through L2:
// read out of the other CTAs' shared memory, 11 bytes per clk and SM, the fold took 5 us.  Every instruction here runs
// once per launch and is fetched cold, 50 clk per 128 bytes of code, so there are few: with rows divided instead of columns, which
// had to go through shared memory on either side, 13000 clk passed from the last P V to the end  (us: 256 queries of 16 heads over
// 2304 keys 18.0 -> 15.5, 512 over 2560 23.5 -> 21.4, 512 of 8 heads over 1512 15.5 -> 12.6.)
// SEVERAL: pairs take several units.  EARLY (SEVERAL, not gated): the epilogue empties the accumulator into registers first (1600 clk), for the
// next unit's P V to go on; in turns, with the way out of the SM between them, it took 3000.  (2 x 5000 tokens of 16/8 heads,
// window 512, 103 -> 96 us.  Gated rows wait for sigmoids, not for the way out: taken early they cost calls of short units 8 %.)
// VISION: causal with vision blocks (p.ids).  Where pairs take several units the next unit's blocks and rows are looked up by warps
// that wait anyway: between two units the look-up cost the softmax warps 2200 clk and the scores behind it as much.  (1531 tokens of
// 16/8 heads with three images 24.4 -> 23.2 us.)
// ONE: not SEVERAL, one unit a pair.  The walks are then left out of every role; small calls waited for them (161 queries of 24/4 heads over
// 202 keys 8.28 -> 7.74 us, gated 9.92 -> 9.33; 64 of 16/8 over 64 6.81 -> 6.29).
template <bool GATE, bool MASKED, int SPLIT = 0, bool SEVERAL = false, bool VISION = false>
__global__ void __launch_bounds__(WideCfg::THREADS, 1)
    sdpa_prefill_wide_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                             const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_out,
                             const __grid_constant__ CUtensorMap tm_gate, const PrefillParams p) {
    using C = WideCfg;
    constexpr int HD = C::HD;
    constexpr bool ONE = !SEVERAL, EARLY = SEVERAL && !GATE;
    static_assert(!(SPLIT && SEVERAL), "a part is a pair's only unit");
    using Cursor = WideCursor<ONE>;
    extern __shared__ __align__(1024) uint8_t smem[];  // (the swizzle pattern follows the address bits)
    uint8_t* sQ = smem;
    uint8_t* sK = sQ + C::Q_BYTES;               // [STAGES]
    uint8_t* sV = sK + C::STAGES * C::K_BYTES;   // [STAGES]
    uint8_t* sOut = sV + C::STAGES * C::V_BYTES;  // output stage
    uint64_t* bars = reinterpret_cast<uint64_t*>(sOut + STAGE_BYTES);
    // [64 head-dim columns] leader: Q and the unit's first K: the first MMAs run while the other columns arrive (96 KB: all of
    // it first, the first scores of a call came 1000 clk later)
    uint64_t* first = bars;
    uint64_t* q_empty = bars + 4;      // both: the tile's last S = Q K^T has completed
    uint64_t* k_full = bars + 5;       // [2] leader: the other K
    uint64_t* k_empty = bars + 7;      // [2] both
    uint64_t* v_full = bars + 9;       // [2] leader
    uint64_t* v_empty = bars + 11;     // [2] both
    uint64_t* s_full = bars + 13;      // [2] both
    uint64_t* p_half = bars + 15;      // [buffer][half] leader: eight warps' probabilities of keys 0-63 / 64-127
    uint64_t* o_full = bars + 19;      // both: one phase per unit
    uint64_t* o_empty = bars + 20;     // leader: eight epilogue warps have read O out
    // [unit & 3] own CTA: the softmax warps have published the unit's row sums.  While the epilogue is still busy with
    // unit n - 1, units n, n + 1 and n + 2 may be through the softmax when they have one key block each (scores are
    // computed one block ahead; the first P V of n + 1 waits for the epilogue of n): with fewer slots a phase could
    // complete twice before the epilogue has looked at it, which a parity wait cannot tell from "not yet".
    uint64_t* fin = bars + 21;
    uint64_t* gate_bar = bars + 25;    // [epilogue warp][buffer] own CTA
    uint64_t* next_full = bars + 33;   // own CTA: the epilogue warps have looked up the next unit's vision blocks
    uint64_t* next_empty = bars + 34;  // the softmax warps have taken them
    uint64_t* gate_late = bars + 35;   // [softmax warp][buffer] own CTA: of the last unit's second half
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + C::NUM_BARS);
    uint32_t* abort_slot = tmem_slot + 1;
    float* fin_vals = reinterpret_cast<float*>(tmem_slot + 4);  // [unit & 3][row] row sum
    WideWork* first_unit = reinterpret_cast<WideWork*>(fin_vals + 4 * 128);
    WideWork* next_place = first_unit + 1;
    int* next_end = reinterpret_cast<int*>(fin_vals + 4 * 128 + 16);  // [row] first key the row does not see
    static_assert(sizeof(WideWork) <= 32, "two units in 64 bytes");

    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);
    const int lane = threadIdx.x & 31;
    const int cta = SPLIT ? (int)cluster_ctarank() : 0;                   // in the cluster, which may hold several pairs
    const int lead = cta & ~1, rank = SPLIT ? cta & 1 : (int)cluster_ctarank();  // the pair's leader; rank in the pair
    const bool leader = rank == 0;

    if (threadIdx.x == 32) {
        prefetch_tensormap(&tm_q);
        prefetch_tensormap(&tm_k);
        prefetch_tensormap(&tm_v);
    }
    if (warp == 0) {  // (a lane a barrier: one thread took them in turn, and what stands in front of the cluster's barrier is on every call's clock)
        for (int i = lane; i < C::NUM_BARS; i += 32) mbar_init(&bars[i], C::arrivals(i));
        fence_mbar_init();
    }
    if (warp == C::PRODUCER_WARP) tmem_alloc_pair(tmem_slot, 512);
    // One warp finds the first unit for all, beside the tensor memory's allocation; its divisions, and the code that every role
    // would fetch for them, took 2500 clk between the kernel's release and its first load.
    constexpr bool blocks_in_memory = MASKED || VISION;
    WideWork w_first{};
    if (warp == C::EPILOGUE_WARP) {
        w_first = wide_place<SPLIT != 0>(p, Cursor(p), rank);
        if (!blocks_in_memory) wide_find_blocks<MASKED, SPLIT != 0, VISION>(p, rank, w_first);
        if (lane == 0) *first_unit = w_first;
    }
    cluster_sync_all();  // both CTAs' barriers exist before anyone arrives on the other's
    // Up to here nothing depends on the kernels in front; everything below may.
    grid_dependency_wait();
    grid_launch_dependents();
    if (threadIdx.x == 0) *abort_slot = *reinterpret_cast<volatile uint32_t*>(p.fault) != 0u ? 1u : 0u;
    // Q and the first K of a unit, 64 head-dim columns after 64; K or V of another block
    auto load_first = [&](const WideWork& w, int st) {
        const uint32_t b_first = map_to_cta(smem_u32(first), lead);
#pragma unroll 1
        for (int c = 0; c < 4; ++c) {
            if (leader && lane == 0) mbar_arrive_expect_tx(&first[c], 2 * (C::Q_CHUNK + C::K_CHUNK));
            __syncwarp();
            tma_load_4d_pair(sQ + c * C::Q_CHUNK, &tm_q, b_first + c * 8, c * 64, w.h, w.q0, w.b);
            tma_load_4d_pair(sK + st * C::K_BYTES + c * C::K_CHUNK, &tm_k, b_first + c * 8, c * 64, w.kvh, w.lo * C::BN + rank * 64, w.b);
        }
    };
    auto load_k = [&](const WideWork& w, int j, int st) {
        const uint32_t b_k = map_to_cta(smem_u32(k_full), lead);
        if (leader && lane == 0) mbar_arrive_expect_tx(&k_full[st], 2 * C::K_BYTES);
        __syncwarp();
#pragma unroll
        for (int c = 0; c < 4; ++c)
            tma_load_4d_pair(sK + st * C::K_BYTES + c * C::K_CHUNK, &tm_k, b_k + st * 8, c * 64, w.kvh, j * C::BN + rank * 64, w.b);
    };
    auto load_v = [&](const WideWork& w, int j, int st) {
        const uint32_t b_v = map_to_cta(smem_u32(v_full), lead);
        if (leader && lane == 0) mbar_arrive_expect_tx(&v_full[st], 2 * C::V_BYTES);
        __syncwarp();
#pragma unroll
        for (int c = 0; c < 2; ++c)
            tma_load_4d_pair(sV + st * C::V_BYTES + c * C::V_CHUNK, &tm_v, b_v + st * 8, rank * 128 + c * 64, w.kvh, j * C::BN, w.b);
    };
    // The first unit's first blocks are asked for before the status word has been looked at (another 500 clk).
    int ahead_k = 0, ahead_v = 0;
    // (The others do not wait for that: issuing takes longer than the status word.)
    static_assert(C::THREADS == 320, "barriers 3 and 4");
    tc_fence_before_sync();
    if (warp == C::PRODUCER_WARP) {
        w_first = *first_unit;
        if (blocks_in_memory) {
            wide_find_blocks<MASKED, SPLIT != 0, VISION>(p, rank, w_first);
            if (lane == 0) *first_unit = w_first;
        }
        __syncwarp();
        asm volatile("bar.arrive 3, 320;" ::: "memory");
        ahead_k = min(w_first.hi - w_first.lo, 2), ahead_v = min(w_first.hi - w_first.lo, 1);
        if (ahead_k > 0) {
            load_first(w_first, 0);
            if (ahead_k > 1) load_k(w_first, w_first.lo + 1, 1);
            load_v(w_first, w_first.lo, 0);
        }
        asm volatile("bar.sync 4, 320;" ::: "memory");
    } else {
        asm volatile("bar.sync 3, 320;" ::: "memory");
        asm volatile("bar.arrive 4, 320;" ::: "memory");
    }
    tc_fence_after_sync();
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, *reinterpret_cast<volatile uint32_t*>(tmem_slot), 0);
    const int total = *abort_slot ? 0 : (int)(blockIdx.x >> 1) < p.few ? p.few_end : p.total_tiles;  // a status is set: walk an empty list
    auto unit_at = [&](const Cursor& cur) {
        if (ONE || cur.i == 0) return *first_unit;
        WideWork w = wide_place<SPLIT != 0>(p, cur, rank);
        wide_find_blocks<MASKED, SPLIT != 0, VISION>(p, rank, w);
        return w;
    };

    // SPLIT 1: columns [col, col + 128) of the part's rows into shared memory, where Q, K and V are through: the f32 tile as
    // [32 columns][row], 128-byte swizzle; and from there, a row of 512 bytes an instruction, to the records.  (By TMA, in
    // boxes of 8 rows x 32 columns, the tile took 4000 clk.)
    constexpr int PART_CHUNK = 128 * 128;
    auto store_part = [&](const WideWork& w, int quarter, float row_l, int col) {
        if (!mbar_wait_warp<2>(o_full, 0)) {
            if (lane == 0) report_fault(p.fault, FAULT_WAIT_O, 0x700u);
            return;
        }
        tc_fence_after_sync();
        const float inv = row_l > 0.f ? 1.0f / row_l : 0.f;
        const uint32_t tO = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + C::COL_O + col;
        const uint32_t tile = smem_u32(smem) + col / 32 * PART_CHUNK, at = tile + (quarter * 32 + lane) * 128;
#pragma unroll 1
        for (int c = 0; c < 4; ++c) {
            uint32_t v[32];
            tmem_ld32(tO + c * 32, v);
            tmem_wait_ld();
#pragma unroll
            for (int i = 0; i < 8; ++i)
                asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(at + c * PART_CHUNK + ((i ^ (lane & 7)) << 4)),
                             "f"(__uint_as_float(v[4 * i]) * inv), "f"(__uint_as_float(v[4 * i + 1]) * inv),
                             "f"(__uint_as_float(v[4 * i + 2]) * inv), "f"(__uint_as_float(v[4 * i + 3]) * inv) : "memory");
        }
        __syncwarp();
        const int end = min(quarter * 32 + 32, p.seq - w.q0);
        const long long step_t = (long long)p.nq * HD;
        float* dst = p.part_o + ((((long long)w.part * p.batch + w.b) * p.seq + w.q0) * p.nq + w.h) * HD + col + lane * 4;
#pragma unroll 1
        for (int i0 = quarter * 32; i0 < end; i0 += 8) {
            float4 v[8];
#pragma unroll
            for (int i = 0; i < 8; ++i)
                v[i] = *reinterpret_cast<const float4*>(smem + (col / 32 + (lane >> 3)) * PART_CHUNK + (i0 + i) * 128 + (((lane & 7) ^ i) << 4));
#pragma unroll
            for (int i = 0; i < 8; ++i)
                if (i0 + i < end) *reinterpret_cast<float4*>(dst + (i0 + i) * step_t) = v[i];
        }
    };

    // SPLIT 2: the parts of a unit divide the columns, 16 at a time, among their CTAs of the same rows: part u finishes the groups
    // [group0(u), group0(u + 1)) of all 128.  A record is [four columns][row], so that a thread, which is a row, stores what the others
    // finish straight from tensor memory and loads what it finishes straight into registers, 512 bytes a warp.
    constexpr int GROUP = 16, GROUPS = HD / GROUP;
    auto group0 = [&](int part) { return part * GROUPS / p.num_splits; };
    auto record_row = [&](const WideWork& w, int part) { return (((long long)part * p.batch + w.b) * p.nq + w.h) * p.seq + w.q0; };
    auto send_part = [&](const WideWork& w, int quarter, float row_l, int half) {  // of columns [128 half, 128 half + 128)
        if (!mbar_wait_warp<2>(o_full, 0)) {
            if (lane == 0) report_fault(p.fault, FAULT_WAIT_O, 0x700u);
            return;
        }
        tc_fence_after_sync();
        const float inv = row_l > 0.f ? 1.0f / row_l : 0.f;
        const uint32_t tO = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + C::COL_O;
        const int g0 = group0(w.part), g1 = group0(w.part + 1), row = quarter * 32 + lane, rows = min(128, p.seq - w.q0);
        float4* dst = reinterpret_cast<float4*>(p.part_o + record_row(w, w.part) * HD) + row;
#pragma unroll 1
        for (int g = half * (GROUPS / 2); g < (half + 1) * (GROUPS / 2); g += 2) {
            const bool first = g < g0 || g >= g1, second = g + 1 < g0 || g + 1 >= g1;  // (a group that another part finishes)
            if (!first && !second) continue;
            uint32_t v[32];
            tmem_ld32(tO + g * GROUP, v);
            tmem_wait_ld();
#pragma unroll
            for (int i = 0; i < 8; ++i)
                if (row < rows && (i < 4 ? first : second))
                    dst[(long long)(g * 4 + i) * rows] = make_float4(__uint_as_float(v[4 * i]) * inv, __uint_as_float(v[4 * i + 1]) * inv, __uint_as_float(v[4 * i + 2]) * inv, __uint_as_float(v[4 * i + 3]) * inv);
        }
    };

    auto store_copies = [&](const OutStage& stage, const uint32_t* words, int n, int col) {  // of this thread's row
        if (stage.t0 + lane >= p.seq) return;
        const long long at = stage.b * p.o_stride_b + (stage.t0 + lane) * p.o_stride_t + (long long)stage.h * HD + col;
        for (int k = 0; k < p.n_copies; ++k) {
            uint4* d4 = reinterpret_cast<uint4*>(reinterpret_cast<uint16_t*>(p.out_copies[k]) + at);
#pragma unroll
            for (int i = 0; i < n / 4; ++i) d4[i] = make_uint4(words[4 * i], words[4 * i + 1], words[4 * i + 2], words[4 * i + 3]);
        }
    };
    // The stage's columns of the warp's 32 rows, which begin at tO, in turns of 32.  (Gated, of which a turn of 16 took 690 clk, 1200 so.
    // us: 1300 tokens of 24/4 heads 33.6 -> 31.5, 2000 57.5 -> 54, 4 x 1500, window 300, 106 -> 97; cold, 200 x 333 of 8/4, 14.4 -> 13.3.)
    // frees: the accumulator may be overwritten behind the last of them.
    auto write_turns = [&](OutStage& stage, uint32_t tO, float inv, bool warp_store, bool frees) -> bool {
        constexpr int SC = 32;
        const int turns = stage.rounds * (64 / SC);
        uint32_t wa[SC], w8[SC / 2];
        tmem_ld(tO, wa);
#pragma unroll 1
        for (int c = 0; c < turns; ++c) {
            if (warp_store && !stage_before<GATE, SC>(stage, &tm_gate, lane, c)) {
                if (lane == 0) report_fault(p.fault, FAULT_WAIT_FULL, 0x600u);
                return false;
            }
            tmem_wait_ld();
            if (frees && c + 1 == turns) {  // O is in registers
                tc_fence_before_sync();
                mbar_arrive_remote_warp(map_to_cta(smem_u32(o_empty), lead));
            }
            auto next = [&]() {
                if (c + 1 < turns) tmem_ld(tO + (c + 1) * SC, wa);
            };
            if (!warp_store) next();
            if (warp_store) {
                stage_turn<GATE>(stage, &tm_out, lane, c, wa, inv, w8, next);
                store_copies(stage, w8, SC / 2, stage.col0 + c * SC);
            }
        }
        return true;
    };

    if (warp == C::PRODUCER_WARP) {
        // ------------------------------------------------------------------ TMA producer
        if (total == 0 && leader && ahead_k > 0) {  // (what has been asked for lands before the CTAs go)
            for (int c = 0; c < 4; ++c) mbar_wait_inline(&first[c], 0);
            if (ahead_k > 1) mbar_wait_inline(&k_full[1], 0);
            mbar_wait_inline(&v_full[0], 0);
        }
        int gk = 0, gv = 0, n = 0;  // K blocks, V blocks and units loaded so far
        bool ok = true;
        auto free_stage = [&](uint64_t* empty, int g) {
            if (g < 2 || mbar_wait_inline(&empty[g & 1], ((g >> 1) - 1) & 1)) return true;
            if (lane == 0) report_fault(p.fault, FAULT_WAIT_EMPTY, 0x100u);
            return false;
        };
        // (vision blocks: the next unit's are looked up while this one's first blocks are worked on)
        Cursor cur(p);
        WideWork w_next{};
        auto look_ahead = [&]() {
            Cursor after = cur;
            after.advance(p);
            if (after.w < total) w_next = unit_at(after);
        };
        for (; ok && cur.w < total; cur.advance(p)) {
            const WideWork w = VISION && cur.i > 0 ? w_next : unit_at(cur);
            if (w.hi == w.lo) {
                if (VISION) look_ahead();
                continue;
            }
            const int have = n == 0 && cur.i == 0 ? ahead_k : 0;  // (asked for above)
            if (have) {
                gk = ahead_k, gv = ahead_v;
            } else {
                if (n > 0 && !mbar_wait_inline(q_empty, (n - 1) & 1)) {
                    if (lane == 0) report_fault(p.fault, FAULT_WAIT_EMPTY, 0x300u);
                    break;
                }
                ok = free_stage(k_empty, gk);
                if (ok) load_first(w, gk++ & 1);
            }
            ++n;
            // in the order of use: K one block ahead of V
            for (int j = w.lo; ok && j < w.hi; ++j) {
                if (have && j == w.lo) {  // (V of the first block, K of the second)
                    if (VISION) look_ahead();
                    continue;
                }
                if (j + 1 < w.hi) {
                    ok = free_stage(k_empty, gk);
                    if (ok) load_k(w, j + 1, gk++ & 1);
                }
                if (ok) ok = free_stage(v_empty, gv);
                if (ok) load_v(w, j, gv++ & 1);
                if (VISION && j == w.lo) look_ahead();
            }
        }
    } else if (warp == C::ISSUER_WARP) {
        // ------------------------------------------------------------------ MMA issuer (for both CTAs)
        if (leader) {
            constexpr uint32_t IDESC_QK = make_idesc_bf16(256, 128, false);
            constexpr uint32_t IDESC_PV = make_idesc_bf16(256, 256, true);
            const uint64_t dQ = make_smem_desc_sw128(smem_u32(sQ), 16, 1024);
            const uint64_t dK = make_smem_desc_sw128(smem_u32(sK), 16, 1024);
            const uint64_t dV = make_smem_desc_sw128(smem_u32(sV), C::V_CHUNK, 1024);
            int gs = 0, gp = 0, nq = 0, no = 0;  // score blocks, P V blocks issued; units whose scores / P V have begun
            uint32_t k_par = 0u;                 // bit st: parity of the stage's k_full
            bool ok = true;
            // S(gs) of the unit's block j
            auto scores = [&](const WideWork& w, int j) -> bool {
                const int st = gs & 1;
                uint64_t da = dQ, db = dK + (uint64_t)(st * (C::K_BYTES >> 4));
                uint32_t acc = 0u;
                auto chunk = [&]() {  // 64 head-dim columns
                    umma_pair_ss_x4<2, 2>(tmem_base + C::COL_S + st * 128, da, db, IDESC_QK, acc);
                    da += C::Q_CHUNK >> 4, db += C::K_CHUNK >> 4, acc = 1u;
                };
                if (j == w.lo) {
#pragma unroll 1
                    for (int c = 0; c < 4; ++c) {
                        if (!mbar_wait_inline(&first[c], nq & 1)) {
                            if (lane == 0) report_fault(p.fault, FAULT_WAIT_Q, nq);
                            return false;
                        }
                        tc_fence_after_sync();
                        chunk();
                    }
                    ++nq;
                } else {
                    if (!mbar_wait_inline(&k_full[st], (k_par >> st) & 1u)) {
                        if (lane == 0) report_fault(p.fault, FAULT_WAIT_K, gs);
                        return false;
                    }
                    k_par ^= 1u << st;
                    tc_fence_after_sync();
#pragma unroll 1
                    for (int c = 0; c < 4; ++c) chunk();
                }
                umma_commit_pair(&s_full[st], lead);
                umma_commit_pair(&k_empty[st], lead);
                if (j + 1 == w.hi) umma_commit_pair(q_empty, lead);
                ++gs;
                return true;
            };
            Cursor cur(p);
            auto next_unit = [&](WideWork& w) -> bool {  // the cursor's unit, or the first one after it with key blocks
                for (; cur.w < total; cur.advance(p)) {
                    w = unit_at(cur);
                    if (w.hi > w.lo) {
                        cur.advance(p);
                        return true;
                    }
                }
                return false;
            };
            WideWork w{}, wn{};
            bool have = next_unit(w);
            if (have) ok = scores(w, w.lo);
            while (have && ok) {
                bool have_next = false;
                for (int j = w.lo; j < w.hi; ++j) {
                    // the next block's scores first: they run while the softmax warps work on this block's
                    if (j + 1 < w.hi) ok = scores(w, j + 1);
                    if (j == w.lo) have_next = next_unit(wn);
                    if (ok && j + 1 == w.hi && have_next) ok = scores(wn, wn.lo);
                    if (!ok) break;
                    const int st = gp & 1;
                    const uint32_t par = (gp >> 1) & 1;
                    if (!mbar_wait_inline(&v_full[st], par)) {
                        if (lane == 0) report_fault(p.fault, FAULT_WAIT_V, gp);
                        ok = false;
                        break;
                    }
                    if (j == w.lo) {
                        if (no > 0 && !mbar_wait_inline(o_empty, (no - 1) & 1)) {
                            if (lane == 0) report_fault(p.fault, FAULT_WAIT_O, 0x100u + no);
                            ok = false;
                            break;
                        }
                        ++no;
                    }
                    // P from tensor memory, 16 keys = 8 columns; V MN-major, 64-column chunks 16 KB apart, 16 keys =
                    // 2048 bytes; the first 64 keys while the softmax warps still exponentiate the other 64
                    uint32_t tP = tmem_base + C::COL_S + st * 128, acc = j > w.lo ? 1u : 0u;
                    uint64_t dv = dV + (uint64_t)(st * (C::V_BYTES >> 4));
#pragma unroll 1
                    for (int half = 0; half < 2; ++half, tP += 32, dv += 512, acc = 1u) {
                        if (!mbar_wait_inline(&p_half[2 * st + half], par)) {
                            if (lane == 0) report_fault(p.fault, FAULT_WAIT_P, gp);
                            ok = false;
                            break;
                        }
                        tc_fence_after_sync();
                        umma_pair_ts_x4<8, 128>(tmem_base + C::COL_O, tP, dv, IDESC_PV, acc);
                    }
                    if (!ok) break;
                    if (j + 1 == w.hi) umma_commit_pair(o_full, lead);
                    umma_commit_pair(&v_empty[st], lead);
                    ++gp;
                }
                w = wn;
                have = have_next;
            }
        }
    } else if (warp >= C::EPILOGUE_WARP) {
        // ------------------------------------------------------------------ epilogue: thread = query row
        const int quarter = warp & 3;
        const int r = quarter * 32 + lane;
        const uint32_t tO = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + C::COL_O;
        [[maybe_unused]] const uint32_t b_empty = map_to_cta(smem_u32(o_empty), lead);
        int n = 0;  // units with key blocks so far
        OutStage stage{sOut + quarter * STAGE_WARP_BYTES, &gate_bar[2 * quarter], 0u, 0, 0, 0, 0, HD / 64};
        Cursor cur(p);
        for (; cur.w < total; cur.advance(p)) {
            const WideWork w = unit_at(cur);
            if (VISION) {  // for the softmax warps, whose look-up would come between two units
                Cursor after = cur;
                after.advance(p);
                if (after.w < total) {
                    const WideWork wn = unit_at(after);
                    const int tn = wn.q0 + quarter * 32 + lane, end = vision_ends(p, tn + p.kv_len - p.seq, tn < p.seq);
                    if (cur.i > 0 && !mbar_wait_warp<2>(next_empty, (cur.i - 1) & 1)) {
                        if (lane == 0) report_fault(p.fault, FAULT_WAIT_EMPTY, 0x500u);
                        break;
                    }
                    next_end[r] = end;
                    if (threadIdx.x == C::EPILOGUE_WARP * 32) *next_place = wn;
                    mbar_arrive_warp(next_full);
                }
            }
            const int t0 = w.q0 + quarter * 32, t = t0 + lane;
            const bool store = t < p.seq, warp_store = t0 < p.seq;  // this row / some row of the warp is stored
            const long long row = ((long long)w.b * p.seq + t) * p.nq + w.h;
            const long long eoff = w.b * p.o_stride_b + t * p.o_stride_t + (long long)w.h * HD;
            if (w.hi == w.lo) {  // nothing visible for the pair: zero output
                if (SPLIT) {
                    if (store) p.part_lse[SPLIT == 2 ? record_row(w, w.part) + quarter * 32 + lane : (long long)w.part * p.batch * p.seq * p.nq + row] = -CUDART_INF_F;
                } else if (store) {
                    for (int c = -1; c < p.n_copies; ++c) {
                        uint4* dst = reinterpret_cast<uint4*>((c < 0 ? p.out : reinterpret_cast<uint16_t*>(p.out_copies[c])) + eoff);
                        for (int i = 0; i < HD / 8; ++i) dst[i] = make_uint4(0u, 0u, 0u, 0u);
                    }
                    if (p.out_lse) p.out_lse[row] = -CUDART_INF_F;
                }
                continue;
            }
            // GATE: the softmax warps take the second half of the last unit's columns: four warps alone wrote them in 12000 clk.  (us: 1000
            // tokens of 16/8 heads 20.2 -> 18.7, 2000 of 8/2 28.9 -> 27.2, 64 10.1 -> 8.4.)
            bool last = false;
            if (GATE && !SPLIT) {
                Cursor after = cur;
                after.advance(p);
                last = after.w >= total;
                stage.rounds = last ? HD / 128 : HD / 64;
            }
            if (!SPLIT && warp_store) stage_open<GATE>(stage, &tm_gate, lane, w.h, t0, w.b);
            if (!mbar_wait_warp<2>(&fin[n & 3], (n >> 2) & 1)) {
                if (lane == 0) report_fault(p.fault, FAULT_WAIT_FULL, 0x500u);
                break;
            }
            const float row_l = fin_vals[(n & 3) * 128 + r];
            if constexpr (SPLIT != 0) {
                if constexpr (SPLIT == 1) store_part(w, quarter, row_l, 0);
                else send_part(w, quarter, row_l, 0);
                break;
            }
            if (!mbar_wait_warp<2>(o_full, n & 1)) {
                if (lane == 0) report_fault(p.fault, FAULT_WAIT_O, n);
                break;
            }
            tc_fence_after_sync();
            ++n;
            const float inv = row_l > 0.f ? 1.0f / row_l : 0.f;
            bool ok = true;
            if constexpr (EARLY) {
                // The whole row into registers as bf16 pairs, so that the next unit may overwrite the accumulator before the last
                // columns have left the SM.
                uint32_t pk[HD / 2], va[32], vb[32];
                const uint64_t inv2 = pack_f32x2(inv, inv);
                auto take = [&](const uint32_t (&v)[32], uint32_t* to) {
#pragma unroll
                    for (int u = 0; u < 16; ++u) {
                        float x0, x1;
                        unpack_f32x2(mul_f32x2(pack_f32x2(__uint_as_float(v[2 * u]), __uint_as_float(v[2 * u + 1])), inv2), x0, x1);
                        to[u] = pack_bf16x2(x0, x1);
                    }
                };
                tmem_ld32(tO, va);
#pragma unroll
                for (int c = 0; c < HD / 32; c += 2) {
                    tmem_wait_ld();
                    tmem_ld32(tO + (c + 1) * 32, vb);
                    take(va, pk + c * 16);
                    tmem_wait_ld();
                    if (c + 2 < HD / 32) tmem_ld32(tO + (c + 2) * 32, va);
                    take(vb, pk + (c + 1) * 16);
                }
                tc_fence_before_sync();
                mbar_arrive_remote_warp(b_empty);
                if (warp_store) {
                    const uint32_t at = smem_u32(stage.buf) + lane * 128;
#pragma unroll
                    for (int c = 0; c < HD / 64; ++c) {
                        stage_before<false>(stage, &tm_gate, lane, 2 * c);
#pragma unroll
                        for (int i = 0; i < 8; ++i)
                            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"((at + (c & 1) * 4096) + ((i ^ (lane & 7)) << 4)),
                                         "r"(pk[c * 32 + 4 * i]), "r"(pk[c * 32 + 4 * i + 1]), "r"(pk[c * 32 + 4 * i + 2]), "r"(pk[c * 32 + 4 * i + 3]) : "memory");
                        stage_send(stage, &tm_out, lane, c);
                    }
                    store_copies(stage, pk, HD / 2, 0);
                }
            } else {
                ok = write_turns(stage, tO, inv, warp_store, !last);
            }
            if (!ok) break;
        }
        if (!SPLIT && lane == 0) bulk_wait_read<0>();  // the stage may go when its last rows have been read
    } else {
        // ------------------------------------------------------------------ softmax: thread = query row
        const int quarter = warp & 3;
        const int r = quarter * 32 + lane;
        const uint32_t lane_sel = static_cast<uint32_t>(quarter * 32) << 16;
        const uint32_t tO = tmem_base + lane_sel + C::COL_O;
        const uint32_t b_half = map_to_cta(smem_u32(p_half), lead);
        const float sl = p.scale_log2;
        const uint64_t sl2 = pack_f32x2(sl, sl);
        const bool causal = (p.mask_type == 3);
        const bool windowed = causal && p.window > 0 && p.window != 0x7fffffff;
        const int off = p.kv_len - p.seq;
        int g = 0, n = 0;  // key blocks and units so far
        bool ok = true;
        uint32_t s0[32], s1[32], s2[32], s3[32];  // the row's 128 scores of the current block
        Cursor cur(p);
        for (; ok && cur.w < total; cur.advance(p)) {
            const bool looked_up = VISION && cur.i > 0;
            int row_end = 0;
            if (looked_up) {
                if (!mbar_wait_inline(next_full, (cur.i - 1) & 1)) {
                    if (lane == 0) report_fault(p.fault, FAULT_WAIT_FULL, 0x700u);
                    break;
                }
                row_end = next_end[r];
            }
            const WideWork w = looked_up ? *next_place : unit_at(cur);
            if (looked_up) mbar_arrive_warp(next_empty);
            if (w.hi == w.lo) {
                if (SPLIT) break;  // (its only one; its place is read again below, not kept through the blocks: a canvas step 17.9 us, 17.6 so)
                continue;
            }
            const int t = w.q0 + r;
            int row_lo = 0, row_hi = p.kv_len;  // visible keys [row_lo, row_hi)
            if (causal) {
                const int diag = t + off;
                row_hi = min(max(diag + 1, 0), p.kv_len);
                if (VISION) row_hi = looked_up ? row_end : vision_ends(p, diag, t < p.seq);
                if (windowed) row_lo = max(0, diag - p.window + 1);
                if (row_lo > row_hi) row_lo = row_hi;
            }
            const RowMask rm{row_lo, row_hi};
            float m = -CUDART_INF_F;  // running max, log2 domain, possibly stale by <= 8
            float l = 0.f;            // row sum
            // (MASKED: a block's class is asked for a block ahead, its bits before its scores are waited for)
            auto class_of = [&](int j) -> uint32_t {
                return MASKED && w.q0 < p.seq && j < w.hi
                           ? reinterpret_cast<const uint8_t*>(p.mask_class + (long long)(w.q0 >> 7) * p.mask_blocks + j)[quarter]
                           : 0u;
            };
            uint32_t cls = class_of(w.lo);
            for (int j = w.lo; j < w.hi; ++j, ++g) {
                const uint32_t next_cls = class_of(j + 1);
                const bool by_bits = (cls & (MASK_HIDDEN | MASK_VALUES)) == MASK_HIDDEN;
                uint4 bits = make_uint4(0u, 0u, 0u, 0u);
                if (MASKED && by_bits) bits = p.mask_bits[((long long)(w.q0 >> 7) * p.mask_blocks + j) * 128 + r];
                const int kc = j * C::BN, st = g & 1;
                const uint32_t tS = tmem_base + lane_sel + C::COL_S + st * 128;
                if (!mbar_wait_inline(&s_full[st], (g >> 1) & 1)) {
                    if (lane == 0) report_fault(p.fault, FAULT_WAIT_S, g);
                    ok = false;
                    break;
                }
                tc_fence_after_sync();
                float bl = sl;  // what the block's scores are scaled by
                uint64_t bl2 = sl2;
                if (MASKED && (cls & MASK_VALUES)) {
                    add_mask_values(tS, p.mask, t, p.seq, kc, p.kv_len, sl);
                    bl = 1.0f, bl2 = pack_f32x2(1.0f, 1.0f);
                }
                tmem_ld32(tS, s0);
                tmem_ld32(tS + 32, s1);
                tmem_ld32(tS + 64, s2);
                tmem_ld32(tS + 96, s3);
                tmem_wait_ld();
                if constexpr (MASKED) {
                    if (by_bits) {
                        select_chunk(s0, bits.x);
                        select_chunk(s1, bits.y);
                        select_chunk(s2, bits.z);
                        select_chunk(s3, bits.w);
                    }
                } else if (!__all_sync(0xffffffffu, rm.lo <= kc && kc + C::BN <= rm.hi)) {  // window edge, diagonal, ragged end
                    mask_chunk(s0, kc, rm);
                    mask_chunk(s1, kc + 32, rm);
                    mask_chunk(s2, kc + 64, rm);
                    mask_chunk(s3, kc + 96, rm);
                }
                float mr[4] = {-CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F};
                chunk_max(s0, mr);
                chunk_max(s1, mr);
                chunk_max(s2, mr);
                chunk_max(s3, mr);
                const float top = fmaxf(fmaxf(mr[0], mr[1]), fmaxf(mr[2], mr[3]));
                const float m_new = fmaxf(m, top * bl);
                if (j == w.lo) {
                    m = m_new;
                } else if (__any_sync(0xffffffffu, m_new > m + 8.0f)) {
                    // Rare: some row's maximum grows by more than 2^8.  Once O += P V of the previous block has landed
                    // (it releases its V stage), rescale those rows of O in tensor memory.
                    const bool need = m_new > m + 8.0f;
                    const float alpha = need ? fast_exp2(m - m_new) : 1.0f;
                    if (!mbar_wait_inline(&v_empty[st ^ 1], ((g - 1) >> 1) & 1)) {
                        if (lane == 0) report_fault(p.fault, FAULT_WAIT_O, 0x200u + g);
                        ok = false;
                        break;
                    }
                    tc_fence_after_sync();
#pragma unroll 1
                    for (int c = 0; c < HD; c += 16) {
                        uint32_t ww[16];
                        tmem_ld16(tO + c, ww);
                        tmem_wait_ld();
#pragma unroll
                        for (int e = 0; e < 16; ++e) ww[e] = __float_as_uint(__uint_as_float(ww[e]) * alpha);
                        tmem_st16(tO + c, ww);
                    }
                    tmem_wait_st();
                    l *= alpha;
                    if (need) m = m_new;
                }
                // Probabilities as bf16, packed over the first 64 of the block's score columns; row sum in fp32.
                // The first 64 keys are announced a chunk late: their stores have landed by then.
                const float m_eff = (m == -CUDART_INF_F) ? 0.f : m;
                const uint64_t nm2 = pack_f32x2(-m_eff, -m_eff);
                uint64_t ls2[2] = {0ull, 0ull};
                // The sum takes the block's largest probability as the second MMA will see it, rounded to bf16: a row that
                // one key dominates would otherwise be off by that rounding whenever m is stale (2^-9, as much as the output's own).
                const float p_top = fast_exp2(fmaf(top, bl, -m_eff));
                l += bf16_round(p_top) - p_top;
                uint32_t pk[16];
                exp_chunk(s0, pk, ls2, bl2, nm2);
                tmem_st16(tS, pk);
                exp_chunk(s1, pk, ls2, bl2, nm2);
                tmem_st16(tS + 16, pk);
                exp_chunk(s2, pk, ls2, bl2, nm2);
                tmem_wait_st();
                tc_fence_before_sync();
                mbar_arrive_remote_warp(b_half + 16 * st);
                tmem_st16(tS + 32, pk);
                exp_chunk(s3, pk, ls2, bl2, nm2);
                tmem_st16(tS + 48, pk);
                cls = next_cls;
                float l0, l1, l2, l3;
                unpack_f32x2(ls2[0], l0, l1);
                unpack_f32x2(ls2[1], l2, l3);
                l += (l0 + l1) + (l2 + l3);
                tmem_wait_st();
                tc_fence_before_sync();
                mbar_arrive_remote_warp(b_half + 16 * st + 8);
            }
            if (ok) {
                fin_vals[(n & 3) * 128 + r] = l;
                // (SPLIT: the place in the output is read again, not kept in registers through the blocks)
                const WideWork u = SPLIT ? *first_unit : w;
                float* lse = SPLIT == 1 ? p.part_lse + (long long)u.part * p.batch * p.seq * p.nq : SPLIT == 2 ? p.part_lse : p.out_lse;
                if (lse && u.q0 + r < p.seq)
                    lse[SPLIT == 2 ? record_row(u, u.part) + r : ((long long)u.b * p.seq + u.q0 + r) * p.nq + u.h] = l > 0.f ? (m + fast_log2(l)) * 0.6931471805599453f : -CUDART_INF_F;
                mbar_arrive_warp(&fin[n & 3]);
                ++n;
                if constexpr (GATE && SPLIT == 0) {
                    Cursor after = cur;
                    after.advance(p);
                    if (after.w >= total) {  // (in what was Q's shared memory)
                        OutStage half{smem + quarter * STAGE_WARP_BYTES, &gate_late[2 * quarter], 0u, 0, 0, 0, HD / 2, HD / 128};
                        const int t0 = w.q0 + quarter * 32;
                        // The unit's last P V has landed: by the V stage that it releases, not by o_full.  A wait on a parity tells two
                        // states of a barrier apart.  Of the stage's these two are left, open or released by this block: the block
                        // before the previous one, which had the stage before, released it ahead of this block's scores, whose MMAs
                        // came behind its P V.  o_full, a phase a unit, may be in three: the unit before still open (a short unit's
                        // scores run ahead of it), or done, or this one done as well, which looks like the first: a wait for the unit
                        // before, and then for this one, ran out where this warp came to it late.
                        if (!mbar_wait_inline(&v_empty[(g - 1) & 1], ((g - 1) >> 1) & 1)) {
                            if (lane == 0) report_fault(p.fault, FAULT_WAIT_O, 0x800u);
                            break;
                        }
                        tc_fence_after_sync();
                        if (t0 < p.seq) stage_open<GATE>(half, &tm_gate, lane, w.h, t0, w.b);
                        write_turns(half, tO + HD / 2, l > 0.f ? 1.0f / l : 0.f, t0 < p.seq, false);
                        if (lane == 0) bulk_wait_read<0>();
                        break;
                    }
                }
                if constexpr (SPLIT != 0) {
                    if constexpr (SPLIT == 1) store_part(*first_unit, quarter, l, HD / 2);
                    else send_part(*first_unit, quarter, l, 1);
                    break;
                }
            }
        }
    }

    __syncwarp();
    tc_fence_before_sync();
    __syncthreads();
    cluster_sync_all();  // neither CTA's barriers or tensor memory go before the other is through with them
    if constexpr (SPLIT == 2) {
        // Every part's records are there; a warp finishes its half of the CTA's columns of 32 rows.
        auto finish = [&](auto parts_tag) {
            constexpr int PARTS = decltype(parts_tag)::value, TAKES = PARTS == 4 ? 2 : PARTS == 3 ? 3 : 4;  // groups a warp takes at most
            const WideWork w = *first_unit;
            const int row = (warp & 3) * 32 + lane, rows = min(128, p.seq - w.q0);
            const bool live = row < rows;
            const int g0 = group0(w.part), g1 = group0(w.part + 1), mid = (g0 + g1 + 1) / 2;
            const int my_first = warp < C::EPILOGUE_WARP ? mid : g0, my_count = (warp < C::EPILOGUE_WARP ? g1 : mid) - my_first;  // groups
            // the others' values, all at once, and the parts' log-sum-exps
            float4 t[PARTS - 1][TAKES][4];
            float weight[PARTS], mx = -CUDART_INF_F, z = 0.f;
            auto other = [&](int s) { return w.part + s < PARTS ? w.part + s : w.part + s - PARTS; };
#pragma unroll
            for (int s = 1; s < PARTS; ++s) {
                const float4* src = reinterpret_cast<const float4*>(p.part_o + record_row(w, other(s)) * HD) + (long long)my_first * 4 * rows + row;
#pragma unroll
                for (int k = 0; k < TAKES; ++k)
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        if (live && k < my_count) t[s - 1][k][i] = __ldcg(src + (k * 4 + i) * rows);
            }
#pragma unroll
            for (int s = 0; s < PARTS; ++s) {  // (of this part first)
                weight[s] = live ? __ldcg(p.part_lse + record_row(w, other(s)) + row) : -CUDART_INF_F;
                mx = fmaxf(mx, weight[s]);
            }
#pragma unroll
            for (int s = 0; s < PARTS; ++s) {
                weight[s] = mx == -CUDART_INF_F ? 0.f : __expf(weight[s] - mx);
                z += weight[s];
            }
            if (p.out_lse && live && my_first == 0)
                p.out_lse[((long long)w.b * p.seq + w.q0 + row) * p.nq + w.h] = z > 0.f ? mx + __logf(z) : -CUDART_INF_F;
            const float iz = z > 0.f ? 1.0f / z : 0.f, row_l = fin_vals[row];
            const float own = row_l > 0.f ? weight[0] * iz / row_l : 0.f;
            // A group at a time: this part's columns as they are, out of tensor memory, and the others' on top.  (One group ahead: all
            // of them held beside the others' values, and through the barrier, made the kernel spill.)  Out through shared memory
            // (Q, K and V are through), so that a store writes whole rows of the warp's columns: a thread's own 16 bytes at a time
            // took 1800 clk.
            constexpr int PITCH = TAKES * GROUP * 2 + 16;
            const uint32_t tile = smem_u32(smem) + warp * 32 * PITCH;
            const long long eoff = w.b * p.o_stride_b + w.q0 * p.o_stride_t + (long long)w.h * HD + my_first * GROUP;
            const uint32_t tO = tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16) + C::COL_O + my_first * GROUP;
            const bool any = w.hi > w.lo;
            uint32_t mine[2][GROUP];
            if (any && my_count > 0) tmem_ld16(tO, mine[0]);
#pragma unroll
            for (int k = 0; k < TAKES; ++k) {
                tmem_wait_ld();
                if (any && k + 1 < my_count) tmem_ld16(tO + (k + 1) * GROUP, mine[(k + 1) & 1]);
                float acc[GROUP];
#pragma unroll
                for (int e = 0; e < GROUP; ++e) acc[e] = own > 0.f ? __uint_as_float(mine[k & 1][e]) * own : 0.f;  // (an empty part's columns may hold anything)
#pragma unroll
                for (int s = 1; s < PARTS; ++s) {
                    const float e = weight[s] * iz;
                    if (e > 0.f) {  // (an empty part's record may hold anything)
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const float4 v = t[s - 1][k][i];
                            acc[4 * i] = fmaf(e, v.x, acc[4 * i]), acc[4 * i + 1] = fmaf(e, v.y, acc[4 * i + 1]);
                            acc[4 * i + 2] = fmaf(e, v.z, acc[4 * i + 2]), acc[4 * i + 3] = fmaf(e, v.w, acc[4 * i + 3]);
                        }
                    }
                }
                uint32_t o[GROUP / 2];
#pragma unroll
                for (int i = 0; i < GROUP / 2; ++i) o[i] = pack_bf16x2(acc[2 * i], acc[2 * i + 1]);
#pragma unroll
                for (int i = 0; i < 2; ++i)
                    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(tile + lane * PITCH + k * 32 + i * 16), "r"(o[4 * i]), "r"(o[4 * i + 1]), "r"(o[4 * i + 2]), "r"(o[4 * i + 3]) : "memory");
            }
            const int per_row = 2 * my_count, magic = (65536 + per_row - 1) / per_row;  // 16-byte pieces of a row (exact for the 256 there are at most)
            const int end = min(32, rows - (warp & 3) * 32);
            auto place_of = [&](int i, int& r, int& c) {  // piece i of the warp's: row, piece of the row; whether there is one
                r = i * magic >> 16, c = i - r * per_row;
                return i < 32 * per_row && r < end;
            };
            [[maybe_unused]] uint4 gate[GATE ? 2 * TAKES : 1];  // all asked for at once
            if constexpr (GATE) {
#pragma unroll
                for (int k = 0; k < 2 * TAKES; ++k) {
                    int r, c;
                    if (place_of(k * 32 + lane, r, c)) gate[k] = *reinterpret_cast<const uint4*>(p.gate + eoff + ((warp & 3) * 32 + r) * p.o_stride_t + c * 8);
                }
            }
            __syncwarp();
#pragma unroll GATE ? 2 * TAKES : 1
            for (int k = 0; k < 2 * TAKES; ++k) {
                int r, c;
                if (!place_of(k * 32 + lane, r, c)) break;
                uint32_t v[4];
                asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(tile + r * PITCH + c * 16));
                if constexpr (GATE) {
                    const uint32_t g[4] = {gate[k].x, gate[k].y, gate[k].z, gate[k].w};
#pragma unroll
                    for (int i = 0; i < 4; ++i)  // bf16(attention) * sigmoid(gate): the rounding order of the two-launch form
                        v[i] = pack_bf16x2(__uint_as_float(v[i] << 16) * sigmoid(__uint_as_float(g[i] << 16)),
                                           __uint_as_float(v[i] & 0xffff0000u) * sigmoid(__uint_as_float(g[i] & 0xffff0000u)));
                }
                const long long at = eoff + ((warp & 3) * 32 + r) * p.o_stride_t + c * 8;
                *reinterpret_cast<uint4*>(p.out + at) = make_uint4(v[0], v[1], v[2], v[3]);
                for (int n = 0; n < p.n_copies; ++n) *reinterpret_cast<uint4*>(reinterpret_cast<uint16_t*>(p.out_copies[n]) + at) = make_uint4(v[0], v[1], v[2], v[3]);
            }
        };
        static_assert(C::MOST_FOLDED == 4, "two to four parts");
        if (warp < C::PRODUCER_WARP && total > 0) {
            if (p.num_splits == 4) finish(std::integral_constant<int, 4>{});
            else if (p.num_splits == 3) finish(std::integral_constant<int, 3>{});
            else finish(std::integral_constant<int, 2>{});
        }
    }
    if (warp == C::PRODUCER_WARP) tmem_dealloc_pair(tmem_base, 512);
}

}  // namespace arc
