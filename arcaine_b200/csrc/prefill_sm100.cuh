// GQA flash-attention prefill kernel for sm_100a, one query tile at a time per CTA: head dim 256 with an additive mask, for
// calls without a workspace for what mask_scan_kernel would read out of it and for parts of a key range that a caller
// asks for (prefill_wide_sm100.cuh does the rest of head dim 256, prefill_pair_sm100.cuh and prefill_chains_sm100.cuh head
// dim 128); and what all prefill kernels share.
//
// One CTA owns a tile of 128 query tokens of one query head and walks all key
// blocks (128 keys).  Q, K and V tiles are staged in shared
// memory by TMA (128-byte swizzle, one 64-element column chunk per copy);
// S = Q K^T and O += P V run on the tcgen05 tensor cores with both accumulators
// in tensor memory; P is written back to tensor memory as bf16 over the S
// columns and fed to the second MMA from there, so probabilities never touch
// shared or global memory.  Softmax is online, fp32.
//
// Warp roles: eight softmax / correction / epilogue warps, two threads per query row
// (warp index mod 4 selects the 32 TMEM lanes, warp index / 4 the 64-key half of each
// block), then one TMA producer warp (also the TMEM owner) and one MMA issuing warp.
//
// Masking in the other kernels follows the reference's rules evaluated inline instead of through a
// (q_len, kv_len) f32 buffer: causal aligned bottom-right with an optional
// window of the W most recent keys, self included
// (src/common/kernels/attention_mask.hpp:12-38); no mask for the bidirectional
// canvas-over-prompt call (src/modeling/diffusion_gemma/attention.cpp:1093-1103).
// Key blocks wholly outside a
// tile's visible band are never loaded (the band idea of gqa_attention,
// src/modeling/diffusion_gemma/attention.cpp:721-769, per CTA).
#pragma once
#include <cuda.h>
#include <math_constants.h>

#include "ptx.cuh"

namespace arc {

struct PrefillParams {
    uint16_t* out;
    const unsigned long long* out_copies;  // n_copies more output buffers (other GPUs' over NVLink), same offsets
    int n_copies;
    const uint16_t* gate;
    const float* mask;
    float* out_lse;
    float* part_o;
    float* part_lse;
    uint32_t* fault;
    int batch, seq, kv_len, nq, nkv;
    long long o_stride_b, o_stride_t;
    float scale_log2;  // scale * log2(e)
    int mask_type, window;
    int num_splits;
    int q_tiles;      // ceil(seq / 128)
    int total_tiles;  // q_tiles * cur_heads * batch * num_splits, dealt round-robin to the persistent CTAs
    int cur_heads;    // head units the tile list walks: nq, or nq / 2 when a CTA takes two query heads at a time
    int head_pair;    // prefill_pair_sm100.cuh: 1 = the CTA's two tiles are the same tokens of two heads of one KV group
    int group;        // nq / nkv
    int group_shift;  // log2(group) if it is a power of two, else -1
    // >= 0 (prefill_chains_sm100.cuh): the launch covers the tail of a two-tile launch's unit list — tile w is head (w & 1)
    // of the head pair with unit index tail_base + (w >> 1), one tile per CTA; -1: the plain tile list
    int tail_base;
    int long_first;  // units in order of falling length
    int step[3];     // digits of the grid's size in the tile list (TileCursor)
    int few, few_end;  // CTA pairs that share the longest units [0, few_end) (WideCursor)
    // The additive mask as mask_scan_kernel has read it (prefill_wide_sm100.cuh; mask_blocks key blocks per row tile)
    const uint32_t* mask_class;  // [row tile][key block]: a byte per 32 rows, MASK_* bits
    const uint4* mask_bits;      // [row tile][key block][row]: one bit per key, set where the mask is 0
    int mask_blocks;
    const int* ids;  // vision-block ids, ids[j] that of key j
};

// A row's visible keys [lo, hi).
struct RowMask {
    int lo, hi;
};

__device__ __forceinline__ float max3f(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// Maximum of one 32-column chunk, folded into four independent running maxima.
__device__ __forceinline__ void chunk_max(const uint32_t (&v)[32], float (&mx)[4]) {
#pragma unroll
    for (int e = 0; e < 32; e += 8)
#pragma unroll
        for (int u = 0; u < 4; ++u) mx[u] = max3f(mx[u], __uint_as_float(v[e + 2 * u]), __uint_as_float(v[e + 2 * u + 1]));
}

// Position of a persistent CTA in the launch's tile list.  Plain order: tile w = ((z * cur_heads) + h) * q_tiles + qt,
// token tiles fastest (neighbouring CTAs share K/V blocks in L2), then query heads, then z = batch * num_splits + split.
// long_first: the tiles with most key blocks first, all heads of a token tile together, and every second wave of CTAs in
// reverse, so that the sums of a CTA's tiles are about equal.  A place in the list is added up from the digits of the
// wave's first place, which move by those of the grid's size (from the host), and of the CTA's place in a wave: divisions
// are few, and ahead of the kernel's wait — where all of a call's CTAs fill the device they are on its clock all the same
// (ten of them were 2.8 us).
struct TileCursor {
    int w, qt, h, z;
    int base_w, base[3];      // first place of the wave: index and digits (fastest first)
    int own_w[2], own[2][3];  // the CTA's place in even / odd waves
    int odd;
    __device__ __forceinline__ void place(const PrefillParams& p) {
        const int rf = p.long_first ? p.cur_heads : p.q_tiles, rm = p.long_first ? p.batch : p.cur_heads;
        w = base_w + (odd ? own_w[1] : own_w[0]);
        int fast = base[0] + (odd ? own[1][0] : own[0][0]), carry = fast >= rf ? 1 : 0;
        fast -= carry * rf;
        int mid = base[1] + (odd ? own[1][1] : own[0][1]) + carry;
        carry = mid >= rm ? 1 : 0;
        mid -= carry * rm;
        const int slow = base[2] + (odd ? own[1][2] : own[0][2]) + carry;
        qt = p.long_first ? p.q_tiles - 1 - slow : fast;
        h = p.long_first ? fast : mid;
        z = p.long_first ? mid : slow;
    }
    __device__ __forceinline__ void init(const PrefillParams& p) {
        const bool tail = p.tail_base >= 0;  // (the grid holds one CTA per tile, and never steps)
        const int heads = tail ? p.cur_heads >> 1 : p.cur_heads;
        const int rf = p.long_first ? heads : p.q_tiles, rm = p.long_first ? p.batch : heads;
        auto digits = [&](int idx, int (&d)[3]) {
            const int rest = idx / rf;
            d[0] = idx - rest * rf;
            d[2] = rest / rm;
            d[1] = rest - d[2] * rm;
        };
        base_w = base[0] = base[1] = base[2] = odd = 0;
        const int first = blockIdx.x;
        own_w[0] = own_w[1] = first;
        digits(tail ? p.tail_base + (first >> 1) : first, own[0]);
        own[1][0] = own[0][0], own[1][1] = own[0][1], own[1][2] = own[0][2];
        if (p.long_first && !tail) {
            own_w[1] = (int)gridDim.x - 1 - first;
            digits(own_w[1], own[1]);
        }
        place(p);
        if (tail) h = h * 2 + (first & 1);
    }
    __device__ __forceinline__ void advance(const PrefillParams& p) {
        const int rf = p.long_first ? p.cur_heads : p.q_tiles, rm = p.long_first ? p.batch : p.cur_heads;
        base_w += gridDim.x;
        base[0] += p.step[0];
        int carry = base[0] >= rf ? 1 : 0;
        base[0] -= carry * rf;
        base[1] += p.step[1] + carry;
        carry = base[1] >= rm ? 1 : 0;
        base[1] -= carry * rm;
        base[2] += p.step[2] + carry;
        odd ^= 1;
        place(p);
    }
};

// One CTA per SM, persistent: it takes tiles (128 query tokens of one query head) round-robin
// and keeps its pipelines running across tile boundaries — the next tile's Q, K and V stream in
// and its first score blocks are computed while the softmax warps still write the previous
// tile's output.  Two score buffers in tensor memory, then O, so S = Q K^T runs one key block ahead of
// the softmax; eight softmax warps (two threads per query row, 64 keys each).
// Eight rather than sixteen softmax warps on purpose: the
// single MMA-issuing thread shares an instruction scheduler with them, and with four busy
// warps per scheduler it could not issue MMAs fast enough to keep the tensor pipe fed.
struct PrefillCfg {
    static constexpr int HD = 256;
    static constexpr int BM = 128;  // query rows per tile
    static constexpr int BN = 128;  // keys per block
    static constexpr int CH = HD / 64;
    static constexpr int CHUNK_BYTES = 128 * 128;  // 128 rows x 64 bf16
    static constexpr int TILE_BYTES = CH * CHUNK_BYTES;
    static constexpr int K_STAGES = 1;
    static constexpr int V_STAGES = 1;
    static constexpr int TMEM_COLS = 512;
    static constexpr int NSB = 2;  // score buffers: S = Q K^T runs NSB-1 blocks ahead of the softmax
    static constexpr int COL_S = 0;                  // NSB buffers of 128 fp32 columns; P (bf16) is written over them
    static constexpr int COL_O = NSB * 128;          // HD fp32 columns
    static constexpr int NUM_BARS = 2 + 2 * K_STAGES + 2 * V_STAGES + 2 * NSB + 2 + 2;
    static constexpr int XCH_FLOATS = 2 * 2 * 128 + 2 * 128;  // row-max exchange (2 phases), row-sum exchange
    static constexpr int SMEM_BYTES = (1 + K_STAGES + V_STAGES) * TILE_BYTES + NUM_BARS * 8 + 16 + XCH_FLOATS * 4 + 1024;
    static constexpr int SOFTMAX_WARPS = 8;
    static constexpr int THREADS = 32 * (SOFTMAX_WARPS + 2);
    static constexpr int MAX_REGS = 168;  // ten warps put three on some scheduler: 3 x 32 x 168 fits its 16384 registers, 176 does not
};

// One unit of work: a tile, or a part of its key range, in the order tile w = ((z * nq) + h) * q_tiles + qt, z = batch *
// num_splits + split.
struct TileWork {
    int q0, h, b, split, kvh;
    int my_lo, n_my;  // key blocks [my_lo, my_lo + n_my)
};

__device__ __forceinline__ TileWork tile_at(const PrefillParams& p, int w) {
    TileWork t;
    const int rest = w / p.q_tiles, z = rest / p.nq;
    t.q0 = (w - rest * p.q_tiles) * PrefillCfg::BM;
    t.h = rest - z * p.nq;
    t.b = z / p.num_splits;
    t.split = z - t.b * p.num_splits;
    t.kvh = p.group_shift >= 0 ? (t.h >> p.group_shift) : t.h / p.group;
    const int blocks = (p.kv_len + PrefillCfg::BN - 1) / PrefillCfg::BN, per = (blocks + p.num_splits - 1) / p.num_splits;
    t.my_lo = t.split * per;
    t.n_my = max(0, min(blocks, t.my_lo + per) - t.my_lo);
    return t;
}

// Score of one key in the log2 domain, with the mask's value for it (natural-log domain).
__device__ __forceinline__ float masked_score(uint32_t raw, float sl, const float* mask_row, int key, int kv_len) {
    return key < kv_len ? __uint_as_float(raw) * sl + mask_row[key] * 1.4426950408889634f : -CUDART_INF_F;
}

// Maximum of 32 keys from key0 on, in four independent ones.
__device__ __forceinline__ void masked_max(const uint32_t (&v)[32], float (&mx)[4], float sl, const float* mask_row, int key0, int kv_len) {
#pragma unroll
    for (int e = 0; e < 32; e += 8)
#pragma unroll
        for (int u = 0; u < 4; ++u)
            mx[u] = max3f(mx[u], masked_score(v[e + 2 * u], sl, mask_row, key0 + e + 2 * u, kv_len),
                          masked_score(v[e + 2 * u + 1], sl, mask_row, key0 + e + 2 * u + 1, kv_len));
}

// exp2 of 32 keys against the running maximum, packed to bf16x2; four independent partial sums.
__device__ __forceinline__ void masked_exp(const uint32_t (&v)[32], uint32_t (&pk)[16], float (&ls)[4], float sl, float m_eff,
                                           const float* mask_row, int key0, int kv_len) {
#pragma unroll
    for (int e = 0; e < 32; e += 2) {
        const float p0 = fast_exp2(masked_score(v[e], sl, mask_row, key0 + e, kv_len) - m_eff);
        const float p1 = fast_exp2(masked_score(v[e + 1], sl, mask_row, key0 + e + 1, kv_len) - m_eff);
        ls[(e >> 1) & 3] += p0 + p1;
        pk[e >> 1] = pack_bf16x2(p0, p1);
    }
}

// Barrier between the two warps that share a set of 32 query rows (warps q and q + 4):
// hardware barrier 1 + q, 64 threads.  Every softmax warp executes the same number of
// pair_syncs per tile, whatever happened to its waits, so neither warp of a pair can be left
// waiting here.
__device__ __forceinline__ void pair_sync(int quarter) {
    asm volatile("bar.sync %0, 64;" ::"r"(quarter + 1) : "memory");
}

// 32 bytes (16 bf16) to q: one 256-bit store where q is 32-byte aligned (a whole DRAM sector), else two
// 128-bit stores.
__device__ __forceinline__ void store_bf16x16(uint16_t* q, const uint32_t (&w)[8]) {
    if ((reinterpret_cast<uintptr_t>(q) & 31u) == 0) {
        asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(q), "r"(w[0]), "r"(w[1]), "r"(w[2]),
                     "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7])
                     : "memory");
    } else {
        *reinterpret_cast<uint4*>(q) = make_uint4(w[0], w[1], w[2], w[3]);
        *reinterpret_cast<uint4*>(q + 8) = make_uint4(w[4], w[5], w[6], w[7]);
    }
}

// The same 32 bytes at element offset `off` of every copy of the output (plain stores; a copy in another
// GPU's memory travels over NVLink while the kernel computes on).
__device__ __forceinline__ void store_copies_bf16x16(const unsigned long long* copies, int n, long long off,
                                                     const uint32_t (&w)[8]) {
    for (int c = 0; c < n; ++c) store_bf16x16(reinterpret_cast<uint16_t*>(copies[c]) + off, w);
}

__global__ void __maxnreg__(PrefillCfg::MAX_REGS)
    sdpa_prefill_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                        const __grid_constant__ CUtensorMap tm_v, const PrefillParams p) {
    using C = PrefillCfg;
    constexpr int HD = C::HD;
    constexpr int KS = C::K_STAGES;
    constexpr int VS = C::V_STAGES;
    constexpr int NSB = C::NSB;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* sQ = smem;
    uint8_t* sK = smem + C::TILE_BYTES;       // [KS] stages
    uint8_t* sV = sK + KS * C::TILE_BYTES;    // [VS] stages
    uint64_t* bars = reinterpret_cast<uint64_t*>(sV + VS * C::TILE_BYTES);
    uint64_t* q_full = bars;
    uint64_t* q_empty = bars + 1;       // the tile's last S = Q K^T has completed: Q may be replaced
    uint64_t* k_full = bars + 2;
    uint64_t* k_empty = k_full + KS;
    uint64_t* v_full = k_empty + KS;
    uint64_t* v_empty = v_full + VS;
    uint64_t* s_full = v_empty + VS;    // [NSB] score buffers
    uint64_t* p_full = s_full + NSB;    // [NSB]
    // [key block & 1]: O += P V of that block has completed
    uint64_t* pv_done = p_full + NSB;
    uint64_t* o_full = pv_done + 2;     // one phase per tile: the tile's last O += P V has completed
    uint64_t* o_empty = o_full + 1;     // one phase per tile: the softmax warps have read O out
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + C::NUM_BARS);
    uint32_t* abort_slot = tmem_slot + 1;
    float* xch_max = reinterpret_cast<float*>(tmem_slot + 4);  // [phase 2][key half 2][row 128]
    float* xch_sum = xch_max + 2 * 2 * 128;                    // [key half 2][row 128]

    // (broadcast, so that the compiler knows them to be the same in every lane and keeps what follows from them —
    // MMA descriptors above all — in uniform registers)
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);
    const int lane = threadIdx.x & 31;
    const long long rows_total = (long long)p.batch * p.seq * p.nq;

    constexpr int PRODUCER_WARP = C::SOFTMAX_WARPS;
    constexpr int MMA_WARP = C::SOFTMAX_WARPS + 1;
    if (threadIdx.x == 0) {
        mbar_init(q_full, 1);
        mbar_init(q_empty, 1);
        for (int s = 0; s < KS; ++s) {
            mbar_init(&k_full[s], 1);
            mbar_init(&k_empty[s], 1);
        }
        for (int s = 0; s < VS; ++s) {
            mbar_init(&v_full[s], 1);
            mbar_init(&v_empty[s], 1);
        }
        for (int s = 0; s < NSB; ++s) {
            mbar_init(&s_full[s], 1);
            mbar_init(&p_full[s], 32 * C::SOFTMAX_WARPS);
        }
        mbar_init(&pv_done[0], 1);
        mbar_init(&pv_done[1], 1);
        mbar_init(o_full, 1);
        mbar_init(o_empty, 32 * C::SOFTMAX_WARPS);
        fence_mbar_init();
    }
    if (warp == PRODUCER_WARP) {
        if (lane == 0) {
            prefetch_tensormap(&tm_q);
            prefetch_tensormap(&tm_k);
            prefetch_tensormap(&tm_v);
        }
        __syncwarp();
        tmem_alloc(tmem_slot, C::TMEM_COLS);
        tmem_relinquish();
    }
    // (the divisions, ahead of the wait: they took 1000 clk between the kernel's release and its first load)
    const TileWork first = tile_at(p, blockIdx.x);
    // Up to here nothing depends on the kernels in front; everything below may.
    grid_dependency_wait();
    grid_launch_dependents();
    if (threadIdx.x == 0) *abort_slot = *reinterpret_cast<volatile uint32_t*>(p.fault) != 0u ? 1u : 0u;
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, *reinterpret_cast<volatile uint32_t*>(tmem_slot), 0);
    // A call that finds a status word set does no work: every role walks an empty tile list and meets
    // the others at the end.
    const int total_tiles = *abort_slot ? 0 : p.total_tiles;

    if (warp == PRODUCER_WARP) {
        // ------------------------------------------------------------------ TMA producer
        if (lane == 0) {
            int gk = 0, gv = 0, tc = 0;  // K blocks, V blocks and non-empty tiles loaded so far
            bool ok = true;
            for (int w = blockIdx.x; ok && w < total_tiles; w += gridDim.x) {
                const TileWork tw = w == (int)blockIdx.x ? first : tile_at(p, w);
                if (tw.n_my == 0) continue;
                if (tc > 0 && !mbar_wait(q_empty, (tc - 1) & 1)) {
                    report_fault(p.fault, FAULT_WAIT_EMPTY, 0x300u);
                    break;
                }
                mbar_arrive_expect_tx(q_full, C::TILE_BYTES);
#pragma unroll
                for (int c = 0; c < C::CH; ++c) tma_load_4d(sQ + c * C::CHUNK_BYTES, &tm_q, q_full, c * 64, tw.h, tw.q0, tw.b);
                int uk = 0, uv = 0;
                // K runs up to K_STAGES blocks ahead of the MMAs, V up to V_STAGES; the two rings
                // are filled in the order the MMAs will need them.
                while (uk < tw.n_my || uv < tw.n_my) {
                    if (uk < tw.n_my && (uk <= uv + 1 || uv >= tw.n_my)) {
                        const int st = gk % KS;
                        if (gk >= KS && !mbar_wait(&k_empty[st], ((gk / KS) - 1) & 1)) {
                            report_fault(p.fault, FAULT_WAIT_EMPTY, 0x100u);
                            ok = false;
                            break;
                        }
                        mbar_arrive_expect_tx(&k_full[st], C::TILE_BYTES);
#pragma unroll
                        for (int c = 0; c < C::CH; ++c)
                            tma_load_4d(sK + st * C::TILE_BYTES + c * C::CHUNK_BYTES, &tm_k, &k_full[st], c * 64, tw.kvh,
                                        (tw.my_lo + uk) * C::BN, tw.b);
                        ++uk;
                        ++gk;
                    } else {
                        const int st = gv % VS;
                        if (gv >= VS && !mbar_wait(&v_empty[st], ((gv / VS) - 1) & 1)) {
                            report_fault(p.fault, FAULT_WAIT_EMPTY, 0x200u);
                            ok = false;
                            break;
                        }
                        mbar_arrive_expect_tx(&v_full[st], C::TILE_BYTES);
#pragma unroll
                        for (int c = 0; c < C::CH; ++c)
                            tma_load_4d(sV + st * C::TILE_BYTES + c * C::CHUNK_BYTES, &tm_v, &v_full[st], c * 64, tw.kvh,
                                        (tw.my_lo + uv) * C::BN, tw.b);
                        ++uv;
                        ++gv;
                    }
                }
                ++tc;
            }
        }
    } else if (warp == MMA_WARP) {
        // ------------------------------------------------------------------ MMA issuer
        // Per tile: the first NSB-1 score blocks; then for every block u:  S(u+NSB-1) into the
        // buffer P(u-1) just left (runs while the softmax warps work on S(u)), then
        // O += P(u) V(u) once P(u) is in tensor memory.  Counters run across tiles, so buffers,
        // stages and barrier phases simply keep rotating.  The whole warp runs the code, one elected lane issues.
        {
            constexpr uint32_t IDESC_QK = make_idesc_bf16(128, 128, false);
            constexpr uint32_t IDESC_PV = make_idesc_bf16(128, HD, true);
            constexpr uint32_t TILE16 = C::TILE_BYTES >> 4, CHUNK16 = C::CHUNK_BYTES >> 4;  // descriptor units
            const uint32_t tO = tmem_base + C::COL_O;
            // Descriptors are built once; per MMA only the start-address field (bytes >> 4, low word) moves.
            const uint64_t dQ = make_smem_desc_sw128(smem_u32(sQ), 16, 1024);
            const uint64_t dK = make_smem_desc_sw128(smem_u32(sK), 16, 1024);
            const uint64_t dV = make_smem_desc_sw128(smem_u32(sV), C::CHUNK_BYTES, 1024);
            // score blocks issued, P V blocks issued, non-empty tiles started; ring positions of gs and gp
            int gs = 0, gp = 0, tc = 0;
            auto issue_qk = [&]() -> bool {
                if (!mbar_wait_inline(&k_full[gs % KS], (gs / KS) & 1)) {
                    report_fault(p.fault, FAULT_WAIT_K, gs);
                    return false;
                }
                tc_fence_after_sync();
                const uint32_t tS = tmem_base + C::COL_S + (gs % NSB) * 128;
                uint64_t da = dQ, db = dK + (uint64_t)((gs % KS) * TILE16);
                uint32_t acc = 0u;
#pragma unroll 1
                for (int c = 0; c < C::CH; ++c, da += CHUNK16, db += CHUNK16, acc = 1u)  // 64 head-dim columns a turn
                    umma_ss_x4<2, 2>(tS, da, db, IDESC_QK, acc);
                umma_commit_warp(&s_full[gs % NSB]);
                umma_commit_warp(&k_empty[gs % KS]);
                ++gs;
                return true;
            };
            bool ok = true;
            for (int w = blockIdx.x; ok && w < total_tiles; w += gridDim.x) {
                const TileWork tw = w == (int)blockIdx.x ? first : tile_at(p, w);
                if (tw.n_my == 0) continue;
                if (!mbar_wait_inline(q_full, tc & 1)) {
                    report_fault(p.fault, FAULT_WAIT_Q, tc);
                    break;
                }
                int issued = 0;  // score blocks of this tile issued so far
                // u < 0: the first scores; the loop is one so that the scores are issued from one place
                for (int u = -(NSB - 1); ok && u < tw.n_my; ++u) {
                    if (issued < tw.n_my) {
                        ok = issue_qk();
                        if (!ok) break;
                        if (++issued == tw.n_my) umma_commit_warp(q_empty);
                    }
                    if (u < 0) continue;
                    // (P comes last: the others have long been there when it does)
                    if (!mbar_wait_inline(&v_full[gp % VS], (gp / VS) & 1)) {
                        report_fault(p.fault, FAULT_WAIT_V, gp);
                        ok = false;
                        break;
                    }
                    if (u == 0 && tc > 0 && !mbar_wait_inline(o_empty, (tc - 1) & 1)) {
                        report_fault(p.fault, FAULT_WAIT_O, 0x100u + tc);
                        ok = false;
                        break;
                    }
                    if (!mbar_wait_inline(&p_full[gp % NSB], (gp / NSB) & 1)) {
                        report_fault(p.fault, FAULT_WAIT_P, gp);
                        ok = false;
                        break;
                    }
                    tc_fence_after_sync();
                    // P from tensor memory: each 32-key chunk keeps its 16 bf16x2 columns at the start
                    // of its own 32 score columns, so 32 keys are two MMAs 8 columns apart.  V is
                    // MN-major: 64-element head-dim chunks 16 KB apart (leading offset), 8-key groups
                    // 1024 bytes apart (stride offset); 16 keys = 2048 bytes.
                    uint32_t tP = tmem_base + C::COL_S + (gp % NSB) * 128, acc = u > 0 ? 1u : 0u;
                    uint64_t dVu = dV + (uint64_t)((gp % VS) * TILE16);
#pragma unroll 1
                    for (int c = 0; c < C::BN / 32; ++c, tP += 32, dVu += 256, acc = 1u)
                        umma_ts_x2<8, 128>(tO, tP, dVu, IDESC_PV, acc);
                    umma_commit_warp(&v_empty[gp % VS]);
                    umma_commit_warp(&pv_done[gp & 1]);
                    ++gp;
                }
                if (ok) umma_commit_warp(o_full);
                ++tc;
            }
        }
    } else {
        // ------------------------------------------------------------------ softmax / epilogue
        // Two threads per query row: warps 0-3 own keys 0-63 of every block (score columns
        // 0-63), warps 4-7 keys 64-127; both threads of a row sit in the same TMEM lane.
        const int kh = warp >> 2;       // 64-key half of each block
        const int quarter = warp & 3;   // TMEM lane quarter
        const int r = quarter * 32 + lane;
        constexpr int OC = HD / 2;  // output columns per thread
        const uint32_t lane_sel = static_cast<uint32_t>(quarter * 32) << 16;
        const uint32_t tS0 = tmem_base + lane_sel + C::COL_S + kh * 64;
        const uint32_t tO = tmem_base + lane_sel + C::COL_O + kh * OC;
        const float sl = p.scale_log2;

        int gb = 0, tc = 0;  // key blocks and non-empty tiles processed so far
        bool ok = true;
        uint32_t va[32], vb[32];  // this thread's 64 scores of the current block

        for (int w = blockIdx.x; w < total_tiles; w += gridDim.x) {
            const TileWork tw = w == (int)blockIdx.x ? first : tile_at(p, w);
            const int t = tw.q0 + r;
            const long long row = ((long long)tw.b * p.seq + t) * p.nq + tw.h;
            if (tw.n_my == 0) {
                // Fewer key blocks than parts: an empty record.
                if (t < p.seq) {
                    float4* dst = reinterpret_cast<float4*>(p.part_o + ((long long)tw.split * rows_total + row) * HD + kh * OC);
                    for (int i = 0; i < OC / 4; ++i) dst[i] = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (kh == 0) p.part_lse[(long long)tw.split * rows_total + row] = -CUDART_INF_F;
                }
                continue;
            }

            const float* mask_row = p.mask + (long long)min(t, p.seq - 1) * p.kv_len;

            float m = -CUDART_INF_F;  // running max, log2 domain, possibly stale by <= 8
            float l = 0.f;            // this thread's share of the row sum

            // Two score buffers leave no room to look ahead: S(i+1) can only be computed once P(i-1) has
            // been consumed, so waiting for it before the exponentials of block i would put the tensor
            // pipe and the softmax in series.  Here every block is taken on its own: maximum, exchange,
            // exponentials; meanwhile the tensor pipe runs O += P(i-1) V(i-1) and S(i+1).
            for (int i = 0; i < tw.n_my; ++i) {
                const int g = gb + i;
                const int kc = (tw.my_lo + i) * C::BN + kh * 64;
                const uint32_t tS = tS0 + (g % NSB) * 128;
                if (ok && !mbar_wait_warp(&s_full[g % NSB], (g / NSB) & 1)) {
                    report_fault(p.fault, FAULT_WAIT_S, g);
                    ok = false;
                }
                if (ok) {
                    tc_fence_after_sync();
                    tmem_ld32(tS, va);
                    tmem_ld32(tS + 32, vb);
                    tmem_wait_ld();
                    float mr[4] = {-CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F};
                    masked_max(va, mr, sl, mask_row, kc, p.kv_len);
                    masked_max(vb, mr, sl, mask_row, kc + 32, p.kv_len);
                    xch_max[(g & 1) * 256 + kh * 128 + r] = fmaxf(fmaxf(mr[0], mr[1]), fmaxf(mr[2], mr[3]));
                }
                pair_sync(quarter);
                if (!ok) continue;
                const float* xm = xch_max + (g & 1) * 256;
                const float m_new = fmaxf(m, fmaxf(xm[r], xm[128 + r]));
                if (i == 0) {
                    m = m_new;  // nothing accumulated yet
                } else if (__any_sync(0xffffffffu, m_new > m + 8.0f)) {
                    // Rare: the row maximum grows by more than 2^8.  Once O += P V of the previous block has
                    // landed, rescale this thread's half of O in tensor memory (the row's other thread takes
                    // the same decision from the same values).
                    const float alpha = (m_new == -CUDART_INF_F) ? 1.0f : fast_exp2(m - m_new);
                    if (!mbar_wait_warp(&pv_done[(g - 1) & 1], ((g - 1) >> 1) & 1)) {
                        report_fault(p.fault, FAULT_WAIT_O, g);
                        ok = false;
                        continue;
                    }
                    tc_fence_after_sync();
                    uint32_t ww[32];
#pragma unroll 1
                    for (int c = 0; c < OC / 32; ++c) {
                        tmem_ld32(tO + c * 32, ww);
                        tmem_wait_ld();
#pragma unroll
                        for (int e = 0; e < 32; ++e) ww[e] = __float_as_uint(__uint_as_float(ww[e]) * alpha);
                        tmem_st32(tO + c * 32, ww);
                    }
                    tmem_wait_st();
                    l *= alpha;
                    m = m_new;
                }
                const float m_eff = (m == -CUDART_INF_F) ? 0.f : m;
                float ls4[4] = {0.f, 0.f, 0.f, 0.f};
                uint32_t pk[16];
                masked_exp(va, pk, ls4, sl, m_eff, mask_row, kc, p.kv_len);
                tmem_st16(tS, pk);
                masked_exp(vb, pk, ls4, sl, m_eff, mask_row, kc + 32, p.kv_len);
                tmem_st16(tS + 32, pk);
                l += (ls4[0] + ls4[1]) + (ls4[2] + ls4[3]);
                tmem_wait_st();
                tc_fence_before_sync();
                mbar_arrive(&p_full[g % NSB]);
            }
            gb += tw.n_my;
            // Row sum = the two threads' shares.
            xch_sum[kh * 128 + r] = l;
            pair_sync(quarter);
            l = xch_sum[r] + xch_sum[128 + r];
            if (ok && !mbar_wait_warp(o_full, tc & 1)) {
                report_fault(p.fault, FAULT_WAIT_O, tc);
                ok = false;
            }
            ++tc;
            if (!ok) continue;
            tc_fence_after_sync();
            const float inv = l > 0.f ? 1.0f / l : 0.f;
            const float lse = l > 0.f ? (m + fast_log2(l)) * 0.6931471805599453f : -CUDART_INF_F;
            const bool store = t < p.seq;
            if (p.num_splits > 1) {
                float* dst = p.part_o + ((long long)tw.split * rows_total + row) * HD + kh * OC;
#pragma unroll 1
                for (int c = 0; c < OC / 32; ++c) {
                    tmem_ld32(tO + c * 32, va);
                    tmem_wait_ld();
                    if (store) {
#pragma unroll
                        for (int e = 0; e < 32; e += 4)
                            *reinterpret_cast<float4*>(dst + c * 32 + e) =
                                make_float4(__uint_as_float(va[e]) * inv, __uint_as_float(va[e + 1]) * inv,
                                            __uint_as_float(va[e + 2]) * inv, __uint_as_float(va[e + 3]) * inv);
                    }
                }
                // O is in registers / on its way out: the next tile may overwrite the accumulator.
                tc_fence_before_sync();
                mbar_arrive(o_empty);
                if (store && kh == 0) p.part_lse[(long long)tw.split * rows_total + row] = lse;
            } else {
                const long long eoff = tw.b * p.o_stride_b + t * p.o_stride_t + (long long)tw.h * HD + kh * OC;
                uint16_t* dst = p.out + eoff;
                const uint16_t* gp = p.gate ? p.gate + eoff : nullptr;
                // One thread writes 256 contiguous bytes of its row.
#pragma unroll 1
                for (int c = 0; c < OC / 32; ++c) {
                    tmem_ld32(tO + c * 32, va);
                    tmem_wait_ld();
                    if (c == OC / 32 - 1) {
                        tc_fence_before_sync();
                        mbar_arrive(o_empty);
                    }
                    if (store) {
#pragma unroll
                        for (int e = 0; e < 32; e += 16) {
                            uint32_t ov[8];
#pragma unroll
                            for (int hh = 0; hh < 2; ++hh) {
                                float o[8];
#pragma unroll
                                for (int u = 0; u < 8; ++u) o[u] = __uint_as_float(va[e + hh * 8 + u]) * inv;
                                if (gp) {
                                    const uint4 gv = *reinterpret_cast<const uint4*>(gp + c * 32 + e + hh * 8);
                                    const uint32_t gw[4] = {gv.x, gv.y, gv.z, gv.w};
#pragma unroll
                                    for (int u = 0; u < 8; ++u) {
                                        const float gf = bf16_bits_to_f32(static_cast<uint16_t>(gw[u >> 1] >> ((u & 1) * 16)));
                                        const float sig = sigmoid(gf);
                                        o[u] = bf16_round(o[u]) * sig;
                                    }
                                }
#pragma unroll
                                for (int u = 0; u < 4; ++u) ov[hh * 4 + u] = pack_bf16x2(o[2 * u], o[2 * u + 1]);
                            }
                            store_bf16x16(dst + c * 32 + e, ov);
                            if (p.n_copies) store_copies_bf16x16(p.out_copies, p.n_copies, eoff + c * 32 + e, ov);
                        }
                    }
                }
                if (store && kh == 0 && p.out_lse) p.out_lse[row] = lse;
            }
        }
    }

    tc_fence_before_sync();
    __syncthreads();
    if (warp == PRODUCER_WARP) tmem_dealloc(tmem_base, C::TMEM_COLS);
}

}  // namespace arc
