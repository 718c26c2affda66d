// GQA flash-attention prefill kernel for sm_100a, head dim 128: one query tile per CTA, its key blocks in two chains.
//
// For calls whose tiles leave SMs idle (prefill_pair_sm100.cuh takes two tiles per CTA), for the last tiles of larger
// ones, for parts of a key range and for additive masks.  A tile on its own is a serial chain per key block — scores,
// softmax, O += P V — of 2200 clk or more, of which the tensor pipe works 1024.  Here the tile's key blocks 0, 2, 4, ...
// and 1, 3, 5, ... are two chains, A and B, each with its softmax warps (a row per thread), row maximum and sum, P and
// accumulator; they share the score buffer in turn as the two tiles of the other kernel do, and are folded at the end.
// (512 queries of 8 heads over 512 keys: 10.1 us as one chain with two threads per row, 6.9 now;
// 1024 over 1024 15.7 and 10.2, 512 of 28 heads over 8192 92 and 52.)
//
// Twelve warps: 0-3 / 4-7 softmax of chain A / B and then the output, 8 TMA producer, 9 issues S = Q K^T, 10 O += P V
// (11 idles).  What is on the clock in a call of a few blocks is everything that runs once, so:
//   - the producer asks for the first Q, K and V before the status word has been looked at (the other warps wait for it,
//     550 clk); if it is set nothing else happens, but the copies are waited for;
//   - all eight softmax warps write the output, a warp 32 rows x 64 columns of both accumulators folded (1000 clk, and as
//     many for its 32 KB to leave the SM; four epilogue warps of their own took 2850 and a TMA store's 800 behind them);
//   - K and V have rings of their own, three stages of K: with K of a block tied to V of the block before it, the fourth
//     block's scores waited 2500 clk for the first block's P V.
//
// Lazy rescaling, bounded waits and the device status word are as in the two-tile kernel.
#pragma once
#include "prefill_wide_sm100.cuh"

namespace arc {

struct ChainsCfg {
    static constexpr int HD = 128;
    static constexpr int BM = 128, BN = 128;  // rows of a tile, keys of a block
    static constexpr int CHUNK_BYTES = 128 * 128;
    static constexpr int TILE_BYTES = 2 * CHUNK_BYTES;
    static constexpr int K_STAGES = 3, V_STAGES = 2;
    static constexpr int COL_S = 0;    // the score buffer, used by the chains in turn
    static constexpr int COL_P = 128;  // + 64 * chain
    static constexpr int COL_O = 256;  // + 128 * chain
    // first[2] q_empty k_full[3] k_empty[3] v_full[2] v_empty[2] s_free s_full[2] p_part[4] pv_done[2] o_full[2] o_empty
    static constexpr int NUM_BARS = 3 + 2 * K_STAGES + 2 * V_STAGES + 1 + 2 + 4 + 2 + 2 + 1;
    static constexpr int SMEM_BYTES = (1 + K_STAGES + V_STAGES) * TILE_BYTES + 8 * 4096 + NUM_BARS * 8 + 16 + 2 * 2 * 128 * 4;  // (8 x 4 KB: output stage)
    static_assert(SMEM_BYTES <= 232448, "more shared memory than a CTA can have");
    static constexpr int PRODUCER_WARP = 8, S_ISSUER_WARP = 9, PV_ISSUER_WARP = 10;
    static constexpr int THREADS = 32 * 12;
    static constexpr int REGS_SOFTMAX = 216, REGS_CONTROL = 64;
    static constexpr int LAUNCH_REGS = (65536 / THREADS) & ~7;
    static_assert((8 * REGS_SOFTMAX + 4 * REGS_CONTROL) * 32 <= THREADS * LAUNCH_REGS, "register budgets exceed what the CTA holds at launch");
};

// One tile (or a part of its key range): key blocks [lo, hi), block lo + i in chain i & 1.
struct ChainsWork {
    int q0, h, b, kvh, lo, hi, part;
    __device__ __forceinline__ int blocks() const { return hi - lo; }
};

template <bool VISION>
__device__ __forceinline__ ChainsWork decode_chains(const PrefillParams& p, const TileCursor& cur) {
    ChainsWork t;
    t.b = cur.z;
    t.part = 0;
    if (p.num_splits > 1) {
        t.b = cur.z / p.num_splits;
        t.part = cur.z - t.b * p.num_splits;
    }
    t.h = cur.h;
    t.kvh = p.group_shift >= 0 ? (cur.h >> p.group_shift) : cur.h / p.group;
    t.q0 = cur.qt * ChainsCfg::BM;
    tile_blocks<VISION>(p, t.q0, t.lo, t.hi);
    if (p.num_splits > 1) {
        const int n = t.hi - t.lo;
        t.hi = t.lo + n * (t.part + 1) / p.num_splits;
        t.lo += n * t.part / p.num_splits;
    }
    return t;
}

// What an additive mask says of the 128 keys from key0 on: bits[c] has a bit per key of chunk c, set where the mask is 0, for the
// lane's row (the warp's begin at row0).  True: other values occur in the warp's rows that do not hide their key.  The
// warp reads a row at a time, 32 keys a load, and a ballot is the chunk's bits.  (A thread reading its own row touched 32 lines
// a load and was 12 KB of code: 1500 x 1500, 16/8 heads, 138 us, from cold caches 193; 32 x 32, 4/1, cold 18.0.)
__device__ __forceinline__ bool read_mask_bits(const float* mask, int row0, int rows, int key0, int kv_len, uint32_t (&bits)[4]) {
    constexpr int AT_ONCE = 8;  // rows, four loads each
    const int lane = threadIdx.x & 31;
    bool values = false;
    bits[0] = bits[1] = bits[2] = bits[3] = 0u;
#pragma unroll 1
    for (int i0 = 0; i0 < 32 && row0 + i0 < rows; i0 += AT_ONCE) {
        float f[AT_ONCE][4];
#pragma unroll
        for (int i = 0; i < AT_ONCE; ++i)
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const int row = row0 + i0 + i, key = key0 + c * 32 + lane;
                f[i][c] = row < rows && key < kv_len ? mask[(long long)row * kv_len + key] : -CUDART_INF_F;
            }
#pragma unroll
        for (int i = 0; i < AT_ONCE; ++i)
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const uint32_t w = __ballot_sync(0xffffffffu, f[i][c] == 0.f);
                if (lane == i0 + i) bits[c] = w;
                values |= f[i][c] != 0.f && !mask_hides(f[i][c]);
            }
    }
    return __any_sync(0xffffffffu, values);
}

// Two bf16 outputs times sigmoid of their gate values: the rounding order of the two-launch form.
__device__ __forceinline__ uint32_t gate_pair(uint32_t attn, uint32_t gate) {
    return pack_bf16x2(__uint_as_float(attn << 16) * sigmoid(__uint_as_float(gate << 16)),
                       __uint_as_float(attn & 0xffff0000u) * sigmoid(__uint_as_float(gate & 0xffff0000u)));
}

// Barrier between the two warps that share a set of 32 query rows (warps q and q + 4): hardware barrier 1 + q, 64 threads.
// Every softmax warp executes the same number of them per tile, whatever happened to its waits.
__device__ __forceinline__ void row_sync(int quarter) { asm volatile("bar.sync %0, 64;" ::"r"(quarter + 1) : "memory"); }

// VISION: causal with vision blocks (p.ids).  MASKED: an additive mask.  num_splits > 1: a unit is a part of the key range,
// whose normalised rows go to the partial records as f32 with their log-sum-exp.
template <bool GATE, bool VISION, bool MASKED>
__global__ void __launch_bounds__(ChainsCfg::THREADS, 1)
    sdpa_prefill_chains_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                               const __grid_constant__ CUtensorMap tm_v, const PrefillParams p) {
    using C = ChainsCfg;
    constexpr int HD = C::HD, KS = C::K_STAGES, VS = C::V_STAGES;
    extern __shared__ __align__(1024) uint8_t smem[];  // (the swizzle pattern follows the address bits)
    uint8_t* sQ = smem;
    uint8_t* sK = sQ + C::TILE_BYTES;         // [KS]
    uint8_t* sV = sK + KS * C::TILE_BYTES;    // [VS]
    uint8_t* sOut = sV + VS * C::TILE_BYTES;  // [softmax warp] 32 rows x 64 columns
    // [64 head-dim columns] Q and the tile's first K: the first MMAs run while the other columns arrive.  (Halves for every
    // block cost more than they bring: 0.80 us a block, not 0.71.)
    uint64_t* first = reinterpret_cast<uint64_t*>(sOut + 8 * 4096);
    uint64_t* q_empty = first + 2;        // the tile's last S = Q K^T has completed
    uint64_t* k_full = q_empty + 1;       // the other K
    uint64_t* k_empty = k_full + KS;
    uint64_t* v_full = k_empty + KS;
    uint64_t* v_empty = v_full + VS;
    uint64_t* s_free = v_empty + VS;      // the softmax warps of the chain that has had the scores last hold them in registers
    uint64_t* s_full = s_free + 1;        // [chain]
    uint64_t* p_part = s_full + 2;        // [chain][part]: P of keys 0-95 / 96-127 of the block is in tensor memory
    uint64_t* pv_done = p_part + 4;       // [chain] O += P V of the block has completed: P may be replaced, O rescaled
    uint64_t* o_full = pv_done + 2;       // [chain] one phase per tile with blocks of the chain: its last O += P V has completed
    uint64_t* o_empty = o_full + 2;       // one phase per tile with blocks: both accumulators have been read
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(o_empty + 1);
    uint32_t* abort_slot = tmem_slot + 1;
    float* fin = reinterpret_cast<float*>(tmem_slot + 4);  // [chain][row sums, row maxima][row]

    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);
    const int lane = threadIdx.x & 31;
    if (threadIdx.x == 32) {
        prefetch_tensormap(&tm_q);
        prefetch_tensormap(&tm_k);
        prefetch_tensormap(&tm_v);
    }
    if (threadIdx.x == 0) {
        mbar_init(&first[0], 1);
        mbar_init(&first[1], 1);
        mbar_init(q_empty, 1);
        for (int i = 0; i < KS; ++i) {
            mbar_init(&k_full[i], 1);
            mbar_init(&k_empty[i], 1);
        }
        for (int i = 0; i < VS; ++i) {
            mbar_init(&v_full[i], 1);
            mbar_init(&v_empty[i], 1);
        }
        mbar_init(s_free, 4);
        for (int s = 0; s < 2; ++s) {
            mbar_init(&s_full[s], 1);
            mbar_init(&p_part[2 * s], 4);
            mbar_init(&p_part[2 * s + 1], 4);
            mbar_init(&pv_done[s], 1);
            mbar_init(&o_full[s], 1);
        }
        mbar_init(o_empty, 8);
        fence_mbar_init();
    }
    if (warp == C::PRODUCER_WARP) {
        tmem_alloc(tmem_slot, 512);
        tmem_relinquish();
    }
    TileCursor cur;  // (with its divisions, ahead of the wait)
    cur.init(p);
    ChainsWork tw{};
    if (!VISION) tw = decode_chains<false>(p, cur);
    __syncthreads();
    // Up to here nothing depends on the kernels in front; everything below may.  (The tail of a two-tile launch runs beside
    // that launch, which let it start only when the kernels before it had completed.)
    if (p.tail_base < 0) grid_dependency_wait();
    grid_launch_dependents();
    if (threadIdx.x == 0) *abort_slot = *reinterpret_cast<volatile uint32_t*>(p.fault) != 0u ? 1u : 0u;
    if (VISION) tw = decode_chains<true>(p, cur);  // (whole warps)
    auto load_first = [&](int st) {  // Q and the first K
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            if (lane == 0) mbar_arrive_expect_tx(&first[c], 2 * C::CHUNK_BYTES);
            __syncwarp();
            tma_load_4d_warp(sQ + c * C::CHUNK_BYTES, &tm_q, &first[c], c * 64, tw.h, tw.q0, tw.b);
            tma_load_4d_warp(sK + st * C::TILE_BYTES + c * C::CHUNK_BYTES, &tm_k, &first[c], c * 64, tw.kvh, tw.lo * C::BN, tw.b);
        }
    };
    auto load = [&](uint8_t* dst, const void* tm, uint64_t* bar, int i) {  // K or V of the tile's block i
        if (lane == 0) mbar_arrive_expect_tx(bar, C::TILE_BYTES);
        __syncwarp();
#pragma unroll
        for (int c = 0; c < 2; ++c) tma_load_4d_warp(dst + c * C::CHUNK_BYTES, tm, bar, c * 64, tw.kvh, (tw.lo + i) * C::BN, tw.b);
    };
    // The first tile's Q, its first two K and its first V
    const int ahead_k = min(tw.blocks(), 2), ahead_v = min(tw.blocks(), 1);
    if (warp == C::PRODUCER_WARP && tw.blocks() > 0) {
        load_first(0);
        if (ahead_k > 1) load(sK + C::TILE_BYTES, &tm_k, &k_full[1], 1);
        load(sV, &tm_v, &v_full[0], 0);
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, *reinterpret_cast<volatile uint32_t*>(tmem_slot), 0);
    const bool aborted = *abort_slot != 0u;
    const int total_tiles = aborted ? 0 : p.total_tiles;  // a status is set: walk an empty list
    auto next_tile = [&]() {
        cur.advance(p);
        if (cur.w < total_tiles) tw = decode_chains<VISION>(p, cur);
    };

    if (warp >= C::PRODUCER_WARP) {
        reg_dealloc<C::REGS_CONTROL>();
        if (warp == C::PRODUCER_WARP) {
            // -------------------------------------------------------------- TMA producer
            if (aborted && tw.blocks() > 0) {  // (what has been asked for lands before the CTA goes)
                for (int i = 0; i < 2; ++i) mbar_wait_inline(&first[i], 0);
                if (ahead_k > 1) mbar_wait_inline(&k_full[1], 0);
                mbar_wait_inline(&v_full[0], 0);
            }
            int gk = 0, gv = 0, n = 0;  // K blocks, V blocks and tiles with blocks loaded so far
            bool ok = true;
            for (; ok && cur.w < total_tiles; next_tile()) {
                if (tw.blocks() == 0) continue;
                int uk = 0, uv = 0;  // of this tile
                // (the first tile of all with blocks may not be the first one)
                if (n == 0 && cur.w == (int)blockIdx.x) {
                    uk = gk = ahead_k, uv = gv = ahead_v;
                } else if (n > 0 && !mbar_wait_inline(q_empty, (n - 1) & 1)) {
                    if (lane == 0) report_fault(p.fault, FAULT_WAIT_EMPTY, 0x300u);
                    break;
                }
                ++n;
                // in the order of use: K up to two blocks ahead of V
                while (uv < tw.blocks()) {
                    if (uk < tw.blocks() && uk <= uv + 1) {
                        const int st = gk % KS;
                        if (gk >= KS && !mbar_wait_inline(&k_empty[st], (gk / KS - 1) & 1)) {
                            if (lane == 0) report_fault(p.fault, FAULT_WAIT_EMPTY, 0x100u);
                            ok = false;
                            break;
                        }
                        if (uk == 0) load_first(st);
                        else load(sK + st * C::TILE_BYTES, &tm_k, &k_full[st], uk);
                        ++uk, ++gk;
                    } else {
                        const int st = gv % VS;
                        if (gv >= VS && !mbar_wait_inline(&v_empty[st], (gv / VS - 1) & 1)) {
                            if (lane == 0) report_fault(p.fault, FAULT_WAIT_EMPTY, 0x200u);
                            ok = false;
                            break;
                        }
                        load(sV + st * C::TILE_BYTES, &tm_v, &v_full[st], uv);
                        ++uv, ++gv;
                    }
                }
            }
        } else if (warp == C::S_ISSUER_WARP) {
            // -------------------------------------------------------------- S = Q K^T, block after block
            // The whole warp runs this code and one lane issues: addresses stay in the uniform datapath.
            constexpr uint32_t IDESC_QK = make_idesc_bf16(128, 128, false);
            constexpr uint32_t TILE16 = C::TILE_BYTES >> 4, CHUNK16 = C::CHUNK_BYTES >> 4;  // descriptor units
            const uint64_t dQ = make_smem_desc_sw128(smem_u32(sQ), 16, 1024);
            const uint64_t dK = make_smem_desc_sw128(smem_u32(sK), 16, 1024);
            int g = 0, st = 0, n = 0;  // blocks so far, their stage; tiles with blocks
            uint32_t k_par = 0u;       // bit st: parity of the stage's k_full
            bool ok = true;
            for (; ok && cur.w < total_tiles; next_tile()) {
                const int blocks = tw.blocks();
                if (blocks == 0) continue;
                for (int i = 0; ok && i < blocks; ++i, ++g) {
                    const uint64_t db = dK + (uint64_t)(st * TILE16);
                    // (the score buffer comes last: what is waited for behind it is on the clock of both chains)
                    ok = i == 0 ? mbar_wait_inline(&first[0], n & 1) : mbar_wait_inline(&k_full[st], (k_par >> st) & 1u);
                    if (i > 0) k_par ^= 1u << st;
                    if (!ok) {
                        if (lane == 0) report_fault(p.fault, FAULT_WAIT_K, g);
                        break;
                    }
                    if (g > 0 && !mbar_wait_inline(s_free, (g - 1) & 1)) {
                        if (lane == 0) report_fault(p.fault, FAULT_WAIT_S, 0x1000u + g);
                        ok = false;
                        break;
                    }
                    tc_fence_after_sync();
                    umma_ss_x4<2, 2>(tmem_base + C::COL_S, dQ, db, IDESC_QK, 0u);  // 64 head-dim columns
                    if (i == 0 && !mbar_wait_inline(&first[1], n & 1)) {
                        if (lane == 0) report_fault(p.fault, FAULT_WAIT_Q, g);
                        ok = false;
                        break;
                    }
                    umma_ss_x4<2, 2>(tmem_base + C::COL_S, dQ + CHUNK16, db + CHUNK16, IDESC_QK, 1u);
                    umma_commit_warp(&s_full[i & 1]);
                    umma_commit_warp(&k_empty[st]);
                    if (i + 1 == blocks) umma_commit_warp(q_empty);
                    if (++st == KS) st = 0;
                }
                ++n;
            }
        } else if (warp == C::PV_ISSUER_WARP) {
            // -------------------------------------------------------------- O += P V
            constexpr uint32_t IDESC_PV = make_idesc_bf16(128, HD, true);
            constexpr uint32_t TILE16 = C::TILE_BYTES >> 4;
            const uint64_t dV = make_smem_desc_sw128(smem_u32(sV), C::CHUNK_BYTES, 1024);
            int g = 0, n = 0;      // blocks and tiles with blocks so far
            uint32_t g_par = 0u;   // bit s: parity of chain s's blocks so far
            bool ok = true;
            for (; ok && cur.w < total_tiles; next_tile()) {
                const int blocks = tw.blocks();
                if (blocks == 0) continue;
                for (int i = 0; i < blocks; ++i, ++g) {
                    const int s = i & 1, st = g & 1;
                    if (!mbar_wait_inline(&v_full[st], (g >> 1) & 1)) {
                        if (lane == 0) report_fault(p.fault, FAULT_WAIT_V, g);
                        ok = false;
                        break;
                    }
                    if (i == 0 && n > 0 && !mbar_wait_inline(o_empty, (n - 1) & 1)) {
                        if (lane == 0) report_fault(p.fault, FAULT_WAIT_O, 0x100u);
                        ok = false;
                        break;
                    }
                    // P from tensor memory: 16 keys are 8 columns of packed bf16.  V is MN-major: 64-element head-dim
                    // chunks 16 KB apart, 8-key groups 1024 bytes apart; 16 keys = 2048 bytes.
                    const uint32_t tO = tmem_base + C::COL_O + s * 128, tP = tmem_base + C::COL_P + s * 64;
                    const uint64_t dv = dV + (uint64_t)(st * TILE16);
                    const uint32_t par = (g_par >> s) & 1u;
                    if (!mbar_wait_inline(&p_part[2 * s], par)) {
                        if (lane == 0) report_fault(p.fault, FAULT_WAIT_P, g);
                        ok = false;
                        break;
                    }
                    tc_fence_after_sync();
                    umma_ts_x4<8, 128>(tO, tP, dv, IDESC_PV, i > 1 ? 1u : 0u);
                    umma_ts_x2<8, 128>(tO, tP + 32, dv + 512, IDESC_PV, 1u);
                    if (!mbar_wait_inline(&p_part[2 * s + 1], par)) {
                        if (lane == 0) report_fault(p.fault, FAULT_WAIT_P, 0x1000u + g);
                        ok = false;
                        break;
                    }
                    tc_fence_after_sync();
                    umma_ts_x2<8, 128>(tO, tP + 48, dv + 768, IDESC_PV, 1u);
                    g_par ^= 1u << s;
                    umma_commit_warp(&pv_done[s]);
                    umma_commit_warp(&v_empty[st]);
                    if (i + 2 >= blocks) umma_commit_warp(&o_full[s]);
                }
                ++n;
            }
        }
    } else {
        // ------------------------------------------------------------------ softmax, then output: thread = query row
        reg_alloc<C::REGS_SOFTMAX>();
        const int s = warp >> 2;
        const int quarter = warp & 3;
        const int r = quarter * 32 + lane;
        const uint32_t lane_sel = static_cast<uint32_t>(quarter * 32) << 16;
        const uint32_t tS = tmem_base + lane_sel + C::COL_S;
        const uint32_t tP = tmem_base + lane_sel + C::COL_P + s * 64;
        const uint32_t tO = tmem_base + lane_sel + C::COL_O;
        const float sl = p.scale_log2;
        const uint64_t sl2 = pack_f32x2(sl, sl);
        const bool causal = (p.mask_type == 3);
        const bool windowed = causal && p.window > 0 && p.window != 0x7fffffff;
        const int off = p.kv_len - p.seq;
        uint8_t* const out_buf = sOut + warp * 4096;
        const bool split = p.num_splits > 1;

        int g = 0, n0 = 0, n1 = 0;  // this chain's key blocks so far; tiles with blocks of chain A / B
        bool ok = true;
        uint32_t s0[32], s1[32], s2[32], s3[32];  // the row's 128 scores of the current block
        for (; cur.w < total_tiles; next_tile()) {
            const int t = tw.q0 + r;
            const bool store = t < p.seq;
            const long long row = ((long long)tw.b * p.seq + t) * p.nq + tw.h;
            const long long prow = (long long)tw.part * p.batch * p.seq * p.nq + row;
            const long long eoff = tw.b * p.o_stride_b + t * p.o_stride_t + (long long)tw.h * HD + s * 64;
            float* const lse_to = s == 0 && store ? (split ? p.part_lse + prow : p.out_lse ? p.out_lse + row : nullptr) : nullptr;
            if (tw.blocks() == 0) {  // nothing visible: zero output, or an empty record
                if (store && !split)
                    for (int c = -1; c < p.n_copies; ++c) {
                        uint4* dst = reinterpret_cast<uint4*>((c < 0 ? p.out : reinterpret_cast<uint16_t*>(p.out_copies[c])) + eoff);
                        for (int i = 0; i < 8; ++i) dst[i] = make_uint4(0u, 0u, 0u, 0u);
                    }
                if (lse_to) *lse_to = -CUDART_INF_F;
                continue;
            }
            if (GATE && store) prefetch_l2(p.gate + eoff);
            int row_lo = 0, row_hi = p.kv_len;  // visible keys [row_lo, row_hi)
            if (causal) {
                const int diag = t + off;
                row_hi = min(max(diag + 1, 0), p.kv_len);
                if (VISION) row_hi = vision_ends(p, diag, t < p.seq);
                if (windowed) row_lo = max(0, diag - p.window + 1);
                if (row_lo > row_hi) row_lo = row_hi;
            }
            const RowMask rm{row_lo, row_hi};

            float m = -CUDART_INF_F;  // running max of the chain, log2 domain, possibly stale by <= 8
            float l = 0.f;            // its sum
            for (int j = tw.lo + s; ok && j < tw.hi; j += 2, ++g) {
                const int kc = j * C::BN;
                uint32_t bits[4];
                bool values = false;
                if (MASKED) values = read_mask_bits(p.mask, t - lane, p.seq, kc, p.kv_len, bits);
                if (!mbar_wait_warp<3>(&s_full[s], g & 1)) {
                    report_fault(p.fault, FAULT_WAIT_S, g);
                    ok = false;
                    break;
                }
                tc_fence_after_sync();
                float bl = sl;  // what the block's scores are scaled by
                uint64_t bl2 = sl2;
                if (MASKED && values) {
                    add_mask_values(tS, p.mask, t, p.seq, kc, p.kv_len, sl);
                    bl = 1.0f, bl2 = pack_f32x2(1.0f, 1.0f);
                }
                const bool full = !MASKED && __all_sync(0xffffffffu, rm.lo <= kc && kc + C::BN <= rm.hi);
                float mr[4] = {-CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F};
                auto mask = [&](uint32_t (&v)[32], int c) {
                    if constexpr (MASKED) {
                        if (!values) select_chunk(v, bits[c]);
                    } else {
                        if (!full) mask_chunk(v, kc + c * 32, rm);  // window edge, diagonal, ragged end
                    }
                };
                tmem_ld32(tS, s0);
                tmem_ld32(tS + 32, s1);
                tmem_wait_ld();
                tmem_ld32(tS + 64, s2);  // lands while the maximum of the first half is taken
                tmem_ld32(tS + 96, s3);
                mask(s0, 0);
                mask(s1, 1);
                chunk_max(s0, mr);
                chunk_max(s1, mr);
                tmem_wait_ld();
                tc_fence_before_sync();
                mbar_arrive_warp(s_free);  // the buffer may take the other chain's scores
                mask(s2, 2);
                mask(s3, 3);
                chunk_max(s2, mr);
                chunk_max(s3, mr);
                const float m_new = fmaxf(m, fmaxf(fmaxf(mr[0], mr[1]), fmaxf(mr[2], mr[3])) * bl);
                // O += P V of the chain's block before has long completed, as a rule: its P may be replaced.
                if (g > 0 && !mbar_wait_warp<3>(&pv_done[s], (g - 1) & 1)) {
                    report_fault(p.fault, FAULT_WAIT_O, 0x200u + g);
                    ok = false;
                    break;
                }
                tc_fence_after_sync();
                const bool need = m_new > m + 8.0f;
                if (j == tw.lo + s) {
                    m = m_new;
                } else if (__any_sync(0xffffffffu, need)) {
                    // Rare: some row's maximum grows by more than 2^8: rescale those rows of O in tensor memory.
                    const float alpha = need ? fast_exp2(m - m_new) : 1.0f;
#pragma unroll 1
                    for (int c = 0; c < HD; c += 16) {
                        uint32_t ww[16];
                        tmem_ld16(tO + s * 128 + c, ww);
                        tmem_wait_ld();
#pragma unroll
                        for (int e = 0; e < 16; ++e) ww[e] = __float_as_uint(__uint_as_float(ww[e]) * alpha);
                        tmem_st16(tO + s * 128 + c, ww);
                    }
                    tmem_wait_st();
                    l *= alpha;
                    if (need) m = m_new;
                }
                // Probabilities as bf16, packed in the chain's 64 columns for P; row sum in fp32.  The first 96 keys are
                // announced half a chunk late: by then their stores have landed and the wait for them costs nothing.
                const float m_eff = (m == -CUDART_INF_F) ? 0.f : m;
                const uint64_t nm2 = pack_f32x2(-m_eff, -m_eff);
                uint64_t ls2[2] = {0ull, 0ull};
                uint32_t pk[16];
                exp_chunk(s0, pk, ls2, bl2, nm2);
                tmem_st16(tP, pk);
                exp_chunk(s1, pk, ls2, bl2, nm2);
                tmem_st16(tP + 16, pk);
                exp_chunk(s2, pk, ls2, bl2, nm2);
                tmem_st16(tP + 32, pk);
                exp_chunk<0, 16>(s3, pk, ls2, bl2, nm2);
                tmem_wait_st();
                tc_fence_before_sync();
                mbar_arrive_warp(&p_part[2 * s]);
                exp_chunk<16, 32>(s3, pk, ls2, bl2, nm2);
                tmem_st16(tP + 48, pk);
                float l0, l1, l2, l3;
                unpack_f32x2(ls2[0], l0, l1);
                unpack_f32x2(ls2[1], l2, l3);
                l += (l0 + l1) + (l2 + l3);
                tmem_wait_st();
                tc_fence_before_sync();
                mbar_arrive_warp(&p_part[2 * s + 1]);
            }

            // ---------------------------------------------------------- output: this warp's 32 rows, columns [64 s, 64 s + 64)
            const bool both = tw.blocks() > 1;  // (a single key block: B has none)
            fin[s * 256 + r] = l;
            fin[s * 256 + 128 + r] = m;
            row_sync(quarter);
            const float l_other = fin[(s ^ 1) * 256 + r], m_other = fin[(s ^ 1) * 256 + 128 + r];
            row_sync(quarter);  // (before the next tile's)
            if (ok && (!mbar_wait_warp<3>(&o_full[0], n0 & 1) || (both && !mbar_wait_warp<3>(&o_full[1], n1 & 1)))) {
                report_fault(p.fault, FAULT_WAIT_O, n0);
                ok = false;
            }
            ++n0, n1 += both;
            if (!ok) continue;
            tc_fence_after_sync();
            const float mx = fmaxf(m, m_other), at0 = mx == -CUDART_INF_F ? 0.f : mx;
            float own = fast_exp2(m - at0), other = fast_exp2(m_other - at0);
            const float sum = l * own + l_other * other, inv = sum > 0.f ? 1.0f / sum : 0.f;
            own *= inv, other *= inv;
            const float fa = s == 0 ? own : other, fb = s == 0 ? other : own;
            if (lse_to) *lse_to = sum > 0.f ? (mx + fast_log2(sum)) * 0.6931471805599453f : -CUDART_INF_F;
            // 32 columns a turn of a rolled loop (this code runs once per tile and is fetched cold, ~50 clk per 128 bytes).
            // A thread's row as it is would go out in 32 lines per store, so the warp turns its tile through shared memory;
            // plain stores then, eight lanes a row: a TMA store took 350 clk to hand over and 800 more until the buffer
            // could go.
            __syncwarp();  // (the tile before has left the buffer)
            const uint32_t at = smem_u32(out_buf) + lane * 128;
            uint32_t a[32], b[32];
            auto fetch = [&](int c) {
                tmem_ld32(tO + s * 64 + c * 32, a);
                if (both) tmem_ld32(tO + 128 + s * 64 + c * 32, b);
            };
            fetch(0);
#pragma unroll 1
            for (int c = 0; c < 2; ++c) {
                tmem_wait_ld();
                float o[32];
#pragma unroll
                for (int e = 0; e < 32; ++e) {
                    const float x = __uint_as_float(a[e]) * fa;
                    o[e] = both ? fmaf(__uint_as_float(b[e]), fb, x) : x;  // (nothing of B's: its columns may hold anything)
                }
                if (c == 0) {
                    fetch(1);
                } else {  // O is in registers: the next tile may overwrite the accumulators
                    tc_fence_before_sync();
                    mbar_arrive_warp(o_empty);
                }
                if (split) {
                    if (store) {
                        float4* dst = reinterpret_cast<float4*>(p.part_o + prow * HD + s * 64 + c * 32);
#pragma unroll
                        for (int i = 0; i < 8; ++i) dst[i] = make_float4(o[4 * i], o[4 * i + 1], o[4 * i + 2], o[4 * i + 3]);
                    }
                    continue;
                }
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at + (((4 * c + i) ^ (lane & 7)) << 4)), "r"(pack_bf16x2(o[8 * i], o[8 * i + 1])),
                                 "r"(pack_bf16x2(o[8 * i + 2], o[8 * i + 3])), "r"(pack_bf16x2(o[8 * i + 4], o[8 * i + 5])),
                                 "r"(pack_bf16x2(o[8 * i + 6], o[8 * i + 7])) : "memory");
            }
            if (split) continue;
            __syncwarp();
            const int row0 = quarter * 32 + (lane >> 3), col = (lane & 7) * 8;  // this lane's first row, its columns of the warp's 64
            const long long out0 = tw.b * p.o_stride_b + (tw.q0 + row0) * p.o_stride_t + (long long)tw.h * HD + s * 64 + col;
            // (Gated two at a time: eight, 64 sigmoids of code that is fetched cold, cost a call of 100 rows 0.1 us less from warm caches
            // and 2.4 more from cold ones: 12.3 and 9.9.)
            constexpr int AT_ONCE = GATE ? 2 : 8;
#pragma unroll AT_ONCE
            for (int i = 0; i < 8; ++i) {
                if (tw.q0 + row0 + 4 * i >= p.seq) break;
                const int rr = (lane >> 3) + 4 * i;
                uint4 v = *reinterpret_cast<const uint4*>(out_buf + rr * 128 + (((lane & 7) ^ (rr & 7)) << 4));
                const long long to = out0 + 4 * i * p.o_stride_t;
                if (GATE) {  // (in L2 since the tile began)
                    const uint4 g4 = *reinterpret_cast<const uint4*>(p.gate + to);
                    v.x = gate_pair(v.x, g4.x), v.y = gate_pair(v.y, g4.y), v.z = gate_pair(v.z, g4.z), v.w = gate_pair(v.w, g4.w);
                }
                *reinterpret_cast<uint4*>(p.out + to) = v;
                for (int k = 0; k < p.n_copies; ++k) *reinterpret_cast<uint4*>(reinterpret_cast<uint16_t*>(p.out_copies[k]) + to) = v;
            }
        }
    }

    __syncwarp();
    tc_fence_before_sync();
    __syncthreads();
    if (warp == C::PRODUCER_WARP) tmem_dealloc(tmem_base, 512);
    // A launch that covers the tail of a two-tile launch's unit list runs beside that launch (programmatic
    // stream serialization) and reads nothing it writes — but whatever follows in the stream waits for this
    // grid only, so this grid does not complete before the one in front of it has: every CTA ends on the
    // grid-dependency wait (a no-op for launches without the attribute).
    if (p.tail_base >= 0) grid_dependency_wait();
}

}  // namespace arc
