// GQA flash-attention prefill kernel for sm_100a, head dim 128: two query tiles per CTA.
//
// A CTA owns two 128-row query tiles, A and B, that walk the same key blocks.  Each tile is a pipeline of its own:
// four softmax warps (one query row per thread, TMEM lane = row, so row maxima and sums never leave the thread), P and
// one accumulator O in tensor memory, one Q buffer in shared memory.  The two share the score buffer, which they use in
// turn (S P_A P_B O_A O_B = 128 + 2 x 64 + 2 x 128 = 512 columns), and the K and V rings, which one producer thread fills
// by TMA, so every key block is fetched once for 256 rows.
//
// Sixteen warps in groups with register budgets of their own (setmaxnreg):
//   warps 0-3 / 4-7   softmax of tile A / B: a thread takes its row's 128 scores out of tensor
//                     memory ONCE and frees the score buffer, masks them in registers where the block needs it, takes
//                     the maximum, exponentiates and writes P (bf16) into the pipeline's own columns;
//   warps 8-11        epilogue: once a tile's last O += P V has landed they read the accumulator
//                     out, normalise, gate and store it, while the softmax warps are already
//                     working on the next tile's first key block;
//   warps 12-15       TMA producer of K / V, issuer of S = Q K^T, issuer of O += P V, TMA producer of Q.
//
// What bounds it.  Per key block and tile 1024 clk of the tensor pipe (64 per M128 N128 K16 MMA, both operand forms)
// and 1024 clk of the ex2 unit (16 a clock), 2048 of either for a pair of blocks, which takes 2490 clk (2 x 8192 tokens of
// 32/16 heads, no mask).  With P written over S, as it was, a pipeline's next scores had to wait for the P V that
// reads them, and a pair of blocks took 2950.  Now they are computed while the block before is exponentiated.  The clock
// gives part of it back: at this density of work the chip holds 1.40 GHz against its power limit, 1.48 before (1833 ->
// 1660 us, 0.95 of what cuBLAS sustains in bf16; window 1024, 4 x 8192 tokens: 572 -> 526 us).  Tried on it and slower: one
// warp for all MMAs (2710 clk: the tensor pipe runs dry while it looks after barriers between two groups), scores strictly
// ahead of P V in the tensor pipe (2-3 %), all 128 scores behind one wait, P announced once a block.
// What made the difference before that (4 x 8192 tokens, window 1024: 691 -> 502 us at full clock):
//   - MMA issue: elect.sync inside the asm statement and warp-uniform operands (an
//     MMA every 64-90 clk instead of every 125);
//   - no turns between the softmax warps: a single warp needs 1200 clk for the exponentials of a block on its own, two on
//     one scheduler 2000 for both, so giving them exclusive turns wasted 40 % of the ex2 unit;
//   - code size: hot code of a scheduler beyond ~8 KB costs ~50 clk per 128 bytes, so masking is one select per score
//     from a bit mask, the epilogue and all MMA loops are rolled, packed fp32 arithmetic halves the rest.  (Re-reading
//     the scores in a rolled loop would be smaller still but measured 2-5 % slower.)
//
// Lazy rescaling: O is rescaled in tensor memory only where a row's maximum grows by more than 2^8.  Calls with few tiles,
// parts of a key range and additive masks are prefill_chains_sm100.cuh's.
#pragma once
#include "prefill_sm100.cuh"

namespace arc {

struct PairCfg {
    static constexpr int HD = 128;
    static constexpr int BM = 128;   // rows per tile; a CTA works on two
    static constexpr int BN = 128;   // keys per block
    static constexpr int CH = HD / 64;
    static constexpr int CHUNK_BYTES = 128 * 128;
    static constexpr int TILE_BYTES = CH * CHUNK_BYTES;
    static constexpr int K_STAGES = 2;
    static constexpr int V_STAGES = 2;
    static constexpr int TMEM_COLS = 512;
    static constexpr int COL_S = 0;    // the score buffer, used by the pipelines in turn
    static constexpr int COL_P = 128;  // + 64 * pipeline
    static constexpr int COL_O = 256;  // + 128 * pipeline
    // q_full[2] q_empty[2] k_first k_first_used kv_full[2] kv_empty[2] s_free then per pipeline:
    // s_full p_part[2] pv_done o_full o_empty fin[2]; then gate[4][2], two per epilogue warp
    static constexpr int NUM_BARS = 4 + 2 + 2 * K_STAGES + 1 + 24;
    static constexpr int FIN_FLOATS = 2 * 2 * 128;  // [tile parity][pipeline][row] row sum
    static constexpr int SMEM_BYTES = (2 + K_STAGES + V_STAGES) * TILE_BYTES + 4 * 8192 + NUM_BARS * 8 + 16 + FIN_FLOATS * 4 + 80;  // (4 x 8 KB: output stage; 80: first unit)
    static_assert(SMEM_BYTES <= 232448, "more shared memory than a CTA can have");
    static constexpr int SOFTMAX_WARPS = 8;   // four per pipeline
    static constexpr int EPILOGUE_WARP = 8;   // four warps
    static constexpr int PRODUCER_WARP = 12;
    static constexpr int S_ISSUER_WARP = 13;  // warp 14 issues the P V MMAs
    static constexpr int Q_PRODUCER_WARP = 15;
    static constexpr int THREADS = 32 * 16;
    // The budgets may only redistribute what the CTA holds at launch (threads x the per-thread
    // count the launch bound gives, 128 for 512 threads): a group that asks for more waits for ever.
    static constexpr int REGS_SOFTMAX = 192;
    static constexpr int REGS_EPILOGUE = 72;
    static constexpr int REGS_CONTROL = 56;
    static constexpr int LAUNCH_REGS = (65536 / THREADS) & ~7;
    static_assert((SOFTMAX_WARPS * REGS_SOFTMAX + 4 * REGS_EPILOGUE + 4 * REGS_CONTROL) * 32 <= THREADS * LAUNCH_REGS,
                  "register budgets exceed what the CTA holds at launch");
};

// One unit of work: two 128-row tiles, and per tile the key blocks [lo, hi) it can see.  With an
// even number of query heads per KV head the tiles are the same 128 tokens of two heads of one KV
// group: both walk exactly the same key blocks, so neither pipeline ever idles while the other
// works on a block only it can see.  Otherwise they are 256 consecutive tokens of one head.
struct PairWork {
    int q0[2], h[2];
    int b, kvh;
    int lo[2], hi[2];
    int ulo, uhi;  // union of the two ranges (contiguous)
    bool live[2];  // the tile has rows below seq
    // Selected without dynamic indexing, so the struct stays in registers.
    __device__ __forceinline__ int q0_of(int s) const { return s ? q0[1] : q0[0]; }
    __device__ __forceinline__ int h_of(int s) const { return s ? h[1] : h[0]; }
    __device__ __forceinline__ int lo_of(int s) const { return s ? lo[1] : lo[0]; }
    __device__ __forceinline__ int hi_of(int s) const { return s ? hi[1] : hi[0]; }
    __device__ __forceinline__ bool live_of(int s) const { return s ? live[1] : live[0]; }
};

// ---------------------------------------------------------------------------
// Vision blocks (a query inside a block of equal non-negative ids also sees the block's later keys).  The ends are looked
// up where they are needed: a launch of its own for one end per row took 4.5 us in front of a kernel of 20.
// ---------------------------------------------------------------------------
// First key after `key` that does not carry `id`.  Whole warps, 128 keys a step.  (512 at once, asked for together with `id`, were
// 5 KB of code in every kernel of head dim 256, which calls without ids jump over: from cold caches a canvas step took 22.1 us,
// 21.4 so.  Prompts of head dim 128, which it did not burden: 3000 tokens of 16/8 heads 31.2 us with it, 29.0 so, cold 38.1 and
// 34.5; one wave of tiles in chains up to 0.4 us faster with it, warm, and 0.5 to 2.5 slower cold.)
__device__ __forceinline__ int run_end(const int* ids, int kv_len, int key, int id) {
    const int lane = threadIdx.x & 31;
    for (int k0 = key + 1;; k0 += 128) {
        bool other[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) other[i] = k0 + 32 * i + lane >= kv_len || ids[k0 + 32 * i + lane] != id;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint32_t found = __ballot_sync(0xffffffffu, other[i]);
            if (found) return k0 + 32 * i + __ffs(found) - 1;
        }
    }
}

// First key the row at key position `self` does not see.  Same position in every lane.
__device__ __forceinline__ int vision_end(const PrefillParams& p, int self) {
    const int plain = min(max(self + 1, 0), p.kv_len);
    if (self < 0 || self + 1 >= p.kv_len) return plain;  // (behind the last key there is nothing to look up)
    const int id = p.ids[self];
    return id >= 0 ? run_end(p.ids, p.kv_len, self, id) : plain;
}

// The same for a warp's 32 consecutive rows, one per lane (row: t < seq).
__device__ __forceinline__ int vision_ends(const PrefillParams& p, int self, bool row) {
    const int lane = threadIdx.x & 31;
    const int id = row && self >= 0 && self < p.kv_len ? p.ids[self] : -1;
    const int next_id = __shfl_down_sync(0xffffffffu, id, 1);  // (all lanes take part; lane 31 does not use it)
    const uint32_t breaks = __ballot_sync(0xffffffffu, lane < 31 && id != next_id);
    const int last_id = __shfl_sync(0xffffffffu, id, 31), last = __shfl_sync(0xffffffffu, self, 31);
    const int end = last_id >= 0 ? run_end(p.ids, p.kv_len, last, last_id) : 0;  // of the block that leaves the warp's rows
    if (id < 0) return min(max(self + 1, 0), p.kv_len);
    const uint32_t ahead = breaks >> lane;
    return ahead ? self + __ffs(ahead) : end;
}

// Key blocks [lo, hi) a 128-row tile starting at token qs can see.  VISION: whole warps.
template <bool VISION>
__device__ __forceinline__ void tile_blocks(const PrefillParams& p, int qs, int& blk_lo, int& blk_hi) {
    const int off = p.kv_len - p.seq;
    blk_lo = 0;
    blk_hi = (p.kv_len + PairCfg::BN - 1) / PairCfg::BN;
    if (p.mask_type == 3) {
        const int q_last = min(qs + PairCfg::BM - 1, p.seq - 1);
        const int last_key = VISION ? vision_end(p, q_last + off) - 1 : min(p.kv_len - 1, q_last + off);  // (monotone in the row)
        blk_hi = last_key >= 0 ? last_key / PairCfg::BN + 1 : 0;
        if (p.window > 0 && p.window != 0x7fffffff) blk_lo = max(0, qs + off - p.window + 1) / PairCfg::BN;
    }
    if (blk_hi < blk_lo) blk_hi = blk_lo;
}

// Every role runs this once per unit, from code that has long left the instruction caches by
// then, so it is kept short: one division at most, and nothing computed twice.
template <bool VISION>
__device__ __forceinline__ PairWork decode_pair(const PrefillParams& p, const TileCursor& cur) {
    PairWork t;
    t.b = cur.z;
    if (p.head_pair) {
        t.h[0] = cur.h * 2;
        t.h[1] = t.h[0] + 1;
        t.q0[0] = t.q0[1] = cur.qt * PairCfg::BM;
        t.kvh = p.group_shift >= 0 ? (t.h[0] >> p.group_shift) : t.h[0] / p.group;
        t.live[0] = t.live[1] = true;  // the tile list only holds tiles with rows
        tile_blocks<VISION>(p, t.q0[0], t.lo[0], t.hi[0]);
        t.lo[1] = t.ulo = t.lo[0];
        t.hi[1] = t.uhi = t.hi[0];
    } else {
        t.h[0] = t.h[1] = cur.h;
        t.q0[0] = cur.qt * 2 * PairCfg::BM;
        t.q0[1] = t.q0[0] + PairCfg::BM;
        t.kvh = p.group_shift >= 0 ? (cur.h >> p.group_shift) : cur.h / p.group;
        t.live[0] = true;
        t.live[1] = t.q0[1] < p.seq;
        tile_blocks<VISION>(p, t.q0[0], t.lo[0], t.hi[0]);
        t.lo[1] = t.hi[1] = 0;
        if (t.live[1]) tile_blocks<VISION>(p, t.q0[1], t.lo[1], t.hi[1]);
        t.ulo = 0x7fffffff;
        t.uhi = 0;
#pragma unroll
        for (int s = 0; s < 2; ++s)
            if (t.hi[s] > t.lo[s]) {
                t.ulo = min(t.ulo, t.lo[s]);
                t.uhi = max(t.uhi, t.hi[s]);
            }
    }
    if (t.uhi == 0) t.ulo = 0;
    return t;
}

// Scores of keys outside the row's visible span [lo, hi) become -inf, in registers: one bit per key of the chunk,
// so that a score costs one select.
__device__ __forceinline__ void mask_chunk(uint32_t (&v)[32], int key0, const RowMask& rm) {
    const int lo = min(max(rm.lo - key0, 0), 32), hi = min(max(rm.hi - key0, 0), 32);
    const uint32_t vis = (uint32_t)((1ull << hi) - (1ull << lo));  // bits [lo, hi); lo > hi cannot be (a span is never negative)
#pragma unroll
    for (int e = 0; e < 32; ++e) v[e] = (vis >> e) & 1u ? v[e] : 0xff800000u;
}

// 2^(score * scale - max) of one chunk (or of its columns [E0, E1)), packed to bf16x2, added up in two pairs of partial sums.  Packed fp32
// arithmetic: the pipe time is that of the scalar forms, the code is half as long.
template <int E0 = 0, int E1 = 32>
__device__ __forceinline__ void exp_chunk(const uint32_t (&v)[32], uint32_t (&pk)[16], uint64_t (&ls2)[2], uint64_t sl2,
                                          uint64_t nm2) {
#pragma unroll
    for (int e = E0; e < E1; e += 2) {
        float x0, x1;
        unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(v[e]), __uint_as_float(v[e + 1])), sl2, nm2), x0, x1);
        const float p0 = fast_exp2(x0), p1 = fast_exp2(x1);
        ls2[(e >> 1) & 1] = add_f32x2(ls2[(e >> 1) & 1], pack_f32x2(p0, p1));
        pk[e >> 1] = pack_bf16x2(p0, p1);
    }
}

// Output of a 128-row tile through shared memory.  Thread = row, so a store of a thread's 16 bytes touches 32 lines per
// warp instruction: written straight to global memory, a tile of 128 x 256 kept the accumulator and the load / store
// unit busy for 9000 clk.  Instead a warp collects its 32 rows, 64 columns a round, in one of two 4 KB buffers (128-byte
// swizzle: lanes of a quarter warp hit different banks) and hands them to TMA, whose stores clip the rows past `seq`;
// gate values come the same way, by TMA into the buffer a round ahead, and are replaced by the products in place.
constexpr int STAGE_WARP_BYTES = 8192;
constexpr int STAGE_BYTES = 4 * STAGE_WARP_BYTES;  // four epilogue warps

struct OutStage {
    uint8_t* buf;        // this warp's 2 x 4 KB, 1024-byte aligned
    uint64_t* gate_bar;  // [2] this warp's, one per buffer
    uint32_t gate_par;   // bit i: parity of buffer i's next gate load
    int h, t0, b;        // head, first of the warp's 32 rows, sequence
    int col0, rounds;    // the columns: [col0, col0 + 64 rounds) of the head
};

// Gate values of round c (columns [64 c, 64 c + 64)) into the round's buffer, which is free.  One lane.
__device__ __forceinline__ void stage_load_gate(const OutStage& s, const void* tm_gate, int c) {
    mbar_arrive_expect_tx(&s.gate_bar[c & 1], 4096);
    tma_load_4d(s.buf + (c & 1) * 4096, tm_gate, &s.gate_bar[c & 1], s.col0 + c * 64, s.h, s.t0, s.b);
}

// Once per tile, before its accumulator is waited for.
template <bool GATE>
__device__ __forceinline__ void stage_open(OutStage& s, const void* tm_gate, int lane, int h, int t0, int b) {
    s.h = h, s.t0 = t0, s.b = b;
    if (lane == 0) {
        bulk_wait_read<0>();
        if (GATE) {
            stage_load_gate(s, tm_gate, 0);
            stage_load_gate(s, tm_gate, 1);
            for (int c = 2; c < s.rounds; ++c) tma_prefetch_4d(tm_gate, s.col0 + c * 64, h, t0, b);  // (the later rounds' into L2)
        }
    }
    __syncwarp();
}

// The epilogue takes STAGE_COLS columns a turn of a rolled loop: its code runs beside the softmax loop out of the same
// instruction cache, and what does not fit beside it costs 50 clk per 128 bytes on every turn.  (Gated, 32 columns a
// turn are 6 KB of code and took 2500 clk, 16 columns 2.5 KB.  On CTA pairs, whose softmax loop is shorter, 32 gated columns are
// the better turn: 1200 clk, and 690 for 16: prefill_wide_sm100.cuh.)
template <bool GATE>
constexpr int STAGE_COLS = GATE ? 16 : 32;

// Before turn k, of N columns.  False: the gate values never came.
template <bool GATE, int N = STAGE_COLS<GATE>>
__device__ __forceinline__ bool stage_before(OutStage& s, const void* tm_gate, int lane, int k) {
    constexpr int TURNS = 64 / N;  // per round
    const int c = k / TURNS, i = c & 1;
    if (k % TURNS == 0) {
        if (GATE) {
            if (!mbar_wait_warp<2>(&s.gate_bar[i], (s.gate_par >> i) & 1u)) return false;
            s.gate_par ^= 1u << i;
        } else if (c >= 2) {
            if (lane == 0) bulk_wait_read<1>();  // round c - 2 has left the buffer
            __syncwarp();
        }
    } else if (GATE && k % TURNS == TURNS / 2 && c >= 1 && c + 1 < s.rounds) {
        if (lane == 0) {
            bulk_wait_read<0>();  // round c - 1 has left its buffer: the one of round c + 1
            stage_load_gate(s, tm_gate, c + 1);
        }
        __syncwarp();
    }
    return true;
}

// Round c of the stage is complete: sent off.
__device__ __forceinline__ void stage_send(const OutStage& s, const void* tm_out, int lane, int c) {
    fence_proxy_async_smem();
    __syncwarp();
    if (lane == 0) {
        tma_store_4d(tm_out, s.buf + (c & 1) * 4096, s.col0 + c * 64, s.h, s.t0, s.b);
        bulk_commit();
    }
}

// Turn k: the accumulator's values times `inv`, gated, as bf16 into the buffer (and into w8 for the caller); after a
// round's last turn the round is sent off.  taken(): called once acc has been used, so that the next turn's values
// can be on their way while this turn's are gated.
template <bool GATE, typename F, int N>
__device__ __forceinline__ void stage_turn(const OutStage& s, const void* tm_out, int lane, int k, const uint32_t (&acc)[N], float inv,
                                           uint32_t (&w8)[N / 2], F&& taken) {
    constexpr int TURNS = 64 / N;
    const int c = k / TURNS;
    const uint32_t row = smem_u32(s.buf) + (c & 1) * 4096 + lane * 128;
    uint32_t at[N / 8], gw[N / 2];
#pragma unroll
    for (int i = 0; i < N / 8; ++i) {
        at[i] = row + ((((k % TURNS) * (N / 8) + i) ^ (lane & 7)) << 4);
        if (GATE)
            asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(gw[4 * i]), "=r"(gw[4 * i + 1]), "=r"(gw[4 * i + 2]), "=r"(gw[4 * i + 3]) : "r"(at[i]));
    }
#pragma unroll
    for (int u = 0; u < N / 2; ++u) w8[u] = pack_bf16x2(__uint_as_float(acc[2 * u]) * inv, __uint_as_float(acc[2 * u + 1]) * inv);
    taken();
#pragma unroll
    for (int i = 0; i < N / 8; ++i) {
        if (GATE) {
            // bf16(attention) * sigmoid(gate): the rounding order of the two-launch form
#pragma unroll
            for (int u = 4 * i; u < 4 * i + 4; ++u) {
                const float a0 = __uint_as_float(w8[u] << 16), a1 = __uint_as_float(w8[u] & 0xffff0000u);
                const float g0 = __uint_as_float(gw[u] << 16), g1 = __uint_as_float(gw[u] & 0xffff0000u);
                w8[u] = pack_bf16x2(a0 * sigmoid(g0), a1 * sigmoid(g1));
            }
        }
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at[i]), "r"(w8[4 * i]), "r"(w8[4 * i + 1]), "r"(w8[4 * i + 2]), "r"(w8[4 * i + 3]) : "memory");
    }
    if (k % TURNS == TURNS - 1) stage_send(s, tm_out, lane, c);
}

// The gated epilogue and the one that also stores copies of the output are instances of their own: code the
// common kernel does not carry.
// VISION: causal with vision blocks (p.ids).
template <bool GATE, bool COPIES, bool VISION = false>
__global__ void __launch_bounds__(PairCfg::THREADS, 1)
    sdpa_prefill_pair_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                             const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_out,
                             const __grid_constant__ CUtensorMap tm_gate, const PrefillParams p) {
    using C = PairCfg;
    constexpr int HD = C::HD;
    constexpr int KS = C::K_STAGES;
    constexpr int VS = C::V_STAGES;
    extern __shared__ __align__(1024) uint8_t smem[];  // (the swizzle pattern follows the address bits)
    uint8_t* sQ = smem;                       // [2] one per pipeline
    uint8_t* sK = smem + 2 * C::TILE_BYTES;   // [KS]
    uint8_t* sV = sK + KS * C::TILE_BYTES;    // [VS]
    uint8_t* sOut = sV + VS * C::TILE_BYTES;  // output stage
    uint64_t* bars = reinterpret_cast<uint64_t*>(sOut + STAGE_BYTES);
    uint64_t* q_full = bars;         // [2]
    uint64_t* q_empty = bars + 2;    // [2] the tile's last S = Q K^T has completed
    uint64_t* k_first = bars + 4;       // the first key block's K
    uint64_t* k_first_used = bars + 5;  // both pipelines' first scores have been computed
    uint64_t* kv_full = bars + 6;       // [2] V of a block and K of the block after it
    uint64_t* kv_empty = bars + 8;      // [2] both have been used by both pipelines
    uint64_t* s_free = kv_empty + 2; // the softmax warps of the pipeline that has had the scores last hold them in registers
    uint64_t* s_full = s_free + 1;   // [2] per pipeline from here on
    uint64_t* p_part = s_full + 2;   // [pipeline][part]: P of keys 0-95 / 96-127 of the block is in tensor memory
    uint64_t* pv_done = p_part + 4;  // O += P V of the block has completed: P may be replaced, O rescaled
    uint64_t* o_full = pv_done + 2;  // one phase per tile: the tile's last O += P V has completed
    uint64_t* o_empty = o_full + 2;  // one phase per tile: the epilogue warps have read O out
    // fin[2 * s + (tile & 1)], one phase per second tile: the softmax warps have published the tile's row sums.  Two barriers per pipeline, used in turn, because a tile of one key block needs no
    // O += P V to finish: with one barrier the softmax warps could complete it for tile n + 1 while a slow
    // epilogue (stores held up) still waits for tile n's completion — and a parity wait cannot tell "twice"
    // from "not yet".  They cannot reach tile n + 2 before the epilogue has taken tile n (the first O += P V
    // of tile n + 1 waits for that), so two are enough.
    uint64_t* fin = o_empty + 2;
    uint64_t* gate_bar = fin + 4;    // [epilogue warp][buffer]
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + C::NUM_BARS);
    uint32_t* abort_slot = tmem_slot + 1;
    float* fin_vals = reinterpret_cast<float*>(tmem_slot + 4);  // [tile parity 2][pipeline 2][row 128] row sum
    TileCursor* cursor = reinterpret_cast<TileCursor*>(fin_vals + C::FIN_FLOATS);  // the CTA's first unit

    // (broadcast, so that the compiler knows them to be the same in every lane and keeps what follows from them —
    // MMA descriptors above all — in uniform registers)
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);
    const int lane = threadIdx.x & 31;

    if (threadIdx.x == 32) {
        prefetch_tensormap(&tm_q);
        prefetch_tensormap(&tm_k);
        prefetch_tensormap(&tm_v);
    }
    if (threadIdx.x == 0) {
        for (int s = 0; s < 2; ++s) {
            mbar_init(&q_full[s], 1);
            mbar_init(&q_empty[s], 1);
            mbar_init(&s_full[s], 1);
            mbar_init(&p_part[2 * s], 4);
            mbar_init(&p_part[2 * s + 1], 4);
            mbar_init(&pv_done[s], 1);
            mbar_init(&o_full[s], 1);
            mbar_init(&o_empty[s], 4);
            mbar_init(&fin[2 * s], 4);
            mbar_init(&fin[2 * s + 1], 4);
        }
        for (int w = 0; w < 8; ++w) mbar_init(&gate_bar[w], 1);
        mbar_init(k_first, 1);
        mbar_init(k_first_used, 1);
        mbar_init(s_free, 4);
        for (int s = 0; s < 2; ++s) {
            mbar_init(&kv_full[s], 1);
            mbar_init(&kv_empty[s], 2);
        }
        fence_mbar_init();
    }
    if (warp == C::PRODUCER_WARP) {
        tmem_alloc(tmem_slot, C::TMEM_COLS);
        tmem_relinquish();
    }
    static_assert(sizeof(TileCursor) <= 80, "the first unit's place in shared memory");
    // (the divisions, once and ahead of the wait: they took 1000 clk between the kernel's release and its first load)
    if (threadIdx.x == 0) {
        TileCursor cur;
        cur.init(p);
        *cursor = cur;
    }
    // Up to here nothing depends on the kernels in front; everything below may.  A launch behind this one (the
    // single-head tail of the unit list) may be scheduled from then on, as SMs free up.
    grid_dependency_wait();
    grid_launch_dependents();
    if (threadIdx.x == 0) *abort_slot = *reinterpret_cast<volatile uint32_t*>(p.fault) != 0u ? 1u : 0u;
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, *reinterpret_cast<volatile uint32_t*>(tmem_slot), 0);
    const int total_tiles = *abort_slot ? 0 : p.total_tiles;  // a status is set: walk an empty list
    constexpr uint32_t TILE16 = C::TILE_BYTES >> 4, CHUNK16 = C::CHUNK_BYTES >> 4;  // descriptor units

    if (warp >= C::PRODUCER_WARP) {
        reg_dealloc<C::REGS_CONTROL>();
        if (warp == C::PRODUCER_WARP) {
            // -------------------------------------------------------------- TMA producer of K and V
            // One stage holds what one step of the issuer takes: V of a key block and K of the block after it — in
            // the next unit, if the block is a unit's last.  K of the very first block comes on its own.
            int r = 0;  // ring position: key blocks whose K has been requested
            bool ok = true;
            auto load = [&](uint8_t* dst, const void* tm, uint64_t* bar, const PairWork& pw, int j) {
#pragma unroll
                for (int c = 0; c < C::CH; ++c)
                    tma_load_4d_warp(dst + c * C::CHUNK_BYTES, tm, bar, c * 64, pw.kvh, j * C::BN, pw.b);
            };
            TileCursor cur = *cursor;
            PairWork last{};  // unit and index of the block requested last
            int last_j = 0;
            for (; ok && cur.w < total_tiles; cur.advance(p)) {
                const PairWork pw = decode_pair<VISION>(p, cur);
                for (int j = pw.ulo; ok && j < pw.uhi; ++j, ++r) {
                    if (r == 0) {
                        if (lane == 0) mbar_arrive_expect_tx(k_first, C::TILE_BYTES);
                        __syncwarp();
                        load(sK, &tm_k, k_first, pw, j);
                    } else {
                        // V of block r - 1 and K of block r; both stages were used by step r - 3 (the first K by the
                        // scores in front of all steps)
                        uint64_t* full = &kv_full[(r - 1) & 1];
                        const bool free = r < 2    ? true
                                          : r == 2 ? mbar_wait_inline(k_first_used, 0u)
                                                   : mbar_wait_inline(&kv_empty[(r - 1) & 1], (((r - 1) >> 1) - 1) & 1);
                        if (!free) {
                            if (lane == 0) report_fault(p.fault, FAULT_WAIT_EMPTY, 0x100u);
                            ok = false;
                            break;
                        }
                        if (lane == 0) mbar_arrive_expect_tx(full, 2 * C::TILE_BYTES);
                        __syncwarp();
                        load(sV + ((r - 1) & 1) * C::TILE_BYTES, &tm_v, full, last, last_j);
                        load(sK + (r & 1) * C::TILE_BYTES, &tm_k, full, pw, j);
                    }
                    last = pw;
                    last_j = j;
                }
            }
            if (ok && r > 0) {  // V of the last block of all
                uint64_t* full = &kv_full[(r - 1) & 1];
                if (r >= 3 && !mbar_wait_inline(&kv_empty[(r - 1) & 1], (((r - 1) >> 1) - 1) & 1)) {
                    if (lane == 0) report_fault(p.fault, FAULT_WAIT_EMPTY, 0x200u);
                } else {
                    if (lane == 0) mbar_arrive_expect_tx(full, C::TILE_BYTES);
                    __syncwarp();
                    load(sV + ((r - 1) & 1) * C::TILE_BYTES, &tm_v, full, last, last_j);
                }
            }
        } else if (warp == C::Q_PRODUCER_WARP) {
            // -------------------------------------------------------------- TMA producer of Q
            // A thread of its own: the next unit's Q tiles are requested the moment the current tiles'
            // last scores are out, whatever the K / V producer is waiting for at that time.
            if (VISION || lane == 0) {  // (the look-up of vision blocks takes the whole warp)
                if (lane == 0) prefetch_tensormap(&tm_q);
                int tq0 = 0, tq1 = 0;  // tiles with key blocks loaded so far, per pipeline
                bool ok = true;
                TileCursor cur = *cursor;
                for (; ok && cur.w < total_tiles; cur.advance(p)) {
                    const PairWork pw = decode_pair<VISION>(p, cur);
#pragma unroll
                    for (int s = 0; s < 2; ++s) {
                        if (pw.hi[s] == pw.lo[s]) continue;
                        int& tq = s ? tq1 : tq0;
                        if (tq > 0 && !(VISION ? mbar_wait_inline(&q_empty[s], (tq - 1) & 1) : mbar_wait<1>(&q_empty[s], (tq - 1) & 1))) {
                            if (lane == 0) report_fault(p.fault, FAULT_WAIT_EMPTY, 0x300u + s);
                            ok = false;
                            break;
                        }
                        if (lane == 0) {
                            mbar_arrive_expect_tx(&q_full[s], C::TILE_BYTES);
#pragma unroll
                            for (int c = 0; c < C::CH; ++c)
                                tma_load_4d(sQ + s * C::TILE_BYTES + c * C::CHUNK_BYTES, &tm_q, &q_full[s], c * 64, pw.h[s],
                                            pw.q0[s], pw.b);
                        }
                        ++tq;
                    }
                    // The unit after this one: its Q rows (one 256-byte piece per token, far apart in
                    // memory) are asked into L2 now, a whole unit ahead of the load that needs them.
                    TileCursor nx = cur;
                    nx.advance(p);
                    if (ok && !VISION && nx.w < total_tiles) {
                        const PairWork pn = decode_pair<false>(p, nx);
#pragma unroll
                        for (int s = 0; s < 2; ++s) {
                            if (pn.hi[s] == pn.lo[s]) continue;
#pragma unroll
                            for (int c = 0; c < C::CH; ++c) tma_prefetch_4d(&tm_q, c * 64, pn.h[s], pn.q0[s], pn.b);
                        }
                    }
                }
            }
        } else if (warp == C::S_ISSUER_WARP) {
            // -------------------------------------------------------------- S = Q K^T of both pipelines
            // The whole warp runs this code and one lane issues: addresses stay in the uniform datapath.
            //
            // The pipelines' scores go through the one buffer in turn: a pipeline's next scores are computed as soon as
            // the other one's softmax warps have taken theirs into registers, which they do when they are through with
            // the block before.  So A's scores of block j + 1 are computed while A exponentiates block j and are there
            // when it is done, and the two are half a period apart by themselves.
            constexpr uint32_t IDESC_QK = make_idesc_bf16(128, 128, false);
            const uint64_t dQ = make_smem_desc_sw128(smem_u32(sQ), 16, 1024);
            const uint64_t dK = make_smem_desc_sw128(smem_u32(sK), 16, 1024);
            static_assert(KS == 2 && VS == 2 && HD == 128, "ring arithmetic assumes two stages and head dim 128");
            int r = 0;            // ring position: key blocks so far
            int ns = 0;           // score blocks so far, of both pipelines
            uint32_t q_par = 0u;  // bit s: parity of pipeline s's tiles so far
            bool ok = true;
            TileCursor cur = *cursor;
            for (; ok && cur.w < total_tiles; cur.advance(p)) {
                const PairWork pw = decode_pair<VISION>(p, cur);
                for (int j = pw.ulo; ok && j < pw.uhi; ++j, ++r) {
                    if (!mbar_wait_inline(r ? &kv_full[(r - 1) & 1] : k_first, r ? ((r - 1) >> 1) & 1 : 0)) {
                        if (lane == 0) report_fault(p.fault, FAULT_WAIT_K, r);
                        ok = false;
                        break;
                    }
#pragma unroll 1
                    for (int s = 0; s < 2; ++s) {
                        if (j < pw.lo_of(s) || j >= pw.hi_of(s)) continue;
                        if (j == pw.lo_of(s)) {
                            if (!mbar_wait_inline(&q_full[s], (q_par >> s) & 1u)) {
                                if (lane == 0) report_fault(p.fault, FAULT_WAIT_Q, s);
                                ok = false;
                                break;
                            }
                            q_par ^= 1u << s;
                        }
                        const uint64_t da = dQ + (uint64_t)(s * TILE16), db = dK + (uint64_t)((r & 1) * TILE16);
                        if (ns > 0 && !mbar_wait_inline(s_free, (ns - 1) & 1)) {
                            if (lane == 0) report_fault(p.fault, FAULT_WAIT_S, 0x1000u + ns);
                            ok = false;
                            break;
                        }
                        ++ns;
                        tc_fence_after_sync();
                        umma_ss_x4<2, 2>(tmem_base + C::COL_S, da, db, IDESC_QK, 0u);  // 64 head-dim columns
                        umma_ss_x4<2, 2>(tmem_base + C::COL_S, da + CHUNK16, db + CHUNK16, IDESC_QK, 1u);
                        umma_commit_warp(&s_full[s]);
                        if (j + 1 == pw.hi_of(s)) umma_commit_warp(&q_empty[s]);
                    }
                    umma_commit_warp(r ? &kv_empty[(r - 1) & 1] : k_first_used);
                }
            }
        } else {
            // -------------------------------------------------------------- O += P V of both pipelines
            constexpr uint32_t IDESC_PV = make_idesc_bf16(128, HD, true);
            const uint64_t dV = make_smem_desc_sw128(smem_u32(sV), C::CHUNK_BYTES, 1024);
            int r = 0;             // ring position: key blocks so far
            uint32_t g_par = 0u;   // bit s: parity of pipeline s's key blocks so far
            uint32_t o_par = 3u;   // bit s: parity to wait for before its next tile's first P V (starts "complete")
            bool ok = true;
            TileCursor cur = *cursor;
            for (; ok && cur.w < total_tiles; cur.advance(p)) {
                const PairWork pw = decode_pair<VISION>(p, cur);
                for (int j = pw.ulo; ok && j < pw.uhi; ++j, ++r) {
                    if (!mbar_wait_inline(&kv_full[r & 1], (r >> 1) & 1)) {
                        if (lane == 0) report_fault(p.fault, FAULT_WAIT_V, r);
                        ok = false;
                        break;
                    }
#pragma unroll 1
                    for (int s = 0; s < 2; ++s) {
                        if (j < pw.lo_of(s) || j >= pw.hi_of(s)) continue;
                        if (j == pw.lo_of(s)) {
                            if (!mbar_wait_inline(&o_empty[s], (o_par >> s) & 1u)) {
                                if (lane == 0) report_fault(p.fault, FAULT_WAIT_O, 0x100u + s);
                                ok = false;
                                break;
                            }
                            o_par ^= 1u << s;
                        }
                        // P from tensor memory: 16 keys are 8 columns of packed bf16.  V is MN-major:
                        // 64-element head-dim chunks 16 KB apart, 8-key groups 1024 bytes apart; 16 keys =
                        // 2048 bytes.  The first 96 keys go to the tensor pipe while the softmax warps are
                        // still busy with the other 32.
                        const uint32_t tO = tmem_base + C::COL_O + s * 128, tP = tmem_base + C::COL_P + s * 64;
                        const uint64_t dv = dV + (uint64_t)((r & 1) * TILE16);
                        const uint32_t par = (g_par >> s) & 1u;
                        if (!mbar_wait_inline(&p_part[2 * s], par)) {
                            if (lane == 0) report_fault(p.fault, FAULT_WAIT_P, r);
                            ok = false;
                            break;
                        }
                        tc_fence_after_sync();
                        umma_ts_x4<8, 128>(tO, tP, dv, IDESC_PV, j > pw.lo_of(s) ? 1u : 0u);
                        umma_ts_x2<8, 128>(tO, tP + 32, dv + 512, IDESC_PV, 1u);
                        if (!mbar_wait_inline(&p_part[2 * s + 1], par)) {
                            if (lane == 0) report_fault(p.fault, FAULT_WAIT_P, 0x1000u + r);
                            ok = false;
                            break;
                        }
                        tc_fence_after_sync();
                        umma_ts_x2<8, 128>(tO, tP + 48, dv + 768, IDESC_PV, 1u);
                        g_par ^= 1u << s;
                        umma_commit_warp(&pv_done[s]);
                        if (j + 1 == pw.hi_of(s)) umma_commit_warp(&o_full[s]);
                    }
                    umma_commit_warp(&kv_empty[r & 1]);
                }
            }
        }
    } else if (warp >= C::EPILOGUE_WARP) {
        // ------------------------------------------------------------------ epilogue
        // Thread = query row (TMEM lane); tiles A and B of every unit in turn.  The accumulator is
        // released as soon as it is in registers, normally before the next tile's first P is ready.
        reg_dealloc<C::REGS_EPILOGUE>();
        const int quarter = warp & 3;
        const int r = quarter * 32 + lane;
        const uint32_t lane_sel = static_cast<uint32_t>(quarter * 32) << 16;
        int tq0 = 0, tq1 = 0;  // tiles with key blocks so far, per pipeline
        bool ok = true;
        OutStage stage{sOut + quarter * STAGE_WARP_BYTES, &gate_bar[2 * quarter], 0u, 0, 0, 0, 0, HD / 64};
        TileCursor cur = *cursor;
        for (; ok && cur.w < total_tiles; cur.advance(p)) {
            const PairWork pw = decode_pair<VISION>(p, cur);
#pragma unroll 1
            for (int s = 0; s < 2 && ok; ++s) {
                const int t0 = pw.q0_of(s) + quarter * 32, t = t0 + lane, h = pw.h_of(s);
                const bool store = pw.live_of(s) && t < p.seq;
                const bool warp_store = pw.live_of(s) && t0 < p.seq;  // some row of the warp is stored
                const long long row = ((long long)pw.b * p.seq + t) * p.nq + h;
                const long long eoff = pw.b * p.o_stride_b + t * p.o_stride_t + (long long)h * HD;
                if (pw.hi_of(s) == pw.lo_of(s)) {
                    // Nothing visible for this tile: zero output.
                    if (store) {
                        for (int c = -1; c < (COPIES ? p.n_copies : 0); ++c) {
                            uint4* dst = reinterpret_cast<uint4*>((c < 0 ? p.out : reinterpret_cast<uint16_t*>(p.out_copies[c])) + eoff);
                            for (int i = 0; i < HD / 8; ++i) dst[i] = make_uint4(0u, 0u, 0u, 0u);
                        }
                        if (p.out_lse) p.out_lse[row] = -CUDART_INF_F;
                    }
                    continue;
                }
                if (warp_store) stage_open<GATE>(stage, &tm_gate, lane, h, t0, pw.b);
                const int tq = s ? tq1 : tq0;
                if (!mbar_wait_warp<2>(&fin[2 * s + (tq & 1)], (tq >> 1) & 1)) {
                    report_fault(p.fault, FAULT_WAIT_FULL, 0x500u + s);
                    ok = false;
                    break;
                }
                const float row_l = fin_vals[((tq & 1) * 2 + s) * 128 + r];
                if (!mbar_wait_warp<2>(&o_full[s], tq & 1)) {
                    report_fault(p.fault, FAULT_WAIT_O, tq);
                    ok = false;
                    break;
                }
                tc_fence_after_sync();
                if (s) ++tq1; else ++tq0;
                const float inv = row_l > 0.f ? 1.0f / row_l : 0.f;
                const uint32_t tO = tmem_base + lane_sel + C::COL_O + s * 128;
                constexpr int SC = STAGE_COLS<GATE>;
                uint32_t wa[SC], w8[SC / 2];
                tmem_ld(tO, wa);
#pragma unroll 1
                for (int c = 0; c < HD / SC; ++c) {
                    if (warp_store && !stage_before<GATE>(stage, &tm_gate, lane, c)) {
                        report_fault(p.fault, FAULT_WAIT_FULL, 0x600u + s);
                        ok = false;
                        break;
                    }
                    tmem_wait_ld();
                    if (c + 1 == HD / SC) {  // O is in registers: the next unit may overwrite the accumulator
                        tc_fence_before_sync();
                        mbar_arrive_warp(&o_empty[s]);
                    }
                    auto next = [&]() {
                        if (c + 1 < HD / SC) tmem_ld(tO + (c + 1) * SC, wa);
                    };
                    if (!warp_store) next();
                    if (warp_store) {
                        stage_turn<GATE>(stage, &tm_out, lane, c, wa, inv, w8, next);
                        if (COPIES && store) {
                            for (int k = 0; k < p.n_copies; ++k) {
                                uint4* d4 = reinterpret_cast<uint4*>(reinterpret_cast<uint16_t*>(p.out_copies[k]) + eoff + c * SC);
#pragma unroll
                                for (int i = 0; i < SC / 8; ++i) d4[i] = make_uint4(w8[4 * i], w8[4 * i + 1], w8[4 * i + 2], w8[4 * i + 3]);
                            }
                        }
                    }
                }
            }
        }
        if (lane == 0) bulk_wait_read<0>();  // the stage may go when its last rows have been read
    } else {
        // ------------------------------------------------------------------ softmax
        // Warps 0-3 serve tile A, warps 4-7 tile B; a thread owns one query row and takes its 128
        // scores of a block out of tensor memory once.
        reg_alloc<C::REGS_SOFTMAX>();
        const int s = warp >> 2;
        const int quarter = warp & 3;
        const int r = quarter * 32 + lane;
        const uint32_t lane_sel = static_cast<uint32_t>(quarter * 32) << 16;
        const uint32_t tS = tmem_base + lane_sel + C::COL_S;
        const uint32_t tP = tmem_base + lane_sel + C::COL_P + s * 64;
        const uint32_t tO = tmem_base + lane_sel + C::COL_O + s * 128;
        const float sl = p.scale_log2;
        const bool causal = (p.mask_type == 3);
        const bool windowed = causal && p.window > 0 && p.window != 0x7fffffff;
        const int off = p.kv_len - p.seq;

        int g = 0, tq = 0;  // key blocks and tiles (with key blocks) of this pipeline so far
        bool ok = true;
        const uint64_t sl2 = pack_f32x2(sl, sl);
        uint32_t s0[32], s1[32], s2[32], s3[32];  // the row's 128 scores of the current block

        TileCursor cur = *cursor;
        for (; ok && cur.w < total_tiles; cur.advance(p)) {
            const PairWork pw = decode_pair<VISION>(p, cur);
            if (pw.uhi == pw.ulo) continue;
            const int t = pw.q0_of(s) + r;
            const int lo = pw.lo_of(s), hi = pw.hi_of(s);
            int row_lo = 0, row_hi = p.kv_len;  // visible keys [row_lo, row_hi)
            if (causal) {
                const int diag = t + off;
                row_hi = min(max(diag + 1, 0), p.kv_len);
                if (VISION) row_hi = vision_ends(p, diag, t < p.seq);
                if (windowed) row_lo = max(0, diag - p.window + 1);
                if (row_lo > row_hi) row_lo = row_hi;
            }
            const RowMask rm{row_lo, row_hi};

            float m = -CUDART_INF_F;  // running max, log2 domain, possibly stale by <= 8
            float l = 0.f;            // row sum
            for (int j = lo; j < hi; ++j, ++g) {
                const int kc = j * C::BN;
                if (!mbar_wait_warp<3>(&s_full[s], g & 1)) {
                    report_fault(p.fault, FAULT_WAIT_S, g);
                    ok = false;
                    break;
                }
                tc_fence_after_sync();
                const bool full = __all_sync(0xffffffffu, rm.lo <= kc && kc + C::BN <= rm.hi);
                float mr[4] = {-CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F};
                tmem_ld32(tS, s0);
                tmem_ld32(tS + 32, s1);
                tmem_wait_ld();
                tmem_ld32(tS + 64, s2);  // lands while the maximum of the first half is taken
                tmem_ld32(tS + 96, s3);
                if (!full) {  // window edge, diagonal, ragged end (two blocks in nine with a 1024-key window)
                    mask_chunk(s0, kc, rm);
                    mask_chunk(s1, kc + 32, rm);
                }
                chunk_max(s0, mr);
                chunk_max(s1, mr);
                tmem_wait_ld();
                tc_fence_before_sync();
                mbar_arrive_warp(s_free);  // the buffer may take the other pipeline's scores
                if (!full) {
                    mask_chunk(s2, kc + 64, rm);
                    mask_chunk(s3, kc + 96, rm);
                }
                chunk_max(s2, mr);
                chunk_max(s3, mr);
                const float m_new = fmaxf(m, fmaxf(fmaxf(mr[0], mr[1]), fmaxf(mr[2], mr[3])) * sl);
                // O += P V of the block before has long completed, as a rule: its P may be replaced.
                if (g > 0 && !mbar_wait_warp<3>(&pv_done[s], (g - 1) & 1)) {
                    report_fault(p.fault, FAULT_WAIT_O, 0x200u + g);
                    ok = false;
                    break;
                }
                tc_fence_after_sync();
                const bool need = m_new > m + 8.0f;
                if (j == lo) {
                    m = m_new;
                } else if (__any_sync(0xffffffffu, need)) {
                    // Rare: some row's maximum grows by more than 2^8: rescale those rows of O in tensor memory.
                    const float alpha = need ? fast_exp2(m - m_new) : 1.0f;
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
                // Probabilities as bf16, packed in the pipeline's 64 columns for P; row sum in fp32.
                // The first 96 keys are announced half a chunk late: by then their stores have landed and the wait
                // for them costs nothing, and their share of O += P V still runs beside the rest.
                const float m_eff = (m == -CUDART_INF_F) ? 0.f : m;
                const uint64_t nm2 = pack_f32x2(-m_eff, -m_eff);
                uint64_t ls2[2] = {0ull, 0ull};
                uint32_t pk[16];
                exp_chunk(s0, pk, ls2, sl2, nm2);
                tmem_st16(tP, pk);
                exp_chunk(s1, pk, ls2, sl2, nm2);
                tmem_st16(tP + 16, pk);
                exp_chunk(s2, pk, ls2, sl2, nm2);
                tmem_st16(tP + 32, pk);
                exp_chunk<0, 16>(s3, pk, ls2, sl2, nm2);
                tmem_wait_st();
                tc_fence_before_sync();
                mbar_arrive_warp(&p_part[2 * s]);
                exp_chunk<16, 32>(s3, pk, ls2, sl2, nm2);
                tmem_st16(tP + 48, pk);
                float l0, l1, l2, l3;
                unpack_f32x2(ls2[0], l0, l1);
                unpack_f32x2(ls2[1], l2, l3);
                l += (l0 + l1) + (l2 + l3);
                tmem_wait_st();
                tc_fence_before_sync();
                mbar_arrive_warp(&p_part[2 * s + 1]);
            }
            if (ok && hi > lo) {
                // The tile's last key block is on its way: hand the row sum to the epilogue warps and go on with
                // the next tile.
                fin_vals[((tq & 1) * 2 + s) * 128 + r] = l;
                if (p.out_lse && pw.live_of(s) && t < p.seq)
                    p.out_lse[((long long)pw.b * p.seq + t) * p.nq + pw.h_of(s)] =
                        l > 0.f ? (m + fast_log2(l)) * 0.6931471805599453f : -CUDART_INF_F;
                mbar_arrive_warp(&fin[2 * s + (tq & 1)]);
                ++tq;
            }
        }
    }

    tc_fence_before_sync();
    __syncthreads();
    if (warp == C::PRODUCER_WARP) tmem_dealloc(tmem_base, C::TMEM_COLS);
}

}  // namespace arc
