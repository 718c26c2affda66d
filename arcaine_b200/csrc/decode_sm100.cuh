// HBM-bound split-KV decode kernel for sm_100a, plus the log-sum-exp merges.
//
// One new query token per sequence attends to that sequence's contiguous KV
// cache rows of (nkv, hd) bf16 (the reference's per-layer cache,
// src/modeling/qwen3_5/cache.hpp:9-14).  The key ranges of all sequences are
// laid end to end and cut into one equal share per CTA (persistent grid, one CTA
// per SM), so the load is balanced whatever the per-sequence lengths are and a
// CTA streams one long contiguous run of cache rows.
//
// Inside a CTA a producer warp streams the cache through a ring of
// shared-memory stages with TMA: the K and V caches are described as 2-D tensors
// (row = one position, all KV heads), and one copy moves a 64-element column
// chunk of a whole stage of rows (16-64 rows, 2-8 KB) with the 128-byte swizzle,
// so ldmatrix reads are bank-conflict free without padding and the copy engine
// sees few, large requests.  Consumer warps each own one KV head
// and a 16-key slice of every stage.  The GQA group of that head (<= 8 query
// heads per n-tile) forms the N dimension of the warp MMAs, so K and V are read
// from HBM and from shared memory exactly once per group:
//     S^T (16 keys x 8 heads) = K_tile (16 x hd) * Q^T (hd x 8)
//     O^T (hd x 8 heads)     += V_tile^T (hd x 16) * P^T (16 x 8)
// Online softmax state (max, sum) is per head = per accumulator column pair,
// reduced across the key rows with warp shuffles.  Each (CTA, sequence) pair a
// share touches yields partial (normalised out, lse) records: one per slice, or —
// for the last segment of a share, which is most of them — one for the CTA, the
// slices folded through shared memory first; the merge kernel folds the records
// and applies the optional sigmoid output gate
// (src/modeling/qwen3_5_moe/kernels.hpp:80-88) while writing bf16.
//
// The reference kernels this replaces read K/V once per query head and never
// split the key range (src/modeling/qwen3_5/kernels.hpp:761-905), or fold the
// group into the MMA rows but launch only nkv*4 work-groups (:910-1054).
#pragma once
#include <cuda.h>
#include <math_constants.h>

#include "ptx.cuh"

namespace arc {

constexpr int DECODE_MAX_BATCH = 2048;

struct DecodeParams {
    const uint16_t* q;
    const int* kv_len;
    const long long* kv_row_offset;
    float* part_o;    // [(slot * slices + slice)][nq][HD]
    float* part_lse;  // [(slot * slices + slice)][nq]
    uint32_t* fault;
    int batch, nq, nkv, kv_len_uniform;
    long long q_stride_b, kv_stride_b, kv_stride_t;
    float scale_log2;
    int nkv_cta;  // KV heads handled by one CTA (grid.y = nkv / nkv_cta)
    int slices;   // 16-key slices per stage; consumer warps = nkv_cta * slices
    int stages;
    int ncta;     // grid.x
    int max_kv_len;            // > 0: no sequence may be longer
    long long kv_rows_total;   // rows addressable from k and v
    // The form that finishes in one launch (sdpa_decode_kernel<.., true>): the results
    const uint16_t* gate;
    uint16_t* out;
    float* out_f32;
    float* out_lse;
    long long o_stride_b;
};

// Prefix sums of the per-sequence lengths into shared memory: cum[b] = keys before sequence b, cum[batch] = total.
// Called by the first warp, which scans 32 sequences a step (one thread adding them up in turn took a microsecond for
// 64); the caller's barrier follows.
template <typename F>
__device__ __forceinline__ void build_len_prefix(int batch, long long* cum, F&& len_of) {
    long long run = 0;
    if (threadIdx.x == 0) cum[0] = 0;
    for (int b0 = 0; b0 < batch; b0 += 32) {
        const int b = b0 + threadIdx.x;
        const int len = b < batch ? len_of(b) : 0;
        long long v = len > 0 ? len : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const long long up = __shfl_up_sync(0xffffffffu, v, o);
            if ((int)threadIdx.x >= o) v += up;
        }
        if (b < batch) cum[b + 1] = run + v;
        run += __shfl_sync(0xffffffffu, v, 31);
    }
}

__device__ __forceinline__ long long share_size(long long total, int ncta, int tile_keys) {
    if (total < (1ll << 30)) {  // (a 64-bit division takes some hundred clk, and every role waits for this one)
        const uint32_t per = ((uint32_t)total + ncta - 1) / (uint32_t)ncta;
        return max(1u, (per + tile_keys - 1) / (uint32_t)tile_keys) * tile_keys;
    }
    const long long per = (total + ncta - 1) / ncta;
    return (per + tile_keys - 1) / tile_keys * tile_keys;
}

__device__ __forceinline__ float sigmoid_gate(float attn, uint16_t gate_bits) {
    const float g = bf16_bits_to_f32(gate_bits);
    return bf16_round(attn) * sigmoid(g);
}

// All consumer warps of the CTA (named barrier 1; the producer warp does not take part).
__device__ __forceinline__ void consumer_sync(int consumer_warps) {
    asm volatile("bar.sync 1, %0;" ::"r"(consumer_warps * 32) : "memory");
}

// CLUSTER: a cluster of CTAs owns one sequence (grid.z) and one group of KV heads (grid.y); its CTAs take a step of the
// sequence's keys each, in order, and equal parts of the rest, fold their slices as above, send the records to the shared memory of the CTAs that finish them
// and write the result: one launch, no records in global memory, no merge kernel.  For calls so small that the
// launches are what they cost; otherwise equal shares over all SMs win.
// What bounds it: a chain of latencies, and behind the last key instructions that run once, fetched cold at 6 clk each.  One token
// of 24/4 heads over 513 keys: 600 clk to the lengths, 1400 to the keys, 1250 for them, and it was 7000 from there to the result
// with records normalised and weighted by their log-sum-exps twice and a barrier of the cluster in between.  Records that travel
// as they are, weights worked out by eight lanes a row, rolled loops and stores that count themselves on an mbarrier of the CTA they
// go to (st.async) take half of that (us): that call 6.2 -> 5.3, 1001 keys 6.7 -> 5.5, 20 sequences of 780 keys 20.3 -> 18.4, 64 of
// 100 to 512 keys, 16/2 heads of 128, 9.0 -> 8.1, twelve of up to 6000 12.3 -> 11.8.
// A CTA's first keys are asked for while the lengths are: they do not depend on them (1630 clk to the lengths when they are on the
// device; us: 16 sequences of 500 keys, 8/4 heads of 128, 6.6 -> 5.9, 32 of 64 to 400, 24/4 of 256, 12.9 -> 11.9, twelve of up to 6000,
// 16/2 of 128, 11.8 -> 11.2, one token over 513 keys 5.34 -> 5.1).  The scores ahead of V, on a barrier of its own, brought nothing.
// ALONE (of CLUSTER): one CTA, which is not launched as a cluster.  (Clusters of a power of two, all of whose CTAs finish columns, had an
// instance of their own with it while records were folded another way; now they are faster as a case of the general one, us: one token of
// 24/4 heads over 256 / 513 / 1001 keys 4.62 / 5.21 / 5.50 -> 4.47 / 5.11 / 5.42, 16 sequences of 500 keys, 8/4 heads of 128, 5.80 -> 5.65.)
template <int HD, int NT, bool CLUSTER, bool ALONE = false>
__global__ void __launch_bounds__(288, 1)
    sdpa_decode_kernel(const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v,
                       const DecodeParams p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));

    const int ncw = p.nkv_cta * p.slices;  // consumer warps
    const int tk = 16 * p.slices;          // keys per stage
    const int row_bytes = p.nkv_cta * HD * 2;
    const int nchunks = p.nkv_cta * (HD / 64);  // 64-element column chunks per row
    const int chunk_bytes = tk * 128;           // one chunk of one stage: tk rows x 128 bytes
    const int tile_bytes = tk * row_bytes;      // one of K / V
    const int stage_bytes = 2 * tile_bytes;

    uint8_t* stage_base = smem;
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + (size_t)p.stages * stage_bytes);
    uint64_t* empty = full + p.stages;
    long long* cum = reinterpret_cast<long long*>(empty + p.stages);

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int head0 = blockIdx.y * p.nkv_cta;  // first KV head of this CTA
    const int G = p.nq / p.nkv;
    // CLUSTER: the first 2^k CTAs of the cluster (all of 1, 2, 4 or 8, four of six) finish an equal number of columns of all
    // heads each.  All CTAs send them what they have, weights still to come: per CTA [query head of the group][column], in front
    // of them [CTA][query head] maximum (log2 domain) and sum, and whether all of the CTA's waits ended well.
    const int dc_log2 = (HD == 256 ? 8 : 7) - (CLUSTER && !ALONE ? 31 - __clz(p.ncta) : 0), dc = 1 << dc_log2;
    const int finishers = HD >> dc_log2;
    const int rows = p.nkv_cta * G, rows2 = (rows + 1) & ~1;
    uint64_t* gathered = empty + p.stages;
    int* gave_up = reinterpret_cast<int*>(gathered + 1);
    float* cflag = reinterpret_cast<float*>(gathered + 2);     // [8]
    float2* cml = reinterpret_cast<float2*>(cflag + 8);         // [8][rows2]
    float* crec = reinterpret_cast<float*>(cml + 8 * rows2);    // [CTA][rows][dc]
    float* cweight = crec + (size_t)p.ncta * rows * dc;         // [rows][8]

    if (threadIdx.x == 32) {
        prefetch_tensormap(&tm_k);
        prefetch_tensormap(&tm_v);
    }
    if (threadIdx.x == 0) {
        for (int s = 0; s < p.stages; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], ncw);
        }
        if constexpr (CLUSTER) {  // what the other CTAs send here, if this one finishes columns
            mbar_init(gathered, 1);
            *gave_up = 0;
        }
        fence_mbar_init();
        if (CLUSTER) mbar_arrive_expect_tx(gathered, (uint32_t)(p.ncta * (4 + rows * (8 + dc * 4))));
    }
    long long g0 = 0, g1 = 0;  // this CTA's keys, counted over the sequences laid end to end (CLUSTER: of its own sequence)
    int b_first = 0, my_len = 0;
    // CLUSTER: a CTA's first step begins at key blockIdx.x * tk, whatever the length, so that its keys are asked for before the length
    // has been looked at; what is left behind the first steps of all is divided evenly.
    int more_keys = 0, more_at = 0;
    bool work = true;
    auto find_share = [&]() {
        if constexpr (CLUSTER) {
            b_first = blockIdx.z;
            const int rest = max(0, my_len - p.ncta * tk), per = ((rest + p.ncta - 1) / p.ncta + 15) / 16 * 16, at = min(rest, (int)blockIdx.x * per);
            more_keys = min(rest, at + per) - at;
            more_at = p.ncta * tk + at;
        } else {
            const long long total = cum[p.batch];
            const long long per = share_size(total, p.ncta, tk);
            g0 = (long long)blockIdx.x * per;
            g1 = min(total, g0 + per);
            for (int b0 = 0; b0 < p.batch - 1; b0 += 32) {  // sequences that end at or before the share's first key
                const int n = __popc(__ballot_sync(0xffffffffu, b0 + lane < p.batch - 1 && cum[b0 + lane + 1] <= g0));
                b_first += n;
                if (n < 32) break;
            }
        }
    };
    // Lengths the host knows, and has checked, need no look at memory: the share is found before the wait.
    const bool known = !p.kv_len && !p.kv_row_offset;
    if (known) {
        my_len = max(0, p.kv_len_uniform);
        if (!CLUSTER && threadIdx.x < 32) build_len_prefix(p.batch, cum, [&](int) { return p.kv_len_uniform; });
        __syncthreads();
        find_share();
    }
    if (CLUSTER) cluster_sync_all();  // every CTA runs: its shared memory may be written
    // The producer's copies of a step.
    auto ask = [&](int st, int row) {
        // A stage always carries tk full rows: rows past the segment end
        // are masked by the consumers, rows past the cache end read as zero.
        if (lane == 0) mbar_arrive_expect_tx(&full[st], (uint32_t)stage_bytes);
        __syncwarp();
        uint8_t* dst = stage_base + (size_t)st * stage_bytes;
        for (int c = lane; c < 2 * nchunks; c += 32) {
            const int is_v = c >= nchunks;
            const int cc = c - is_v * nchunks;
            tma_load_2d(dst + (size_t)is_v * tile_bytes + (size_t)cc * chunk_bytes, is_v ? &tm_v : &tm_k,
                        &full[st], head0 * HD + cc * 64, row);
        }
    };
    // Up to here nothing depends on the kernels in front; everything below may.
    grid_dependency_wait();
    int asked = 0;
    // (Not where the sequence is known to end in front of it.)
    bool no_step = known && my_len <= (int)blockIdx.x * tk;
    if (CLUSTER && warp == ncw && !p.kv_row_offset && !no_step) {
        ask(0, (int)((long long)blockIdx.z * p.kv_stride_b) + (int)blockIdx.x * tk);
        asked = 1;
    }
    grid_launch_dependents();  // the merge kernel may be scheduled now; it waits for this grid before reading
    const uint32_t fault = threadIdx.x == 0 ? *reinterpret_cast<volatile uint32_t*>(p.fault) : 0u;  // (set: no result is written)
    long long own_row = CLUSTER ? (long long)blockIdx.z * p.kv_stride_b : 0ll;  // first row of the cluster's sequence
    if (!known) {
        // The status word, the lengths and the row offsets are asked for together: each is a trip to L2 or HBM.
        // Lengths and row offsets live on the device, so this is where they can be checked: a sequence that reaches past the
        // cache (the copies would read zero rows and fold them in as score-0 keys) or past the stated bound stops the
        // launch with a status instead of a wrong result.  Every CTA checks all sequences and so none of them works.
        // (The first warp checks and adds up what it has asked for once: a second look was a second trip.)
        bool bad = fault != 0u;
        const int own_len = CLUSTER && p.kv_len ? p.kv_len[blockIdx.z] : p.kv_len_uniform;
        if (CLUSTER && p.kv_row_offset) own_row = p.kv_row_offset[blockIdx.z];
        auto checked_len = [&](int b) {
            const int len = p.kv_len ? p.kv_len[b] : p.kv_len_uniform;
            const long long row0 = p.kv_row_offset ? p.kv_row_offset[b] : (long long)b * p.kv_stride_b;
            if ((len > 0 && (row0 < 0 || row0 + len > p.kv_rows_total)) || (p.max_kv_len > 0 && len > p.max_kv_len)) {
                report_fault(p.fault, FAULT_BAD_KV_RANGE, (uint32_t)b);
                bad = true;
            }
            return len;
        };
        if (!CLUSTER && threadIdx.x < 32) build_len_prefix(p.batch, cum, checked_len);
        if (CLUSTER)
            for (int b = threadIdx.x; b < p.batch; b += blockDim.x) checked_len(b);
        work = !__syncthreads_or(bad);
        if (CLUSTER && work) my_len = max(0, own_len);
        if (work) find_share();
    }
    if (!CLUSTER && g0 >= g1) return;
    no_step |= p.kv_row_offset && my_len <= (int)blockIdx.x * tk;  // (CLUSTER: nothing has been asked for, and there are no keys)
    // keys before sequence b / up to its end, in the count g0 and g1 use
    auto seq_begin = [&](int b) { return CLUSTER ? 0ll : cum[b]; };
    auto seq_end = [&](int b) { return CLUSTER ? (long long)my_len : cum[b + 1]; };
    constexpr int RS = HD + 4;  // floats from one head's row of a warp's record to the next

    if (warp == ncw) {
        // ------------------------------------------------------------------ producer
        int it = 0;
        bool ok = true;
        int b = b_first;
        long long g = g0;
        if constexpr (CLUSTER) {
            const int steps = no_step ? 0 : 1 + (more_keys + tk - 1) / tk;
            for (it = asked; it < steps; ++it) {
                const int st = it % p.stages;
                if (it >= p.stages && !mbar_wait_warp(&empty[st], ((it / p.stages) - 1) & 1)) {
                    if (lane == 0) report_fault(p.fault, FAULT_WAIT_EMPTY, it);
                    break;
                }
                ask(st, (int)own_row + (it == 0 ? (int)blockIdx.x * tk : more_at + (it - 1) * tk));
            }
        }
        while (!CLUSTER && ok && g < g1) {
            while (seq_end(b) <= g) ++b;
            const long long seg_end = min(g1, seq_end(b));
            const long long row0 = (p.kv_row_offset ? p.kv_row_offset[b] : (long long)b * p.kv_stride_b) + (g - seq_begin(b));
            const int seg_keys = (int)(seg_end - g);
            for (int k0 = 0; k0 < seg_keys; k0 += tk, ++it) {
                const int st = it % p.stages;
                if (it >= p.stages && !mbar_wait_warp(&empty[st], ((it / p.stages) - 1) & 1)) {
                    if (lane == 0) report_fault(p.fault, FAULT_WAIT_EMPTY, it);
                    ok = false;
                    break;
                }
                ask(st, (int)(row0 + k0));
            }
            g = seg_end;
        }
        // Drain: every copy issued above has landed before the CTA retires.
        if (lane == 0) {
            for (int back = 1; back <= p.stages && back <= it; ++back) {
                const int j = it - back;
                mbar_wait(&full[j % p.stages], (j / p.stages) & 1);
            }
        }
    } else if (warp < ncw) {
        // ------------------------------------------------------------------ consumers
        const int hl = warp % p.nkv_cta;  // local KV head
        const int slice = warp / p.nkv_cta;
        const int kvh = head0 + hl;
        const int g4 = lane >> 2;  // accumulator row group
        const int q4 = lane & 3;   // accumulator column pair
        const float sl = p.scale_log2;

        int it = 0;
        bool ok = true;
        bool folded = false;  // this warp has been through the two barriers of the in-CTA fold
        int b = b_first;
        long long g = g0;
        while (CLUSTER || (ok && g < g1)) {  // (CLUSTER: once, keys or not)
            while (!CLUSTER && seq_end(b) <= g) ++b;
            const long long seg_end = CLUSTER ? 0 : min(g1, seq_end(b));
            const int seg_keys = CLUSTER ? (no_step ? 0 : tk + more_keys) : (int)(seg_end - g);  // (CLUSTER: a first step, full or not)

            // Q^T fragments (B operand, hd x 8 heads) for this head's GQA group.
            uint32_t qf[NT][HD / 16][2];
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
                const int n = nt * 8 + g4;
                const bool valid = n < G;
                const uint16_t* qp = p.q + (long long)b * p.q_stride_b + ((long long)kvh * G + (valid ? n : 0)) * HD + q4 * 2;
#pragma unroll
                for (int kk = 0; kk < HD / 16; ++kk) {
                    qf[nt][kk][0] = valid ? *reinterpret_cast<const uint32_t*>(qp + kk * 16) : 0u;
                    qf[nt][kk][1] = valid ? *reinterpret_cast<const uint32_t*>(qp + kk * 16 + 8) : 0u;
                }
            }
            float m[NT][2], l[NT][2];
            float o[NT][HD / 16][4];
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
                m[nt][0] = m[nt][1] = -CUDART_INF_F;
                l[nt][0] = l[nt][1] = 0.f;
#pragma unroll
                for (int mt = 0; mt < HD / 16; ++mt) o[nt][mt][0] = o[nt][mt][1] = o[nt][mt][2] = o[nt][mt][3] = 0.f;
            }

            for (int k0 = 0; k0 < seg_keys; k0 += tk, ++it) {
                const int st = it % p.stages;
                if (!mbar_wait_warp(&full[st], (it / p.stages) & 1)) {
                    if (lane == 0) report_fault(p.fault, FAULT_WAIT_FULL, it);
                    ok = false;
                    break;
                }
                const int nk = CLUSTER && k0 == 0 ? min(max(my_len - (int)blockIdx.x * tk, 0), tk) : min(tk, seg_keys - k0);
                const int nvalid = min(16, nk - slice * 16);  // keys of this warp's slice
                if (nvalid > 0) {
                    // Swizzled addressing: 16-byte unit u of row r sits at unit u ^ (r & 7).
                    const uint32_t sK = smem_u32(stage_base + (size_t)st * stage_bytes) + hl * (HD / 64) * chunk_bytes;
                    const uint32_t sV = sK + tile_bytes;
                    const int key_k = slice * 16 + (lane & 15);
                    const int key_v = slice * 16 + (lane & 7) + (lane >> 4) * 8;
                    const uint32_t a_k = sK + key_k * 128;
                    const uint32_t a_v = sV + key_v * 128;
                    const int xk = key_k & 7, hk = lane >> 4;
                    const int xv = key_v & 7, hv = (lane >> 3) & 1;
                    if (nvalid < 16) {
                        // Rows past the segment end may hold anything (another sequence, or
                        // never-written cache); clear this warp's V rows so 0 * x stays 0.
                        for (int i = lane; i < (16 - nvalid) * (HD / 8); i += 32) {
                            const int key = slice * 16 + nvalid + i / (HD / 8);
                            const int u = i % (HD / 8);
                            const uint32_t a = sV + (u >> 3) * chunk_bytes + key * 128 + (u & 7) * 16;
                            asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};" ::"r"(a), "r"(0u) : "memory");
                        }
                        fence_proxy_async_smem();
                        __syncwarp();
                    }

                    // Fragments are fetched AHEAD at a time and a batch before their MMAs: fetched one by one, each MMA
                    // waited 40 clk for its own, and the 32 of a step of 16 keys at head dim 256 took 1400 clk (now 800).
                    constexpr int AHEAD = HD * NT > 256 ? 2 : 4, BATCHES = HD / 16 / AHEAD;
                    constexpr int CHAINS = NT == 1 ? 4 : 2;  // independent sums of S
                    uint32_t fr[2][AHEAD][4];
                    auto fetch_k = [&](int bt) {
#pragma unroll
                        for (int i = 0; i < AHEAD; ++i) {
                            const int kk = bt * AHEAD + i;
                            ldmatrix_x4(fr[bt & 1][i], a_k + (kk >> 2) * chunk_bytes + ((((kk & 3) * 2 + hk) ^ xk) << 4));
                        }
                    };
                    auto fetch_v = [&](int bt) {
#pragma unroll
                        for (int i = 0; i < AHEAD; ++i) {
                            const int mt = bt * AHEAD + i;
                            ldmatrix_x4_trans(fr[bt & 1][i], a_v + (mt >> 2) * chunk_bytes + ((((mt & 3) * 2 + hv) ^ xv) << 4));
                        }
                    };
                    float acc[NT][CHAINS][4];
#pragma unroll
                    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                        for (int hh = 0; hh < CHAINS; ++hh) acc[nt][hh][0] = acc[nt][hh][1] = acc[nt][hh][2] = acc[nt][hh][3] = 0.f;
                    fetch_k(0);
#pragma unroll
                    for (int bt = 0; bt < BATCHES; ++bt) {
                        if (bt + 1 < BATCHES) fetch_k(bt + 1);
                        else if (NT == 1) fetch_v(0);  // (an even number of batches: into the other half)
#pragma unroll
                        for (int i = 0; i < AHEAD; ++i) {
                            const int kk = bt * AHEAD + i;
#pragma unroll
                            for (int nt = 0; nt < NT; ++nt) mma_bf16_16816(acc[nt][kk % CHAINS], fr[bt & 1][i], qf[nt][kk][0], qf[nt][kk][1]);
                        }
                    }
                    static_assert(BATCHES % 2 == 0, "the first batch of V goes where the last one of K is not");
                    const bool v_lo = g4 < nvalid, v_hi = g4 + 8 < nvalid;
                    uint32_t pb[NT][2];
                    bool any_rescale = false;
                    float alpha[NT][2];
#pragma unroll
                    for (int nt = 0; nt < NT; ++nt) {
                        float x[4];
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            float s = acc[nt][0][e] + acc[nt][1][e];
                            if constexpr (CHAINS == 4) s += acc[nt][2][e] + acc[nt][3][e];
                            s *= sl;
                            x[e] = ((e < 2) ? v_lo : v_hi) ? s : -CUDART_INF_F;
                        }
                        float pr[4];
#pragma unroll
                        for (int u = 0; u < 2; ++u) {
                            float mx = fmaxf(x[u], x[u + 2]);
                            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 4));
                            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
                            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
                            const float m_new = fmaxf(m[nt][u], mx);
                            const float m_eff = (m_new == -CUDART_INF_F) ? 0.f : m_new;
                            alpha[nt][u] = (m_new == -CUDART_INF_F) ? 1.f : fast_exp2(m[nt][u] - m_new);
                            pr[u] = fast_exp2(x[u] - m_eff);
                            pr[u + 2] = fast_exp2(x[u + 2] - m_eff);
                            l[nt][u] = l[nt][u] * alpha[nt][u] + pr[u] + pr[u + 2];
                            m[nt][u] = m_new;
                            any_rescale |= alpha[nt][u] != 1.f;
                        }
                        pb[nt][0] = movmatrix_trans(pack_bf16x2(pr[0], pr[1]));
                        pb[nt][1] = movmatrix_trans(pack_bf16x2(pr[2], pr[3]));
                    }
                    if (__any_sync(0xffffffffu, any_rescale)) {
#pragma unroll
                        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                            for (int mt = 0; mt < HD / 16; ++mt) {
                                o[nt][mt][0] *= alpha[nt][0];
                                o[nt][mt][1] *= alpha[nt][1];
                                o[nt][mt][2] *= alpha[nt][0];
                                o[nt][mt][3] *= alpha[nt][1];
                            }
                    }
                    if (NT > 1) fetch_v(0);
#pragma unroll
                    for (int bt = 0; bt < BATCHES; ++bt) {
                        if (bt + 1 < BATCHES) fetch_v(bt + 1);
#pragma unroll
                        for (int i = 0; i < AHEAD; ++i)
#pragma unroll
                            for (int nt = 0; nt < NT; ++nt) mma_bf16_16816(o[nt][bt * AHEAD + i], fr[bt & 1][i], pb[nt][0], pb[nt][1]);
                    }
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(&empty[st]);
            }

            if constexpr (CLUSTER) {
                // Everything from here on runs once a call, from instructions fetched cold, so it is kept short: records as they
                // are, weights worked out once, by eight lanes a row, loops that are not unrolled.
                float* rec = reinterpret_cast<float*>(stage_base);                     // [warp][NT * 8 heads][RS]
                float2* rec_ml = reinterpret_cast<float2*>(rec + (size_t)ncw * NT * 8 * RS);  // [warp][NT * 8]
                float* rec_w = reinterpret_cast<float*>(rec_ml + ncw * NT * 8);
                static_assert(NT * 8 * (RS + 3) <= 2 * 16 * HD, "a warp's records, sums and weights in its slices of K and V of two stages");
                if (lane == 0 && (!ok || !work || fault != 0u)) *reinterpret_cast<volatile int*>(gave_up) = 1;  // (no result is written)
                consumer_sync(ncw);  // every warp is through with the stages; no copy is in flight any more
#pragma unroll
                for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        float ls = l[nt][u];
                        ls += __shfl_xor_sync(0xffffffffu, ls, 4);
                        ls += __shfl_xor_sync(0xffffffffu, ls, 8);
                        ls += __shfl_xor_sync(0xffffffffu, ls, 16);
                        const int n = warp * NT * 8 + nt * 8 + q4 * 2 + u;
                        if (g4 == 0) rec_ml[n] = make_float2(m[nt][u], ls);
                        float* dst = rec + (size_t)n * RS + g4;
#pragma unroll
                        for (int mt = 0; mt < HD / 16; ++mt) {
                            dst[mt * 16] = o[nt][mt][u];
                            dst[mt * 16 + 8] = o[nt][mt][u + 2];
                        }
                    }
                consumer_sync(ncw);
                const uint32_t bar = smem_u32(gathered);
                // (st.async is for clusters: plain stores where a CTA is alone.)
#pragma unroll 1
                for (int n0 = slice * 4; n0 < G; n0 += p.slices * 4) {  // four rows of the KV head a turn, a lane per slice
                    const int n = n0 + (lane >> 3), s = lane & 7, at = (s * p.nkv_cta + hl) * NT * 8 + n;
                    const bool some = n < G && s < p.slices;
                    const float2 ml = some ? rec_ml[at] : make_float2(-CUDART_INF_F, 0.f);
                    float mx = ml.x;
#pragma unroll
                    for (int o = 4; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
                    const float wt = ml.x == -CUDART_INF_F ? 0.f : fast_exp2(ml.x - mx);
                    float z = wt * ml.y;
#pragma unroll
                    for (int o = 4; o > 0; o >>= 1) z += __shfl_xor_sync(0xffffffffu, z, o);
                    // (2^-6, taken back with the CTAs' weights: up to 64 records are added up before their sum of weights is
                    // divided by, and values that a record of its own can hold must not run over in between.)
                    if (some) rec_w[at] = wt * 0.015625f;
                    float2* to = cml + blockIdx.x * rows2 + hl * G + n;
                    if (n < G && s < finishers) {
                        if (ALONE) *to = make_float2(mx, z);
                        else st_async_f32x2(map_to_cta(smem_u32(to), s), make_float2(mx, z), map_to_cta(bar, s));
                    }
                }
                if (warp == 0 && lane < finishers) {
                    const float good = *reinterpret_cast<volatile int*>(gave_up) ? 0.f : 1.f;
                    if (ALONE) cflag[0] = good;
                    else st_async_f32(map_to_cta(smem_u32(cflag + blockIdx.x), lane), good, map_to_cta(bar, lane));
                }
                consumer_sync(ncw);
#pragma unroll 1
                for (int i = slice; i < G * (HD / 128); i += p.slices) {  // half a row (head dim 256) a turn
                    const int n = i / (HD / 128), d = i % (HD / 128) * 128 + lane * 4;
                    const float* src = rec + (size_t)(hl * NT * 8 + n) * RS + d;
                    const float* wts = rec_w + hl * NT * 8 + n;
                    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 2
                    for (int s = 0; s < p.slices; ++s) {
                        const float wt = *wts;
                        const float4 v = *reinterpret_cast<const float4*>(src);
                        acc.x = fmaf(wt, v.x, acc.x), acc.y = fmaf(wt, v.y, acc.y), acc.z = fmaf(wt, v.z, acc.z), acc.w = fmaf(wt, v.w, acc.w);
                        src += (size_t)p.nkv_cta * NT * 8 * RS, wts += p.nkv_cta * NT * 8;
                    }
                    float* at = crec + (size_t)(blockIdx.x * rows + hl * G + n) * dc + (d & (dc - 1));
                    const int to = d >> dc_log2;
                    if (ALONE) *reinterpret_cast<float4*>(at) = acc;
                    else st_async_f32x4(map_to_cta(smem_u32(at), to), acc, map_to_cta(bar, to));
                }
                break;
            }
            // Partial record of this (CTA, sequence, slice): normalised out + natural-log lse.
            // The last segment of the share (for most CTAs the only one) is folded across the slices inside
            // the CTA first: the stages are free by then, so each warp leaves its record in shared memory,
            // and the warps of a KV head combine them into ONE record per (CTA, sequence), stored in slice
            // 0's slot; the other slices' slots stay unwritten.  The merge kernel then reads
            // `slices` times fewer records.  Earlier segments (a sequence boundary inside the share) write
            // one record per slice.
            const bool fold_here = p.slices > 1 && seg_end == g1;  // CTA-uniform
            // (rows four floats longer than HD: the four lanes that write the same column of different heads hit different banks)
            float* rec = reinterpret_cast<float*>(stage_base);     // [warp][NT * 8 heads][RS]
            float* rec_lse = rec + (size_t)ncw * NT * 8 * RS;      // [warp][NT * 8]
            if (fold_here) {
                consumer_sync(ncw);  // every warp is through with the stages; no copy is in flight any more
                folded = true;
            }
            if (ok) {
                const long long part = ((long long)blockIdx.x + b) * p.slices + slice;
#pragma unroll
                for (int nt = 0; nt < NT; ++nt) {
                    float inv[2];
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        float ls = l[nt][u];
                        ls += __shfl_xor_sync(0xffffffffu, ls, 4);
                        ls += __shfl_xor_sync(0xffffffffu, ls, 8);
                        ls += __shfl_xor_sync(0xffffffffu, ls, 16);
                        inv[u] = ls > 0.f ? 1.f / ls : 0.f;
                        const int n = nt * 8 + q4 * 2 + u;
                        const float lse = ls > 0.f ? (m[nt][u] + fast_log2(ls)) * 0.6931471805599453f : -CUDART_INF_F;
                        if (g4 == 0) {
                            if (fold_here) rec_lse[warp * NT * 8 + n] = lse;
                            else if (n < G) p.part_lse[part * p.nq + (long long)kvh * G + n] = lse;
                        }
                    }
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        const int n = nt * 8 + q4 * 2 + u;
                        if (fold_here || n < G) {
                            float* dst = fold_here ? rec + ((size_t)warp * NT * 8 + n) * RS
                                                   : p.part_o + (part * p.nq + (long long)kvh * G + n) * HD;
#pragma unroll
                            for (int mt = 0; mt < HD / 16; ++mt) {
                                dst[mt * 16 + g4] = o[nt][mt][u] * inv[u];
                                dst[mt * 16 + g4 + 8] = o[nt][mt][u + 2] * inv[u];
                            }
                        }
                    }
                }
            }
            if (fold_here) {
                consumer_sync(ncw);  // all records of the CTA are in shared memory
                // The `slices` (at most eight) warps of this KV head take its rows in turn; the weights of a row's records
                // are worked out once, a lane each.
                const long long row0 = ((long long)blockIdx.x + b) * p.slices * p.nq + (long long)kvh * G;
                for (int n = slice; n < G; n += p.slices) {
                    const float li = lane < p.slices ? rec_lse[(lane * p.nkv_cta + hl) * NT * 8 + n] : -CUDART_INF_F;
                    float mx = li;
#pragma unroll
                    for (int o = 4; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
                    mx = __shfl_sync(0xffffffffu, mx, 0);
                    float z = mx > -CUDART_INF_F ? __expf(li - mx) : 0.f;
                    const float e = z;
#pragma unroll
                    for (int o = 4; o > 0; o >>= 1) z += __shfl_xor_sync(0xffffffffu, z, o);
                    z = __shfl_sync(0xffffffffu, z, 0);
                    const float weight = z > 0.f ? e / z : 0.f;
                    float4 acc[HD / 128];
#pragma unroll
                    for (int j = 0; j < HD / 128; ++j) acc[j] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
                    for (int sidx = 0; sidx < p.slices; ++sidx) {
                        const float wt = __shfl_sync(0xffffffffu, weight, sidx);
                        const float* src = rec + ((size_t)(sidx * p.nkv_cta + hl) * NT * 8 + n) * RS + lane * 4;
#pragma unroll
                        for (int j = 0; j < HD / 128; ++j) {  // (an empty slice's record holds zeros)
                            const float4 ov = *reinterpret_cast<const float4*>(src + 128 * j);
                            acc[j].x = fmaf(wt, ov.x, acc[j].x);
                            acc[j].y = fmaf(wt, ov.y, acc[j].y);
                            acc[j].z = fmaf(wt, ov.z, acc[j].z);
                            acc[j].w = fmaf(wt, ov.w, acc[j].w);
                        }
                    }
                    const float rec_l = z > 0.f ? mx + __logf(z) : -CUDART_INF_F;
#pragma unroll
                    for (int j = 0; j < HD / 128; ++j) *reinterpret_cast<float4*>(p.part_o + (row0 + n) * HD + lane * 4 + 128 * j) = acc[j];
                    if (lane == 0) p.part_lse[row0 + n] = rec_l;
                }
            }
            g = seg_end;
        }
        // A warp that gave up a wait never reached the fold: it still meets the others at both barriers.
        if (!CLUSTER && !folded && p.slices > 1) {
            consumer_sync(ncw);
            consumer_sync(ncw);
        }
    }
    if constexpr (CLUSTER) {
        // This CTA's columns, two a thread, once every record is in its own shared memory.  (Nothing is sent to a CTA that
        // finishes none, and what this one has sent is waited for by those it went to: no barrier of the cluster here.)
        if (!ALONE && (int)(blockIdx.x << dc_log2) >= HD) return;
        const int items = rows * (dc / 2), b = blockIdx.z;
        auto offset_of = [&](int item) {
            return (long long)b * p.o_stride_b + (long long)(head0 * G + (item >> (dc_log2 - 1))) * HD + blockIdx.x * dc + (item & (dc / 2 - 1)) * 2;
        };
        uint32_t gw = p.gate && (int)threadIdx.x < items ? *reinterpret_cast<const uint32_t*>(p.gate + offset_of(threadIdx.x)) : 0u;
        __syncwarp();
        // Whether the records came is settled for the whole CTA before any warp goes on: each warp waits by its own clock, and
        // one that gave up stood at the cluster's barrier while another, whose last look found them, stood at the CTA's.
        const bool came = ALONE || mbar_wait_cluster(gathered, 0);
        if (!__syncthreads_and(came)) {
            if (!came && lane == 0) report_fault(p.fault, FAULT_WAIT_FULL, 0x10000u);
            cluster_sync_all();  // (what is still under way here arrives before the other CTAs have gone)
            return;
        }
        const bool fine = __all_sync(0xffffffffu, (lane & 7) >= p.ncta || cflag[lane & 7] != 0.f);  // (the same in every warp)
        // The CTAs' weights of a row: eight lanes.
#pragma unroll 1
        for (int n0 = warp * 4; n0 < rows; n0 += (ncw + 1) * 4) {
            const int n = n0 + (lane >> 3), c = lane & 7;
            const float2 ml = n < rows && c < p.ncta ? cml[c * rows2 + n] : make_float2(-CUDART_INF_F, 0.f);
            float mx = ml.x;
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
            const float wt = ml.x == -CUDART_INF_F ? 0.f : fast_exp2(ml.x - mx);
            float z = wt * ml.y;
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) z += __shfl_xor_sync(0xffffffffu, z, o);
            if (n < rows) {
                // (A sum of weights that is no number, as scores make it that are none, goes on to the log-sum-exp: -inf beside such
                // a row would say that it is empty, and who merges it with others would leave it out.)
                cweight[n * 8 + c] = z == 0.f ? 0.f : __fdividef(wt * 64.f, z);
                if (p.out_lse && fine && blockIdx.x == 0 && c == 0)
                    p.out_lse[(long long)b * p.nq + head0 * G + n] = z == 0.f ? -CUDART_INF_F : fmaf(mx, 0.6931471805599453f, logf(z));
            }
        }
        __syncthreads();
        if (!fine) return;
#pragma unroll 1
        for (int item = threadIdx.x; item < items; item += blockDim.x) {
            const int n = item >> (dc_log2 - 1), d = (item & (dc / 2 - 1)) * 2;
            const long long eoff = offset_of(item);
            if (p.gate && item != (int)threadIdx.x) gw = *reinterpret_cast<const uint32_t*>(p.gate + eoff);
            float a0 = 0.f, a1 = 0.f;
#pragma unroll 2
            for (int c = 0; c < p.ncta; ++c) {
                const float wt = cweight[n * 8 + c];
                const float2 v = *reinterpret_cast<const float2*>(crec + (size_t)(c * rows + n) * dc + d);
                a0 = fmaf(wt, v.x, a0);
                a1 = fmaf(wt, v.y, a1);
            }
            const long long row = (long long)b * p.nq + head0 * G + n;
            if (p.out_f32) *reinterpret_cast<float2*>(p.out_f32 + row * HD + blockIdx.x * dc + d) = make_float2(a0, a1);
            if (p.out) {
                if (p.gate) {
                    a0 = sigmoid_gate(a0, (uint16_t)(gw & 0xffffu));
                    a1 = sigmoid_gate(a1, (uint16_t)(gw >> 16));
                }
                *reinterpret_cast<uint32_t*>(p.out + eoff) = pack_bf16x2(a0, a1);
            }
        }
    }
}

// ---------------------------------------------------------------------------
// Merge of the decode partials.  grid = (nq, batch, column blocks); every warp of a
// block recomputes the share boundaries the decode kernel used, which say where the
// records of its sequence are: CTAs [c_first, c_last], record index (cta + b)*slices + s.
// ---------------------------------------------------------------------------
struct DecodeMergeParams {
    const float* part_o;
    const float* part_lse;
    const int* kv_len;
    const uint16_t* gate;
    uint16_t* out;
    float* out_f32;
    float* out_lse;
    int batch, nq, kv_len_uniform;
    int ncta, slices;
    long long o_stride_b;
    // Sequence-sharded decode over NVLink peer memory (x_world > 1): every rank's exchange
    // buffer base address; this rank's index; a step counter that grows by one per call.
    const unsigned long long* x_peers;
    int x_world, x_rank;
    uint32_t x_step;
    long long x_wait_cycles;  // bound of the wait for the other ranks' records
    uint32_t* fault;
};

// Layout of one rank's exchange buffer: [2 parities][world sources][rows] records of HD + 2 words, a word
// being 8 bytes = (value bits, step).  Every value travels with the step number it belongs to, so a
// receiver recognises a word as soon as it lands: no fence between data and a separate flag, one NVLink
// crossing per exchange instead of three (stores, their acknowledgement, the flag).  Words HD and HD + 1
// hold the row's log-sum-exp and padding.  8-byte stores are single transactions; a 16-byte store may be
// split, which is fine because each half carries its own step.
constexpr int XCHG_MAX_WORLD = 16;  // ranks of one exchange (one NVSwitch box has 8)
__host__ __device__ inline size_t xchg_record_words(int hd) { return (size_t)hd + 2; }
__host__ __device__ inline size_t xchg_total_bytes(int world, long long rows, int hd) {
    return (size_t)2 * world * rows * xchg_record_words(hd) * 8;
}

__device__ __forceinline__ void st_volatile_v4(uint4* p, uint4 v) {
    asm volatile("st.volatile.global.v4.u32 [%0], {%1, %2, %3, %4};" ::"l"(p), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
__device__ __forceinline__ uint4 ld_volatile_v4(const uint4* p) {
    uint4 v;
    asm volatile("ld.volatile.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
    return v;
}


constexpr int MERGE_THREADS = 256;

// XCHG: the instance that also exchanges records with other GPUs.  It keeps every source's values in
// registers; the plain merge — hundreds of small blocks for a large batch — stays lean.
// COLS: columns of the row a block takes.  All of them, unless the rows are so few that most SMs would idle: one token of
// 24 heads over 6760 keys has 106 records in each of 24 rows, 100 KB a block, and took 7.5 us from the decode kernel's
// end; 64 columns a block, every load of a batch in flight with the log-sum-exps, take 3.9.
// (Whole rows of 256: four blocks per SM, 64 sequences of 24 heads are 1536 of them.  At 128 columns the registers that
// would take are worth more: 12 sequences of 16 heads 14.8 us, with four blocks per SM 15.6.)
template <int HD, bool XCHG, int COLS>
__global__ void __launch_bounds__(MERGE_THREADS, XCHG || COLS < 256 ? 1 : 4) sdpa_decode_merge_kernel(const DecodeMergeParams p) {
    // One row of output per block; what the block does before its one barrier every warp does for itself — where the
    // row's records are, their maximum and weights — because that is a handful of loads, while three block-wide
    // reductions and a list in shared memory made this kernel's tail 5 us.
    constexpr int NW = MERGE_THREADS / 32;
    constexpr int LPR = COLS / 4 < 32 ? COLS / 4 : 32, VPL = COLS / LPR;  // lanes of a record, their output values
    constexpr int TEAMS = NW * 32 / LPR;                                  // records the block takes at a time
    __shared__ float acc_sm[TEAMS * COLS];
    const int h = blockIdx.x, b = blockIdx.y, col0 = XCHG ? 0 : blockIdx.z * COLS;
    const int team = threadIdx.x / LPR, tl = threadIdx.x % LPR;
    const int lane = threadIdx.x & 31;
    // (The decode kernel released this one after its own wait for the kernels in front: the lengths are final.)
    long long k_begin = 0, total = 0, k_len = 0;
    if (!p.kv_len) {
        k_len = max(0, p.kv_len_uniform);
        k_begin = (long long)b * k_len;
        total = (long long)p.batch * k_len;
    } else {
        for (int i = lane; i < p.batch; i += 32) {
            const int len = max(0, p.kv_len[i]);
            total += len;
            if (i < b) k_begin += len;
            if (i == b) k_len = len;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            total += __shfl_xor_sync(0xffffffffu, total, o);
            k_begin += __shfl_xor_sync(0xffffffffu, k_begin, o);
            k_len += __shfl_xor_sync(0xffffffffu, k_len, o);
        }
    }
    // requests for the lines the end will need
    if (p.gate && p.out && threadIdx.x < HD * 2 / 128)
        prefetch_l2(p.gate + (long long)b * p.o_stride_b + (long long)h * HD + threadIdx.x * 64);
    const long long per = share_size(total, p.ncta, 16 * p.slices);
    const long long k_end = k_begin + k_len;
    grid_dependency_wait();                                            // from here on the partial records are read
    grid_launch_dependents();
    const uint32_t fault = threadIdx.x == 0 ? *reinterpret_cast<volatile uint32_t*>(p.fault) : 0u;
    float acc[VPL];
#pragma unroll
    for (int j = 0; j < VPL; ++j) acc[j] = 0.f;
    float lse = -CUDART_INF_F, inv = 0.f;
    if (k_len > 0) {  // block-uniform
        const bool small = total < (1ll << 30);
        const int c_first = small ? (int)((uint32_t)k_begin / (uint32_t)per) : (int)(k_begin / per);
        const int c_last = small ? (int)((uint32_t)(k_end - 1) / (uint32_t)per) : (int)((k_end - 1) / per);
        const long long part0 = ((long long)c_first + b) * p.slices;
        // Which records exist follows from the shares: a share whose last segment is this sequence's folded its slices
        // into slice 0's record — every share but possibly the last, whose slices wrote one record each if the
        // sequence ends before the share does.
        const int n_full = c_last - c_first;
        const int n_rec = n_full + (k_end == min(total, (c_last + 1) * per) ? 1 : p.slices);
        auto rec_of = [&](int j) { return part0 + (j < n_full ? (long long)j * p.slices : (long long)n_full * p.slices + (j - n_full)); };
        const float* lses = p.part_lse + h;
        // The records are dealt to the teams in turn, U at a time; a lane owns VPL consecutive output values.  Always the
        // same order of additions.  The first batch and all log-sum-exps (eight a lane; more is rare) are asked for
        // together: one trip to L2.
        constexpr int U = VPL == 8 ? 2 : 4, MINE = 8;
        float wu[U];
        float4 ov[U][VPL / 4];
        auto load_batch = [&](int j0) {
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int j = j0 + u * TEAMS;
                wu[u] = -CUDART_INF_F;
                if (j < n_rec) {
                    const long long rec = rec_of(j);
                    wu[u] = lses[rec * p.nq];
                    const float* src = p.part_o + (rec * p.nq + h) * HD + col0 + tl * VPL;
#pragma unroll
                    for (int i = 0; i < VPL / 4; ++i) ov[u][i] = *reinterpret_cast<const float4*>(src + 4 * i);
                }
            }
        };
        load_batch(team);
        float mine[MINE], mx = -CUDART_INF_F;
#pragma unroll
        for (int i = 0; i < MINE; ++i) mine[i] = lane + 32 * i < n_rec ? lses[rec_of(lane + 32 * i) * p.nq] : -CUDART_INF_F;
#pragma unroll
        for (int i = 0; i < MINE; ++i) mx = fmaxf(mx, mine[i]);
        for (int j = lane + 32 * MINE; j < n_rec; j += 32) mx = fmaxf(mx, lses[rec_of(j) * p.nq]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        if (mx > -CUDART_INF_F) {
            float z = 0.f;
#pragma unroll
            for (int i = 0; i < MINE; ++i) z += __expf(mine[i] - mx);  // exp(-inf) = 0: an empty slice
            for (int j = lane + 32 * MINE; j < n_rec; j += 32) z += __expf(lses[rec_of(j) * p.nq] - mx);
            for (int j0 = team; j0 < n_rec; j0 += TEAMS * U) {
                if (j0 != team) load_batch(j0);
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    if (wu[u] == -CUDART_INF_F) continue;  // an empty slice's record may hold anything
                    const float w = __expf(wu[u] - mx);
#pragma unroll
                    for (int i = 0; i < VPL / 4; ++i) {
                        acc[4 * i] = fmaf(w, ov[u][i].x, acc[4 * i]);
                        acc[4 * i + 1] = fmaf(w, ov[u][i].y, acc[4 * i + 1]);
                        acc[4 * i + 2] = fmaf(w, ov[u][i].z, acc[4 * i + 2]);
                        acc[4 * i + 3] = fmaf(w, ov[u][i].w, acc[4 * i + 3]);
                    }
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) z += __shfl_xor_sync(0xffffffffu, z, o);
            inv = 1.f / z;
            lse = mx + __logf(z);
        }
    }
#pragma unroll
    for (int j = 0; j < VPL; ++j) acc_sm[team * COLS + tl * VPL + j] = acc[j];
    if (__syncthreads_or(fault != 0u)) return;  // a status is set: no work
    const long long row = (long long)b * p.nq + h;
    if (p.out_lse && threadIdx.x == 0 && col0 == 0) p.out_lse[row] = lse;
    const int d = col0 + threadIdx.x * 2;
    float a0 = 0.f, a1 = 0.f;
    if (threadIdx.x < COLS / 2) {
#pragma unroll
        for (int w = 0; w < TEAMS; ++w) {
            const float2 v = *reinterpret_cast<const float2*>(acc_sm + w * COLS + threadIdx.x * 2);
            a0 += v.x;
            a1 += v.y;
        }
        a0 *= inv;
        a1 *= inv;
        if (p.out_f32) *reinterpret_cast<float2*>(p.out_f32 + row * HD + d) = make_float2(a0, a1);
    }
    if (XCHG && p.x_world > 1) {
        // Sequence-sharded: this rank's (out, lse) of the row goes straight into every rank's exchange
        // buffer over NVLink as plain peer stores of (value, step) words.  Then the block waits — for a
        // bounded time — until the words of every source rank show this step, and folds the records.
        // Thread t < HD / 2 sends and receives values 2t, 2t + 1 (one 16-byte store / load); thread HD / 2
        // does the same for the log-sum-exp word and hands the sources' values round through shared memory.
        const long long rows = (long long)p.batch * p.nq;
        const int par = (int)(p.x_step & 1u);
        const size_t rw = xchg_record_words(HD) / 2;  // 16-byte units per record
        const size_t slot = ((size_t)par * p.x_world + p.x_rank) * rows + row;
        const bool sender = threadIdx.x <= HD / 2;
        if (sender) {
            const uint4 word = threadIdx.x < HD / 2 ? make_uint4(__float_as_uint(a0), p.x_step, __float_as_uint(a1), p.x_step)
                                                    : make_uint4(__float_as_uint(lse), p.x_step, 0u, p.x_step);
            for (int dst = 0; dst < p.x_world; ++dst)
                st_volatile_v4(reinterpret_cast<uint4*>(p.x_peers[dst]) + slot * rw + threadIdx.x, word);
        }
        const uint4* mine = reinterpret_cast<const uint4*>(p.x_peers[p.x_rank]);
        __shared__ int x_timeout;
        __shared__ float x_lse[XCHG_MAX_WORLD];
        if (threadIdx.x == 0) x_timeout = 0;
        __syncthreads();
        float b0 = 0.f, b1 = 0.f, z = 0.f;
        float2 rv[XCHG_MAX_WORLD];  // this thread's two values from every source
        if (sender) {
            const long long t0 = clock64();
            bool gave_up = false;
#pragma unroll
            for (int src = 0; src < XCHG_MAX_WORLD; ++src) {
                if (src >= p.x_world) break;
                const uint4* w = mine + (((size_t)par * p.x_world + src) * rows + row) * rw + threadIdx.x;
                uint4 v = ld_volatile_v4(w);
                while (!gave_up && (v.y != p.x_step || v.w != p.x_step)) {
                    if (clock64() - t0 > p.x_wait_cycles) {  // the peer never came
                        report_fault(p.fault, FAULT_WAIT_PEER, (uint32_t)src);
                        x_timeout = 1;
                        gave_up = true;
                        break;
                    }
                    v = ld_volatile_v4(w);
                }
                rv[src] = make_float2(__uint_as_float(v.x), __uint_as_float(v.z));
                if (threadIdx.x == HD / 2) x_lse[src] = rv[src].x;
            }
        }
        __syncthreads();  // x_lse[] and x_timeout are visible
        if (x_timeout) return;
        float mx = -CUDART_INF_F;
        for (int src = 0; src < p.x_world; ++src) mx = fmaxf(mx, x_lse[src]);
        if (mx > -CUDART_INF_F && threadIdx.x < HD / 2) {
#pragma unroll
            for (int src = 0; src < XCHG_MAX_WORLD; ++src) {
                if (src >= p.x_world) break;
                const float li = x_lse[src];
                if (li == -CUDART_INF_F) continue;
                const float wgt_s = __expf(li - mx);
                z += wgt_s;
                b0 = fmaf(wgt_s, rv[src].x, b0);
                b1 = fmaf(wgt_s, rv[src].y, b1);
            }
            b0 /= z;
            b1 /= z;
        }
        a0 = b0;
        a1 = b1;
    }
    if (threadIdx.x < COLS / 2) {
        if (p.out) {
            const long long eoff = (long long)b * p.o_stride_b + (long long)h * HD + d;
            if (p.gate) {
                const uint32_t gw = *reinterpret_cast<const uint32_t*>(p.gate + eoff);
                a0 = sigmoid_gate(a0, (uint16_t)(gw & 0xffffu));
                a1 = sigmoid_gate(a1, (uint16_t)(gw >> 16));
            }
            *reinterpret_cast<uint32_t*>(p.out + eoff) = pack_bf16x2(a0, a1);
        }
    }
}

// ---------------------------------------------------------------------------
// Merge of `num_parts` uniformly strided partial sets: part_o (parts, rows, hd),
// part_lse (parts, rows), consecutive parts o_part_stride / lse_part_stride
// elements apart (so one packed record per part works too).  One warp per row.  Used for split prefill tiles and
// for records gathered from other GPUs.  out rows are contiguous (rows, hd)
// unless seq > 0, in which case row = (b, t, h) is scattered with the
// given strides (prefill output layout).
// ---------------------------------------------------------------------------
struct UniformMergeParams {
    const float* part_o;
    const float* part_lse;
    const uint16_t* gate;
    uint16_t* out;
    float* out_f32;
    float* out_lse;
    long long rows;
    long long o_part_stride, lse_part_stride;  // elements between consecutive parts
    int num_parts;
    int seq, nq;  // seq > 0: strided (b, t, h) addressing of out / gate
    long long o_stride_b, o_stride_t;
    const unsigned long long* out_copies;  // n_copies more output buffers, same offsets (prefill: other GPUs' buffers)
    int n_copies;
};

// U consecutive parts of a row, `VPL` values a lane: log-sum-exp and values asked for together.
template <int HD, int U>
__device__ __forceinline__ void load_parts(const UniformMergeParams& p, long long row, int i0, float (&li)[U], float4 (&ov)[U][HD / 128]) {
    const float* src = p.part_o + row * HD + (threadIdx.x & 31) * (HD / 32);
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const bool in = i0 + u < p.num_parts;
        li[u] = in ? p.part_lse[(long long)(i0 + u) * p.lse_part_stride + row] : -CUDART_INF_F;
#pragma unroll
        for (int j = 0; j < HD / 128; ++j)
            ov[u][j] = in ? *reinterpret_cast<const float4*>(src + (long long)(i0 + u) * p.o_part_stride + 4 * j) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
}

// Adds them to the row's sums, which are relative to the maximum so far.
template <int HD, int U>
__device__ __forceinline__ void fold_parts(const float (&li)[U], const float4 (&ov)[U][HD / 128], float& mx, float& z, float (&acc)[HD / 32]) {
    float m_new = mx;
#pragma unroll
    for (int u = 0; u < U; ++u) m_new = fmaxf(m_new, li[u]);
    if (m_new == -CUDART_INF_F) return;  // nothing but empty parts so far
    const float old = __expf(mx - m_new);
    mx = m_new;
    z *= old;
#pragma unroll
    for (int j = 0; j < HD / 32; ++j) acc[j] *= old;
#pragma unroll
    for (int u = 0; u < U; ++u) {
        if (li[u] == -CUDART_INF_F) continue;  // an empty part's record may hold anything
        const float w = __expf(li[u] - mx);
        z += w;
#pragma unroll
        for (int j = 0; j < HD / 128; ++j) {
            acc[4 * j] = fmaf(w, ov[u][j].x, acc[4 * j]);
            acc[4 * j + 1] = fmaf(w, ov[u][j].y, acc[4 * j + 1]);
            acc[4 * j + 2] = fmaf(w, ov[u][j].z, acc[4 * j + 2]);
            acc[4 * j + 3] = fmaf(w, ov[u][j].w, acc[4 * j + 3]);
        }
    }
}

// The row's gate values (bf16 pairs) of this lane; eoff: offset of the row in out and gate.
template <int HD>
__device__ __forceinline__ void load_gate_row(const UniformMergeParams& p, long long eoff, uint32_t (&gw)[HD / 64]) {
#pragma unroll
    for (int j = 0; j < HD / 64; ++j) gw[j] = p.gate ? *reinterpret_cast<const uint32_t*>(p.gate + eoff + (threadIdx.x & 31) * (HD / 32) + 2 * j) : 0u;
}

template <int HD>
__device__ __forceinline__ void store_folded(const UniformMergeParams& p, long long row, long long eoff, float mx, float z, float (&acc)[HD / 32],
                                             const uint32_t (&gw)[HD / 64]) {
    constexpr int VPL = HD / 32;
    const int lane = threadIdx.x & 31, d = lane * VPL;
    const float inv = z > 0.f ? 1.f / z : 0.f;
#pragma unroll
    for (int j = 0; j < VPL; ++j) acc[j] *= inv;
    if (p.out_f32) {
#pragma unroll
        for (int j = 0; j < VPL / 4; ++j)
            *reinterpret_cast<float4*>(p.out_f32 + row * HD + d + 4 * j) = make_float4(acc[4 * j], acc[4 * j + 1], acc[4 * j + 2], acc[4 * j + 3]);
    }
    if (p.out_lse && lane == 0) p.out_lse[row] = z > 0.f ? mx + __logf(z) : -CUDART_INF_F;
    if (p.out) {
        uint32_t packed[VPL / 2];
#pragma unroll
        for (int j = 0; j < VPL / 2; ++j) {
            float a0 = acc[2 * j], a1 = acc[2 * j + 1];
            if (p.gate) {
                a0 = sigmoid_gate(a0, (uint16_t)(gw[j] & 0xffffu));
                a1 = sigmoid_gate(a1, (uint16_t)(gw[j] >> 16));
            }
            packed[j] = pack_bf16x2(a0, a1);
        }
        for (int c = -1; c < p.n_copies; ++c) {
            uint16_t* o = (c < 0 ? p.out : reinterpret_cast<uint16_t*>(p.out_copies[c])) + eoff + d;
            if (VPL == 8) *reinterpret_cast<uint4*>(o) = make_uint4(packed[0], packed[1], packed[VPL / 2 - 2], packed[VPL / 2 - 1]);
            else *reinterpret_cast<uint2*>(o) = make_uint2(packed[0], packed[1]);
        }
    }
}

// One warp per row (a block per row spent its time being scheduled: thousands of 64-thread blocks).  What bounds it is
// the trips to L2: the parts are taken U at a time.  (Log-sum-exp and values in two trips, four parts at a time: the
// merge of six parts of 2048 rows took 2.6 us more than that of four.)
constexpr int UMERGE_ROWS = 8;  // rows per block

template <int HD, int U>
__global__ void __launch_bounds__(32 * UMERGE_ROWS) sdpa_uniform_merge_kernel(const UniformMergeParams p) {
    const long long row = (long long)blockIdx.x * UMERGE_ROWS + (threadIdx.x >> 5);
    long long eoff = row * HD;
    if (p.seq > 0) {
        const unsigned r = (unsigned)row, tb = r / (unsigned)p.nq, hh = r - tb * (unsigned)p.nq;
        const unsigned bb = tb / (unsigned)p.seq, t = tb - bb * (unsigned)p.seq;
        eoff = bb * p.o_stride_b + t * p.o_stride_t + (long long)hh * HD;
    }
    grid_dependency_wait();  // launched behind the kernel that writes the partials, possibly before it has finished
    grid_launch_dependents();
    if (row >= p.rows) return;
    uint32_t gw[HD / 64];
    load_gate_row<HD>(p, eoff, gw);
    float mx = -CUDART_INF_F, z = 0.f, acc[HD / 32];
#pragma unroll
    for (int j = 0; j < HD / 32; ++j) acc[j] = 0.f;
    for (int i0 = 0; i0 < p.num_parts; i0 += U) {
        float li[U];
        float4 ov[U][HD / 128];
        load_parts<HD, U>(p, row, i0, li, ov);
        fold_parts<HD, U>(li, ov, mx, z, acc);
    }
    store_folded<HD>(p, row, eoff, mx, z, acc, gw);
}

// a[i] = bf16(f32(a[i]) * sigmoid(f32(gate[i]))) : src/modeling/qwen3_5_moe/kernels.hpp:80-88
__global__ void mul_sigmoid_kernel(uint16_t* a, const uint16_t* gate, long long n) {
    grid_dependency_wait();
    grid_launch_dependents();
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        const float g = bf16_bits_to_f32(gate[i]);
        const float sig = sigmoid(g);
        a[i] = __bfloat16_as_ushort(__float2bfloat16_rn(bf16_bits_to_f32(a[i]) * sig));
    }
}

// Additive causal / sliding-window mask : src/common/kernels/attention_mask.hpp:12-38; with
// block_ids (one int per absolute position, -1 = text) tokens of the same non-negative block also
// see each other's future: fill_causal_mask_with_block_ids, attention_mask.hpp:44-73.
// Bound by the stores: a thread writes four consecutive keys of one row, 16 bytes at once where the row allows it, and
// divides nothing (one element per thread and a division per element took 13 us for 1000 x 1300).  SHORT: rows share a block
// (blockDim.y of them; one each took 69 us for 70000 x 64.  An instance of its own: the general one was 0.5 us slower with it).
template <bool IDS, bool SHORT>
__global__ void fill_causal_mask_kernel(float* mask, const int* block_ids, int q_len, int kv_len, int past_offset, int window) {
    grid_dependency_wait();
    grid_launch_dependents();
    const int j0 = (blockIdx.x * blockDim.x + threadIdx.x) * 4;
    if (j0 >= kv_len) return;
    const int first = past_offset - (kv_len - q_len);  // absolute position of key 0
    for (int qi = SHORT ? blockIdx.y * blockDim.y + threadIdx.y : blockIdx.y; qi < q_len; qi += SHORT ? gridDim.y * blockDim.y : gridDim.y) {
        const int q_global = past_offset + qi;
        const int qb = IDS ? block_ids[q_global] : -1;
        float v[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int kv_global = first + j0 + e;
            const bool same_block = IDS && qb >= 0 && kv_global >= 0 && j0 + e < kv_len && qb == block_ids[kv_global];
            const bool causal = !same_block && kv_global > q_global;
            const bool too_far = (window != 0x7fffffff) && (kv_global < q_global - window + 1);
            v[e] = (causal || too_far) ? -CUDART_INF_F : 0.0f;
        }
        float* dst = mask + (long long)qi * kv_len + j0;
        if (j0 + 4 <= kv_len && (reinterpret_cast<uintptr_t>(dst) & 15u) == 0) {
            *reinterpret_cast<float4*>(dst) = make_float4(v[0], v[1], v[2], v[3]);
        } else {
            for (int e = 0; e < 4 && j0 + e < kv_len; ++e) dst[e] = v[e];
        }
    }
}

}  // namespace arc
