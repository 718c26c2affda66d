// C ABI of the sm_100a attention library: argument validation, launch plans,
// TMA tensor maps and kernel launches.  Nothing here allocates device memory or
// synchronises a stream (except the explicit status query); scratch is provided
// by the caller and sized by the *_workspace_bytes functions.
#include "../../include/arc_sdpa.h"

#include <cuda.h>
#include <cuda_runtime.h>

#include <atomic>
#include <cmath>
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <type_traits>
#include <mutex>

#include "decode_sm100.cuh"
#include "prefill_pair_sm100.cuh"
#include "qkv_prepare_sm100.cuh"
#include "prefill_sm100.cuh"
#include "prefill_wide_sm100.cuh"
#include "prefill_chains_sm100.cuh"

namespace arc {

// Per-device status word written by kernels whose bounded waits give up.
__device__ uint32_t g_fault_words[2];

constexpr int kMaxDevices = 64;
// The decode kernel keeps a few bytes of static shared memory; the dynamic part
// may use the opt-in maximum minus this reserve.
constexpr int kDecodeStaticSmem = 1024;

// What the device holds of the CTA pairs of prefill_wide_sm100.cuh at once (the defaults: a B200).
struct WideRoom {
    static constexpr int MOST_FOLDED = WideCfg::MOST_FOLDED;
    int pairs = 74;
    int folded[MOST_FOLDED + 1] = {0, 0, 33, 22, 15};  // clusters of that many pairs
    int clusters(int parts) const { return parts <= MOST_FOLDED ? folded[parts] : 0; }
};

struct DeviceState {
    std::atomic<bool> ready{false};  // set (release) once everything below is written
    uint32_t* fault = nullptr;
    int sm_count = 0;
    int smem_optin = 0;
    int decode_clusters[9] = {};  // [size]: clusters of the one-launch decode the device holds at once
    WideRoom wide;
};

static DeviceState g_dev[kMaxDevices];
static std::mutex g_mu;
static std::atomic<uint64_t> g_launches{0};

using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static EncodeTiledFn g_encode = nullptr;

// Text of the most recent failing CUDA call on this thread (for diagnostics).
static thread_local char g_last_error[256] = "";

static int cuda_fail(const char* what, cudaError_t e) {
    std::snprintf(g_last_error, sizeof(g_last_error), "%s: %s", what, cudaGetErrorString(e));
    cudaGetLastError();
    return ARC_ERR_CUDA;
}

#define ARC_CUDA(call)                                      \
    do {                                                    \
        cudaError_t e_ = (call);                            \
        if (e_ != cudaSuccess) return cuda_fail(#call, e_); \
    } while (0)

template <typename K>
static cudaError_t opt_in_smem(K kernel, int bytes) {
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
}

// How many clusters of `size` CTAs of a kernel the device holds at once (0: none).
template <typename K>
static int clusters_at_once(K kernel, int size, int sm_count, int threads, int smem) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(sm_count / size * size));  // the answer is capped by the grid asked about
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = (size_t)smem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)size;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return n;
}

// The instances of the kernels of head dim 128 for a call; the common ones carry nothing they do not need.
using PairKernel = void (*)(CUtensorMap, CUtensorMap, CUtensorMap, CUtensorMap, CUtensorMap, PrefillParams);
static PairKernel pair_kernel(bool gate, bool copies, bool vision) {
    if (vision) return gate ? sdpa_prefill_pair_kernel<true, true, true> : copies ? sdpa_prefill_pair_kernel<false, true, true> : sdpa_prefill_pair_kernel<false, false, true>;
    if (copies) return gate ? sdpa_prefill_pair_kernel<true, true> : sdpa_prefill_pair_kernel<false, true>;
    return gate ? sdpa_prefill_pair_kernel<true, false> : sdpa_prefill_pair_kernel<false, false>;
}
using ChainsKernel = void (*)(CUtensorMap, CUtensorMap, CUtensorMap, PrefillParams);
static ChainsKernel chains_kernel(bool gate, bool vision, bool masked) {
    if (masked) return gate ? sdpa_prefill_chains_kernel<true, false, true> : sdpa_prefill_chains_kernel<false, false, true>;
    if (vision) return gate ? sdpa_prefill_chains_kernel<true, true, false> : sdpa_prefill_chains_kernel<false, true, false>;
    return gate ? sdpa_prefill_chains_kernel<true, false, false> : sdpa_prefill_chains_kernel<false, false, false>;
}

using WideKernel = void (*)(CUtensorMap, CUtensorMap, CUtensorMap, CUtensorMap, CUtensorMap, PrefillParams);
static WideKernel wide_kernel(bool gate, bool masked, int split, bool several, bool vision) {  // (several: units per CTA pair)
    if (split == 2 && gate) return masked ? sdpa_prefill_wide_kernel<true, true, 2> : vision ? sdpa_prefill_wide_kernel<true, false, 2, false, true> : sdpa_prefill_wide_kernel<true, false, 2>;
    if (split == 2) return masked ? sdpa_prefill_wide_kernel<false, true, 2> : vision ? sdpa_prefill_wide_kernel<false, false, 2, false, true> : sdpa_prefill_wide_kernel<false, false, 2>;
    if (split == 1) return masked ? sdpa_prefill_wide_kernel<false, true, 1> : vision ? sdpa_prefill_wide_kernel<false, false, 1, false, true> : sdpa_prefill_wide_kernel<false, false, 1>;
    if (several || vision) {  // (979 tokens with four images, one unit a pair: 17.4 us, 17.75 without the walks)
        if (masked) return gate ? sdpa_prefill_wide_kernel<true, true, 0, true> : sdpa_prefill_wide_kernel<false, true, 0, true>;
        if (vision) return gate ? sdpa_prefill_wide_kernel<true, false, 0, true, true> : sdpa_prefill_wide_kernel<false, false, 0, true, true>;
        return gate ? sdpa_prefill_wide_kernel<true, false, 0, true> : sdpa_prefill_wide_kernel<false, false, 0, true>;
    }
    if (masked) return gate ? sdpa_prefill_wide_kernel<true, true> : sdpa_prefill_wide_kernel<false, true>;
    return gate ? sdpa_prefill_wide_kernel<true, false> : sdpa_prefill_wide_kernel<false, false>;
}

// One-time set-up for the current device: status-word address, SM count, and the
// dynamic shared memory opt-in of every kernel.
static int device_state(DeviceState** out) {
    int dev = 0;
    ARC_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kMaxDevices) return ARC_ERR_CUDA;
    DeviceState& s = g_dev[dev];
    if (!s.ready.load(std::memory_order_acquire)) {
        std::lock_guard<std::mutex> lock(g_mu);
        if (!s.ready.load(std::memory_order_relaxed)) {
            void* sym = nullptr;
            ARC_CUDA(cudaGetSymbolAddress(&sym, g_fault_words));
            s.fault = static_cast<uint32_t*>(sym);
            ARC_CUDA(cudaDeviceGetAttribute(&s.sm_count, cudaDevAttrMultiProcessorCount, dev));
            ARC_CUDA(cudaDeviceGetAttribute(&s.smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
            if (!g_encode) {
                void* fn = nullptr;
                cudaDriverEntryPointQueryResult qres = cudaDriverEntryPointSymbolNotFound;
                ARC_CUDA(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres));
                if (qres != cudaDriverEntryPointSuccess || fn == nullptr) {
                    std::snprintf(g_last_error, sizeof(g_last_error), "cuTensorMapEncodeTiled not found in the driver");
                    return ARC_ERR_CUDA;
                }
                g_encode = reinterpret_cast<EncodeTiledFn>(fn);
            }
            for (int i = 0; i < 8; ++i) {
                ARC_CUDA(opt_in_smem(pair_kernel(i & 1, i & 2, i & 4), PairCfg::SMEM_BYTES));
                ARC_CUDA(opt_in_smem(chains_kernel(i & 1, i & 2, i & 4), ChainsCfg::SMEM_BYTES));
            }
            ARC_CUDA(opt_in_smem(sdpa_prefill_kernel, PrefillCfg::SMEM_BYTES));
            for (int i = 0; i < 48; ++i) ARC_CUDA(opt_in_smem(wide_kernel(i & 1, i & 2, i / 16, i & 4, i & 8), WideCfg::SMEM_BYTES));
            s.wide.pairs = clusters_at_once(sdpa_prefill_wide_kernel<false, false>, 2, s.sm_count, WideCfg::THREADS, WideCfg::SMEM_BYTES);
            for (int parts = 2; parts <= WideRoom::MOST_FOLDED; ++parts)
                s.wide.folded[parts] = clusters_at_once(sdpa_prefill_wide_kernel<false, false, 2>, 2 * parts, s.sm_count, WideCfg::THREADS, WideCfg::SMEM_BYTES);
            if (s.wide.pairs < 1) {
                std::snprintf(g_last_error, sizeof(g_last_error), "the device cannot hold a CTA pair of the prefill kernel");
                return ARC_ERR_CUDA;
            }
            ARC_CUDA(opt_in_smem(sdpa_decode_kernel<128, 1, false>, s.smem_optin - kDecodeStaticSmem));
            ARC_CUDA(opt_in_smem(sdpa_decode_kernel<128, 1, true>, s.smem_optin - kDecodeStaticSmem));
            ARC_CUDA(opt_in_smem(sdpa_decode_kernel<128, 1, true, true>, s.smem_optin - kDecodeStaticSmem));
            ARC_CUDA(opt_in_smem(sdpa_decode_kernel<128, 2, false>, s.smem_optin - kDecodeStaticSmem));
            ARC_CUDA(opt_in_smem(sdpa_decode_kernel<128, 2, true>, s.smem_optin - kDecodeStaticSmem));
            ARC_CUDA(opt_in_smem(sdpa_decode_kernel<128, 2, true, true>, s.smem_optin - kDecodeStaticSmem));
            ARC_CUDA(opt_in_smem(sdpa_decode_kernel<256, 1, false>, s.smem_optin - kDecodeStaticSmem));
            ARC_CUDA(opt_in_smem(sdpa_decode_kernel<256, 1, true>, s.smem_optin - kDecodeStaticSmem));
            ARC_CUDA(opt_in_smem(sdpa_decode_kernel<256, 1, true, true>, s.smem_optin - kDecodeStaticSmem));
            ARC_CUDA(opt_in_smem(sdpa_decode_kernel<256, 2, false>, s.smem_optin - kDecodeStaticSmem));
            ARC_CUDA(opt_in_smem(sdpa_decode_kernel<256, 2, true>, s.smem_optin - kDecodeStaticSmem));
            ARC_CUDA(opt_in_smem(sdpa_decode_kernel<256, 2, true, true>, s.smem_optin - kDecodeStaticSmem));
            for (int size = 1; size <= 8; ++size)
                s.decode_clusters[size] = clusters_at_once(sdpa_decode_kernel<256, 1, true>, size, s.sm_count, 288, s.smem_optin - kDecodeStaticSmem);
            s.ready.store(true, std::memory_order_release);
        }
    }
    *out = &s;
    return ARC_OK;
}

// Launch `kernel` behind the previous kernel of `stream` with programmatic serialization: its CTAs may be scheduled and
// run up to their grid_dependency_wait() while that kernel is still running, which takes the launch latency and the
// prologue off the critical path (2-3 us of a small call).  Every kernel of the library is launched this way, and every
// one of them waits before it touches global memory and only then releases the kernel behind it
// (grid_launch_dependents): so when a kernel may run, everything in front of its predecessor has completed, and no grid
// completes before the one in front of it has.  cluster > 1: in clusters of that many CTAs along x.
template <typename... KArgs, typename... Args>
static cudaError_t launch_dependent(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, int cluster,
                                    Args... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = (unsigned)cluster;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = cluster > 1 ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, kernel, KArgs(args)...);
}

static bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// (hd, heads, tokens, batch) view of a token-major bf16 tensor; box = 64 x 1 x box_rows x 1, 128-byte swizzle.
static int make_tile_map(CUtensorMap* tm, const void* base, int hd, int heads, int tokens, int batch,
                         int64_t stride_t, int64_t stride_b, int box_rows = 128) {
    cuuint64_t dims[4] = {(cuuint64_t)hd, (cuuint64_t)heads, (cuuint64_t)tokens, (cuuint64_t)batch};
    cuuint64_t sb = (cuuint64_t)(batch > 1 ? stride_b : stride_t * (int64_t)tokens) * 2u;
    cuuint64_t strides[3] = {(cuuint64_t)hd * 2u, (cuuint64_t)stride_t * 2u, sb};
    cuuint32_t box[4] = {64u, 1u, (cuuint32_t)box_rows, 1u};
    cuuint32_t estr[4] = {1u, 1u, 1u, 1u};
    CUresult r = g_encode(tm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(base), dims, strides, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        std::snprintf(g_last_error, sizeof(g_last_error), "cuTensorMapEncodeTiled failed with CUresult %d", (int)r);
        return ARC_ERR_CUDA;
    }
    return ARC_OK;
}

// Output and gate as the epilogue warps see them: boxes of 64 columns x 32 rows.
static int make_out_maps(CUtensorMap* to, CUtensorMap* tg, const arc_sdpa_prefill_params* p) {
    const int rc = make_tile_map(to, p->out, p->hd, p->nq, p->seq, p->batch, p->o_stride_t, p->o_stride_b, 32);
    if (rc != ARC_OK || !p->gate) {
        *tg = *to;
        return rc;
    }
    return make_tile_map(tg, p->gate, p->hd, p->nq, p->seq, p->batch, p->o_stride_t, p->o_stride_b, 32);
}

// (nkv*hd, rows) view of a KV cache whose rows are `stride_t` elements apart;
// box = 64 columns x `box_rows` rows, 128-byte swizzle; rows past `rows` read as zero.
static int make_cache_map(CUtensorMap* tm, const void* base, int row_elems, int64_t rows, int64_t stride_t,
                          int box_rows) {
    cuuint64_t dims[2] = {(cuuint64_t)row_elems, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)stride_t * 2u};
    cuuint32_t box[2] = {64u, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1u, 1u};
    CUresult r = g_encode(tm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        std::snprintf(g_last_error, sizeof(g_last_error), "cuTensorMapEncodeTiled (cache) failed with CUresult %d", (int)r);
        return ARC_ERR_CUDA;
    }
    return ARC_OK;
}

// ---------------------------------------------------------------------------
// Prefill plan
// ---------------------------------------------------------------------------
struct PrefillPlan {
    int q_tiles = 0;
    int splits = 1;
    long long rows = 0;
    size_t ws_bytes = 0;    // what must be there: partial records of key-range splits
    size_t mask_bytes = 0;  // behind it, if it is there: the classes and bits of an additive mask
};

// Key blocks that token tile qt (128 rows) of a call sees, block ids apart.
static int tile_key_blocks(const arc_sdpa_prefill_params* p, int qt) {
    const int blocks = (p->kv_len + 127) / 128, off = p->kv_len - p->seq;
    if (p->mask_type != ARC_MASK_CAUSAL) return blocks;
    const int last = std::min(p->kv_len - 1, std::min(qt * 128 + 127, p->seq - 1) + off);
    const int hi = last >= 0 ? last / 128 + 1 : 0, lo = p->window > 0 && p->window != 0x7fffffff ? std::max(0, qt * 128 + off - p->window + 1) / 128 : 0;
    return std::max(0, hi - lo);
}

// Head dim 256: units of the CTA pairs' list.
static long long wide_units(const arc_sdpa_prefill_params* p, int q_tiles) {
    const bool head_pair = ((p->nq / p->nkv) & 1) == 0;
    return (head_pair ? (long long)q_tiles * (p->nq / 2) : (long long)((p->seq + 255) / 256) * p->nq) * p->batch;
}

// Do the parts of a unit fold themselves, as one cluster?  Two and three do where all clusters fit at once; four where the library chose
// them and there is neither gate nor additive mask (the merge launch gates for nothing, and is as good where most blocks are hidden).
// Four that the caller asked for keep the two launches, and the bits, that they had before four could fold themselves: who gives a
// count, unlike who leaves it to the library, may count on either.
static bool folds_itself(const arc_sdpa_prefill_params* p, int parts, long long units, const WideRoom& room) {
    if (parts > 3 && (p->num_splits != 0 || p->gate || p->mask_type == ARC_MASK_EXPLICIT)) return false;
    return units <= room.clusters(parts);
}

// How many parts the key range of each unit is worth when the units alone would leave pairs idle: what a call takes besides what all
// calls have in common (us; n pairs; rows: the part of a tile's 128 that there are, where they are stored).  Fitted to 20 to 512
// rows of 4 to 24 heads over 384 to 8000 keys in every number of parts.  (256 queries of 16 heads over 2304 keys: 25.6 whole, 17.1 in
// two parts, 15.6 in three, 18.2 in four with a merge; of 8 heads 25.5, 13.7 in four.  Gated, 128 of 8 heads over 700 keys: 13.8 whole,
// 10.7 in three parts, 12.1 in five; three sequences of 45 queries, 4 heads, over 1000: 10.8 in three, 10.0 in four, 10.6 in eight.)
struct WideCosts {
    double block, block_n;                          // a part's key blocks, each
    double whole;                                   // the epilogue of whole units
    double fold, fold_4, fold_n, fold_rows;         // parts that fold themselves: two or three, four, per pair, per pair and rows
    double merge, merge_more, merge_n, merge_rows;  // a merge launch: up to four parts, more, per pair, per pair and rows
};
constexpr WideCosts kWidePlain = {1.11, 0.0022, 0.0, 0.6, 1.2, 0.0, 0.045, 2.2, 2.2, 0.0, 0.073};
constexpr WideCosts kWideGated = {1.4, 0.0, 1.8, 1.7, 1.7, 0.02, 0.012, 1.5, 1.8, 0.026, 0.06};
// (Of an additive mask's blocks some are hidden, which is not known here: a block counts less.)
constexpr WideCosts kWideMasked = {1.11, 0.0022, 0.0, 1.8, 1.8, 0.0, 0.045, 2.2, 2.2, 0.0, 0.073};
constexpr WideCosts kWideMaskedGated = {1.13, 0.0, 1.4, 2.0, 2.0, 0.012, 0.028, 2.5, 2.5, 0.018, 0.042};

static int choose_wide_splits(const arc_sdpa_prefill_params* p, int q_tiles, const WideRoom& room) {
    const long long units = wide_units(p, q_tiles);
    if (units * 2 > room.pairs) return 1;
    const bool masked = p->mask_type == ARC_MASK_EXPLICIT;
    const bool windowed = p->mask_type == ARC_MASK_CAUSAL && p->window > 0 && p->window < p->kv_len && !p->block_ids;
    int most = (p->kv_len + 127) / 128;  // key blocks of the longest unit
    // What an additive mask hides is not known here.  Over the few blocks of a window the parts of 2048 rows cost 5 us more
    // than they save (256 queries of 8 heads over 2304 keys: 16.4 us whole and 21.1; with all keys seen 30.3 and 23.9); 1024
    // rows are even (64 queries of 16 heads over 4096 keys: 15.9 and 15.6; 45 and 20).  A longer cache is worth it in any case (a
    // bias per key, 128 queries of 16 heads over 4096 keys: 116 us whole).
    if (masked && most <= 24 && (long long)p->batch * p->seq * p->nq > 1024) return 1;
    if (windowed) {
        most = std::min(most, (p->window + 255) / 128 + 1);
        // (That is the most that a window can cover, up to two more than it does.  Gated calls, whose epilogue and merge weigh more, are
        // divided by what it does: 256 queries of 8 heads over 1500 keys, window 533, 11.5 us in three parts, 13.2 in four.  For the others
        // the bound is the better guess: 63 of 24 heads over 1000 keys 9.9 in four, 10.4 in three.)
        if (p->gate) {
            const int tiles = ((p->nq / p->nkv) & 1) == 0 ? 1 : 2;  // token tiles of a unit
            int seen = 0;
            for (int qt = 0; qt < q_tiles; qt += tiles) {
                const int last = std::min(q_tiles, qt + tiles) - 1, blocks = tile_key_blocks(p, last);
                seen = std::max(seen, blocks + (last > qt && blocks > 0 ? 1 : 0));
            }
            most = std::min(most, seen);
        }
    }
    // Two blocks are not divided: the second one's scores run under the first one's softmax (128 queries of 8 heads over 256 keys: 7.6
    // whole, 7.95 in two parts).
    if (most <= 2) return 1;
    const WideCosts& c = masked ? (p->gate ? kWideMaskedGated : kWideMasked) : p->gate ? kWideGated : kWidePlain;
    const double rows = std::min<int>(p->seq, 128) / 128.0;
    // Behind a window a unit's first two blocks are tested key by key, which shows where one part has both.  (45 queries of 8 heads over
    // 663 keys, window 533: 9.8 in three parts of two blocks, 9.1 in six, 9.0 in four, whose first is one; without a window 9.05, 9.04, 8.9.)
    const auto edge = [&](int parts) { return windowed && most / parts >= 2 ? 1.0 : 0.0; };
    int best = 1;
    double least = c.block * most + c.whole + edge(1);
    for (int s = 2; s <= 8 && s <= most && units * s <= room.pairs; ++s) {
        const double n = (double)(units * s), blocks = (c.block + c.block_n * n) * ((most + s - 1) / s) + edge(s);
        const double t = blocks + (folds_itself(p, s, units, room) ? (s == 4 ? c.fold_4 : c.fold) + (c.fold_n + c.fold_rows * rows) * n
                                                                   : (s > 4 ? c.merge_more : c.merge) + (c.merge_n + c.merge_rows * rows) * n);
        if (t < least) least = t, best = s;
    }
    return best;
}

static int plan_prefill(const arc_sdpa_prefill_params* p, int sm_count, const WideRoom& room, PrefillPlan* plan) {
    if (!p) return ARC_ERR_NULL_POINTER;
    if (p->batch <= 0 || p->seq <= 0 || p->kv_len <= 0 || p->nq <= 0 || p->nkv <= 0 || p->nq % p->nkv != 0)
        return ARC_ERR_BAD_SHAPE;
    if (p->hd != 128 && p->hd != 256) return ARC_ERR_UNSUPPORTED_HEAD_DIM;
    if (!(p->scale > 0.f) || !std::isfinite(p->scale)) return ARC_ERR_BAD_SHAPE;
    if (p->mask_type != ARC_MASK_NONE && p->mask_type != ARC_MASK_EXPLICIT && p->mask_type != ARC_MASK_CAUSAL)
        return ARC_ERR_BAD_SHAPE;
    if (p->num_splits < 0) return ARC_ERR_BAD_SHAPE;
    plan->q_tiles = (p->seq + 127) / 128;
    plan->rows = (long long)p->batch * p->seq * p->nq;
    const int kv_blocks = (p->kv_len + 127) / 128;
    int splits = p->num_splits;
    const long long tiles = (long long)plan->q_tiles * p->nq * p->batch;
    const bool scanned_mask = p->mask_type == ARC_MASK_EXPLICIT && p->hd == 256 && p->num_splits <= 1;
    if (splits == 0 && p->hd == 256) splits = choose_wide_splits(p, plan->q_tiles, room);
    if (splits == 0) {
        // Head dim 128: split the key range when the tiles alone leave most SMs idle and there are enough key blocks to pay
        // for folding the parts again, into as many parts as take least: a key block is 0.71 us, records and merge 0.028 a part.
        // (8 tiles of 12 / 16 / 32 blocks: 12.4 / 16.1 / 28.9 us whole, 10.6 / 11.3 / 14.5 in four parts, 10.5 / 10.7 / 12.3 in
        // eight; 32 tiles of 16: 16.8 whole, 16.2 in two, 13.5 in four.)
        splits = 1;
        if (tiles * 2 <= sm_count && kv_blocks >= 10) {
            double least = 1e30;
            for (int s = 2; s <= 8 && 2 * s <= kv_blocks && tiles * s <= sm_count; ++s) {
                const double t = 0.71 * ((kv_blocks + s - 1) / s) + 0.028 * (double)(tiles * s);
                if (t < least) least = t, splits = s;
            }
        }
    }
    if (splits > kv_blocks) splits = kv_blocks;
    if (splits > 64) splits = 64;
    plan->splits = splits;
    plan->ws_bytes = splits > 1 ? (size_t)splits * plan->rows * ((size_t)p->hd + 1) * sizeof(float) : 0;
    plan->ws_bytes = (plan->ws_bytes + 15) & ~(size_t)15;
    if (scanned_mask) plan->mask_bytes = (size_t)plan->q_tiles * kv_blocks * (128 * sizeof(uint4) + sizeof(uint32_t));
    if (p->block_ids && (p->mask_type != ARC_MASK_CAUSAL || p->block_ids_offset < 0)) return ARC_ERR_BAD_SHAPE;
    return ARC_OK;
}

// The parts of a split key range, folded, gated and stored.
template <int HD>
static int launch_fold(const arc_sdpa_prefill_params* p, const PrefillPlan& plan, const PrefillParams& kp, cudaStream_t stream) {
    UniformMergeParams mp{};
    mp.part_o = kp.part_o;
    mp.part_lse = kp.part_lse;
    mp.gate = kp.gate;
    mp.out = kp.out;
    mp.out_f32 = nullptr;
    mp.out_lse = p->out_lse;
    mp.rows = plan.rows;
    mp.num_parts = plan.splits;
    mp.o_part_stride = plan.rows * HD;
    mp.lse_part_stride = plan.rows;
    mp.seq = p->seq;
    mp.nq = p->nq;
    mp.o_stride_b = p->o_stride_b;
    mp.o_stride_t = p->o_stride_t;
    mp.out_copies = kp.out_copies;
    mp.n_copies = kp.n_copies;
    ARC_CUDA(launch_dependent(plan.splits <= 4 ? sdpa_uniform_merge_kernel<HD, 4> : sdpa_uniform_merge_kernel<HD, 8>, dim3((unsigned)((plan.rows + UMERGE_ROWS - 1) / UMERGE_ROWS)),
                              dim3(32 * UMERGE_ROWS), 0, stream, 1, mp));
    g_launches.fetch_add(1, std::memory_order_relaxed);
    return ARC_OK;
}

// What the SM (or CTA pair) with most to do takes for its share of the units [u0, u1) (`heads` per token tile and sequence, of
// `tiles` token tiles each), which are dealt to `sms` of them longest first and every second wave in reverse, a unit taking
// per_block for each of its key blocks and per_unit.  The load is linear in the SM's index between the ends of the waves, so
// these are what is looked at.
static double longest_sorted_share(const arc_sdpa_prefill_params* p, long long u0, long long u1, int heads, int tiles, long long sms, double per_block, double per_unit) {
    const int q_tiles = (p->seq + 127) / 128;
    const long long units = u1 - u0, waves = (units + sms - 1) / sms, rest = units - (waves - 1) * sms;
    const long long per = (long long)heads * p->batch, edge = (waves & 1) ? rest : sms - rest;
    double most = 0.0;
    for (long long x : {0ll, sms - 1, edge - 1, edge}) {
        if (x < 0 || x >= sms) continue;
        double sum = 0.0;
        for (long long i = 0; i < waves; ++i) {
            const long long u = i * sms + ((i & 1) ? sms - 1 - x : x);
            if (u < units) sum += per_block * tile_key_blocks(p, std::min(q_tiles - 1, (int)((q_tiles + tiles - 1) / tiles - 1 - (u0 + u) / per) * tiles + tiles - 1)) + per_unit;
        }
        most = std::max(most, sum);
    }
    return most;
}

// The same of all `units` units, or, dealt in plain order, as if all were as long as the longest.
static double longest_share(const arc_sdpa_prefill_params* p, long long units, int heads, int tiles, long long sms, bool by_length, double per_block, double per_unit) {
    const long long waves = (units + sms - 1) / sms;
    if (!by_length || waves > 16) return (double)waves * (per_block * tile_key_blocks(p, (p->seq + 127) / 128 - 1) + per_unit);
    return longest_sorted_share(p, 0, units, heads, tiles, sms, per_block, per_unit);
}

// Longest first, all heads and sequences of a token tile run side by side: do the keys and values that they read together stay in
// L2 (126 MB)?  All of them may, where there are few waves or no window; behind a window it is the window's and those of the tiles under
// way that are read at one time.  In plain order the shorter first tiles of a windowed call fall to some CTAs only, however many waves
// there are, where the count of token tiles and the grid share a factor: 5 to 20 % between the fullest CTA and the mean.  (us, plain and
// longest first, window 1024 unless said: 8192 tokens of 24/4 heads of 256 184 and 177; 2 x 8192 of 28/4 of 128, window 2048, 399
// and 378; 4 x 6000 of 16/8, window 300, 120 and 111; but 4 x 8192 of 32/16, whose windows are 48 MB, 534 and 577.)
static bool stays_in_l2(const arc_sdpa_prefill_params* p, bool few_waves) {
    const bool windowed = p->window > 0 && p->window < p->kv_len;
    const long long key = (long long)p->batch * p->nkv * p->hd * 4;
    if (windowed && std::min<long long>(p->kv_len, (long long)p->window + 512) * key <= 24ll << 20) return true;
    return (few_waves || !windowed) && p->kv_len * key <= 96ll << 20;
}

// Digits of a grid of `ctas` in the tile list, fastest first (TileCursor).
static void set_step(PrefillParams* kp, long long ctas) {
    const long long rf = kp->long_first ? kp->cur_heads : kp->q_tiles, rm = kp->long_first ? kp->batch : kp->cur_heads;
    kp->step[0] = (int)(ctas % rf);
    kp->step[1] = (int)(ctas / rf % rm);
    kp->step[2] = (int)(ctas / rf / rm);
}

template <int HD>
static int launch_prefill(const arc_sdpa_prefill_params* p, const PrefillPlan& plan, DeviceState* ds,
                          cudaStream_t stream) {
    CUtensorMap tq, tk, tv, to, tg;
    int rc;
    if ((rc = make_tile_map(&tq, p->q, HD, p->nq, p->seq, p->batch, p->q_stride_t, p->q_stride_b)) != ARC_OK) return rc;
    if ((rc = make_tile_map(&tk, p->k, HD, p->nkv, p->kv_len, p->batch, p->k_stride_t, p->k_stride_b)) != ARC_OK) return rc;
    if ((rc = make_tile_map(&tv, p->v, HD, p->nkv, p->kv_len, p->batch, p->v_stride_t, p->v_stride_b)) != ARC_OK) return rc;

    PrefillParams kp{};
    kp.out = static_cast<uint16_t*>(p->out);
    kp.out_copies = reinterpret_cast<const unsigned long long*>(p->out_copies);
    kp.n_copies = p->out_copies ? p->out_copy_count : 0;
    kp.gate = static_cast<const uint16_t*>(p->gate);
    kp.mask = p->mask_type == ARC_MASK_EXPLICIT ? p->mask : nullptr;
    kp.out_lse = p->out_lse;
    kp.part_o = plan.splits > 1 ? static_cast<float*>(p->workspace) : nullptr;
    kp.part_lse = kp.part_o ? kp.part_o + (size_t)plan.splits * plan.rows * HD : nullptr;
    const bool wide = HD == 256 && (plan.splits == 1 || p->mask_type != ARC_MASK_EXPLICIT || plan.mask_bytes > 0);
    if (p->block_ids) kp.ids = p->block_ids + p->block_ids_offset;
    kp.fault = ds->fault;
    kp.batch = p->batch;
    kp.seq = p->seq;
    kp.kv_len = p->kv_len;
    kp.nq = p->nq;
    kp.nkv = p->nkv;
    kp.o_stride_b = p->o_stride_b;
    kp.o_stride_t = p->o_stride_t;
    kp.scale_log2 = p->scale * 1.4426950408889634f;
    kp.mask_type = p->mask_type;
    kp.window = p->window;
    kp.num_splits = plan.splits;
    kp.group = p->nq / p->nkv;
    kp.group_shift = -1;
    kp.tail_base = -1;
    for (int sh = 0; sh < 31; ++sh)
        if ((1 << sh) == kp.group) kp.group_shift = sh;

    const bool masked = kp.mask_type == ARC_MASK_EXPLICIT && kp.mask != nullptr;
    // Head dim 128: two query tiles per CTA (prefill_pair_sm100.cuh), or one in two chains of key blocks
    // (prefill_chains_sm100.cuh), whichever covers the tiles faster; the latter for additive masks and parts of a key range.
    // ARC_SDPA_PREFILL_KERNEL=single|pair overrides the choice (for A/B measurements).
    if constexpr (HD == 128) {
        static const int forced = [] {
            const char* e = std::getenv("ARC_SDPA_PREFILL_KERNEL");
            if (!e) return 0;
            return std::strcmp(e, "pair") == 0 ? 2 : (std::strcmp(e, "single") == 0 ? 1 : 0);
        }();
        const bool split = plan.splits > 1;
        // A CTA takes two 128-row tiles: the same tokens of two heads of one KV group when the group
        // size is even (both tiles then see exactly the same key blocks), else 256 tokens of one head.
        const bool head_pair = ((p->nq / p->nkv) & 1) == 0;
        const long long pair_tiles = head_pair ? (long long)plan.q_tiles * (p->nq / 2) * p->batch
                                               : (long long)((p->seq + 255) / 256) * p->nq * p->batch;
        const long long single_tiles = (long long)plan.q_tiles * p->nq * p->batch * plan.splits;
        const long long sms = ds->sm_count;
        // The pairs left over after the last whole wave of CTAs may be cut into their two heads when every SM then
        // gets at most one of them: a second launch (a tile per CTA, scheduled behind this
        // one as SMs free up) takes them, and no SM runs a whole pair while the others idle.  It pays for a few calls in a
        // hundred, of three waves and more (4 x 1728 tokens of 32/16 heads, no mask, by the measure below: 97.9 cut, 101.5 whole, 105.0 in
        // chains); in others chains cover the tiles more evenly.
        const long long full_waves = pair_tiles / sms, left = pair_tiles - full_waves * sms;
        // Under a causal mask tiles differ in length and go longest first, as at head dim 256 below, with the same limit.
        const auto by_length = [&](long long units) {
            return !split && p->mask_type == ARC_MASK_CAUSAL && units > sms && stays_in_l2(p, units < 8 * sms);
        };
        // In steps of a key block of a pair (1.37 us): launches, loads and output apart, a pair's unit takes its blocks and
        // half a step, a tile in chains 0.52 a block and 0.8.  A second launch for the tail adds 3.6 (it starts when the first
        // one's CTAs end).  (16 heads, 1152 queries, 512 / 2048 keys: 8.7 / 17.2 us in chains, 11.4 / 27.9 in pairs; 2304
        // queries 14 / 32, 13 / 31; 2000 causal queries of 28 heads: 29 in pairs, 31 in chains.)
        bool use_pair = false, cut_tail = false;
        if (!split && !masked && forced != 1 && (forced == 2 || single_tiles > sms)) {
            const int heads = head_pair ? p->nq / 2 : p->nq, tiles = head_pair ? 1 : 2;
            const bool sorted = by_length(pair_tiles);
            double cost_pair = longest_share(p, pair_tiles, heads, tiles, sms, sorted, 1.0, 0.5);
            if (head_pair && full_waves > 0 && left > 0 && 2 * left <= sms) {
                const int first = sorted ? plan.q_tiles - 1 - (int)(full_waves * sms / ((long long)heads * p->batch)) : plan.q_tiles - 1;  // the tail's longest
                const double cost_cut = longest_share(p, full_waves * sms, heads, 1, sms, sorted, 1.0, 0.5) + 3.6 + 0.52 * tile_key_blocks(p, first);
                cut_tail = cost_cut < cost_pair;
                cost_pair = std::min(cost_pair, cost_cut);
            }
            use_pair = forced == 2 || cost_pair <= longest_share(p, single_tiles, p->nq, 1, sms, by_length(single_tiles), 0.52, 0.8);
        }
        if ((use_pair ? pair_tiles : single_tiles) > 0x7fffffffLL) return ARC_ERR_TOO_LARGE;
        kp.long_first = by_length(use_pair ? pair_tiles : single_tiles);
        PrefillParams cp = kp;  // tiles one by one
        cp.head_pair = 0;
        cp.cur_heads = p->nq;
        cp.q_tiles = plan.q_tiles;
        cp.total_tiles = (int)single_tiles;
        auto launch_chains = [&](long long ctas) -> int {
            set_step(&cp, ctas);
            ARC_CUDA(launch_dependent(chains_kernel(cp.gate && !split, cp.ids != nullptr, masked), dim3((unsigned)ctas), dim3(ChainsCfg::THREADS),
                                      (size_t)ChainsCfg::SMEM_BYTES, stream, 1, tq, tk, tv, cp));
            g_launches.fetch_add(1, std::memory_order_relaxed);
            return ARC_OK;
        };
        if (!use_pair) {
            if ((rc = launch_chains(std::min(single_tiles, sms))) != ARC_OK) return rc;
            return split ? launch_fold<HD>(p, plan, kp, stream) : ARC_OK;
        }
        kp.head_pair = head_pair ? 1 : 0;
        kp.cur_heads = head_pair ? p->nq / 2 : p->nq;
        kp.q_tiles = head_pair ? plan.q_tiles : (p->seq + 255) / 256;
        const long long pair_units = cut_tail ? full_waves * sms : pair_tiles;
        kp.total_tiles = (int)pair_units;
        set_step(&kp, std::min(pair_units, sms));
        if ((rc = make_out_maps(&to, &tg, p)) != ARC_OK) return rc;
        ARC_CUDA(launch_dependent(pair_kernel(kp.gate != nullptr, kp.n_copies > 0, kp.ids != nullptr), dim3((unsigned)std::min(pair_units, sms)), dim3(PairCfg::THREADS),
                                  (size_t)PairCfg::SMEM_BYTES, stream, 1, tq, tk, tv, to, tg, kp));
        g_launches.fetch_add(1, std::memory_order_relaxed);
        if (!cut_tail) return ARC_OK;
        cp.tail_base = (int)pair_units;
        cp.total_tiles = (int)(2 * left);
        return launch_chains(2 * left);
    }

    // Head dim 256, whole tiles, no additive mask: pairs of CTAs (prefill_wide_sm100.cuh) take 2300-2500 clk per key block
    // and pair of tiles where a CTA on its own takes 3700 per tile.
    // (a caller who brings no workspace for the scanned mask gets the one-tile kernel, which reads the mask itself)
    if (wide &&
        (!masked || (plan.mask_bytes > 0 && plan.q_tiles < 16384 && p->workspace && aligned16(p->workspace) && p->workspace_bytes >= plan.ws_bytes + plan.mask_bytes))) {
        if (masked) {
            kp.mask_blocks = (p->kv_len + 127) / 128;
            uint4* bits = reinterpret_cast<uint4*>(static_cast<unsigned char*>(p->workspace) + plan.ws_bytes);
            uint32_t* cls = reinterpret_cast<uint32_t*>(bits + (size_t)plan.q_tiles * kp.mask_blocks * 128);
            ARC_CUDA(launch_dependent(mask_scan_kernel, dim3((unsigned)kp.mask_blocks, (unsigned)plan.q_tiles * 4), dim3(512), 0, stream, 1,
                                      kp.mask, (int)p->seq, (int)p->kv_len, kp.mask_blocks, cls, reinterpret_cast<uint32_t*>(bits)));
            g_launches.fetch_add(1, std::memory_order_relaxed);
            kp.mask_bits = bits;
            kp.mask_class = cls;
        }
        const bool split = plan.splits > 1;
        kp.head_pair = ((p->nq / p->nkv) & 1) == 0;
        kp.cur_heads = kp.head_pair ? p->nq / 2 : p->nq;
        kp.q_tiles = kp.head_pair ? plan.q_tiles : (p->seq + 255) / 256;
        const long long units = wide_units(p, plan.q_tiles) * plan.splits;
        if (units > 0x3fffffffLL) return ARC_ERR_TOO_LARGE;
        kp.total_tiles = (int)units;
        // Under a causal mask (as most additive ones are, too) units differ in length and go longest first then, unless K and V would
        // not stay in L2.  (1531 tokens, window 1024, 96 units on 74 pairs: 36.5 -> 27 us.)
        kp.long_first = !split && p->mask_type != ARC_MASK_NONE && units > ds->wide.pairs && stays_in_l2(p, units < 8LL * ds->wide.pairs);
        // A few waves: with k whole ones, the pairs that get k units may as well have the longest and leave the rest, which are
        // shorter, to those that get k + 1.  (2048 queries over 5049 keys, 24 heads: 192 units of 25 to 40 blocks on 74 pairs, the fullest with
        // 96 blocks in one list and 91 so, 84 on average: 153 -> 147 us, gated 165 -> 158; 1664 tokens of 24/4 34.0 -> 32.5.  Vision prompts of
        // 96 to 160 units, and 8192 tokens of 24/4 behind a window of 1024, as fast either way.)
        const long long pairs = ds->wide.pairs, whole = units / pairs, extra = units % pairs;
        if (kp.long_first && !masked && extra > 0 && whole <= 8) {
            const int tiles = kp.head_pair ? 1 : 2;
            const long long few = pairs - extra, end = whole * few;
            const double as_one = longest_sorted_share(p, 0, units, kp.cur_heads, tiles, pairs, 1.0, 1.0);
            if (std::max(longest_sorted_share(p, 0, end, kp.cur_heads, tiles, few, 1.0, 1.0), longest_sorted_share(p, end, units, kp.cur_heads, tiles, extra, 1.0, 1.0)) < as_one)
                kp.few = (int)few, kp.few_end = (int)end;
        }
        if ((rc = make_tile_map(&tk, p->k, HD, p->nkv, p->kv_len, p->batch, p->k_stride_t, p->k_stride_b, 64)) != ARC_OK) return rc;
        if (split) {
            to = tg = tq;  // (not used)
        } else if ((rc = make_out_maps(&to, &tg, p)) != ARC_OK) {
            return rc;
        }
        // (a cluster is placed inside one GPC, so fewer fit than pairs / parts)
        const bool fold = split && folds_itself(p, plan.splits, wide_units(p, plan.q_tiles), ds->wide);
        const WideKernel kernel = wide_kernel(kp.gate != nullptr, masked, fold ? 2 : split ? 1 : 0, units > ds->wide.pairs, kp.ids != nullptr);
        ARC_CUDA(launch_dependent(kernel,
                                  dim3((unsigned)(2 * (split || units < ds->wide.pairs ? units : ds->wide.pairs))), dim3(WideCfg::THREADS),
                                  (size_t)WideCfg::SMEM_BYTES, stream, fold ? 2 * plan.splits : 2, tq, tk, tv, to, tg, kp));
        g_launches.fetch_add(1, std::memory_order_relaxed);
        return split && !fold ? launch_fold<HD>(p, plan, kp, stream) : ARC_OK;
    }

    kp.q_tiles = plan.q_tiles;
    kp.cur_heads = p->nq;
    kp.head_pair = 0;
    // Persistent grid: one CTA per SM (fewer if there are fewer tiles), tiles dealt round-robin.
    const long long total_tiles = (long long)plan.q_tiles * p->nq * p->batch * plan.splits;
    if (total_tiles > 0x7fffffffLL) return ARC_ERR_TOO_LARGE;
    kp.total_tiles = (int)total_tiles;
    const unsigned ctas = (unsigned)(total_tiles < ds->sm_count ? total_tiles : ds->sm_count);
    ARC_CUDA(launch_dependent(sdpa_prefill_kernel, dim3(ctas), dim3(PrefillCfg::THREADS), (size_t)PrefillCfg::SMEM_BYTES, stream, 1, tq, tk, tv, kp));
    g_launches.fetch_add(1, std::memory_order_relaxed);

    return plan.splits > 1 ? launch_fold<HD>(p, plan, kp, stream) : ARC_OK;
}

// ---------------------------------------------------------------------------
// Decode plan
// ---------------------------------------------------------------------------
struct DecodePlan {
    int nkv_cta = 1, groups = 1, slices = 1, stages = 2, ncta = 1, nt = 1;
    int smem_bytes = 0;
    long long parts = 0;
    size_t ws_bytes = 0;
    bool cluster = false;  // one launch: a cluster of `ncta` CTAs per sequence and group of KV heads
};

// Slices of 16 keys in a stage of `kb` KB of a CTA that works on `nkv_cta` KV heads, a consumer warp for each and head.
static int most_slices(int hd, int nkv_cta, int kb) {
    return std::max(1, std::min(kb * 1024 / (32 * nkv_cta * hd * 2), 8 / nkv_cta));
}

// Shared memory of a CTA that works on `nkv_cta` KV heads (and holds `extra` bytes): stages, bytes.  False: not even two stages fit.
static bool size_decode_cta(int hd, int nkv_cta, int slices, int batch, int extra, int smem_optin, DecodePlan* plan) {
    const int row_bytes = nkv_cta * hd * 2;
    const int stage_bytes = 2 * 16 * slices * row_bytes;
    const int fixed = 1024 + 2 * 8 * 8 + (batch + 2) * 8 + extra;
    int stages = (smem_optin - kDecodeStaticSmem - fixed) / stage_bytes;
    if (stages > 4) stages = 4;
    plan->nkv_cta = nkv_cta;
    plan->slices = slices;
    plan->stages = stages;
    plan->smem_bytes = stages * stage_bytes + fixed;
    return stages >= 2;
}

// One launch or two?  A cluster of up to eight CTAs per sequence and group of heads finishes alone: 4.1 us (4.7 with the lengths on the
// device) and the longer of two times: of the CTAs with the longest sequence, at the 93 GB/s one CTA pulls at head dim 256 (four
// consumer warps) and 105 at 128 (eight), and of all bytes at what so many CTAs get out of the memory (less when a CTA's heads fill a
// row of 2 KB: one slice, as few warps as heads).  Equal shares over all SMs read the total at 7 TB/s, but cost 7.2 us (8 with the
// lengths on the device) and 0.1 us per sequence for the second launch and the records.  (Measured over
// batches of 1 to 64 and lengths of 64 to 8192 for five head layouts: one token over 513 keys, 24/4 heads: 6.7 and 5.1 us,
// 64 sequences of 512 keys, 16/2 heads: 17.8 and 9.9.  With 5.2, as it was before the records' way was shortened, one token over 2929 and
// 3768 keys, 24/4 heads, took 9.7 and 9.9 by shares, 7.6 and 8.4 so.)  Lengths on the device are not known here: the longest sequence is
// taken to be as long as its bound says, or twice the mean of a packed cache, the others half of that.  If they are not and
// one sequence holds nearly all keys, its cluster works alone: 20000 keys among 31 sequences of 400 took 52 to 228 us where
// shares take 16 to 34.  So the form is left alone where that could cost more than 24 us and 1.3 times what shares do.
static void plan_decode_cluster(const arc_sdpa_decode_params* p, const DeviceState& ds, int nkv_cta, DecodePlan* plan) {
    if (p->num_ctas != 0 || p->xchg_world > 1 || p->kv_rows_total == 0 || p->batch > 1024) return;
    const int G = p->nq / p->nkv;
    int heads = 0, csize = 0;  // the smallest group of heads and then the largest cluster that are all resident at once
    for (int c = 1; c <= nkv_cta && !heads; ++c)
        if (p->nkv % c == 0 && (long long)p->batch * (p->nkv / c) <= ds.decode_clusters[1]) heads = c;
    for (int size = 8; heads && size >= 1 && !csize; --size)
        if ((long long)p->batch * (p->nkv / heads) <= ds.decode_clusters[size]) csize = size;
    if (!csize) return;
    double longest = (double)p->kv_len_uniform, total = longest * p->batch;
    if (p->kv_len) {
        longest = (double)(p->max_kv_len > 0 ? p->max_kv_len : p->kv_rows_total);
        if (p->kv_row_offset && p->batch > 1 && longest > 2.0 * (double)p->kv_rows_total / p->batch)
            longest = 2.0 * (double)p->kv_rows_total / p->batch;
        total = longest * (0.5 * p->batch + 0.5);
    }
    // Three, five, six or seven CTAs at head dim 128 where the longest sequence then takes fewer steps than in two or four, at
    // 256 where it would be too long for these.  (12 sequences of 200 to 6000 keys, 16/2 heads of 128: 12.5 us in fours, 11.5 in
    // sixes; 24 of 100 to 900, 8/1, two steps either way: 7.1 in fours, 7.4 in sixes.  Head dim 256, with six warps a CTA, 24/4: 6
    // of 300 to 2000 10.3 and 11.2; 5 packed ones of 300 to 3000: 16.8 by shares, 11.5 in sevens.)
    const int most_ctas = csize;
    int finishers = 1;  // CTAs that finish columns: the largest power of two there is
    while (finishers * 2 <= csize) finishers *= 2;
    const long long keys = (long long)std::min(longest, 1e9), step = 16 * most_slices(p->hd, heads, 64);
    if (p->hd == 256 || (keys + csize * step - 1) / (csize * step) >= (keys + finishers * step - 1) / (finishers * step)) csize = finishers;
    const double per_key = p->nkv * p->hd * 4.0;
    auto t_shares = [&](double k) { return (p->kv_len ? 8.0 : 7.2) + 0.1 * p->batch + k * per_key / 7.0e6; };
    auto worth_it = [&](int size, double more) {  // (more: us that it has to gain besides)
        const double ctas = (double)p->batch * (p->nkv / heads) * size;
        const double all = heads * p->hd >= 1024 ? 6.0e6 : 6.9e6 - 6e3 * (ds.sm_count - ctas);
        const double per_longest = heads * p->hd * 4.0 / size / (p->hd == 256 ? 93e3 : 105e3);
        auto t_cluster = [&](double most, double k) { return more + (p->kv_len ? 4.7 : 4.1) + std::max(most * per_longest, k * per_key / all); };
        if (t_cluster(longest, total) > t_shares(total)) return false;
        if (!p->kv_len) return true;
        const double most = p->max_kv_len > 0 ? std::min((double)p->max_kv_len, (double)p->kv_rows_total) : (double)p->kv_rows_total;
        const double wide_group = G <= 8 ? 1.0 : p->hd == 256 ? 4.0 : 1.6;  // (two tiles of heads a warp: the rates are that much lower)
        return t_cluster(most * wide_group, most) <= std::max(24.0, 1.3 * t_shares(most));
    };
    // (A power of two of CTAs where there could be more has to be well worth it: five sequences of up to 2233 keys, 16/8 heads of 256, take 14.7
    // us in twos and 12.7 in threes.)
    if (!worth_it(csize, csize < most_ctas ? (p->kv_len ? 0.5 : 1.1) : 0.0)) {
        csize = most_ctas;
        if (!worth_it(csize, 0.0)) return;
    }
    // A step of a CTA is one 16-key slice for each of its warps.  Head dim 256 has room for six a head in two stages instead of
    // four in three: taken where the longest sequence then needs fewer steps, a step of s slices counted as 2 + s.  (One token
    // of 24/4 heads over 513 keys, 65 a CTA: 6.74 us in two steps, 6.37 in one; 701: 6.82 and 6.38; 1501: 7.56 and 7.26; over
    // 1001 keys four slices fill two steps, six read half as much again for nothing: 6.84 and 7.08.)
    // That is with five or six query heads a KV head, which six warps fold in one turn and four in two, or more than eight.  With
    // others the fold of six takes 0.6 us longer where a cluster folds (two tokens of 16/8 heads over 780 keys 6.0 us in fours, 6.8 in
    // sixes, of 16/2 over 1500 8.2 and 8.7, four of 16/8 over 1500 12.4 and 12.9), 0.2 where a CTA is alone, and up to four heads
    // do not make up for that but where a third of the steps goes (16 of 16/8 over 200 / 260 keys 10.3 / 11.3 and 10.7 / 10.9).
    // Fewer than 100 single CTAs need the third stage over many steps (20 of 24/4 over 780 keys 17.8 and 19.0; 30 22.1 and 21.9).
    int slices = most_slices(p->hd, heads, 64);
    const int wide = most_slices(p->hd, heads, 96);
    if (p->hd == 256 && wide > slices) {
        const long long units = ((long long)std::min(longest, 1e9) + csize * 16 - 1) / (csize * 16);  // 16-key slices of a CTA
        const long long steps = (units + slices - 1) / slices, wide_steps = (units + wide - 1) / wide;
        const bool alone = csize == 1, few = alone && (long long)p->batch * (p->nkv / heads) < 100 && steps > 9;
        if (G > 8 || G == 5 || G == 6 || (alone && G > 4)) {
            if (wide_steps * (2 + wide) <= steps * (2 + slices) && (G > 8 || !few)) slices = wide;
        } else if (alone && !few && 3 * wide_steps < 2 * steps) {
            slices = wide;
        }
    }
    DecodePlan one = *plan;
    // (The records the CTA finishes have a place of their own: they come while it still works.  Its warps' records go where
    // the stages were, of which there are at least two.)
    const int rows = heads * G;
    const int extra = 64 + 8 * ((rows + 1) & ~1) * 8 + csize * rows * (p->hd / finishers) * 4 + rows * 32;
    if (!size_decode_cta(p->hd, heads, slices, 0, extra, ds.smem_optin, &one)) return;
    one.cluster = true;
    one.groups = p->nkv / heads;
    one.ncta = csize;
    *plan = one;
}

static int plan_decode(const arc_sdpa_decode_params* p, const DeviceState& ds, DecodePlan* plan) {
    const int sm_count = ds.sm_count, smem_optin = ds.smem_optin;
    if (!p) return ARC_ERR_NULL_POINTER;
    if (p->batch <= 0 || p->nq <= 0 || p->nkv <= 0 || p->nq % p->nkv != 0) return ARC_ERR_BAD_SHAPE;
    if (p->batch > DECODE_MAX_BATCH) return ARC_ERR_TOO_LARGE;
    if (p->hd != 128 && p->hd != 256) return ARC_ERR_UNSUPPORTED_HEAD_DIM;
    if (!(p->scale > 0.f) || !std::isfinite(p->scale)) return ARC_ERR_BAD_SHAPE;
    if (!p->kv_len && p->kv_len_uniform < 0) return ARC_ERR_BAD_SHAPE;
    if (p->kv_rows_total < 0 || p->kv_rows_total > 0x7fffffffLL) return ARC_ERR_BAD_SHAPE;
    // An empty cache (a sequence-sharded rank whose slice holds no keys) is fine as long as the
    // host-side length says so too.
    if (p->kv_rows_total == 0 && (p->kv_len || p->kv_len_uniform != 0)) return ARC_ERR_BAD_SHAPE;
    if (p->max_kv_len < 0) return ARC_ERR_BAD_SHAPE;
    if (p->max_kv_len > 0 && !p->kv_len && p->kv_len_uniform > p->max_kv_len) return ARC_ERR_BAD_SHAPE;
    if (!p->kv_len && !p->kv_row_offset && p->kv_len_uniform > 0 &&
        (int64_t)(p->batch - 1) * p->kv_stride_b + p->kv_len_uniform > p->kv_rows_total)
        return ARC_ERR_BAD_SHAPE;  // everything is known on the host: refuse at once
    const int G = p->nq / p->nkv;
    if (G > 16) return ARC_ERR_UNSUPPORTED_GQA;
    plan->nt = G > 8 ? 2 : 1;
    // Heads per CTA: the largest divisor of nkv whose row (all its heads) is <= 2 KB.
    const int max_heads = 1024 / p->hd;  // 8 for hd 128, 4 for hd 256
    int nkv_cta = 1;
    for (int c = 1; c <= p->nkv && c <= max_heads; ++c)
        if (p->nkv % c == 0) nkv_cta = c;
    if (!size_decode_cta(p->hd, nkv_cta, most_slices(p->hd, nkv_cta, 64), p->batch, 0, smem_optin, plan)) return ARC_ERR_TOO_LARGE;
    plan->groups = p->nkv / nkv_cta;
    int ncta = p->num_ctas > 0 ? p->num_ctas : sm_count / plan->groups;
    if (ncta < 1) ncta = 1;
    if (ncta > 1024) ncta = 1024;
    plan->ncta = ncta;
    plan->parts = ((long long)ncta + p->batch) * plan->slices;
    plan->ws_bytes = (size_t)plan->parts * p->nq * ((size_t)p->hd + 1) * sizeof(float);
    plan_decode_cluster(p, ds, nkv_cta, plan);  // (the workspace asked for stays that of the form above)
    return ARC_OK;
}

template <int HD>
static int launch_decode(const arc_sdpa_decode_params* p, const DecodePlan& plan, DeviceState* ds,
                         cudaStream_t stream) {
    CUtensorMap tk, tv;
    int rc;
    const bool empty_cache = p->kv_rows_total == 0;  // nothing to read: only the merge runs (all records empty)
    if (!empty_cache) {
        if ((rc = make_cache_map(&tk, p->k, p->nkv * HD, p->kv_rows_total, p->kv_stride_t, 16 * plan.slices)) != ARC_OK) return rc;
        if ((rc = make_cache_map(&tv, p->v, p->nkv * HD, p->kv_rows_total, p->kv_stride_t, 16 * plan.slices)) != ARC_OK) return rc;
    }
    DecodeParams kp{};
    kp.q = static_cast<const uint16_t*>(p->q);
    kp.kv_len = p->kv_len;
    kp.kv_row_offset = reinterpret_cast<const long long*>(p->kv_row_offset);
    kp.part_o = static_cast<float*>(p->workspace);
    kp.part_lse = kp.part_o + (size_t)plan.parts * p->nq * HD;
    kp.fault = ds->fault;
    kp.batch = p->batch;
    kp.nq = p->nq;
    kp.nkv = p->nkv;
    kp.kv_len_uniform = p->kv_len_uniform;
    kp.q_stride_b = p->q_stride_b;
    kp.kv_stride_b = p->kv_stride_b;
    kp.kv_stride_t = p->kv_stride_t;
    kp.scale_log2 = p->scale * 1.4426950408889634f;
    kp.nkv_cta = plan.nkv_cta;
    kp.slices = plan.slices;
    kp.stages = plan.stages;
    kp.ncta = plan.ncta;
    kp.max_kv_len = p->max_kv_len;
    kp.kv_rows_total = p->kv_rows_total;

    dim3 grid((unsigned)plan.ncta, (unsigned)plan.groups, 1);
    const unsigned threads = 32u * (unsigned)(plan.nkv_cta * plan.slices + 1);
    if (plan.cluster) {
        kp.gate = static_cast<const uint16_t*>(p->gate);
        kp.out = static_cast<uint16_t*>(p->out);
        kp.out_f32 = p->out_f32;
        kp.out_lse = p->out_lse;
        kp.o_stride_b = p->o_stride_b;
        const bool alone = plan.ncta == 1;
        auto kernel = plan.nt == 1 ? (alone ? sdpa_decode_kernel<HD, 1, true, true> : sdpa_decode_kernel<HD, 1, true>)
                                   : (alone ? sdpa_decode_kernel<HD, 2, true, true> : sdpa_decode_kernel<HD, 2, true>);
        grid.z = (unsigned)p->batch;
        ARC_CUDA(launch_dependent(kernel, grid, dim3(threads), (size_t)plan.smem_bytes, stream, plan.ncta, tk, tv, kp));
        g_launches.fetch_add(1, std::memory_order_relaxed);
        return ARC_OK;
    }
    if (!empty_cache) {
        ARC_CUDA(launch_dependent(plan.nt == 1 ? sdpa_decode_kernel<HD, 1, false> : sdpa_decode_kernel<HD, 2, false>, grid, dim3(threads),
                                  (size_t)plan.smem_bytes, stream, 1, tk, tv, kp));
        g_launches.fetch_add(1, std::memory_order_relaxed);
    }

    DecodeMergeParams mp{};
    mp.part_o = kp.part_o;
    mp.part_lse = kp.part_lse;
    mp.kv_len = p->kv_len;
    mp.gate = static_cast<const uint16_t*>(p->gate);
    mp.out = static_cast<uint16_t*>(p->out);
    mp.out_f32 = p->out_f32;
    mp.out_lse = p->out_lse;
    mp.batch = p->batch;
    mp.nq = p->nq;
    mp.kv_len_uniform = p->kv_len_uniform;
    mp.ncta = plan.ncta;
    mp.slices = plan.slices;
    mp.o_stride_b = p->o_stride_b;
    mp.x_peers = reinterpret_cast<const unsigned long long*>(p->xchg_peers);
    mp.x_world = p->xchg_world;
    mp.x_rank = p->xchg_rank;
    mp.x_step = p->xchg_step;
    mp.x_wait_cycles = p->xchg_wait_cycles > 0 ? p->xchg_wait_cycles : 2000000000LL;
    mp.fault = ds->fault;
    const bool xchg = mp.x_world > 1;
    // 64 columns a block while that leaves at most one block per SM; with more, every block would repeat the search for
    // the records for less work of its own.
    const bool narrow = !xchg && (long long)p->nq * p->batch * (HD / 64) <= ds->sm_count;
    const dim3 mgrid((unsigned)p->nq, (unsigned)p->batch, narrow ? HD / 64 : 1);
    ARC_CUDA(launch_dependent(xchg     ? sdpa_decode_merge_kernel<HD, true, HD>
                              : narrow ? sdpa_decode_merge_kernel<HD, false, 64>
                                       : sdpa_decode_merge_kernel<HD, false, HD>, mgrid,
                              dim3(MERGE_THREADS), 0, stream, 1, mp));
    g_launches.fetch_add(1, std::memory_order_relaxed);
    return ARC_OK;
}

}  // namespace arc

// ===========================================================================
// extern "C"
// ===========================================================================
using namespace arc;

extern "C" const char* arc_sdpa_status_string(int status) {
    switch (status) {
        case ARC_OK: return "ok";
        case ARC_ERR_BAD_SHAPE: return "bad shape or parameter";
        case ARC_ERR_ALIGNMENT: return "pointer or stride not 16-byte aligned";
        case ARC_ERR_UNSUPPORTED_HEAD_DIM: return "head_dim must be 128 or 256";
        case ARC_ERR_WORKSPACE_TOO_SMALL: return "workspace missing or too small";
        case ARC_ERR_CUDA: return "CUDA call failed";
        case ARC_ERR_COLLECTIVE: return "collective failed";
        case ARC_ERR_DEVICE_WAIT_TIMEOUT: return "a bounded device-side wait gave up";
        case ARC_ERR_NULL_POINTER: return "required pointer is null";
        case ARC_ERR_UNSUPPORTED_GQA: return "more than 16 query heads per KV head";
        case ARC_ERR_TOO_LARGE: return "size beyond a fixed limit";
        case ARC_ERR_DEVICE_BAD_RANGE: return "a device-side kv_len or kv_row_offset reaches past the cache";
        default: return "unknown status";
    }
}

extern "C" size_t arc_sdpa_prefill_workspace_bytes(const arc_sdpa_prefill_params* p) {
    DeviceState* ds = nullptr;
    const bool known = device_state(&ds) == ARC_OK;
    PrefillPlan plan;
    if (plan_prefill(p, known ? ds->sm_count : 148, known ? ds->wide : WideRoom{}, &plan) != ARC_OK) return 0;
    return plan.ws_bytes + plan.mask_bytes;
}

extern "C" int arc_sdpa_prefill(const arc_sdpa_prefill_params* p, void* stream) {
    if (!p) return ARC_ERR_NULL_POINTER;
    if (!p->q || !p->k || !p->v || !p->out) return ARC_ERR_NULL_POINTER;
    if (p->mask_type == ARC_MASK_EXPLICIT && !p->mask) return ARC_ERR_NULL_POINTER;
    if (p->out_copy_count < 0 || p->out_copy_count > 15 || (p->out_copy_count > 0 && !p->out_copies)) return ARC_ERR_BAD_SHAPE;
    DeviceState* ds = nullptr;
    int rc = device_state(&ds);
    if (rc != ARC_OK) return rc;
    PrefillPlan plan;
    if ((rc = plan_prefill(p, ds->sm_count, ds->wide, &plan)) != ARC_OK) return rc;
    if (p->hd == 256 && p->num_splits == 0 && plan.splits > 1 && (!p->workspace || !aligned16(p->workspace) || p->workspace_bytes < plan.ws_bytes)) {
        arc_sdpa_prefill_params whole = *p;  // no room for the parts of a split the caller has not asked for: none, then
        whole.num_splits = 1;
        if ((rc = plan_prefill(&whole, ds->sm_count, ds->wide, &plan)) != ARC_OK) return rc;
    }
    if (!aligned16(p->q) || !aligned16(p->k) || !aligned16(p->v) || !aligned16(p->out) ||
        (p->gate && !aligned16(p->gate)))
        return ARC_ERR_ALIGNMENT;
    const int64_t strides[8] = {p->q_stride_b, p->q_stride_t, p->k_stride_b, p->k_stride_t,
                                p->v_stride_b, p->v_stride_t, p->o_stride_b, p->o_stride_t};
    for (int64_t s : strides)
        if (s < 0 || (s & 7) != 0) return ARC_ERR_ALIGNMENT;
    if (p->q_stride_t < (int64_t)p->nq * p->hd || p->o_stride_t < (int64_t)p->nq * p->hd ||
        p->k_stride_t < (int64_t)p->nkv * p->hd || p->v_stride_t < (int64_t)p->nkv * p->hd)
        return ARC_ERR_BAD_SHAPE;
    if (plan.ws_bytes > 0) {
        if (!p->workspace || p->workspace_bytes < plan.ws_bytes) return ARC_ERR_WORKSPACE_TOO_SMALL;
        if (!aligned16(p->workspace)) return ARC_ERR_ALIGNMENT;
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    return p->hd == 128 ? launch_prefill<128>(p, plan, ds, st) : launch_prefill<256>(p, plan, ds, st);
}

extern "C" size_t arc_sdpa_decode_workspace_bytes(const arc_sdpa_decode_params* p) {
    DeviceState* ds = nullptr;
    if (device_state(&ds) != ARC_OK) return 0;
    DecodePlan plan;
    if (plan_decode(p, *ds, &plan) != ARC_OK) return 0;
    return plan.ws_bytes;
}

extern "C" size_t arc_sdpa_exchange_bytes(int32_t world, int32_t batch, int32_t nq, int32_t hd) {
    if (world <= 0 || batch <= 0 || nq <= 0 || hd <= 0) return 0;
    return xchg_total_bytes(world, (long long)batch * nq, hd);
}

extern "C" int arc_sdpa_decode(const arc_sdpa_decode_params* p, void* stream) {
    if (!p) return ARC_ERR_NULL_POINTER;
    if (!p->q || ((!p->k || !p->v) && p->kv_rows_total != 0)) return ARC_ERR_NULL_POINTER;
    if (!p->out && !p->out_f32) return ARC_ERR_NULL_POINTER;
    DeviceState* ds = nullptr;
    int rc = device_state(&ds);
    if (rc != ARC_OK) return rc;
    DecodePlan plan;
    if ((rc = plan_decode(p, *ds, &plan)) != ARC_OK) return rc;
    if (!aligned16(p->q) || (p->kv_rows_total != 0 && (!aligned16(p->k) || !aligned16(p->v))) || (p->out && !aligned16(p->out)) ||
        (p->gate && !aligned16(p->gate)) || (p->out_f32 && !aligned16(p->out_f32)))
        return ARC_ERR_ALIGNMENT;
    if ((p->q_stride_b & 7) || (p->o_stride_b & 7) || (p->kv_stride_t & 7) || p->kv_stride_t < (int64_t)p->nkv * p->hd ||
        p->q_stride_b < 0 || p->o_stride_b < 0 || p->kv_stride_b < 0)
        return ARC_ERR_ALIGNMENT;
    if (p->gate && !p->out) return ARC_ERR_NULL_POINTER;
    if (p->xchg_world > 1) {
        if (!p->xchg_peers || !p->out) return ARC_ERR_NULL_POINTER;
        if (p->xchg_rank < 0 || p->xchg_rank >= p->xchg_world || p->xchg_world > XCHG_MAX_WORLD) return ARC_ERR_BAD_SHAPE;
    }
    if (!p->workspace || p->workspace_bytes < plan.ws_bytes) return ARC_ERR_WORKSPACE_TOO_SMALL;
    if (!aligned16(p->workspace)) return ARC_ERR_ALIGNMENT;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    return p->hd == 128 ? launch_decode<128>(p, plan, ds, st) : launch_decode<256>(p, plan, ds, st);
}

// ---------------------------------------------------------------------------
// Decode without any caller-provided or allocated scratch.
//
// Some callers have nowhere to get a workspace from: a serving process whose
// memory planner has already handed every free byte of the GPU to its own arena
// (Arcaine's per-GPU arena works that way), or a thin foreign-function caller
// that owns no device allocator at all; and cudaMalloc on a decode loop would
// also stall the whole device.  For them the split-KV partial records live in
// the fixed array below, which is part of the library image: every GPU that
// loads the library carries these 8 MiB until the process exits.
//
// In host code the array's name is only a handle; the device address is looked
// up once per device (with that device current) and that address is what the
// kernels receive.
// ---------------------------------------------------------------------------
static __device__ __align__(256) unsigned char g_static_scratch[ARC_STATIC_SCRATCH_BYTES];
static std::atomic<void*> g_static_scratch_addr[arc::kMaxDevices];

static int static_scratch_address(void** out) {
    int dev = 0;
    ARC_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= arc::kMaxDevices) return ARC_ERR_CUDA;
    void* ptr = g_static_scratch_addr[dev].load(std::memory_order_acquire);
    if (ptr == nullptr) {
        std::lock_guard<std::mutex> lock(arc::g_mu);
        ptr = g_static_scratch_addr[dev].load(std::memory_order_relaxed);
        if (ptr == nullptr) {
            ARC_CUDA(cudaGetSymbolAddress((void**)&ptr, g_static_scratch));
            g_static_scratch_addr[dev].store(ptr, std::memory_order_release);
        }
    }
    *out = ptr;
    return ARC_OK;
}

extern "C" int arc_sdpa_decode_static(const arc_sdpa_decode_params* p, void* stream) {
    if (!p) return ARC_ERR_NULL_POINTER;
    void* scratch = nullptr;
    int rc = static_scratch_address(&scratch);
    if (rc != ARC_OK) return rc;
    arc_sdpa_decode_params q = *p;
    q.workspace = nullptr;
    q.workspace_bytes = 0;
    const size_t need = arc_sdpa_decode_workspace_bytes(&q);
    if (need > (size_t)ARC_STATIC_SCRATCH_BYTES) {
        std::snprintf(g_last_error, sizeof(g_last_error),
                      "arc_sdpa_decode_static: this shape needs %zu bytes of scratch, the built-in array holds %zu",
                      need, (size_t)ARC_STATIC_SCRATCH_BYTES);
        return ARC_ERR_TOO_LARGE;
    }
    q.workspace = scratch;
    q.workspace_bytes = ARC_STATIC_SCRATCH_BYTES;
    return arc_sdpa_decode(&q, stream);
}

extern "C" int arc_sdpa_merge(const float* part_out, const float* part_lse, int32_t num_parts, int64_t rows,
                              int32_t hd, int64_t part_out_stride, int64_t part_lse_stride, const void* gate,
                              void* out_bf16, float* out_f32, float* out_lse, void* stream) {
    if (!part_out || !part_lse) return ARC_ERR_NULL_POINTER;
    if (!out_bf16 && !out_f32) return ARC_ERR_NULL_POINTER;
    if (num_parts <= 0 || rows <= 0 || rows > 0x7fffffffLL) return ARC_ERR_BAD_SHAPE;
    if (hd != 128 && hd != 256) return ARC_ERR_UNSUPPORTED_HEAD_DIM;
    if (gate && !out_bf16) return ARC_ERR_NULL_POINTER;
    if (!aligned16(part_out) || (out_bf16 && !aligned16(out_bf16)) || (out_f32 && !aligned16(out_f32)) ||
        (gate && !aligned16(gate)))
        return ARC_ERR_ALIGNMENT;
    UniformMergeParams mp{};
    mp.part_o = part_out;
    mp.part_lse = part_lse;
    mp.gate = static_cast<const uint16_t*>(gate);
    mp.out = static_cast<uint16_t*>(out_bf16);
    mp.out_f32 = out_f32;
    mp.out_lse = out_lse;
    mp.rows = rows;
    mp.num_parts = num_parts;
    mp.seq = 0;
    mp.o_part_stride = part_out_stride > 0 ? part_out_stride : rows * hd;
    mp.lse_part_stride = part_lse_stride > 0 ? part_lse_stride : rows;
    if ((mp.o_part_stride & 3) != 0) return ARC_ERR_ALIGNMENT;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const unsigned blocks = (unsigned)((rows + UMERGE_ROWS - 1) / UMERGE_ROWS);
    ARC_CUDA(launch_dependent(hd == 128 ? sdpa_uniform_merge_kernel<128, 4> : sdpa_uniform_merge_kernel<256, 4>, dim3(blocks),
                              dim3(32 * UMERGE_ROWS), 0, st, 1, mp));
    g_launches.fetch_add(1, std::memory_order_relaxed);
    return ARC_OK;
}

extern "C" int arc_mul_sigmoid_inplace(void* a, const void* gate, int64_t n, void* stream) {
    if (!a || !gate) return ARC_ERR_NULL_POINTER;
    if (n < 0) return ARC_ERR_BAD_SHAPE;
    if (n == 0) return ARC_OK;
    long long blocks = (n + 255) / 256;
    if (blocks > 148 * 16) blocks = 148 * 16;
    ARC_CUDA(launch_dependent(mul_sigmoid_kernel, dim3((unsigned)blocks), dim3(256), 0, static_cast<cudaStream_t>(stream), 1,
                              static_cast<uint16_t*>(a), static_cast<const uint16_t*>(gate), (long long)n));
    g_launches.fetch_add(1, std::memory_order_relaxed);
    return ARC_OK;
}

extern "C" int arc_qkv_prepare(const arc_qkv_prepare_params* p, void* stream) {
    if (!p) return ARC_ERR_NULL_POINTER;
    if (p->batch <= 0 || p->seq < 0 || p->nq < 0 || p->nkv < 0) return ARC_ERR_BAD_SHAPE;
    if (p->hd != 128 && p->hd != 256 && p->hd != 512) return ARC_ERR_UNSUPPORTED_HEAD_DIM;
    if (p->n_active_pairs < 0 || p->n_active_pairs > p->hd / 2) return ARC_ERR_BAD_SHAPE;
    if ((p->rope_cos == nullptr) != (p->rope_sin == nullptr)) return ARC_ERR_NULL_POINTER;
    if (p->n_active_pairs > 0 && !p->rope_cos && !(p->theta > 0.f)) return ARC_ERR_BAD_SHAPE;
    if (p->k_src && !p->k_dst) return ARC_ERR_NULL_POINTER;
    if (p->v_dst && !p->v_src && !p->k_src) return ARC_ERR_NULL_POINTER;
    if (!p->q && !p->k_src && !p->v_dst) return ARC_OK;
    if (p->seq == 0) return ARC_OK;
    // Shared K/V projection (v_src NULL): V comes from the raw K rows, so K must not be rewritten
    // in place — another warp may already have normalised and rotated the row V is read from.
    if (p->v_dst && !p->v_src && p->k_dst == p->k_src) return ARC_ERR_BAD_SHAPE;
    const int row_count = (p->q ? p->nq : 0) + (p->k_src ? p->nkv : 0) + (p->v_dst ? p->nkv : 0);
    if (row_count == 0) return ARC_OK;  // pointers given, but no heads
    auto aligned = [](const void* x) { return (reinterpret_cast<uintptr_t>(x) & 15u) == 0; };
    if (!aligned(p->q) || !aligned(p->k_src) || !aligned(p->v_src) || !aligned(p->k_dst) || !aligned(p->v_dst) ||
        !aligned(p->q_weight) || !aligned(p->k_weight))
        return ARC_ERR_ALIGNMENT;
    const int64_t strides[] = {p->q_stride_b, p->q_stride_t, p->k_src_stride_b, p->k_src_stride_t, p->v_src_stride_b,
                               p->v_src_stride_t, p->k_dst_stride_b, p->k_dst_stride_t, p->v_dst_stride_b, p->v_dst_stride_t};
    for (int64_t st : strides)
        if (st < 0 || st % 8 != 0) return ARC_ERR_ALIGNMENT;
    // a token's heads must fit between two tokens
    const int64_t qrow = (int64_t)p->nq * p->hd, kvrow = (int64_t)p->nkv * p->hd;
    if ((p->q && p->q_stride_t < qrow) || (p->k_src && (p->k_src_stride_t < kvrow || p->k_dst_stride_t < kvrow)) ||
        (p->v_src && p->v_src_stride_t < kvrow) || (p->v_dst && p->v_dst_stride_t < kvrow))
        return ARC_ERR_BAD_SHAPE;
    DeviceState* ds = nullptr;
    int rc = device_state(&ds);
    if (rc != ARC_OK) return rc;

    QkvPrepareParams kp{};
    kp.q = static_cast<uint16_t*>(p->q);
    kp.k_src = static_cast<const uint16_t*>(p->k_src);
    kp.v_src = static_cast<const uint16_t*>(p->v_src);
    kp.k_dst = static_cast<uint16_t*>(p->k_dst);
    kp.v_dst = static_cast<uint16_t*>(p->v_dst);
    kp.q_weight = static_cast<const uint16_t*>(p->q_weight);
    kp.k_weight = static_cast<const uint16_t*>(p->k_weight);
    kp.rope_cos = p->rope_cos;
    kp.rope_sin = p->rope_sin;
    kp.pos_offset = p->pos_offset;
    kp.batch = p->batch;
    kp.seq = p->seq;
    kp.nq = p->nq;
    kp.nkv = p->nkv;
    kp.nap = p->n_active_pairs;
    kp.q_stride_b = p->q_stride_b;
    kp.q_stride_t = p->q_stride_t;
    kp.ks_stride_b = p->k_src_stride_b;
    kp.ks_stride_t = p->k_src_stride_t;
    kp.vs_stride_b = p->v_src_stride_b;
    kp.vs_stride_t = p->v_src_stride_t;
    kp.kd_stride_b = p->k_dst_stride_b;
    kp.kd_stride_t = p->k_dst_stride_t;
    kp.vd_stride_b = p->v_dst_stride_b;
    kp.vd_stride_t = p->v_dst_stride_t;
    kp.rope_stride_b = p->rope_stride_b;
    kp.pos0 = p->pos0;
    kp.theta = p->theta;
    kp.eps = p->eps;
    kp.rot_half = p->rot_half > 0 ? p->rot_half : p->hd / 2;
    kp.freq_denom = p->freq_denom > 0 ? p->freq_denom : p->hd;
    kp.mrope_pos = p->mrope_positions;
    kp.sec1 = p->mrope_section[1];
    kp.sec2 = p->mrope_section[2];
    kp.v_copy = p->v_copy ? 1 : 0;
    if (kp.rot_half != p->hd / 2) {
        const int rh = kp.rot_half;
        if (rh < 8 || (rh & (rh - 1)) != 0 || rh > p->hd / 4 || p->n_active_pairs > rh) return ARC_ERR_BAD_SHAPE;
    }
    const bool qwen = kp.rot_half != p->hd / 2 || kp.freq_denom != p->hd || kp.mrope_pos != nullptr || kp.v_copy;
    // A warp takes a token at a time, or a part of a token's passes: whatever gives the last warp the fewest passes,
    // the start of a unit (the token's angles) counted as 0.7 of one; whole tokens where there are several for every warp.
    const long long tokens = (long long)p->batch * p->seq;
    if (tokens > 0x7fffffffLL) return ARC_ERR_TOO_LARGE;
    const int passes = (row_count + 512 / p->hd - 1) / (512 / p->hd);
    const long long warps = (long long)ds->sm_count * (qwen ? PREP_CTAS<true> : PREP_CTAS<false>) * PREP_WARPS;
    int chunk = passes, chunks = 1;
    long long best = 0;
    for (int c = passes; tokens < 4 * warps; c = (c + 1) / 2) {
        const int n = (passes + c - 1) / c;
        const long long cost = (tokens * n + warps - 1) / warps * (10 * c + 7);
        if (best == 0 || cost < best) best = cost, chunk = c, chunks = n;
        if (c == 1) break;
    }
    if (tokens * chunks + warps > 0x7fffffffLL) return ARC_ERR_TOO_LARGE;
    const long long units = tokens * chunks;
    const unsigned ctas = (unsigned)((units < warps ? units : warps) + PREP_WARPS - 1) / PREP_WARPS;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    auto launch = [&](auto hd_tag, auto qwen_tag) {
        constexpr int H = decltype(hd_tag)::value;
        constexpr bool Q = decltype(qwen_tag)::value;
        return launch_dependent(qkv_prepare_kernel<H, Q>, dim3(ctas), dim3(32 * PREP_WARPS), 0, st, 1, kp, chunk, chunks);
    };
    auto launch_hd = [&](auto qwen_tag) {
        if (p->hd == 128) return launch(std::integral_constant<int, 128>{}, qwen_tag);
        if (p->hd == 256) return launch(std::integral_constant<int, 256>{}, qwen_tag);
        return launch(std::integral_constant<int, 512>{}, qwen_tag);
    };
    ARC_CUDA(qwen ? launch_hd(std::true_type{}) : launch_hd(std::false_type{}));
    g_launches.fetch_add(1, std::memory_order_relaxed);
    return ARC_OK;
}

static int fill_mask(float* mask, const int32_t* block_ids, int32_t q_len, int32_t kv_len, int32_t past_offset,
                     int32_t sliding_window, void* stream);

extern "C" int arc_fill_causal_mask(float* mask, int32_t q_len, int32_t kv_len, int32_t past_offset,
                                    int32_t sliding_window, void* stream) {
    return fill_mask(mask, nullptr, q_len, kv_len, past_offset, sliding_window, stream);
}

extern "C" int arc_fill_causal_mask_with_block_ids(float* mask, const int32_t* block_ids, int32_t q_len,
                                                   int32_t kv_len, int32_t past_offset, int32_t sliding_window,
                                                   void* stream) {
    // Positions past_offset - (kv_len - q_len) .. past_offset + q_len - 1 are looked up.
    if (block_ids && past_offset - (kv_len - q_len) < 0) return ARC_ERR_BAD_SHAPE;
    return fill_mask(mask, block_ids, q_len, kv_len, past_offset, sliding_window, stream);
}

static int fill_mask(float* mask, const int32_t* block_ids, int32_t q_len, int32_t kv_len, int32_t past_offset,
                     int32_t sliding_window, void* stream) {
    if (!mask) return ARC_ERR_NULL_POINTER;
    if (q_len < 0 || kv_len < 0) return ARC_ERR_BAD_SHAPE;
    if (q_len == 0 || kv_len == 0) return ARC_OK;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    // a block writes 1024 keys of a row, or several rows that are shorter; a grid's y extent ends at 65535, longer masks loop
    unsigned x = 256;
    while (x > 1 && (int64_t)x * 2 >= kv_len) x /= 2;
    const unsigned y = 256 / x;
    // Four times as many rows a block where the blocks are more than three or four fills of the device (1184 blocks): it
    // is their scheduling that such a fill waits for (2048 x 4048 9.35 us, 5.43 so; 70000 x 64 5.36 and 3.55; 1000 x 1300,
    // 2000 blocks, 3.6 either way, but the attention behind it 27.4 and 28.5).
    const int64_t cols = ((int64_t)kv_len + 4 * x - 1) / (4 * x);
    int64_t rows = ((int64_t)q_len + y - 1) / y;
    if (cols * rows > 4096) rows = (rows + 3) / 4;
    const dim3 grid((unsigned)cols, (unsigned)(rows < 65535 ? rows : 65535));
    auto kernel = y > 1 ? (block_ids ? fill_causal_mask_kernel<true, true> : fill_causal_mask_kernel<false, true>)
                        : (block_ids ? fill_causal_mask_kernel<true, false> : fill_causal_mask_kernel<false, false>);
    ARC_CUDA(launch_dependent(kernel, grid, dim3(x, y), 0, st, 1,
                              mask, block_ids, (int)q_len, (int)kv_len, (int)past_offset, (int)sliding_window));
    g_launches.fetch_add(1, std::memory_order_relaxed);
    return ARC_OK;
}

extern "C" int arc_sdpa_device_status(uint32_t* fault_code, uint32_t* fault_detail) {
    DeviceState* ds = nullptr;
    int rc = device_state(&ds);
    if (rc != ARC_OK) return rc;
    uint32_t w[2] = {0, 0};
    if (cudaDeviceSynchronize() != cudaSuccess) return ARC_ERR_CUDA;
    if (cudaMemcpy(w, ds->fault, sizeof(w), cudaMemcpyDeviceToHost) != cudaSuccess) return ARC_ERR_CUDA;
    if (fault_code) *fault_code = w[0];
    if (fault_detail) *fault_detail = w[1];
    if (w[0] == 0) return ARC_OK;
    return w[0] == FAULT_BAD_KV_RANGE ? ARC_ERR_DEVICE_BAD_RANGE : ARC_ERR_DEVICE_WAIT_TIMEOUT;
}

extern "C" int arc_sdpa_clear_device_status(void) {
    DeviceState* ds = nullptr;
    int rc = device_state(&ds);
    if (rc != ARC_OK) return rc;
    if (cudaDeviceSynchronize() != cudaSuccess) return ARC_ERR_CUDA;
    return cudaMemset(ds->fault, 0, 2 * sizeof(uint32_t)) == cudaSuccess ? ARC_OK : ARC_ERR_CUDA;
}

extern "C" const char* arc_sdpa_last_error(void) { return g_last_error; }

extern "C" uint64_t arc_sdpa_launch_count(void) { return g_launches.load(std::memory_order_relaxed); }
