// What runs just before attention, as one HBM-bound kernel: RMSNorm (+ RoPE) of the projected
// Q and K rows, unit-RMS norm of V, and the append of K and V into the KV cache.
//
// The reference does this with separate launches per tensor and two memcpys into the cache
// (src/modeling/diffusion_gemma/attention.cpp:529-610 for the norms and RoPE, :1017-1020 for the
// cache append; the kernels are src/common/kernels/rms_norm.hpp:9-49 and
// src/modeling/diffusion_gemma/attention_kernels.hpp:99-153).  Here every element is read once
// and written once: Q in place, K and V straight to their cache rows.
//
// Arithmetic and rounding order follow the reference: the normalised value v * rsqrt(mean(v^2) +
// eps) * weight is rounded to bf16 first, and the rotation
//   x[p] = x0 c - x1 s,  x[p + hd/2] = x0 s + x1 c,   p < n_active_pairs
// works on those rounded values.  cos / sin come from a caller table (seq x n_active_pairs, as
// the reference's RopeTable) or are computed per token: angle = (offset + token) / theta^(2p/hd).
//
// Mapping: a warp on its own takes a unit of work — a token, or a part of a token's rows where there are few tokens — and
// walks it 32 / (hd / 16) rows a pass: a lane holds eight consecutive elements of a row's first half and the matching
// eight of the second half (16-byte loads), so a rotation pair never leaves the lane and a warp covers 4 / 2 / 1 rows at
// once for head dim 128 / 256 / 512.  The token's cos / sin are worked out once, a pair per lane, into shared memory of
// the warp's own; nothing but the norm weights and the frequencies is shared, so there is one barrier in all.
//
// What bounds it: for prompts the instructions of a pass (about 250 for 2 KB moved) as much as HBM.  Hence pointers
// per unit instead of per row, carries instead of divisions between units, weights and angles read from shared memory
// (in registers they cost the third CTA per SM: 208 us), one pass of loads ahead (two: 198 us).  For a few tokens it is
// the latency of one pass, so their rows are spread over all warps.  4 x 8192 tokens, 32/16 heads of 128 (1.07 GB):
// 206 -> 193 us against a CTA per four tokens with angles behind a barrier per round; 64 tokens, 24/4 heads of 256:
// 10.4 -> 3.3 us.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "ptx.cuh"

namespace arc {

struct QkvPrepareParams {
    uint16_t* q;            // (batch, seq, nq, hd) in place, or nullptr
    const uint16_t* k_src;  // (batch, seq, nkv, hd) projected K, or nullptr
    const uint16_t* v_src;  // projected V; nullptr with v_dst set: V is taken from k_src (before its norm)
    uint16_t* k_dst;        // cache row of the first token (may equal k_src)
    uint16_t* v_dst;        // or nullptr
    const uint16_t* q_weight;  // [hd] or nullptr (unit scale)
    const uint16_t* k_weight;
    const float* rope_cos;  // (seq, nap) or nullptr: computed inline
    const float* rope_sin;
    const int* pos_offset;  // [batch] position of each sequence's first token, or nullptr: pos0
    int batch, seq, nq, nkv, nap;
    long long q_stride_b, q_stride_t;
    long long ks_stride_b, ks_stride_t, vs_stride_b, vs_stride_t;
    long long kd_stride_b, kd_stride_t, vd_stride_b, vd_stride_t;
    long long rope_stride_b;  // elements between the tables of two sequences (0: shared)
    int pos0;
    float theta, eps;
    // Qwen3.5 multi-axis RoPE (src/modeling/qwen3_5/kernels.hpp:576-617): pairs (f, f + rot_half) inside the
    // first 2 * rot_half values of a row, frequency exponent 2 f / freq_denom, position taken from one of
    // three axes per frequency.  rot_half == hd / 2 with no positions is the plain form.
    int rot_half, freq_denom;
    const int* mrope_pos;  // (batch, 3, seq) or nullptr
    int sec1, sec2;        // sections of axes 1 and 2
    int v_copy;            // V rows are copied, not normalised
};

__device__ __forceinline__ int mrope_axis(int f, int sec1, int sec2) {
    if (f >= 1 && f < sec1 * 3 && f % 3 == 1) return 1;
    if (f >= 2 && f < sec2 * 3 && f % 3 == 2) return 2;
    return 0;
}

__device__ __forceinline__ void unpack8(const uint4& raw, float (&f)[8]) {
    const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        f[2 * i] = __uint_as_float(w[i] << 16);
        f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
}

__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
    return make_uint4(pack_bf16x2(f[0], f[1]), pack_bf16x2(f[2], f[3]), pack_bf16x2(f[4], f[5]), pack_bf16x2(f[6], f[7]));
}

// Rows of a token per pass of a warp.
template <int HD>
constexpr int PREP_RPW = 512 / HD;
constexpr int PREP_WARPS = 8;
// CTAs per SM (the Qwen3.5 form does not fit 80 registers).
template <bool QWEN>
constexpr int PREP_CTAS = QWEN ? 2 : 3;

// QWEN: the Qwen3.5 form (pairs rot_half apart, per-axis positions, V copied); the common instance does not carry its
// branches.  chunk: passes per unit; chunks: units per token.
template <int HD, bool QWEN>
__global__ void __launch_bounds__(32 * PREP_WARPS, PREP_CTAS<QWEN>) qkv_prepare_kernel(const QkvPrepareParams p, const int chunk, const int chunks) {
    constexpr int LPR = HD / 16;    // lanes per row
    constexpr int RPW = PREP_RPW<HD>;
    __shared__ float s_inv[HD / 2];                      // rotation frequencies
    __shared__ __align__(16) float s_cos[PREP_WARPS][HD / 2], s_sin[PREP_WARPS][HD / 2];  // per warp: the token's angles
    __shared__ __align__(16) float s_w[2][HD];           // norm weights of Q and K (1 where there are none: the product is then exact)
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int sub = lane / LPR;     // which of the pass's rows
    const int li = lane % LPR;      // position inside the row
    if (p.nap > 0 && !p.rope_cos) {
        for (int pr = threadIdx.x; pr < p.nap; pr += blockDim.x)
            s_inv[pr] = 1.0f / powf(p.theta, 2.0f * pr / static_cast<float>(QWEN ? p.freq_denom : HD));
    }
    grid_dependency_wait();  // (the frequencies above depend on no kernel in front)
    grid_launch_dependents();
    for (int i = threadIdx.x; i < HD; i += blockDim.x) {
        s_w[0][i] = p.q_weight ? bf16_bits_to_f32(p.q_weight[i]) : 1.0f;
        s_w[1][i] = p.k_weight ? bf16_bits_to_f32(p.k_weight[i]) : 1.0f;
    }

    const int rows_q = p.q ? p.nq : 0;
    const int rows_k = p.k_src && p.k_dst ? p.nkv : 0;
    const int rows_v = p.v_dst ? p.nkv : 0;
    const int rows = rows_q + rows_k + rows_v;
    const int units = p.batch * p.seq * chunks;  // the host keeps this below 2^31
    const int stride = gridDim.x * PREP_WARPS;

    // A unit and its rows [r0, r1).  Row r of the token sits r * HD elements behind the pointer of its part (so K's
    // pointer is set back by Q's rows, V's by Q's and K's), this lane's columns included.
    struct Unit {
        int id, b, t, c, r0, r1;
    };
    auto set_rows = [&](Unit& u) {
        u.r0 = u.c * chunk * RPW;
        u.r1 = u.id < units ? min(rows, u.r0 + chunk * RPW) : u.r0;
    };
    auto first_unit = [&]() {
        Unit u;
        u.id = blockIdx.x * PREP_WARPS + warp;
        const int tk = u.id / chunks;
        u.c = u.id - tk * chunks;
        u.b = tk / p.seq;
        u.t = tk - u.b * p.seq;
        set_rows(u);
        return u;
    };
    // `stride` units on, by carries instead of divisions
    const int stk = stride / chunks, sc = stride - stk * chunks, sb = stk / p.seq, stt = stk - sb * p.seq;
    auto advance = [&](Unit& u) {
        u.id += stride;
        u.c += sc;
        const int c1 = u.c >= chunks ? 1 : 0;
        u.c -= c1 * chunks;
        u.t += stt + c1;
        const int c2 = u.t >= p.seq ? 1 : 0;
        u.t -= c2 * p.seq;
        u.b += sb + c2;
        set_rows(u);
    };
    const int k0 = rows_q, v0 = rows_q + rows_k;  // first K row, first V row
    // The walk of the loads, a pass ahead of the work: unit fu, rows from fr on.
    Unit fu = first_unit();
    int fr = 0;
    const uint16_t *fq, *fk, *fv;
    auto begin_loads = [&]() {
        fr = fu.r0;
        fq = p.q + fu.b * p.q_stride_b + fu.t * p.q_stride_t + li * 8;
        const uint16_t* kr = p.k_src + fu.b * p.ks_stride_b + fu.t * p.ks_stride_t + li * 8;
        fk = kr - k0 * HD;
        fv = (p.v_src ? p.v_src + fu.b * p.vs_stride_b + fu.t * p.vs_stride_t + li * 8 : kr) - v0 * HD;
    };
    auto fetch = [&](uint4& lo, uint4& hi) {
        if (fr < fu.r1) {
            const int r = fr + sub;
            lo = hi = make_uint4(0u, 0u, 0u, 0u);
            if (r < fu.r1) {
                const uint16_t* src = (r < k0 ? fq : r < v0 ? fk : fv) + r * HD;
                lo = *reinterpret_cast<const uint4*>(src);
                hi = *reinterpret_cast<const uint4*>(src + HD / 2);
            }
            fr += RPW;
            if (fr >= fu.r1 && fu.id < units - stride) {  // the next unit's first rows follow at once
                advance(fu);
                begin_loads();
            }
        }
    };
    begin_loads();
    uint4 nl, nh;
    nl = nh = make_uint4(0u, 0u, 0u, 0u);
    fetch(nl, nh);
    __syncthreads();  // frequencies and weights, while the first rows are on their way

    for (Unit u = first_unit(); u.id < units; advance(u)) {
        uint32_t turns = 0;  // bit e: element e is rotated
        const int dl = QWEN ? p.rot_half >> 3 : 0;
        const bool split = QWEN && p.rot_half != HD / 2;  // pairs inside the row's first half
        const int pr0 = split ? (li & (dl - 1)) * 8 : li * 8;
        if (p.nap > 0 && u.r0 < rows_q + rows_k) {
            __syncwarp();
            for (int pr = lane; pr < p.nap; pr += 32) {
                float cv, sv;
                if (p.rope_cos) {
                    const long long ti = (long long)u.b * p.rope_stride_b + (long long)u.t * p.nap + pr;
                    cv = p.rope_cos[ti];
                    sv = p.rope_sin[ti];
                } else {
                    const int pos = (QWEN && p.mrope_pos)
                                        ? p.mrope_pos[((long long)u.b * 3 + mrope_axis(pr, p.sec1, p.sec2)) * p.seq + u.t]
                                        : (p.pos_offset ? p.pos_offset[u.b] : p.pos0) + u.t;
                    sincosf(static_cast<float>(pos) * s_inv[pr], &sv, &cv);
                }
                s_cos[warp][pr] = cv;
                s_sin[warp][pr] = sv;
            }
            __syncwarp();
            const int n = min(max(p.nap - pr0, 0), 8);
            turns = split && li >= 2 * dl ? 0u : (1u << n) - 1u;
        }
        uint16_t* dq = p.q + u.b * p.q_stride_b + u.t * p.q_stride_t + li * 8;
        uint16_t* dk = p.k_dst + u.b * p.kd_stride_b + u.t * p.kd_stride_t + li * 8 - k0 * HD;
        uint16_t* dv = p.v_dst + u.b * p.vd_stride_b + u.t * p.vd_stride_t + li * 8 - v0 * HD;
        for (int r0 = u.r0; r0 < u.r1; r0 += RPW) {
            const uint4 rl = nl, rh = nh;
            fetch(nl, nh);
            const int r = r0 + sub;
            const bool is_v = r >= v0;
            uint16_t* dst = (r < k0 ? dq : r < v0 ? dk : dv) + r * HD;
            uint4 ol = rl, oh = rh;
            if (!(QWEN && p.v_copy && r0 >= v0)) {  // (rows of the warp that are only copied need no norm)
                float lo[8], hi[8];
                unpack8(rl, lo);
                unpack8(rh, hi);
                float ss = 0.f;
#pragma unroll
                for (int e = 0; e < 8; ++e) ss += lo[e] * lo[e] + hi[e] * hi[e];
#pragma unroll
                for (int o = LPR / 2; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
                const float rms_inv = rsqrtf(ss / static_cast<float>(HD) + p.eps);
#pragma unroll
                for (int e = 0; e < 8; ++e) lo[e] *= rms_inv, hi[e] *= rms_inv;
                if (r0 < v0) {  // some row of the pass is a Q or K row
                    const float* w = s_w[r < k0 ? 0 : 1] + li * 8;
#pragma unroll
                    for (int e = 0; e < 8; e += 4) {
                        const float4 a = *reinterpret_cast<const float4*>(w + e), b = *reinterpret_cast<const float4*>(w + HD / 2 + e);
                        if (r0 + RPW <= v0 || !is_v) {
                            lo[e] *= a.x, lo[e + 1] *= a.y, lo[e + 2] *= a.z, lo[e + 3] *= a.w;
                            hi[e] *= b.x, hi[e + 1] *= b.y, hi[e + 2] *= b.z, hi[e + 3] *= b.w;
                        }
                    }
                }
                ol = pack8(lo);
                oh = pack8(hi);
                if (r0 < v0 && p.nap > 0) {
                    unpack8(ol, lo);  // the rotation works on the rounded values
                    unpack8(oh, hi);
                    float c[8], s[8];  // (from nap on whatever was there: not used)
#pragma unroll
                    for (int e = 0; e < 8; e += 4) {
                        const float4 cv = *reinterpret_cast<const float4*>(&s_cos[warp][pr0 + e]), sv = *reinterpret_cast<const float4*>(&s_sin[warp][pr0 + e]);
                        c[e] = cv.x, c[e + 1] = cv.y, c[e + 2] = cv.z, c[e + 3] = cv.w;
                        s[e] = sv.x, s[e + 1] = sv.y, s[e + 2] = sv.z, s[e + 3] = sv.w;
                    }
                    if (split) {
                        // Pairs (f, f + rot_half) both sit in the row's first half, rot_half / 8 lanes apart: the
                        // partner's values come by shuffle (every lane takes part; only the rotary lanes update).
                        const bool first = (li & dl) == 0;
#pragma unroll
                        for (int e = 0; e < 8; ++e) {
                            const float other = __shfl_xor_sync(0xffffffffu, lo[e], dl);
                            if ((turns >> e) & 1u) lo[e] = first ? lo[e] * c[e] - other * s[e] : other * s[e] + lo[e] * c[e];
                        }
                    } else if (p.nap == HD / 2) {
#pragma unroll
                        for (int e = 0; e < 8; ++e) {
                            const float x0 = lo[e], x1 = hi[e];
                            lo[e] = x0 * c[e] - x1 * s[e];
                            hi[e] = x0 * s[e] + x1 * c[e];
                        }
                    } else {
#pragma unroll
                        for (int e = 0; e < 8; ++e) {
                            const float x0 = lo[e], x1 = hi[e];
                            const bool on = (turns >> e) & 1u;
                            lo[e] = on ? x0 * c[e] - x1 * s[e] : x0;
                            hi[e] = on ? x0 * s[e] + x1 * c[e] : x1;
                        }
                    }
                    if (r0 + RPW <= v0) {
                        ol = pack8(lo);
                        oh = pack8(hi);
                    } else if (!is_v) {  // (V rows beside K rows are not rotated)
                        ol = pack8(lo);
                        oh = pack8(hi);
                    }
                }
                if (QWEN && p.v_copy && is_v) ol = rl, oh = rh;
            }
            if (r < u.r1) {
                *reinterpret_cast<uint4*>(dst) = ol;
                *reinterpret_cast<uint4*>(dst + HD / 2) = oh;
            }
        }
    }
}

}  // namespace arc
