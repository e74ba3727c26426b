// What the two beam-search kernels share: sort keys, the learned stop, the gather of a code row.
#pragma once

#include "beam_args.h"

namespace tann {

constexpr int kBeamThreads = 128;

// State written by thread 0 (or benignly by any thread) and read by the block after a barrier.
// Counters every thread can derive identically (valid, visited, merges since the last Bloom
// rebuild) are kept in registers instead.
struct BeamCtl {
    uint32_t first_full;
    uint32_t nsel, stop, stop_scan;
    // learned stop state (:2252-2258)
    uint32_t ls_stage, ls_has_prev, ls_topk_changed;
    float ls_prev_dk, ls_prev_boundary;
    uint32_t ls_prev_ids[32];
};

// Candidates and frontier entries are 64-bit keys in shared memory: high word = order-preserving
// bits of the distance, low word = packed node id (bit 31 = expanded). Comparing two keys with
// bit 31 masked off is the reference's CandidateLess (distance, then raw id).
constexpr unsigned long long kInvalidKey = 0xff800000ffffffffull;  // (+inf, 0xffffffff)
constexpr unsigned long long kCmpMask = 0xffffffff7fffffffull;
__device__ __forceinline__ float KeyDist(unsigned long long k) { return FromOrderedBits((uint32_t)(k >> 32)); }
__device__ __forceinline__ uint32_t KeyPackedId(unsigned long long k) { return (uint32_t)k; }
__device__ __forceinline__ uint32_t KeyRawId(unsigned long long k) { return RawId((uint32_t)k); }

__device__ __forceinline__ uint32_t CountBitsInRange(const uint32_t* bits, uint32_t b, uint32_t e) {
    uint32_t n = 0;
    for (uint32_t i = b; i < e; ++i) n += (bits[i >> 5] >> (i & 31)) & 1u;
    return n;
}
__device__ __forceinline__ uint32_t FindFirstSetBit(const uint32_t* bits, uint32_t limit) {
    const uint32_t words = (limit + 31) / 32;
    for (uint32_t w = 0; w < words; ++w) {
        uint32_t word = bits[w];
        if (w + 1 == words && (limit & 31)) word &= (1u << (limit & 31)) - 1u;
        if (word) return w * 32 + __ffs(word) - 1;
    }
    return limit;
}

// Learned stop on one thread; returns true when the traversal has to stop.
static __device__ __forceinline__ bool LearnedStop(const TannLearnedStop& ls, BeamCtl& s, uint32_t valid, uint32_t visited,
                            uint32_t expanded, const unsigned long long* cand, const uint32_t* unexp,
                            uint32_t top_l) {
    while (s.ls_stage < ls.num_stages) {
        const uint32_t p = ls.stage_prefixes[s.ls_stage];
        if (p == 0 || p >= top_l || p < ls.top_k) { ++s.ls_stage; continue; }
        if (valid < top_l || valid < p || valid < ls.top_k || expanded < p) break;
        const float dk = KeyDist(cand[ls.top_k - 1]);
        const float boundary = KeyDist(cand[p - 1]);
        const uint32_t next64_end = min(p + 64u, top_l);
        const uint32_t next256_end = min(p + 256u, top_l);
        const uint32_t next64_span = next64_end > p ? next64_end - p : 1u;
        const uint32_t next256_span = next256_end > p ? next256_end - p : 1u;
        const uint32_t gap32_index = min(max(ls.top_k - 1u, 31u), p - 1u);
        const bool has_prev = s.ls_has_prev != 0;
        float f[TANN_STOP_FEATURES];
        f[0] = ls.feature_mask[0] ? (float)p * ls.inv_top_l : 0.0f;
        f[1] = ls.feature_mask[1] ? (float)expanded * ls.inv_top_l : 0.0f;
        f[2] = ls.feature_mask[2] ? (float)visited * ls.inv_top_l : 0.0f;
        const bool need_best = ls.feature_mask[3] || (ls.feature_mask[4] && ls.next64_flag_mode);
        uint32_t best = top_l;
        if (need_best) {
            best = FindFirstSetBit(unexp, top_l);
            f[3] = ls.feature_mask[3] ? (float)best * ls.inv_top_l : 0.0f;
        } else {
            f[3] = 0.0f;
        }
        if (ls.feature_mask[4]) {
            if (ls.next64_flag_mode) f[4] = best < next64_end ? 1.0f : 0.0f;
            else f[4] = (float)CountBitsInRange(unexp, p, next64_end) / (float)next64_span;
        } else {
            f[4] = 0.0f;
        }
        f[5] = ls.feature_mask[5] ? (float)CountBitsInRange(unexp, p, next256_end) / (float)next256_span
                                  : 0.0f;
        f[6] = ls.feature_mask[6] ? dk : 0.0f;
        f[7] = ls.feature_mask[7] ? (boundary - dk) : 0.0f;
        f[8] = ls.feature_mask[8] ? (KeyDist(cand[gap32_index]) - dk) : 0.0f;
        f[9] = (ls.feature_mask[9] && has_prev) ? (s.ls_prev_dk - dk) : 0.0f;
        f[10] = (ls.feature_mask[10] && has_prev) ? (s.ls_prev_boundary - boundary) : 0.0f;
        if (!ls.feature_mask[11]) {
            f[11] = 0.0f;
        } else if (ls.topk_churn_flag_mode) {
            f[11] = s.ls_topk_changed ? 1.0f : 0.0f;
        } else if (!has_prev) {
            f[11] = 1.0f;
        } else {
            uint32_t changed = 0;
            for (uint32_t i = 0; i < ls.top_k; ++i) {
                const uint32_t cur = KeyRawId(cand[i]);
                bool found = false;
                for (uint32_t j = 0; j < ls.top_k; ++j)
                    if (s.ls_prev_ids[j] == cur) { found = true; break; }
                changed += found ? 0u : 1u;
            }
            f[11] = (float)changed / (float)ls.top_k;
        }
        float logit = ls.bias;
#pragma unroll
        for (int i = 0; i < TANN_STOP_FEATURES; ++i) logit = fmaf(f[i], ls.weights[i], logit);
        s.ls_prev_dk = dk;
        s.ls_prev_boundary = boundary;
        s.ls_has_prev = 1;
        s.ls_topk_changed = 0;
        if (ls.feature_mask[11] && !ls.topk_churn_flag_mode)
            for (uint32_t i = 0; i < ls.top_k; ++i) s.ls_prev_ids[i] = KeyRawId(cand[i]);
        if (logit < ls.threshold_logit) {
            if (ls.shadow_mode) { s.ls_stage = ls.num_stages; break; }
            return true;
        }
        ++s.ls_stage;
    }
    return false;
}

// The code row of a node as 32-bit words (specialised chunk counts only): loading is split from
// summing so that the loads can be issued before a barrier and consumed after it.
template <int kM>
__device__ __forceinline__ void LoadCodeWords(const uint8_t* row, uint32_t (&w)[kM > 0 ? kM / 4 : 1]) {
    const uint4* r4 = reinterpret_cast<const uint4*>(row);
#pragma unroll
    for (int i = 0; i < kM / 16; ++i) {
        const uint4 v = __ldg(r4 + i);
        w[4 * i + 0] = v.x; w[4 * i + 1] = v.y; w[4 * i + 2] = v.z; w[4 * i + 3] = v.w;
    }
}

// Row n of an array: the plain form knows there is one shard.
template <bool kOneShard>
__device__ __forceinline__ const uint8_t* Row(const TannShards& s, uint64_t n, uint64_t row_bytes) {
    if constexpr (kOneShard) return static_cast<const uint8_t*>(s.base[0]) + n * row_bytes;
    else return ShardRow(s, n, row_bytes);
}

}  // namespace tann
