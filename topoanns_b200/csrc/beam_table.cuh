// The query's PQ table in shared memory and the sum of a code row over it, shared by the beam-search kernels for chunk counts
// that are multiples of 16.
//
// The table lies as [code][chunk], 32 chunks = 32 banks. Lane l reads chunk c ^ l at step c, so the 32 lanes of a look-up
// fall on 32 banks whatever their codes are (a table per chunk in a row of 256 entries: 2 to 3.5 wavefronts per look-up). The
// reference's tree (16, 8, 4, 2, 1 over the chunks of a group of 32) pairs chunk i with chunk i ^ 16, then i ^ 8, ...;
// floating-point addition commutes, so permuting the chunks by any xor leaves every partial sum of the tree, and the
// result, bit for bit the same.
#pragma once

#include "beam_common.cuh"

namespace tann {

// The 16-byte pieces of a code row, in the order in which lane `lane` uses them (bit 4 of the lane exchanges the two pieces
// of a group of 32 chunks).
template <int kM>
__device__ __forceinline__ void LoadCodesXor(const uint8_t* row, uint32_t lane, uint32_t (&w)[kM / 4]) {
    const uint4* r4 = reinterpret_cast<const uint4*>(row);
#pragma unroll
    for (int i = 0; i < kM / 16; ++i) {
        const int piece = (i | 1) * 16 < kM ? (int)((uint32_t)i ^ (lane >> 4)) : i;
        const uint4 v = __ldg(r4 + piece);
        w[4 * i + 0] = v.x; w[4 * i + 1] = v.y; w[4 * i + 2] = v.z; w[4 * i + 3] = v.w;
    }
}
// Bits 2 and 3 of the lane exchange the words of a piece: word j then holds chunks 4 (j ^ lane / 4) + {0..3}.
template <int kM>
__device__ __forceinline__ void PermuteXor(uint32_t lane, uint32_t (&w)[kM / 4]) {
    const bool b3 = (lane & 8u) != 0, b2 = (lane & 4u) != 0;
#pragma unroll
    for (int i = 0; i < kM / 16; ++i) {
        const uint32_t a = w[4 * i], b = w[4 * i + 1], c = w[4 * i + 2], d = w[4 * i + 3];
        const uint32_t a1 = b3 ? c : a, c1 = b3 ? a : c, b1 = b3 ? d : b, d1 = b3 ? b : d;
        w[4 * i] = b2 ? b1 : a1; w[4 * i + 1] = b2 ? a1 : b1;
        w[4 * i + 2] = b2 ? d1 : c1; w[4 * i + 3] = b2 ? c1 : d1;
    }
}

// What a lane needs to turn a byte of a code word into the byte offset of its table entry with one dp4a: step c of a group
// reads chunk c ^ lane, i.e. byte (c ^ lane) & 3 of the permuted word c / 4, at code * 128 + 4 (c ^ lane).
struct LaneOffsets {
    uint32_t chunk[32], row[4];
    __device__ __forceinline__ explicit LaneOffsets(uint32_t lane) {
#pragma unroll
        for (uint32_t c = 0; c < 32; ++c) chunk[c] = (c ^ lane) << 2;
#pragma unroll
        for (uint32_t b = 0; b < 4; ++b) row[b] = 128u << (8u * ((b ^ lane) & 3u));
    }
};
template <int kM>
__device__ __forceinline__ float AdcXor(const unsigned char* lut, const uint32_t (&w)[kM / 4], const LaneOffsets& o) {
    float total = 0.0f;
#pragma unroll
    for (int base = 0; base < kM; base += 32) {
        const int n = (kM - base) < 32 ? (kM - base) : 32;
        const unsigned char* t = lut + base * 1024;
        float2 x[16];
#pragma unroll
        for (int c = 0; c < n; ++c) {
            // groups of 16 chunks: rows of 64 bytes, lanes l and l + 16 read the same chunk
            const uint32_t at = n == 32 ? __dp4a(w[(base + c) / 4], o.row[c & 3], o.chunk[c])
                                        : __dp4a(w[(base + c) / 4], o.row[c & 3] >> 1, o.chunk[c] & 0x3cu);
            const float v = *reinterpret_cast<const float*>(t + at);
            if ((c & 1) == 0) x[c / 2].x = v; else x[c / 2].y = v;
        }
#pragma unroll
        for (int off = 8; off >= 1; off >>= 1) {
#pragma unroll
            for (int i = 0; i < off; ++i)
                if (i + off < n / 2) x[i] = __fadd2_rn(x[i], x[i + off]);
        }
        const float s = x[0].x + x[0].y;
        total = (base == 0) ? s : total + s;
    }
    return total;
}

// ---- the query's table, [code][chunk] per group of 32 (16) chunks --------------------------------------------------------
// Packed pivots (PackPivots): per group, pair of codes and chunk the kSub dims of both codes interleaved, so that a lane
// reads its chunk's values of two codes in one contiguous piece and the packed FP32 operations take them as they come.
template <int kSub>
__device__ __forceinline__ void PairEntries(const float* __restrict__ src, const float (&nq)[kSub], float2& acc) {
    float t[2 * kSub];
#pragma unroll
    for (int i = 0; i < kSub / 2; ++i) *reinterpret_cast<float4*>(t + 4 * i) = __ldg(reinterpret_cast<const float4*>(src) + i);
    acc = make_float2(0.0f, 0.0f);
#pragma unroll
    for (int s = 0; s < kSub; ++s) {
        const float2 df = __fadd2_rn(make_float2(t[2 * s], t[2 * s + 1]), make_float2(nq[s], nq[s]));
        acc = __ffma2_rn(df, df, acc);
    }
}
template <int kM, int kSub>
__device__ __forceinline__ void TableFromPacked(float* lut, const float* sq, const float* __restrict__ packed, uint32_t tid) {
    const uint32_t lane = tid & 31, warp = tid >> 5;
#pragma unroll
    for (int g = 0; g * 32 < kM; ++g) {
        const bool full = (g + 1) * 32 <= kM;
        const uint32_t width = full ? 32u : 16u;
        const uint32_t m = full ? lane : (lane & 15u), half = full ? 0u : lane >> 4;
        float nq[kSub];
#pragma unroll
        for (int s = 0; s < kSub; ++s) nq[s] = -sq[(g * 32 + m) * kSub + s];
        float* t = lut + g * 32 * kCentroids + m;
        const float* src = packed + (size_t)g * 32 * kCentroids * kSub + m * kSub * 2;
        // pairs of codes: warp, warp + 4, ... (both halves of a warp take a pair each in a group of 16 chunks)
        const uint32_t pairs = full ? 128u : 64u;
        constexpr int kAhead = kSub >= 8 ? 4 : (kSub >= 4 ? 8 : 16);
        for (uint32_t p0 = warp; p0 < pairs; p0 += 4 * kAhead) {
            float2 acc[kAhead];
#pragma unroll
            for (int u = 0; u < kAhead; ++u) {
                const uint32_t cp = full ? p0 + 4 * u : 2 * (p0 + 4 * u) + half;
                PairEntries<kSub>(src + (size_t)cp * width * kSub * 2, nq, acc[u]);
            }
#pragma unroll
            for (int u = 0; u < kAhead; ++u) {
                const uint32_t cp = full ? p0 + 4 * u : 2 * (p0 + 4 * u) + half;
                // in a group of 16 the two halves write codes of different parity at a time: 32 banks
                t[(2 * cp + half) * width] = half ? acc[u].y : acc[u].x;
                t[(2 * cp + (half ^ 1u)) * width] = half ? acc[u].x : acc[u].y;
            }
        }
    }
}
// The packed layout is for chunks of one width. Every warp checks all chunks, so that a block decides as one.
template <int kM>
__device__ __forceinline__ bool EqualChunks(const uint32_t* offsets, uint32_t dim, uint32_t lane) {
    bool equal = dim % kM == 0;
#pragma unroll
    for (uint32_t m = 0; m <= kM; m += 32)
        if (m + lane <= kM) equal = equal && __ldg(offsets + m + lane) == (m + lane) * (dim / kM);
    return __all_sync(kFull, equal);
}
// From the column-major pivots (any chunk widths), or copied from a caller's [M][256] table.
template <int kM>
__device__ __forceinline__ void TableFromColumns(float* lut, const float* sq, const BeamArgs& a, const float* given, uint32_t tid) {
    const uint32_t lane = tid & 31, warp = tid >> 5;
#pragma unroll 1
    for (int g = 0; g * 32 < kM; ++g) {
        const bool full = (g + 1) * 32 <= kM;
        const uint32_t width = full ? 32u : 16u;
        const uint32_t m = full ? lane : (lane & 15u), half = full ? 0u : lane >> 4;
        const uint32_t chunk = g * 32 + m;
        float* t = lut + g * 32 * kCentroids + m;
        const uint32_t k0 = given ? 0u : __ldg(a.ix.pq_chunk_offsets + chunk), k1 = given ? 0u : __ldg(a.ix.pq_chunk_offsets + chunk + 1);
        const uint32_t step = full ? 16u : 32u;
#pragma unroll 4
        for (uint32_t c0 = (full ? warp : 2 * warp + half) * 4; c0 < kCentroids; c0 += step) {
            float4 acc = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (given) {
                acc = __ldg(reinterpret_cast<const float4*>(given + (size_t)chunk * kCentroids + c0));
            } else {
                for (uint32_t k = k0; k < k1; ++k) {
                    const float4 v = __ldg(reinterpret_cast<const float4*>(a.ix.pq_tables_col_major + (size_t)k * kCentroids + c0));
                    const float sv = sq[k];
                    float df = v.x - sv; acc.x = fmaf(df, df, acc.x);
                    df = v.y - sv; acc.y = fmaf(df, df, acc.y);
                    df = v.z - sv; acc.z = fmaf(df, df, acc.z);
                    df = v.w - sv; acc.w = fmaf(df, df, acc.w);
                }
            }
            t[(c0 + 0) * width] = acc.x;
            t[(c0 + 1) * width] = acc.y;
            t[(c0 + 2) * width] = acc.z;
            t[(c0 + 3) * width] = acc.w;
        }
    }
}

// Table of query q (tid: 0 to 127; sq: room for the query's values); `sync` is a barrier of these 128 threads.
template <int kM, typename Sync>
__device__ __forceinline__ void BuildTable(float* lut, float* sq, const BeamArgs& a, uint64_t q, uint32_t tid, Sync sync) {
    const uint32_t d = a.ix.dim;
    const float* given = a.lut != nullptr ? a.lut + q * (uint64_t)kM * kCentroids : nullptr;
    const bool packed = a.pivots_packed != nullptr && EqualChunks<kM>(a.ix.pq_chunk_offsets, d, tid & 31);
    if (given == nullptr)   // src/search/pq_query_tables.cu:33-52
        for (uint32_t i = tid; i < d; i += 128) sq[i] = LoadAsFloat<float>(a.queries, a.query_kind, q * d + i) - __ldg(a.ix.pq_centroid + i);
    sync();
    if (packed && d == 2 * kM) TableFromPacked<kM, 2>(lut, sq, a.pivots_packed, tid);
    else if (packed && d == 4 * kM) TableFromPacked<kM, 4>(lut, sq, a.pivots_packed, tid);
    else if (packed && d == 8 * kM) TableFromPacked<kM, 8>(lut, sq, a.pivots_packed, tid);
    else TableFromColumns<kM>(lut, sq, a, given, tid);
    sync();
}

// Smallest key of a warp (all lanes call; every lane returns it).
__device__ __forceinline__ unsigned long long WarpMinKey(unsigned long long k) {
    const uint32_t hi = __reduce_min_sync(kFull, (uint32_t)(k >> 32));
    const uint32_t lo = __reduce_min_sync(kFull, (uint32_t)(k >> 32) == hi ? (uint32_t)k : 0xffffffffu);
    return ((unsigned long long)hi << 32) | lo;
}

}  // namespace tann
