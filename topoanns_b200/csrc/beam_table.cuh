// The query's PQ table in shared memory and the sum of a code row over it, shared by the beam-search kernels for 32, 48 and 96 chunks.
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
// Eight lanes read 128 consecutive bytes of a row of pivots (four codes each), and a lane does so for the rows of kPer chunks. The
// table wants the chunks of a code side by side: writing chunk (step + lane) mod kPer at each step puts the 32 lanes on 32 banks,
// for which a lane's kPer results are first rotated by its number (selects between registers, log2 kPer rounds).
// What bounds it is the stream of dim KB of pivots per query out of L2. Whole calls of 2 k queries with top_l 64: 10 M x 128 uint8 390 ->
// 327 us, 1 M x 768 float32 1176 -> 792 us against one row per lane (32 rows per request); against pivots that a launch in front laid
// out anew 352 -> 352 and 921 -> 851 us.
template <int kPer>
__device__ __forceinline__ void RotateByLane(float4 (&v)[kPer], uint32_t by) {
#pragma unroll
    for (int b = 1; b < kPer; b <<= 1) {
        const bool on = (by & b) != 0;
        float4 w[kPer];
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            const float4 x = v[j], y = v[(j + b) % kPer];
            w[j] = make_float4(on ? y.x : x.x, on ? y.y : x.y, on ? y.z : x.z, on ? y.w : x.w);
        }
#pragma unroll
        for (int j = 0; j < kPer; ++j) v[j] = w[j];
    }
}
__device__ __forceinline__ void AddSquares(float4& acc, const float4 v, float nq) {
    const float2 n = make_float2(nq, nq);
    const float2 a = __fadd2_rn(make_float2(v.x, v.y), n), b = __fadd2_rn(make_float2(v.z, v.w), n);
    const float2 lo = __ffma2_rn(a, a, make_float2(acc.x, acc.y)), hi = __ffma2_rn(b, b, make_float2(acc.z, acc.w));
    acc = make_float4(lo.x, lo.y, hi.x, hi.y);
}
// The entries of a group of 4 * kPer chunks. sub: dims of every chunk (0: chunks of different widths).
template <int kPer>
__device__ __forceinline__ void GroupTable(float* lut, const float* sq, const BeamArgs& a, const float* given, uint32_t sub, uint32_t chunk0, uint32_t tid) {
    const uint32_t p = tid & 7u, first = chunk0 + ((tid & 31u) >> 3) * kPer;
    constexpr uint32_t width = kPer * 4;
    float* t = lut + chunk0 * kCentroids + (first - chunk0);
#pragma unroll 1
    for (uint32_t c0 = (tid >> 5) * 32u + p * 4u; c0 < kCentroids; c0 += 128u) {
        float4 acc[kPer];
#pragma unroll
        for (int j = 0; j < kPer; ++j) acc[j] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (given != nullptr) {
#pragma unroll
            for (int j = 0; j < kPer; ++j) acc[j] = __ldg(reinterpret_cast<const float4*>(given + (size_t)(first + j) * kCentroids + c0));
        } else if (sub != 0) {
            const float* rows = a.ix.pq_tables_col_major + (size_t)first * sub * kCentroids + c0;
            const float* q = sq + first * sub;
#pragma unroll 1
            for (uint32_t s = 0; s < sub; ++s) {
                float4 v[kPer];
#pragma unroll
                for (int j = 0; j < kPer; ++j) v[j] = __ldg(reinterpret_cast<const float4*>(rows + (size_t)(j * sub + s) * kCentroids));
#pragma unroll
                for (int j = 0; j < kPer; ++j) AddSquares(acc[j], v[j], -q[j * sub + s]);
            }
        } else {
#pragma unroll 1
            for (int j = 0; j < kPer; ++j) {
                const uint32_t k1 = __ldg(a.ix.pq_chunk_offsets + first + j + 1);
                float4 x = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 4
                for (uint32_t k = __ldg(a.ix.pq_chunk_offsets + first + j); k < k1; ++k)
                    AddSquares(x, __ldg(reinterpret_cast<const float4*>(a.ix.pq_tables_col_major + (size_t)k * kCentroids + c0)), -sq[k]);
#pragma unroll
                for (int u = 0; u < kPer; ++u)
                    if (u == j) acc[u] = x;
            }
        }
        RotateByLane<kPer>(acc, p);
#pragma unroll
        for (int s = 0; s < kPer; ++s) {
            const uint32_t m = (s + p) % kPer;
            // rows of 16 chunks: lanes p and p + 4 write the same chunk, of codes of different parity
            const bool odd = kPer == 4 && (p & 4u) != 0;
            const float4 x = acc[s];
            t[(c0 + (odd ? 1u : 0u)) * width + m] = odd ? x.y : x.x;
            t[(c0 + (odd ? 0u : 1u)) * width + m] = odd ? x.x : x.y;
            t[(c0 + (odd ? 3u : 2u)) * width + m] = odd ? x.w : x.z;
            t[(c0 + (odd ? 2u : 3u)) * width + m] = odd ? x.z : x.w;
        }
    }
}
// Dims of every chunk, or 0 when the chunks are of different widths. Every warp looks at all chunks, so that a block decides as one.
template <int kM>
__device__ __forceinline__ uint32_t EqualWidth(const uint32_t* offsets, uint32_t dim, uint32_t lane) {
    bool equal = dim % kM == 0;
#pragma unroll
    for (uint32_t m = 0; m <= kM; m += 32)
        if (m + lane <= kM) equal = equal && __ldg(offsets + m + lane) == (m + lane) * (dim / kM);
    return __all_sync(kFull, equal) ? dim / kM : 0u;
}
// Table of query q, built from the pivots or copied from the caller's [M][256] table (tid: 0 to 127; sq: room for the query's
// values); `sync` is a barrier of these 128 threads.
template <int kM, typename Sync>
__device__ __forceinline__ void BuildTable(float* lut, float* sq, const BeamArgs& a, uint64_t q, uint32_t tid, Sync sync) {
    const uint32_t d = a.ix.dim;
    const float* given = a.lut != nullptr ? a.lut + q * (uint64_t)kM * kCentroids : nullptr;
    uint32_t sub = 0;
    if (given == nullptr) {   // src/search/pq_query_tables.cu:33-52
        sub = EqualWidth<kM>(a.ix.pq_chunk_offsets, d, tid & 31);
        for (uint32_t i = tid; i < d; i += 128) sq[i] = LoadAsFloat<float>(a.queries, a.query_kind, q * d + i) - __ldg(a.ix.pq_centroid + i);
    }
    sync();
#pragma unroll 1
    for (uint32_t chunk0 = 0; chunk0 + 32 <= kM; chunk0 += 32) GroupTable<8>(lut, sq, a, given, sub, chunk0, tid);
    if constexpr (kM % 32 != 0) GroupTable<4>(lut, sq, a, given, sub, kM / 32 * 32, tid);
    sync();
}

// Smallest key of a warp (all lanes call; every lane returns it).
__device__ __forceinline__ unsigned long long WarpMinKey(unsigned long long k) {
    const uint32_t hi = __reduce_min_sync(kFull, (uint32_t)(k >> 32));
    const uint32_t lo = __reduce_min_sync(kFull, (uint32_t)(k >> 32) == hi ? (uint32_t)k : 0xffffffffu);
    return ((unsigned long long)hi << 32) | lo;
}

}  // namespace tann
