// Beam search for lists of 32, 64, 128 or 256 entries (the candidate capacity), search widths of 1 and 2, 32, 48 or 96 chunks, at
// most 256 frontier slots per step: the common case of the path. One query per block of five warps; the traversal is the
// reference kernel's (src/search/topology_search_kernel.cu:2190-2664) step by step, and the records are bit for bit those of
// the general kernels.
//
// A step ("push") is one dependent chain - memory round trip, visited filter, table sums, list, next memory round trip - and
// with four or five queries per SM both the chain's length and the instructions it issues bound the kernel. Hence:
//
// * Four slot warps own the frontier slots (adjacency ids, code rows, visited filter, table sums). A fifth, the list warp,
//   holds the sorted list in registers (kList keys per lane, rank = register * 32 + lane) and does the list work alone: no
//   shared-memory list, no merge barriers, and each of its instructions is issued once instead of by every warp.
// * Early selection. The next nodes are the smallest among the list's unexpanded entries (known before the push) and the
//   push's new keys below the list's last one. The list warp picks them right behind the one barrier after the table sums;
//   the slot warps issue the next loads and the list warp merges the new keys meanwhile: a sort of 32 keys across the
//   lanes, one split against the end of the list and a bitonic merge.
//
// Keys: distance bits (order-preserving) << 32 | id << 2 | state, so that one 64-bit comparison orders copies of one node
// (they have the same distance) as a merged list holds them: newest first. Copies within the first top_l ranks come from one
// push only (anything else there is in the visited filter); when the last selected node has copies that were not selected,
// these become kTwin and stay behind it. Copies behind rank top_l are revisits: they are new (kNew) and lie in front of the
// older ones, expanded or not. Whether a new key enters a full list is decided without the states: a tie with the entry that it
// would displace keeps the old one (:1338-1424).
#pragma once

#include "beam_table.cuh"

namespace tann {

constexpr uint32_t kSlotThreads = 128, kShortThreads = 160;
constexpr uint32_t kNew = 0, kExpanded = 1, kTwin = 2, kLate = 3;
constexpr unsigned long long kNoKey = 0xff800000ffffffffull;   // (+inf, no id): behind every key that enters a list

__device__ __forceinline__ void SlotSync() { asm volatile("bar.sync 1, 128;" ::: "memory"); }
__device__ __forceinline__ void BlockSync() { asm volatile("bar.sync 0, 160;" ::: "memory"); }

// Merges 32 keys (one per lane, descending) into the ascending list, which keeps the smallest of both.
template <int kList>
__device__ __forceinline__ void MergeIntoList(unsigned long long (&list)[kList], unsigned long long k, uint32_t lane, unsigned long long mask) {
    // The list's last 32 ascending against the new keys descending: the smaller halves, with the rest, form a bitonic sequence.
    // This is also the test of an eager merge, new key number x against the entry x places in front of the last, and with the
    // states masked out a tie keeps the old entry, as there.
    if (k < (list[kList - 1] & mask)) list[kList - 1] = k;
#pragma unroll
    for (int stride = kList / 2; stride > 0; stride >>= 1) {
#pragma unroll
        for (int r = 0; r < kList; ++r) {
            if ((r & stride) == 0) {
                const unsigned long long x = list[r], y = list[r + stride];
                const bool swap = y < x;
                list[r] = swap ? y : x;
                list[r + stride] = swap ? x : y;
            }
        }
    }
#pragma unroll
    for (uint32_t stride = 16; stride > 0; stride >>= 1) {
        const bool keep_max = (lane & stride) != 0;
#pragma unroll
        for (int r = 0; r < kList; ++r) {
            const unsigned long long o = __shfl_xor_sync(kFull, list[r], stride);
            if ((o > list[r]) == keep_max) list[r] = o;
        }
    }
}

__device__ __forceinline__ Cand RecordOf(unsigned long long k) {
    Cand c;
    c.dist = FromOrderedBits((uint32_t)(k >> 32));
    const uint32_t low = (uint32_t)k;
    c.id = low == 0xffffffffu ? kInvalid : (low >> 2) | ((low & 3u) == kExpanded ? kExpandedBit : 0u);
    return c;
}

// Sorts a list that is sorted except for the states of copies: neighbours are exchanged until none is out of order.
template <int kList>
__device__ __forceinline__ void SortCopies(unsigned long long (&list)[kList], uint32_t lane) {
    bool any;
    do {
        bool mine = false;
#pragma unroll
        for (int r = 0; r < kList; ++r) {   // ranks 2 i and 2 i + 1
            const unsigned long long o = __shfl_xor_sync(kFull, list[r], 1);
            if ((lane & 1u) ? o > list[r] : o < list[r]) { list[r] = o; mine = true; }
        }
        unsigned long long before[kList], behind[kList];
#pragma unroll
        for (int r = 0; r < kList; ++r) {
            before[r] = __shfl_sync(kFull, list[r], (lane + 31u) & 31u);
            behind[r] = __shfl_sync(kFull, list[r], (lane + 1u) & 31u);
        }
#pragma unroll
        for (int r = 0; r < kList; ++r) {   // ranks 2 i + 1 and 2 i + 2
            const unsigned long long b = lane == 0u ? (r == 0 ? 0ull : before[r - (r > 0)]) : before[r];
            const unsigned long long f = lane == 31u ? (r == kList - 1 ? ~0ull : behind[r + (r < kList - 1)]) : behind[r];
            if ((lane & 1u) ? f < list[r] : b > list[r]) { list[r] = (lane & 1u) ? f : b; mine = true; }
        }
        any = __any_sync(kFull, mine);
    } while (any);
}

struct ShortLayout {
    uint32_t bloom, fkey, total;
    __host__ __device__ ShortLayout(uint32_t M, uint32_t rounds) {
        bloom = M * kCentroids * 4;
        fkey = bloom + kBloomWords * 4;                      // new keys of a push, two pushes in turn
        total = fkey + 2 * kSlotThreads * rounds * 8;
    }
};

// kKind: 0 = codes gathered by id, 1 = neighbour-code layout, 2 = codes and adjacency in node-id-range shards.
// kR: slots per thread (ceil(W * degree / 128)). kList: list registers per lane of the list warp.
template <int kM, int kR, int kKind, int kList>
__global__ void __launch_bounds__(kShortThreads, kM <= 32 ? 5 : (kM <= 48 ? 4 : 2))
beam_short_kernel(const __grid_constant__ BeamArgs a) {
    constexpr bool kNbr = kKind == 1;
    constexpr bool kOneShard = kKind != 2;
    constexpr uint32_t kFresh = kSlotThreads * kR;   // new keys per push at most
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const ShortLayout lay(kM, kR);
    uint32_t* bloom = reinterpret_cast<uint32_t*>(smem_raw + lay.bloom);
    unsigned long long* fkey = reinterpret_cast<unsigned long long*>(smem_raw + lay.fkey);
    __shared__ unsigned long long s_thr;       // last key of the list; a new key behind it cannot enter
    __shared__ __align__(16) uint32_t s_count[4];   // per slot warp: new keys of the push | passing slots << 16
    __shared__ __align__(16) unsigned long long s_sort[32];
    __shared__ unsigned long long s_open_key[2], s_end[2];   // of the list warp: its first unexpanded keys and their ranks; ranks L - 1, L - 2
    __shared__ uint32_t s_open_rank[2];
    __shared__ uint32_t s_nsel, s_node[2];     // nodes selected (0 ends the search)
    const uint64_t q = blockIdx.x;
    const uint32_t W = a.p.search_width, deg = a.ix.degree, slots = W * deg;
    const uint32_t entry_begin = a.entry_offsets[q];
    const uint32_t num_entries = a.entry_offsets[q + 1] - entry_begin;
    const uint32_t entry_pushes = (num_entries + slots - 1) / slots;
    constexpr uint32_t C = 32u * kList;        // the candidate capacity

    if (warp < 4) {
        // ================================================ slot warps ========================================================
        const uint32_t N = (uint32_t)a.ix.num_nodes;   // below 2^30 (checked by the launcher)
        const uint32_t lt = (1u << lane) - 1u;
        uint32_t my_k[kR], my_j[kR];          // this thread's slots: node my_k, neighbour my_j
        uint32_t id[kR], words[kR][kM / 4];
#pragma unroll
        for (int r = 0; r < kR; ++r) {
            const uint32_t s = r * kSlotThreads + tid;
            my_k[r] = s / deg;
            my_j[r] = s - my_k[r] * deg;
            id[r] = (s < slots && s < num_entries) ? __ldg(a.entry_ids + entry_begin + s) : kInvalid;
        }
        // dim <= kBloomWords (checked by the launcher)
        BuildTable<kM>(reinterpret_cast<float*>(smem_raw), reinterpret_cast<float*>(bloom), a, q, tid, SlotSync);
        for (uint32_t i = tid; i < kBloomWords / 4; i += kSlotThreads) reinterpret_cast<uint4*>(bloom)[i] = make_uint4(0, 0, 0, 0);
        const LaneOffsets offs(lane);
        BlockSync();
        uint32_t push = 0, hash_iter = 0, nslots = slots;
        while (entry_pushes != 0) {
            // ---- visited tests, table sums -----------------------------------------------------------------------------------
            if (!kNbr || push < entry_pushes) {
#pragma unroll
                for (int r = 0; r < kR; ++r)
                    if (id[r] < N) LoadCodesXor<kM>(Row<kOneShard>(a.ix.codes, id[r], kM), lane, words[r]);
            }
            // (a threshold from before the last merge is an upper bound: the list warp sorts out the rest)
            const unsigned long long thr = *reinterpret_cast<volatile unsigned long long*>(&s_thr);
            BloomBits bits[kR];
            bool pass[kR];
            unsigned long long key[kR];
#pragma unroll
            for (int r = 0; r < kR; ++r) {
                bits[r] = BloomPositions(id[r]);
                pass[r] = id[r] < N;
                // an id that is neither the padding value nor a node of the index is skipped and reported
                if (!pass[r] && id[r] != kInvalid && a.status != nullptr) atomicOr(a.status, TANN_STATUS_BEAM_ID_RANGE);
            }
            if (hash_iter == 0 && push != 0) BlockSync();   // the list warp has rebuilt the filter
            pass[0] = pass[0] && !BloomTest(bits[0], bloom);
            bool first_added = false;
            if constexpr (kR > 1) {
                if (nslots > kSlotThreads) {
                    // the reference's 128 threads walk the slots in rounds of 128: the tests of a round see the adds of the
                    // rounds before it (src/search/topology_search_kernel.cu:2543-2564)
                    SlotSync();
                    if (pass[0]) BloomAdd(bits[0], bloom);
                    SlotSync();
                    first_added = true;
                    pass[1] = pass[1] && !BloomTest(bits[1], bloom);
                }
            }
#pragma unroll
            for (int r = 0; r < kR; ++r) {
                PermuteXor<kM>(lane, words[r]);
                key[r] = ((unsigned long long)OrderedBits(AdcXor<kM>(smem_raw, words[r], offs)) << 32) | (id[r] << 2);
            }
            // ---- the new keys that can enter the list ------------------------------------------------------------------------
            uint32_t mine = 0;
            unsigned long long* segment = fkey + (push & 1u) * kFresh + warp * (32u * kR);
#pragma unroll
            for (int r = 0; r < kR; ++r) {
                const bool surv = pass[r] && key[r] < thr;
                const uint32_t b = __ballot_sync(kFull, surv);
                if (surv) segment[(mine & 0xffffu) + __popc(b & lt)] = key[r];
                mine += __popc(b) + (__popc(__ballot_sync(kFull, pass[r])) << 16);
            }
            if (lane == 0) s_count[warp] = mine;
            BlockSync();
            // ---- visited marks, while the list warp selects -------------------------------------------------------------------
            ++push;
            if (++hash_iter >= 3) {
                // every third merge the filter is rebuilt from the first top_l ranks (:2394-2411,2636-2654); this push's marks
                // would be wiped with the rest
                hash_iter = 0;
#pragma unroll 2
                for (uint32_t i = tid; i < kBloomWords / 4; i += kSlotThreads) reinterpret_cast<uint4*>(bloom)[i] = make_uint4(0, 0, 0, 0);
            } else {
#pragma unroll
                for (int r = 0; r < kR; ++r)
                    if (pass[r] && !(kR > 1 && r == 0 && first_added)) BloomAdd(bits[r], bloom);
            }
            BlockSync();
            // ---- the next push's loads ---------------------------------------------------------------------------------------
            if (push < entry_pushes) {
#pragma unroll
                for (int r = 0; r < kR; ++r) {
                    const uint32_t s = r * kSlotThreads + tid, e = push * slots + s;
                    id[r] = (s < slots && e < num_entries) ? __ldg(a.entry_ids + entry_begin + e) : kInvalid;
                }
            } else {
                const uint32_t nsel = s_nsel;
                if (nsel == 0) break;
                nslots = nsel * deg;
#pragma unroll
                for (int r = 0; r < kR; ++r) {
                    id[r] = kInvalid;
                    if (my_k[r] < nsel) {
                        const uint32_t node = s_node[my_k[r]];
                        const uint32_t* row = node < a.ix.adjacency_cached_rows
                                                  ? a.ix.adjacency_cache + (uint64_t)node * deg
                                                  : reinterpret_cast<const uint32_t*>(Row<kOneShard>(a.ix.adjacency, node, (uint64_t)deg * 4));
                        id[r] = __ldg(row + my_j[r]);
                        // the slot's code row sits at (node, j): both loads share one round trip
                        if constexpr (kNbr)
                            LoadCodesXor<kM>(Row<kOneShard>(a.ix.neighbor_codes, node, (uint64_t)deg * kM) + (size_t)my_j[r] * kM, lane, words[r]);
                    }
                }
            }
        }
        if (entry_pushes == 0) {
            for (uint32_t i = tid; i < C; i += kSlotThreads) a.out_cand[q * (uint64_t)C + i] = RecordOf(kNoKey);
            if (tid < 8) a.out_stats[q * 8 + tid] = tid == 5 ? 0xffffffffu : 0u;
        }
    } else {
        // ================================================ list warp =========================================================
        const uint32_t L = a.p.top_l;
        unsigned long long list[kList];
#pragma unroll
        for (int r = 0; r < kList; ++r) list[r] = kNoKey;
        if (lane == 0) {
            s_thr = kNoKey;
            s_nsel = 0;
        }
        uint32_t valid = 0, visited = 0, expanded = 0, iterations = 0, first_full = 0xffffffffu, hash_iter = 0;
        // The first two unexpanded entries of the list and their ranks, and the keys of ranks L - 1 and L - 2: a new key below
        // them lies within the first L ranks, alone or behind one other new key.
        unsigned long long un_key_0 = kNoKey, un_key_1 = kNoKey, at_end_0 = kNoKey, at_end_1 = L > 1 ? kNoKey : 0ull;
        uint32_t un_pos_0 = 0, un_pos_1 = 0;
        constexpr uint32_t kSeg = 32u * kR;
        BlockSync();
        for (uint32_t push = 0; entry_pushes != 0; ++push) {
            BlockSync();   // the push's new keys are there
            const unsigned long long* fresh = fkey + (push & 1u) * kFresh;
            const uint4 c4 = *reinterpret_cast<const uint4*>(s_count);
            const uint32_t counts = c4.x + c4.y + c4.z + c4.w, n = counts & 0xffffu, fv = counts >> 16;
            const uint32_t e0 = c4.x & 0xffffu, e1 = e0 + (c4.y & 0xffffu), e2 = e1 + (c4.z & 0xffffu);
            // new key i: the warps' segments one behind the other
            const auto new_key = [&](uint32_t i) {
                const uint32_t at = i + (i >= e2 ? 3u * kSeg - e2 : (i >= e1 ? 2u * kSeg - e1 : (i >= e0 ? kSeg - e0 : 0u)));
                return i < n ? fresh[at] : kNoKey;
            };
            const bool more = push + 1 < entry_pushes;   // the next push takes entries again
            // ---- selection -----------------------------------------------------------------------------------------------------
            const unsigned long long k0 = new_key(lane);
            uint32_t nsel = 0, list_end = 0;
            unsigned long long done_key = 0ull;   // the largest new key selected (the smaller ones all are) ...
            uint32_t done = 0;                    // ... how many copies of it ...
            unsigned long long last_old = 0ull;   // ... and the last list entry selected
            if (!more && expanded < a.p.max_expansions) {
                unsigned long long m0 = k0, m1 = kNoKey;   // the two least of this lane's keys
#pragma unroll 1
                for (uint32_t i = 32u; i < n; i += 32u) {
                    const unsigned long long k = new_key(i + lane);
                    m1 = k < m0 ? m0 : (k < m1 ? k : m1);
                    m0 = k < m0 ? k : m0;
                }
                const unsigned long long s0 = WarpMinKey(m0);
                const uint32_t holders = __ballot_sync(kFull, m0 == s0);
                const bool owner = m0 == s0 && (holders & ((1u << lane) - 1u)) == 0u;
                const unsigned long long s1 = WarpMinKey(owner ? m1 : m0);
                const bool new_first = s0 < un_key_0;
                if (new_first ? s0 < at_end_0 : un_key_0 < kNoKey) {
                    nsel = 1;
                    uint32_t id0, id1 = 0;
                    if (new_first) { done_key = s0; done = 1; id0 = (uint32_t)s0 >> 2; }
                    else { last_old = un_key_0; list_end = un_pos_0 + 1u; id0 = (uint32_t)last_old >> 2; }
                    if (W == 2) {
                        const unsigned long long s = new_first ? s1 : s0, u = new_first ? un_key_0 : un_key_1;
                        const uint32_t u_pos = new_first ? un_pos_0 + 1u : un_pos_1;
                        if (s < u) {
                            if (s < (new_first ? at_end_1 : at_end_0)) {
                                nsel = 2;
                                id1 = (uint32_t)s >> 2;
                                done = s == done_key ? 2u : 1u;
                                done_key = s;
                            }
                        } else if (u < kNoKey && u_pos < L) {
                            nsel = 2;
                            id1 = (uint32_t)u >> 2;
                            last_old = u;
                            list_end = (new_first ? un_pos_0 : un_pos_1) + 1u;
                        }
                    }
                    if (lane < 2) s_node[lane] = lane == 0 ? id0 : id1;
                }
            }
            if (lane == 0) s_nsel = nsel;
            BlockSync();   // the selection is there
            const bool last_push = !more && nsel == 0;
            // ---- merge, behind the next push's loads ------------------------------------------------------------------------------
            if (list_end != 0u) {   // every unexpanded entry up to there was selected; a twin of the last one stays behind it
#pragma unroll
                for (int r = 0; r < kList; ++r) {
                    if (r * 32u + lane < list_end) list[r] = (list[r] & ~3ull) | kExpanded;
                    else if (((list[r] ^ last_old) >> 2) == 0ull) list[r] = (list[r] & ~3ull) | kTwin;
                }
            }
            // The merge below takes 32 keys at a time. Where several such merges meet a full list that may hold copies of theirs (behind
            // rank L), a later one must not displace an old copy that an earlier one left in its place: until the last of them
            // new copies are kLate, behind the old ones, and so the first to drop out.
            const bool late = n > 32u && C > L && valid != 0u && (uint64_t)valid + fv > C;
            const uint32_t nv = (uint32_t)min((uint64_t)C, (uint64_t)valid + fv);
            if (first_full == 0xffffffffu && nv >= L) first_full = push < entry_pushes ? 0u : iterations;
            visited += fv;
            valid = nv;
            iterations += nsel != 0u ? 1u : 0u;
            expanded += nsel;
            uint32_t copies = 0;
#pragma unroll 1
            for (uint32_t c = 0; c < n; c += 32u) {
                unsigned long long k = c == 0 ? k0 : new_key(c + lane);
                if (done != 0u) {
                    const uint32_t same = __ballot_sync(kFull, k == done_key);
                    if (k < done_key) k |= kExpanded;
                    else if (k == done_key) k |= copies + __popc(same & ((1u << lane) - 1u)) < done ? kExpanded : kTwin;
                    copies += __popc(same);
                }
                if (late && ((uint32_t)k & 3u) == kNew) k |= kLate;
                // descending order by rank counting
                s_sort[lane] = k;
                __syncwarp();
                uint32_t rank = 0;
                const uint32_t m = min(n - c, 32u);
#pragma unroll 1
                for (uint32_t j = 0; j < m; j += 8u) {
                    const ulonglong2* p = reinterpret_cast<const ulonglong2*>(s_sort + j);
                    const ulonglong2 a0 = p[0], a1 = p[1], a2 = p[2], a3 = p[3];
                    rank += (a0.x < k ? 1u : 0u) + (a0.y < k ? 1u : 0u) + (a1.x < k ? 1u : 0u) + (a1.y < k ? 1u : 0u);
                    rank += (a2.x < k ? 1u : 0u) + (a2.y < k ? 1u : 0u) + (a3.x < k ? 1u : 0u) + (a3.y < k ? 1u : 0u);
                }
                rank += __popc(__match_any_sync(kFull, rank) & ((1u << lane) - 1u));   // equal keys: any order
                __syncwarp();
                s_sort[31u - rank] = k;
                __syncwarp();
                MergeIntoList<kList>(list, s_sort[lane], lane, late ? ~0ull : ~3ull);
                __syncwarp();
            }
            if (late) {
#pragma unroll
                for (int r = 0; r < kList; ++r)
                    if (((uint32_t)list[r] & 3u) == kLate && list[r] != kNoKey) list[r] &= ~3ull;
                SortCopies<kList>(list, lane);
            }
            if (last_push) break;
            if (lane == 31u) *reinterpret_cast<volatile unsigned long long*>(&s_thr) = list[kList - 1];
            if (++hash_iter >= 3) {
                hash_iter = 0;
#pragma unroll
                for (int r = 0; r < kList; ++r)
                    if (r * 32u + lane < L && list[r] != kNoKey) BloomAdd((uint32_t)list[r] >> 2, bloom);
                BlockSync();   // the filter is complete
            }
            // the first unexpanded ranks below L
            uint32_t open = 0;
#pragma unroll
            for (int r = 0; r < kList; ++r) {
                const uint32_t rank = r * 32u + lane;
                const bool mine = rank < L && list[r] != kNoKey && ((uint32_t)list[r] & 3u) != kExpanded;
                const uint32_t b = __ballot_sync(kFull, mine);
                const uint32_t order = open + __popc(b & ((1u << lane) - 1u));
                if (mine && order < W) { s_open_key[order] = list[r]; s_open_rank[order] = rank; }
                if (rank == L - 1u) s_end[0] = list[r];
                if (rank + 2u == L) s_end[1] = list[r];
                open += __popc(b);
            }
            __syncwarp();
            un_key_0 = open > 0u ? s_open_key[0] : kNoKey;
            un_pos_0 = s_open_rank[0];
            un_key_1 = W == 2u && open > 1u ? s_open_key[1] : kNoKey;
            un_pos_1 = s_open_rank[1];
            at_end_0 = s_end[0];
            if (L > 1u) at_end_1 = s_end[1];
            __syncwarp();
        }
        if (entry_pushes == 0) return;
        // ---- results ------------------------------------------------------------------------------------------------------------
        Cand* out = a.out_cand + q * (uint64_t)C;
#pragma unroll
        for (int r = 0; r < kList; ++r) out[r * 32u + lane] = RecordOf(list[r]);
        if (lane == 0) {
            uint32_t* st = a.out_stats + q * 8;
            st[0] = visited; st[1] = expanded; st[2] = 0; st[3] = iterations;
            st[4] = valid; st[5] = first_full; st[6] = 0; st[7] = 0;
        }
    }
}

typedef void (*BeamKernelFn)(const BeamArgs);
template <int kM, int kList>
BeamKernelFn PickShortOf(uint32_t rounds, int kind) {
    if (rounds == 1)
        return kind == 2 ? beam_short_kernel<kM, 1, 2, kList> : (kind == 1 ? beam_short_kernel<kM, 1, 1, kList> : beam_short_kernel<kM, 1, 0, kList>);
    return kind == 2 ? beam_short_kernel<kM, 2, 2, kList> : (kind == 1 ? beam_short_kernel<kM, 2, 1, kList> : beam_short_kernel<kM, 2, 0, kList>);
}

}  // namespace tann
