// Beam search for steps of up to 256 frontier slots that the register list does not take (wider searches, lists of up to 1024 entries, the
// learned stop): 32, 48 or 96 chunks, one query per 128-thread block, the list in shared memory. Table, early selection and records as
// in beam_short.cuh; the merge is shared by the block: a new key's place is its rank among the new keys plus its lower bound
// in the list, the taken places form a bitmap, and the entry of any other place p is old entry p - (taken places below p).
// The same pass yields the bitmap of unexpanded ranks.
#pragma once

#include "beam_table.cuh"

namespace tann {

constexpr uint32_t kTakenWords = 32;   // places of a list

// Where the parts of a block's shared memory start, in bytes; shared by the launcher and the kernel.
struct LongLayout {
    uint32_t bloom, list, other, fkey, place, words, total;
    __host__ __device__ LongLayout(uint32_t M, uint32_t rounds, uint32_t list_len, bool two_lists) {
        bloom = M * kCentroids * 4;
        list = bloom + kBloomWords * 4;
        other = list + list_len * 8;                      // second list, when there is one
        fkey = (other + (two_lists ? list_len * 8 : 0) + 15u) & ~15u;
        place = fkey + kBeamThreads * rounds * 8 + 32;    // new keys, and invalid ones behind the last
        words = (place + kBeamThreads * rounds * 2 + 15u) & ~15u;
        total = words + (kTakenWords + 32) * 4;           // taken places, unexpanded ranks
    }
};

// What warp 0 tells the block about the selection of the next nodes.
struct LongPicks {
    uint32_t count;        // nodes selected; 0 = the search ends
    uint32_t new_picks;    // how many of them are new keys: the first of those in order
    uint32_t list_end;     // 1 + rank of the last selected list entry (0: none)
    uint32_t pad;
    uint32_t node[TANN_MAX_SEARCH_WIDTH];
};

// kKind: 0 = codes gathered by id, 1 = neighbour-code layout, 2 = codes and adjacency in node-id-range shards.
// kR: slots per thread (ceil(W * degree / 128)). kLate: the learned stop looks at the merged list before nodes are selected.
template <int kM, int kR, int kKind, bool kLate>
__global__ void __launch_bounds__(kBeamThreads, kM <= 32 ? 5 : (kM <= 48 ? 4 : 2))
beam_long_kernel(const __grid_constant__ BeamArgs a) {
    constexpr bool kNbr = kKind == 1;
    constexpr bool kOneShard = kKind != 2;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const uint32_t C = a.p.candidate_capacity, L = a.p.top_l, W = a.p.search_width, deg = a.ix.degree;
    const uint32_t slots = W * deg;
    const uint64_t N = a.ix.num_nodes;
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const LongLayout lay(kM, kR, a.list_len, a.two_lists != 0);
    float* lut = reinterpret_cast<float*>(smem_raw);
    uint32_t* bloom = reinterpret_cast<uint32_t*>(smem_raw + lay.bloom);
    unsigned long long* fkey = reinterpret_cast<unsigned long long*>(smem_raw + lay.fkey);
    uint16_t* place = reinterpret_cast<uint16_t*>(smem_raw + lay.place);
    uint32_t* taken = reinterpret_cast<uint32_t*>(smem_raw + lay.words);
    uint32_t* unexp = taken + kTakenWords;
    __shared__ uint32_t s_count[2];       // new keys | passing slots << 16 of a push, two pushes in turn
    __shared__ uint32_t s_flag;
    __shared__ __align__(16) LongPicks picks;
    __shared__ BeamCtl ctl;
    const LaneOffsets offs(lane);
    const uint32_t lt = (1u << lane) - 1u;
    const uint32_t UW = (L + 31) / 32;
    uint32_t my_k[kR], my_j[kR];          // this thread's slots: node my_k, neighbour my_j
#pragma unroll
    for (int r = 0; r < kR; ++r) {
        my_k[r] = (r * kBeamThreads + tid) / deg;
        my_j[r] = r * kBeamThreads + tid - my_k[r] * deg;
    }
    for (uint64_t q = blockIdx.x; q < a.num_queries; q += gridDim.x) {
    const uint32_t entry_begin = a.entry_offsets[q];
    const uint32_t num_entries = a.entry_offsets[q + 1] - entry_begin;

    // ---- the query's table ---------------------------------------------------------------------------------------------
    __syncthreads();   // the query before is done
    // dim <= kBloomWords (checked by the launcher)
    BuildTable<kM>(lut, reinterpret_cast<float*>(bloom), a, q, tid, [] { __syncthreads(); });

    const uint32_t list_len = a.list_len;
    const bool two_lists = a.two_lists != 0;
    {
        unsigned long long* cur = reinterpret_cast<unsigned long long*>(smem_raw + lay.list);
        unsigned long long* nxt = two_lists ? reinterpret_cast<unsigned long long*>(smem_raw + lay.other) : cur;
        for (uint32_t i = tid; i < kBloomWords / 4; i += kBeamThreads) reinterpret_cast<uint4*>(bloom)[i] = make_uint4(0, 0, 0, 0);
        if (tid < kTakenWords + 32) taken[tid] = 0u;
        if (tid < 2) s_count[tid] = 0;
        if (tid == 0) {
            s_flag = 0;
            picks.count = 0; picks.new_picks = 0; picks.list_end = 0;
        }
        if constexpr (kLate) {
            // the learned stop reads ranks up to `valid`, which are invalid from `mv` on
            for (uint32_t i = tid; i < list_len; i += kBeamThreads) cur[i] = nxt[i] = kInvalidKey;
            if (tid == 0) {
                ctl.ls_stage = 0; ctl.ls_has_prev = 0; ctl.ls_topk_changed = 0;
                ctl.ls_prev_dk = __int_as_float(0x7f800000);
                ctl.ls_prev_boundary = __int_as_float(0x7f800000);
            }
            if (tid < 32) ctl.ls_prev_ids[tid] = kInvalid;
        }
        // block-uniform state, identical in every thread
        uint32_t valid = 0, visited = 0, hash_iter = 0, expanded = 0, iterations = 0, mv = 0;
        uint32_t first_full = 0xffffffffu, entries_done = 0, nslots = slots, parity = 0;
        // of warp 0, lane x: the x-th unexpanded entry of the list, and its rank
        unsigned long long un_key = kInvalidKey;
        uint32_t un_pos = 0;
        bool from_entries = num_entries != 0, stop = num_entries == 0;
        uint32_t id[kR], words[kR][kM / 4];
#pragma unroll
        for (int r = 0; r < kR; ++r) {
            const uint32_t s = r * kBeamThreads + tid;
            id[r] = (s < slots && s < num_entries) ? __ldg(a.entry_ids + entry_begin + s) : kInvalid;
        }
        __syncthreads();
        while (!stop) {
            // ---- visited tests, table sums ---------------------------------------------------------------------------------
            const uint32_t rounds = kR == 1 ? 1u : (nslots + kBeamThreads - 1) / kBeamThreads;
            if (!kNbr || from_entries) {
#pragma unroll
                for (int r = 0; r < kR; ++r)
                    if (id[r] < N) LoadCodesXor<kM>(Row<kOneShard>(a.ix.codes, id[r], kM), lane, words[r]);
            }
            BloomBits bits[kR];
            bool pass[kR];
            unsigned long long key[kR];
#pragma unroll
            for (int r = 0; r < kR; ++r) {
                bits[r] = BloomPositions(id[r]);
                pass[r] = id[r] < N;
                // an id that is neither the padding value nor a node of the index is skipped and reported
                if (id[r] != kInvalid && !pass[r] && a.status != nullptr) atomicOr(a.status, TANN_STATUS_BEAM_ID_RANGE);
                if (r == 0) pass[r] = pass[r] && !BloomTest(bits[r], bloom);
            }
            if (kR > 1 && rounds > 1) {
                // the reference's 128 threads walk the slots in rounds of 128: the tests of a round see the adds of the
                // rounds before it (src/search/topology_search_kernel.cu:2543-2564)
                __syncthreads();
                if (pass[0]) BloomAdd(bits[0], bloom);
                __syncthreads();
                if constexpr (kR > 1) pass[1] = pass[1] && !BloomTest(bits[1], bloom);
            }
#pragma unroll
            for (int r = 0; r < kR; ++r) {
                PermuteXor<kM>(lane, words[r]);
                key[r] = ((unsigned long long)OrderedBits(AdcXor<kM>(smem_raw, words[r], offs)) << 32) | id[r];
            }
            // ---- which new keys can enter the list -------------------------------------------------------------------------
            // A NaN distance (its key is behind the invalid one) never enters, as in the general form: its slot counts as visited
            // and as valid, so that `valid` may run ahead of `mv`.
            const unsigned long long thr = mv == list_len ? (cur[list_len - 1] & kCmpMask) : kInvalidKey;
            uint32_t ballots[kR], mine = 0;
#pragma unroll
            for (int r = 0; r < kR; ++r) {
                ballots[r] = __ballot_sync(kFull, pass[r] && key[r] < thr);
                mine += __popc(ballots[r]) + (__popc(__ballot_sync(kFull, pass[r])) << 16);
            }
            uint32_t base = 0;
            if (lane == 0) base = atomicAdd(&s_count[parity], mine);
            base = __shfl_sync(kFull, base, 0) & 0xffffu;
#pragma unroll
            for (int r = 0; r < kR; ++r)
                if ((ballots[r] >> lane) & 1u) fkey[base + (r == 1 ? __popc(ballots[0]) : 0u) + __popc(ballots[r] & lt)] = key[r];
            __syncthreads();
            const uint32_t counts = s_count[parity];
            const uint32_t n = counts & 0xffffu, fv = counts >> 16;
            parity ^= 1u;
            const uint32_t nv = (uint32_t)min((uint64_t)C, (uint64_t)valid + fv);
            if (first_full == 0xffffffffu && nv >= L) first_full = from_entries ? 0u : iterations;
            visited += fv;
            entries_done += from_entries ? slots : 0u;
            const bool more = from_entries && entries_done < num_entries;   // the next push takes entries again
            // ---- early selection, by warp 0 ------------------------------------------------------------------------------------
            if (!kLate && !more && warp == 0) {
                uint32_t nsel = 0, new_picks = 0, list_end = 0, pick = kInvalid;
                if (expanded < a.p.max_expansions) {
                    // of the new keys a lane looks at (usually one), the least; used = those selected already
                    unsigned long long least = kInvalidKey;
                    uint32_t at_s = 0, used = 0, un_taken = 0;
                    for (uint32_t s = 0; s * 32u < n; ++s) {
                        const unsigned long long k = s * 32u + lane < n ? fkey[s * 32u + lane] : kInvalidKey;
                        if (k < least) { least = k; at_s = s; }
                    }
                    unsigned long long s_min = n != 0 ? WarpMinKey(least) : kInvalidKey;
                    while (nsel < W) {
                        const unsigned long long u = __shfl_sync(kFull, un_key, un_taken);
                        if (s_min < kInvalidKey && s_min <= u) {
                            // inside the first L ranks: fewer than L - new_picks list entries are below it
                            const uint32_t at = L - 1u - new_picks;
                            if (new_picks >= L || !(at >= mv || s_min <= (cur[at] & kCmpMask))) break;
                            if (mv + n > list_len) {
                                // a tie with the entry it would displace: not accepted, nor is any larger new key
                                const uint32_t last = list_len - 1u - new_picks;
                                if (last < mv && s_min >= (cur[last] & kCmpMask)) { s_min = kInvalidKey; continue; }
                            }
                            if (lane == nsel) pick = (uint32_t)s_min & kRawMask;
                            ++new_picks;
                            if (++nsel < W) {
                                const uint32_t owner = __ffs(__ballot_sync(kFull, least == s_min)) - 1;
                                if (lane == owner) {
                                    used |= 1u << at_s;
                                    least = kInvalidKey;
                                    if (n > 32u) {
                                        for (uint32_t s = 0; s * 32u < n; ++s) {
                                            const unsigned long long k = (s * 32u + lane < n && !((used >> s) & 1u)) ? fkey[s * 32u + lane] : kInvalidKey;
                                            if (k < least) { least = k; at_s = s; }
                                        }
                                    }
                                }
                                s_min = WarpMinKey(least);
                            }
                        } else if (u < kInvalidKey) {
                            const uint32_t pos = __shfl_sync(kFull, un_pos, un_taken);
                            if (pos + new_picks >= L) break;
                            if (lane == nsel) pick = (uint32_t)u & kRawMask;
                            list_end = pos + 1u;
                            ++un_taken;
                            ++nsel;
                        } else {
                            break;
                        }
                    }
                }
                if (lane < nsel) picks.node[lane] = pick;
                if (lane == 0) { picks.count = nsel; picks.new_picks = new_picks; picks.list_end = list_end; }
            }
            if (!kLate && !more) __syncthreads();
            uint32_t new_picks = 0, list_end = 0;
            const auto issue_nodes = [&]() {
                const uint32_t nsel = picks.count;
                nslots = nsel * deg;
                ++iterations;
                expanded += nsel;
#pragma unroll
                for (int r = 0; r < kR; ++r) {
                    id[r] = kInvalid;
                    if (my_k[r] < nsel) {
                        const uint32_t node = picks.node[my_k[r]];
                        const uint32_t* row = node < a.ix.adjacency_cached_rows
                                                  ? a.ix.adjacency_cache + (uint64_t)node * deg
                                                  : reinterpret_cast<const uint32_t*>(Row<kOneShard>(a.ix.adjacency, node, (uint64_t)deg * 4));
                        id[r] = __ldg(row + my_j[r]);
                        // the slot's code row sits at (node, j): both loads share one round trip
                        if constexpr (kNbr)
                            LoadCodesXor<kM>(Row<kOneShard>(a.ix.neighbor_codes, node, (uint64_t)deg * kM) + (size_t)my_j[r] * kM, lane, words[r]);
                    }
                }
            };
            from_entries = more;
            if (more) {
#pragma unroll
                for (int r = 0; r < kR; ++r) {
                    const uint32_t s = r * kBeamThreads + tid, e = entries_done + s;
                    id[r] = (s < slots && e < num_entries) ? __ldg(a.entry_ids + entry_begin + e) : kInvalid;
                }
                nslots = slots;
            } else if (!kLate) {
                new_picks = picks.new_picks;
                list_end = picks.list_end;
                if (picks.count == 0) stop = true; else issue_nodes();
            }
            if constexpr (kLate) list_end = picks.list_end;   // selected after the last merge
            // ---- behind the loads: visited marks, merge ------------------------------------------------------------------
            ++hash_iter;
            const bool rebuild = hash_iter >= 3;
            if (rebuild) {
                // every third merge the filter is rebuilt from the first L ranks (:2394-2411,2636-2654): this push's marks
                // would be wiped with the rest
                hash_iter = 0;
                for (uint32_t i = tid; i < kBloomWords / 4; i += kBeamThreads) reinterpret_cast<uint4*>(bloom)[i] = make_uint4(0, 0, 0, 0);
            } else {
#pragma unroll
                for (int r = 0; r < kR; ++r)
                    if (pass[r] && !(kR > 1 && r == 0 && rounds > 1)) BloomAdd(bits[r], bloom);
            }
            const uint32_t total = mv + n;
            while (n != 0) {   // once, unless a new key ties with the last entry of a full list
                // Places of the new keys, one lane per key (warps 1 to 3): keys of this push below it, plus list entries below it.
                for (uint32_t c = warp - 1u; c * 32u < n && warp != 0; c += 3u) {
                    const uint32_t i = c * 32u + lane;
                    if (lane < 4u) fkey[n + lane] = kInvalidKey;   // the loop below takes four keys at a time
                    const unsigned long long k = i < n ? fkey[i] : kInvalidKey;
                    __syncwarp();
                    uint32_t rank = 0;
#pragma unroll 1
                    for (uint32_t j = 0; j < n; j += 4) {
                        const ulonglong2 ka = *reinterpret_cast<const ulonglong2*>(fkey + j);
                        const ulonglong2 kb = *reinterpret_cast<const ulonglong2*>(fkey + j + 2);
                        rank += (ka.x < k) ? 1u : 0u;
                        rank += (ka.y < k) ? 1u : 0u;
                        rank += (kb.x < k) ? 1u : 0u;
                        rank += (kb.y < k) ? 1u : 0u;
                    }
                    uint32_t below = 0;
                    if (mv != 0) {
#pragma unroll 1
                        for (uint32_t b = 1u << (31 - __clz(mv)); b > 0; b >>= 1) {
                            const uint32_t t = below + b;
                            if (t <= mv && (cur[t - 1] & kCmpMask) < k) below = t;
                        }
                    }
                    if (i < n) {
                        uint32_t pos = rank + below;
                        const uint32_t places = list_len;
                        // copies of one node in the same push have equal keys: they take neighbouring places
                        while (pos < places && ((atomicOr(&taken[pos >> 5], 1u << (pos & 31u)) >> (pos & 31u)) & 1u) != 0u) { ++pos; ++rank; }
                        place[i] = (uint16_t)min(pos, places);
                        if (total > list_len && pos < places && below < mv && (cur[below] & kCmpMask) == k) {
                            // A full list takes a new key only while it is below the entry it would displace
                            // (:1338-1424): at the end of the list a tie keeps the old entries.
                            uint32_t upto = below + 1;
                            while (upto < mv && (cur[upto] & kCmpMask) == k) ++upto;
                            if (rank + upto >= list_len) { s_flag = 1; place[i] |= 0x8000u; }
                        }
                        if constexpr (kLate) if (pos < a.p.learned_stop.top_k) ctl.ls_topk_changed = 1;
                    }
                }
                __syncthreads();
                if (s_flag == 0u) break;
                // rare: take the rejected keys out and place the others again
                __syncthreads();
                if (tid == 0) s_flag = 0;
                for (uint32_t i = tid; i < n; i += kBeamThreads)
                    if (place[i] & 0x8000u) fkey[i] = kInvalidKey;
                if (tid < kTakenWords) taken[tid] = 0u;
                __syncthreads();
            }
            // Places [0, span) of the list: one that no new key took holds the old entry with as many untaken places in
            // front of it.
            const uint32_t span = min(total, list_len);
            const uint32_t rows = (span + 31u) / 32u;
            for (uint32_t hi = (rows + 3u) / 4u; hi > 0;) {   // from the end, up to four rows per warp at a time
                const uint32_t take = min(hi, 4u), first = hi - take;
                unsigned long long keep[4];
                uint32_t old_at = 0;   // bit u: keep[u] holds an entry
#pragma unroll
                for (uint32_t u = 0; u < 4; ++u) {
                    const uint32_t w = (first + u) * 4u + warp;
                    if (u < take && w < rows) {
                        const uint32_t word = taken[w], p = w * 32u + lane;
                        const uint32_t below = __reduce_add_sync(kFull, lane < w ? (uint32_t)__popc(taken[lane]) : 0u);
                        const uint32_t in_front = below + __popc(word & lt);
                        bool un;
                        if ((word >> lane) & 1u) {
                            un = in_front >= new_picks;
                        } else {
                            un = false;
                            if (p < span) {
                                const uint32_t o = p - in_front;
                                unsigned long long k = cur[o];
                                if (o < list_end) k |= kExpandedBit;   // every unexpanded entry up to there was selected
                                un = ((uint32_t)k & kExpandedBit) == 0u;
                                keep[u] = k;
                                old_at |= 1u << u;
                            }
                        }
                        const uint32_t un_word = __ballot_sync(kFull, un && p < L);
                        if (lane == 0 && w < UW) unexp[w] = un_word;
                    }
                }
                if (!two_lists) __syncthreads();   // every thread has read its entries of the list it now writes
#pragma unroll
                for (uint32_t u = 0; u < 4; ++u) {
                    if ((old_at >> u) & 1u) {
                        const uint32_t p = (first + u) * kBeamThreads + tid;
                        nxt[p] = keep[u];
                    }
                }
                hi = first;
            }
            for (uint32_t i = tid; i < n; i += kBeamThreads) {
                const uint32_t p = place[i];
                if (p < span) {
                    unsigned long long k = fkey[i];
                    // the first new_picks of the new keys are the ones selected: those with fewer new keys in front
                    if (new_picks != 0) {
                        uint32_t before = __popc(taken[p >> 5] & ((1u << (p & 31u)) - 1u));
                        for (uint32_t w = 0; w < (p >> 5) && before < new_picks; ++w) before += __popc(taken[w]);
                        if (before < new_picks) k |= kExpandedBit;
                    }
                    nxt[p] = k;
                }
            }
            mv = span;
            valid = nv;
            if (two_lists) { unsigned long long* t = cur; cur = nxt; nxt = t; }
            __syncthreads();
            if (tid < kTakenWords) taken[tid] = 0u;   // written again behind the next barrier
            if (tid == 0) s_count[parity ^ 1u] = 0;
            if (rebuild)
                for (uint32_t p = tid; p < min(mv, L); p += kBeamThreads) BloomAdd((uint32_t)cur[p] & kRawMask, bloom);
            if constexpr (kLate) {
                if (!from_entries) {
                    if (expanded >= a.p.max_expansions || valid == 0) {
                        stop = true;
                    } else {
                        if (tid == 0)
                            ctl.stop = LearnedStop(a.p.learned_stop, ctl, valid, visited, expanded, cur, unexp, L) ? 1u : 0u;
                        __syncthreads();
                        stop = ctl.stop != 0u;
                    }
                }
            }
            if (!stop && warp == 0 && (!kLate || !from_entries)) {
                // the first W unexpanded ranks of the list
                uint32_t word = lane < UW ? unexp[lane] : 0u, found = 0;
                un_pos = 0;
                for (uint32_t live = __ballot_sync(kFull, word != 0u); live != 0u && found < W; ++found) {
                    const uint32_t w = __ffs(live) - 1u;
                    const uint32_t bit = __ffs(__shfl_sync(kFull, word, w)) - 1u;
                    if (lane == found) un_pos = w * 32u + bit;
                    if (lane == w) word &= word - 1u;
                    live = __ballot_sync(kFull, word != 0u);
                }
                un_key = lane < found ? cur[un_pos] : kInvalidKey;
                if constexpr (kLate) {
                    if (lane < found) picks.node[lane] = (uint32_t)un_key & kRawMask;
                    const uint32_t last = __shfl_sync(kFull, un_pos, found != 0u ? found - 1u : 0u);
                    if (lane == 0) { picks.count = found; picks.list_end = found != 0u ? last + 1u : 0u; }
                }
            }
            if constexpr (kLate) {
                __syncthreads();   // the selection is complete
                if (!stop && !from_entries && picks.count == 0) stop = true;
            }
            if (rebuild && !kLate) __syncthreads();   // the filter is complete
            if constexpr (kLate) {
                if (!stop && !from_entries) issue_nodes();
            }
        }
        // ---- results ---------------------------------------------------------------------------------------------------------
        __syncthreads();
        Cand* out = a.out_cand + q * (uint64_t)C;
        for (uint32_t i = tid; i < C; i += kBeamThreads) {
            unsigned long long k = kInvalidKey;
            if (i < mv) k = cur[i];
            Cand c;
            c.dist = KeyDist(k);
            c.id = KeyPackedId(k);
            out[i] = c;
        }
        if (tid == 0) {
            uint32_t* st = a.out_stats + q * 8;
            st[0] = visited; st[1] = expanded; st[2] = 0; st[3] = iterations;
            st[4] = valid; st[5] = first_full; st[6] = 0; st[7] = 0;
        }
    }
    }
}

typedef void (*BeamKernelFn)(const BeamArgs);
template <int kM>
BeamKernelFn PickLongOf(uint32_t rounds, int kind, bool late) {
    if (rounds == 1) {
        if (late) return kind == 2 ? nullptr : (kind == 1 ? beam_long_kernel<kM, 1, 1, true> : beam_long_kernel<kM, 1, 0, true>);
        // (48 chunks: steps of up to 128 slots come here with the learned stop only)
        if constexpr (kM != 48) return kind == 2 ? beam_long_kernel<kM, 1, 2, false> : (kind == 1 ? beam_long_kernel<kM, 1, 1, false> : beam_long_kernel<kM, 1, 0, false>);
        return nullptr;
    }
    if (kind == 2) return late ? nullptr : beam_long_kernel<kM, 2, 2, false>;
    if (kind == 1) return late ? beam_long_kernel<kM, 2, 1, true> : beam_long_kernel<kM, 2, 1, false>;
    return late ? beam_long_kernel<kM, 2, 0, true> : beam_long_kernel<kM, 2, 0, false>;
}

}  // namespace tann
