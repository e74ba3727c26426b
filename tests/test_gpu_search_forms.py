"""The forms of the beam search and of the pq2 refine that a call is sent to by its sizes, at the edges of their ranges."""
import dataclasses

import numpy as np
import pytest
import torch

from oracle import oracle as orc
from topoanns_b200 import capi, search

from gpu_support import assert_candidates_equal, device_index, fixed_entries, np_u32, small_index

pytestmark = pytest.mark.gpu


def _index(chunks):
    if chunks == 32:
        return small_index()
    if chunks == 48:
        return small_index(name="cfg3", num_nodes=12000, components=60, num_queries=128)
    return small_index(name="cfg5", num_nodes=6000, components=30, num_queries=64)


# top_l on both sides of each list width of the register form (32, 64, 128, 256 ranks) and beyond it; capacities from the list
# itself to one that keeps a long unsorted tail; steps of up to 128 and up to 256 slots
@pytest.mark.parametrize("chunks", [32, 48, 96])
@pytest.mark.parametrize("top_l,width,top_n", [(1, 1, 1), (5, 2, 5), (16, 2, 192), (32, 2, 32), (33, 1, 33), (64, 3, 300), (65, 2, 65),
                                               (100, 4, 75), (128, 2, 512), (129, 2, 129), (200, 3, 300), (256, 2, 256), (257, 2, 64)])
def test_beam_search_at_the_edges_of_the_list_widths(chunks, top_l, width, top_n):
    s, host = _index(chunks)
    width = min(width, 256 // host["adjacency"].shape[1])
    q = s.queries.cuda().contiguous()
    rng = np.random.default_rng(top_l)
    entries = np.concatenate([[s.medoid], rng.choice(host["codes"].shape[0], 149, replace=False)])
    eo, ei = fixed_entries(q.shape[0], entries.tolist())
    p = search.TopologySearchParams(top_k=1, top_l=top_l, search_width=width, max_expansions=2048)
    cap = p.capacity(top_n)
    want, want_stats = None, None
    for layout in ("plain", "neighbor_codes"):
        ix = device_index(s)
        lut = search.lut_build(ix, q)
        if want is None:
            want, want_stats = orc.beam_search(host["adjacency"], host["codes"], lut.cpu().numpy(), np_u32(eo), np_u32(ei),
                                               top_l=top_l, search_width=width, max_expansions=2048, capacity=cap)
        if layout == "neighbor_codes":
            ix = search.inline_neighbor_codes(ix)
        cand, stats = search.beam_search(ix, p, eo, ei, queries=q, capacity=cap)
        assert_candidates_equal(cand, stats, want, want_stats)


# on both sides of the batch sizes from which the shared-memory list takes steps of up to 128 slots: one wave of the general form,
# per_sm blocks on an SM (0: at every size)
@pytest.mark.parametrize("chunks,top_l,width,top_n,learned,per_sm", [(32, 400, 2, 64, False, 4), (32, 300, 1, 512, True, 4), (32, 64, 2, 512, True, 4),
                                                                     (48, 64, 2, 64, True, 3), (48, 100, 1, 16, True, 3), (96, 100, 2, 300, False, 1),
                                                                     (96, 600, 1, 64, True, 1), (96, 64, 2, 64, True, 0), (96, 200, 2, 64, True, 0)])
def test_shared_memory_list_from_the_second_wave_on(chunks, top_l, width, top_n, learned, per_sm):
    s, _ = _index(chunks)
    ix = device_index(s)
    line = per_sm * torch.cuda.get_device_properties(0).multi_processor_count
    p = search.TopologySearchParams(top_k=10, top_l=top_l, search_width=width, max_expansions=1024,
                                    learned_stop=_learned_stop(top_l) if learned else None)
    cap = p.capacity(top_n)
    for batch in ((line, line + 1) if line else (33,)):
        q = s.queries.cuda().float().repeat(batch // s.queries.shape[0] + 1, 1)[:batch].contiguous()
        eo, ei = fixed_entries(batch, [s.medoid, 17, 400])
        want, want_stats = search.beam_search(_general_form(ix), p, eo, ei, queries=q, capacity=cap)
        for form in (ix, search.inline_neighbor_codes(dataclasses.replace(ix))):
            got, got_stats = search.beam_search(form, p, eo, ei, queries=q, capacity=cap)
            assert_candidates_equal(got, got_stats, np_u32(want), np_u32(want_stats))


def _shared_neighbours(chunks, degree, nodes=3000, window=160, seed=5):
    """A graph in which parents share many neighbours, so that one push brings copies of a node and later ones bring it again; the
    codes are random, so that the copies end up anywhere in the list."""
    rng = np.random.default_rng(seed)
    adjacency = np.stack([(i + rng.permutation(window)[:degree] - window // 2) % nodes for i in range(nodes)]).astype(np.uint32)
    adjacency[:, :4] = rng.integers(0, nodes, (nodes, 4))
    codes = rng.integers(0, 256, (nodes, chunks)).astype(np.uint8)
    ix = search.device_index_from_arrays(
        adjacency=adjacency, codes=codes, vectors=np.zeros((nodes, chunks), np.float32),
        pq_tables_row_major=rng.normal(size=(256, chunks)).astype(np.float32), pq_centroid=np.zeros(chunks, np.float32),
        pq_chunk_offsets=np.arange(chunks + 1, dtype=np.uint32))
    return ix, adjacency, codes, rng


# lists that end at top_l and lists that go on behind it, where copies of one node in different states (expanded or not) meet the
# end of the list; steps of up to 128 and of up to 256 slots, entries that repeat
@pytest.mark.parametrize("chunks,degree,window,batch", [(32, 32, 80, 3000), (48, 64, 160, 400), (96, 32, 80, 400), (32, 128, 200, 400),
                                                        (48, 96, 160, 300), (96, 128, 200, 300)])
@pytest.mark.parametrize("top_l,width,capacity", [(5, 2, 8), (5, 1, 32), (16, 2, 32), (32, 2, 32), (32, 1, 128), (32, 2, 128), (33, 2, 64),
                                                  (64, 2, 64), (64, 2, 256), (100, 2, 128), (128, 2, 256), (128, 2, 512), (200, 1, 256),
                                                  (256, 2, 256)])
def test_copies_of_a_node_across_the_end_of_the_list(chunks, degree, window, batch, top_l, width, capacity):
    ix, adjacency, codes, rng = _shared_neighbours(chunks, degree, window=window)
    q = torch.from_numpy(rng.normal(size=(batch, chunks)).astype(np.float32)).cuda()
    eo, ei = fixed_entries(batch, [3, 700, 700, 1500, 3])
    lut = search.lut_build(ix, q)
    want, want_stats = orc.beam_search(adjacency, codes, lut.cpu().numpy(), np_u32(eo), np_u32(ei), top_l=top_l, search_width=width,
                                       max_expansions=1024, capacity=capacity)
    p = search.TopologySearchParams(top_k=1, top_l=top_l, search_width=width, max_expansions=1024)
    for form in (ix, search.inline_neighbor_codes(dataclasses.replace(ix))):
        cand, stats = search.beam_search(form, p, eo, ei, lut=lut, capacity=capacity)
        assert_candidates_equal(cand, stats, want, want_stats)


@pytest.mark.parametrize("top_l", [16, 33, 100, 256])
@pytest.mark.parametrize("batch", [100, 700])
def test_pq2_refine_inside_the_searcher_matches_the_table_form(top_l, batch):
    """A searcher refines without tables, small batches by one block per query and larger ones with the pivots in shared memory;
    the separate entry point reads tables. The sums are the same operations in the same order: equal bits."""
    s, host = small_index(name="cfg3", num_nodes=12000, components=60, num_queries=128)
    ix = device_index(s)
    q = s.queries.cuda().repeat(6, 1)[:batch].contiguous()
    t2, c2 = s.pq2_tables.cuda().float().contiguous(), s.pq2_centroid.cuda().float().contiguous()
    cross = search.pq2_cross_terms(ix.pq_chunk_offsets, s.pq_tables.cuda().float().contiguous(), ix.pq_centroid, t2, c2)
    p2 = search.Pq2Resources(codes=s.pq2_codes.cuda().contiguous(), tables_col_major=t2.t().contiguous(), centroid=c2,
                             chunk_offsets=ix.pq_chunk_offsets, error_bounds=s.pq2_error_bounds.cuda().contiguous(),
                             cross_terms=cross)
    top_n = min(top_l, 64)
    tp = search.TopologySearchParams(top_k=10, top_l=top_l, search_width=2, max_expansions=2048)
    rp = search.RerankExactParams(top_k=10, top_n=top_n, rank_tile_size=16, use_pq2_bound_filter=True)
    eo, ei = fixed_entries(batch, [s.medoid])
    cand, stats = search.beam_search(ix, tp, eo, ei, queries=q, capacity=tp.capacity(top_n))
    lut2 = search.lut_build(ix, q, tables_col_major=p2.tables_col_major, centroid=c2)
    refined = search.pq2_refine(cand, stats, top_l, p2.codes, lut2, base_codes=ix.codes, cross_terms=cross)
    d, i, _, _ = search.rerank_exact(ix, rp, refined, q, p2.error_bounds)
    want_d, want_i = search.topk_pack(d, i, 10)
    sr = search.Searcher(ix, batch, tp.capacity(top_n), top_n, 1)
    sr.set_pq2(p2, top_l)
    got_i, got_d = sr.run_host(q.cpu().numpy(), tp, rp, np.array([s.medoid], np.uint32))[:2]
    sr.close()
    assert np.array_equal(got_i, np_u32(want_i))
    assert np.array_equal(got_d.view(np.uint32), np_u32(want_d))


def _general_form(ix):
    """The same index with the neighbour codes in two node-id-range shards: a layout that the general kernels take alone."""
    ix = search.inline_neighbor_codes(dataclasses.replace(ix))
    ix.rows_per_shard = (ix.num_nodes + 1) // 2
    base = ix.neighbor_codes.data_ptr()
    ix.neighbor_codes_bases = [base, base + ix.rows_per_shard * ix.degree * ix.num_chunks]
    return ix


def _learned_stop(top_l):
    ls = capi.LearnedStop()
    ls.enabled, ls.num_stages, ls.top_k, ls.inv_top_l = 1, 3, 10, 1.0 / top_l
    for i, p in enumerate((12, 16, 24)):
        ls.stage_prefixes[i] = p
    for i in range(12):
        ls.feature_mask[i], ls.weights[i] = 1, 1e-4 * (i - 5)
    ls.bias = 1.0
    return ls


# chunks of 1, 3, 4, 6 and 8 dims, and chunks of different widths (the last ones one dim wide)
@pytest.mark.parametrize("chunks,dim", [(32, 32), (32, 96), (32, 128), (32, 100), (48, 48), (48, 144), (48, 101), (96, 96), (96, 576),
                                        (96, 768), (96, 301)])
@pytest.mark.parametrize("top_l,width,capacity", [(64, 2, 64), (40, 4, 64)])
def test_table_built_in_the_kernel_gives_the_same_records_as_a_given_one(chunks, dim, top_l, width, capacity):
    """The sums are the same operations in the same order: equal bits. width 4 on a degree of 64: the shared-memory list."""
    degree = 64 if width == 4 else 32
    ix, _, _, rng = _shared_neighbours(chunks, degree)
    widths = np.full(chunks, dim // chunks)
    if dim % chunks:
        widths[:] = 1
        widths[:chunks // 2] += rng.multinomial(dim - chunks, np.full(chunks // 2, 2.0 / chunks))
    ix.dim = dim
    ix.pq_chunk_offsets = torch.from_numpy(np.concatenate([[0], np.cumsum(widths)]).astype(np.int32)).cuda()
    ix.pq_tables_col_major = torch.from_numpy(rng.normal(size=(dim, 256)).astype(np.float32)).cuda()
    ix.pq_centroid = torch.from_numpy(rng.normal(size=dim).astype(np.float32)).cuda()
    q = torch.from_numpy(rng.normal(size=(100, dim)).astype(np.float32)).cuda()
    eo, ei = fixed_entries(100, [3, 700])
    p = search.TopologySearchParams(top_k=1, top_l=top_l, search_width=width, max_expansions=512)
    want, want_stats = search.beam_search(ix, p, eo, ei, lut=search.lut_build(ix, q), capacity=capacity)
    got, got_stats = search.beam_search(ix, p, eo, ei, queries=q, capacity=capacity)
    assert_candidates_equal(got, got_stats, np_u32(want), np_u32(want_stats))
    general, general_stats = search.beam_search(_general_form(ix), p, eo, ei, queries=q, capacity=capacity)
    assert_candidates_equal(got, got_stats, np_u32(general), np_u32(general_stats))


# Distances that are NaN are not listed (no comparison with them holds), infinite ones are, by id. Where a list has them, the
# count of valid entries runs ahead of the list.
@pytest.mark.parametrize("chunks", [32, 48])
@pytest.mark.parametrize("top_l,width,top_n,learned", [(300, 2, 64, False), (400, 1, 1024, False), (64, 4, 64, False), (64, 2, 64, True),
                                                       (100, 2, 512, True), (200, 4, 256, True)])
def test_distances_that_are_not_finite_in_long_lists(chunks, top_l, width, top_n, learned):
    _not_finite(chunks, top_l, width, top_n, learned)


@pytest.mark.parametrize("chunks", [32, 48])
@pytest.mark.parametrize("top_l,width,top_n", [(32, 2, 16), (16, 2, 256), (64, 1, 64), (100, 2, 128), (100, 2, 512), (256, 2, 256)])
def test_distances_that_are_not_finite_in_short_lists(chunks, top_l, width, top_n):
    _not_finite(chunks, top_l, width, top_n, False)


def _not_finite(chunks, top_l, width, top_n, learned):
    s, _ = _index(chunks)
    ix = device_index(s)
    q = s.queries.cuda().float()[:12].clone()   # (the index is shared by other tests)
    lut = search.lut_build(ix, q)
    rng = np.random.default_rng(top_l)
    lut[1, 3] = float("nan")                    # every distance
    lut[2, 5, rng.permutation(256)[:128].tolist()] = float("nan")   # half of them
    lut[3, 7, ::3] = float("inf")
    lut[4] = 3e38                               # sums that overflow
    lut[5, 0, ::2], lut[5, 1, ::2] = float("nan"), float("inf")
    lut[6, :, 200:] = float("nan")
    lut[7, 9, :250] = float("nan")              # the list stays far shorter than the count of valid entries
    qn = q.clone()
    qn[1, 3], qn[2, 5], qn[3, 7], qn[4], qn[5, 0], qn[5, 1] = float("nan"), float("inf"), -float("inf"), 3e38, float("nan"), float("inf")
    eo, ei = fixed_entries(12, [s.medoid, 17, 400])
    p = search.TopologySearchParams(top_k=10, top_l=top_l, search_width=width, max_expansions=512,
                                    learned_stop=_learned_stop(top_l) if learned else None)
    cap = p.capacity(top_n)
    for entries in ((eo, ei), fixed_entries(12, [s.medoid]), fixed_entries(12, range(50, 201))):
        for kw in (dict(lut=lut), dict(queries=qn)):
            want, want_stats = search.beam_search(_general_form(ix), p, *entries, capacity=cap, **kw)
            for form in (ix, search.inline_neighbor_codes(dataclasses.replace(ix))):
                got, got_stats = search.beam_search(form, p, *entries, capacity=cap, **kw)
                assert_candidates_equal(got, got_stats, np_u32(want), np_u32(want_stats))
            w = np_u32(want)
            assert (w[1, :, 1] == 0xFFFFFFFF).all() and np_u32(want_stats)[1, 4] == min(cap, entries[1].numel() // 12)
            assert not np.isnan(w[:, :, 0].view(np.float32)).any()


# on both sides of the batch sizes from which the pivots lie in shared memory (5 queries per SM up to 48 chunks, 20 up to 64)
@pytest.mark.parametrize("chunks,dim,per_sm", [(16, 64, 5), (32, 64, 5), (48, 96, 5), (64, 128, 20), (96, 192, 20)])
@pytest.mark.parametrize("top_l", [16, 100])
def test_pq2_refine_at_the_lines_between_its_forms(chunks, dim, per_sm, top_l):
    ix, _, codes, rng = _shared_neighbours(chunks, 32)
    ix.dim = dim
    ix.pq_chunk_offsets = torch.arange(0, dim + 1, dim // chunks, dtype=torch.int32, device="cuda")
    normal = lambda *shape: torch.from_numpy(rng.normal(size=shape).astype(np.float32)).cuda()
    ix.pq_tables_col_major, ix.pq_centroid = normal(dim, 256), normal(dim)
    pages = search.device_index_from_arrays(adjacency=np.zeros((3000, 1), np.int32), codes=codes, vectors=rng.normal(size=(3000, dim)).astype(np.float32),
                                            pq_tables_row_major=np.zeros((256, dim), np.float32), pq_centroid=np.zeros(dim, np.float32),
                                            pq_chunk_offsets=np.arange(0, dim + 1, dim // chunks, dtype=np.uint32))
    ix.vector_pages, ix.vector_bytes, ix.vectors_per_page = pages.vector_pages, pages.vector_bytes, pages.vectors_per_page
    p2 = search.Pq2Resources(codes=torch.from_numpy(codes[::-1].copy()).cuda(), tables_col_major=normal(dim, 256), centroid=normal(dim),
                             chunk_offsets=ix.pq_chunk_offsets, error_bounds=normal(3000).abs(), cross_terms=normal(chunks, 256, 256))
    tp = search.TopologySearchParams(top_k=10, top_l=top_l, search_width=2, max_expansions=64)
    rp = search.RerankExactParams(top_k=10, top_n=16, rank_tile_size=16, use_pq2_bound_filter=True)
    line = per_sm * torch.cuda.get_device_properties(0).multi_processor_count
    for batch in (line - 1, line):
        q = normal(batch, dim)
        eo, ei = fixed_entries(batch, [7])
        cand, stats = search.beam_search(ix, tp, eo, ei, queries=q, capacity=tp.capacity(16))
        lut2 = search.lut_build(ix, q, tables_col_major=p2.tables_col_major, centroid=p2.centroid)
        refined = search.pq2_refine(cand, stats, top_l, p2.codes, lut2, base_codes=ix.codes, cross_terms=p2.cross_terms)
        d, i, _, _ = search.rerank_exact(ix, rp, refined, q, p2.error_bounds)
        want_d, want_i = search.topk_pack(d, i, 10)
        sr = search.Searcher(ix, batch, tp.capacity(16), 16, 1)
        sr.set_pq2(p2, top_l)
        got_i, got_d = sr.run_host(q.cpu().numpy(), tp, rp, np.array([7], np.uint32))[:2]
        sr.close()
        assert np.array_equal(got_i, np_u32(want_i))
        assert np.array_equal(got_d.view(np.uint32), np_u32(want_d))
