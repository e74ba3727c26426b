"""The batched graph search as its users call it, over the range of sizes and options it serves.

Four indexes with the shapes of the benchmark configurations: 10 M x 128 uint8 (degree 64, PQ 32, RVQ entries), 100 k x 128
uint8 (degree 32, PQ 32, medoid entry), 4 M x 96 float32 (degree 64, PQ 48 + residual pq2, RVQ entries) and 1 M x 768 float32
(degree 64, PQ 96, RVQ entries). An index is what a serving process loads once and keeps: it is generated from its own fixed
seed and kept for the life of the process. The queries - what changes from call to call - come from the case's seed, drawn
from the same mixture as the index.

Four ways in: `host` (one blocking call, host buffers in and out), `pipelined` (four searchers submitted in turn, then waited
for), `device` (queries and results stay on the GPU) and `staged` (the separate entry points, every intermediate returned).
"""
from __future__ import annotations

import dataclasses
import math

import numpy as np
import torch

from topoanns_b200 import capi, search, synth

TOP_K = 10
LANES = 4          # searchers of the pipelined way in
MAX_BATCH = 10_000

# name -> (configuration, what differs from its stated size)
INDEXES = {
    "u8": ("cfg2", dict()),
    "u8_small": ("cfg1", dict()),
    "f96": ("cfg3", dict(num_nodes=4_000_000, components=4_000)),
    "f768": ("cfg5", dict(num_nodes=1_000_000, components=1_000)),
}
FLOATS = ("f96", "f768")


def _case(name, index, way, batch, top_l, top_n, *, width=2, queries="float32", entries=128, neighbor_codes=False, pq2=False,
          tile=0, stop="none", traversal_stop=False, pinned=False):
    """queries: the dtype the caller holds; entries: RVQ entries per query, 0 = the medoid; pq2: residual refine and bound
    filter; stop: rerank stop ("none", "early", "learned"); pinned: page-locked host buffers."""
    c = dict(index=index, way=way, batch=batch, top_l=top_l, top_n=top_n, width=width, queries=queries, entries=entries,
             neighbor_codes=neighbor_codes, pq2=pq2, tile=tile, stop=stop, traversal_stop=traversal_stop, pinned=pinned)
    return dict(c, name=name) if name else c


def listed():
    return [
        # one user's query at a time: latency
        _case("one_query", "u8", "host", 1, 64, 32, neighbor_codes=True),
        # a short, odd batch of uint8 queries, odd list sizes, the memory-lean layout
        _case("odd_batch_u8_queries", "u8", "host", 37, 100, 75, queries="uint8"),
        # the small configuration as stated: 1 k queries, medoid entry, L = 64, rerank_top_n = 32
        _case("small_index_medoid", "u8_small", "host", 1000, 64, 32, queries="uint8", entries=0, pinned=True),
        # the benchmark's operating point, one blocking call on page-locked buffers
        _case("batch_10k", "u8", "host", 10_000, 16, 192, neighbor_codes=True, pinned=True),
        # the same point as a serving process runs it: several searchers in flight
        _case("serving_4x10k", "u8", "pipelined", 10_000, 16, 192, neighbor_codes=True, pinned=True),
        # queries and results on the device, without the neighbour-code layout
        _case("device_10k", "u8", "device", 10_000, 64, 32),
        # the long end of the list-size sweep
        _case("deep_list", "u8", "host", 2000, 512, 32, neighbor_codes=True, pinned=True),
        # search width 4 (256 frontier slots per step), with the learned stop of the traversal
        _case("wide_frontier", "u8", "device", 1003, 200, 128, width=4, traversal_stop=True),
        # float vectors: residual refine, bound filter, short rerank tiles
        _case("float_pq2", "f96", "host", 10_000, 64, 64, pq2=True, tile=16, pinned=True),
        # the deep float point with the learned rerank stop
        _case("float_deep_learned_stop", "f96", "device", 10_000, 256, 256, pq2=True, tile=16, stop="learned"),
        # every stage by its own entry point, tables built beforehand
        _case("staged_float", "f96", "staged", 500, 64, 64, pq2=True, tile=32),
        # wide embeddings
        _case("wide_vectors", "f768", "host", 3000, 128, 64),
    ]


def _expanded(c):
    return c["top_l"] + 2.0


def _visited(c):
    _, cfg = _config(c["index"])
    return max(c["entries"], 1) + 0.65 * cfg.degree * _expanded(c)


def _passes(c):
    return c["batch"] * (LANES if c["way"] == "pipelined" else 1)


def _cost(c):
    """A rough figure of a case's time, to keep drawn cases below the largest listed one."""
    _, cfg = _config(c["index"])
    vb = cfg.dim * (1 if cfg.kind == "uint8" else 4)
    refine = c["top_l"] * cfg.pq_chunks * 2 if c["pq2"] else 0
    wide = 4.0 if c["width"] * cfg.degree > 128 else 1.0   # steps of more than 128 slots
    return _passes(c) * (wide * _visited(c) * cfg.pq_chunks + 64.0 * cfg.dim + 0.5 * c["top_n"] * vb + refine)


def draw(rng):
    def log_int(lo, hi):
        return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))

    index = rng.choice(["u8", "u8", "u8_small", "f96", "f96", "f768"])
    way = rng.choice(["host", "host", "pipelined", "device", "device", "staged"])
    batch = log_int(1, MAX_BATCH if way != "staged" else 1000)
    top_l = log_int(16, 512)
    top_n = log_int(16, 512)
    width = rng.choice([1, 2, 2, 2, 4])
    entries = 0 if index == "u8_small" else rng.choice([32, 128, 128, 100])
    pq2 = index == "f96" and (way == "staged" or rng.random() < 0.6)
    if pq2:
        top_n = min(top_n, top_l)   # the refined list holds top_l entries
    c = _case("", index, way, batch, top_l, top_n, width=width,
              queries="uint8" if index in ("u8", "u8_small") and way != "staged" and rng.random() < 0.4 else "float32",
              entries=entries, neighbor_codes=index == "u8" and rng.random() < 0.6, pq2=pq2,
              tile=rng.choice([16, 32, 64]) if pq2 else 0,
              stop=rng.choice(["none", "learned", "early"]) if pq2 and way != "staged" and top_n >= 48 else "none",
              traversal_stop=way != "staged" and rng.random() < 0.15, pinned=rng.random() < 0.5)
    most = 0.8 * max(_cost(x) for x in listed())
    if _cost(c) > most:
        c["batch"] = max(1, int(c["batch"] * most / _cost(c)))
    return c


# ---- what a program keeps: the index and its models ------------------------------------------------------------------------

_kept = {}


def _config(name):
    base, kw = INDEXES[name]
    # one query of the generator's own: the cases draw theirs with more_queries()
    cfg = dataclasses.replace(synth.CONFIGS[base], num_queries=1, **kw)
    return base, cfg


def _index(name):
    """The index, its RVQ model and its pq2 data on the GPU, with and without the neighbour-code layout."""
    if name in _kept:
        return _kept[name]
    _, cfg = _config(name)
    was = torch.are_deterministic_algorithms_enabled(), torch.is_deterministic_algorithms_warn_only_enabled()
    torch.use_deterministic_algorithms(True, warn_only=True)   # the same index in every process
    try:
        s = synth.build(cfg, "cuda")
    finally:
        torch.use_deterministic_algorithms(was[0], warn_only=was[1])
    ix = search.device_index_from_synth(s)
    k = dict(cfg=cfg, plain=ix, medoid=s.medoid, centres=s.extras["centres"], basis=s.extras["basis"],
             rvq=search.rvq_model_from_synth(s) if cfg.rvq else None)
    if name == "u8":
        k["nbr"] = search.inline_neighbor_codes(dataclasses.replace(ix))
    if s.pq2_tables is not None:
        t1, t2 = s.pq_tables.float().contiguous(), s.pq2_tables.float().contiguous()
        c2 = s.pq2_centroid.float().contiguous()
        k["pq2"] = search.Pq2Resources(
            codes=s.pq2_codes.contiguous(), tables_col_major=t2.t().contiguous(), centroid=c2,
            chunk_offsets=ix.pq_chunk_offsets, error_bounds=s.pq2_error_bounds.contiguous(),
            cross_terms=search.pq2_cross_terms(ix.pq_chunk_offsets, t1, ix.pq_centroid, t2, c2))
    del s
    torch.cuda.empty_cache()
    _kept[name] = k
    return k


def _traversal_stop(top_l):
    """A synthetic model: stop once the prefix that has been expanded outweighs the distance spread of the list."""
    ls = capi.LearnedStop()
    stages = [p for p in (16, 24, 32, 48, 64, 96, 128, 192, 256, 384) if TOP_K <= p < top_l]
    ls.enabled, ls.num_stages, ls.top_k = int(bool(stages)), len(stages), TOP_K
    ls.topk_churn_flag_mode, ls.next64_flag_mode = 1, 0
    for i, p in enumerate(stages):
        ls.stage_prefixes[i] = p
    for i in range(12):
        ls.feature_mask[i] = 1
    # share of the list expanded, unexpanded share of the next 64 ranks, change of the top-k since the last stage
    ls.weights[1], ls.weights[4], ls.weights[11] = -2.0, 0.5, 1.0
    ls.bias, ls.threshold_logit, ls.inv_top_l = 1.0, 0.0, 1.0 / top_l
    return ls


def _rerank_stop(budget):
    """A synthetic model on the share of the budget scored and the top-k churn."""
    ls = capi.RerankLearnedStop()
    stages = [p for p in (16, 32, 48, 64, 96, 128, 192, 256, 384, 512) if p < budget]
    ls.enabled, ls.num_stages, ls.top_k, ls.bootstrap_prefix = 1, len(stages), TOP_K, 16
    for i, p in enumerate(stages):
        ls.stage_prefixes[i] = p
    while ls.initial_stage_index < ls.num_stages and ls.stage_prefixes[ls.initial_stage_index] <= 16:
        ls.initial_stage_index += 1
    ls.linear_weights[1], ls.linear_weights[6], ls.bias, ls.threshold_logit = -2.5, 1.0, 1.0, 0.0
    ls.inv_budget_top_n, ls.inv_top_k = 1.0 / budget, 1.0 / TOP_K
    return ls


class _DeviceArray:
    """A searcher's result buffer as a torch-readable array; the buffer lives as long as its searcher, which is kept."""

    def __init__(self, owner, ptr, shape, kind):
        self.owner = owner
        self.__cuda_array_interface__ = dict(data=(int(ptr), False), shape=shape, typestr=kind, version=3)


def _host_array(shape, dtype, pinned):
    if not pinned:
        return np.empty(shape, dtype)
    t = torch.empty(int(np.prod(shape)) * np.dtype(dtype).itemsize, dtype=torch.uint8).pin_memory()
    return t.numpy().view(dtype).reshape(shape)


def prepare(case, seed):
    k = _index(case["index"])
    cfg, batch = k["cfg"], case["batch"]
    lanes = LANES if case["way"] == "pipelined" else 1
    q = synth.more_queries(cfg, k["centres"], batch * lanes, seed, k["basis"])
    q = q.to(torch.uint8 if case["queries"] == "uint8" else torch.float32).view(lanes, batch, cfg.dim).contiguous()
    tp = search.TopologySearchParams(top_k=TOP_K, top_l=case["top_l"], search_width=case["width"], max_expansions=4096,
                                     learned_stop=_traversal_stop(case["top_l"]) if case["traversal_stop"] else None)
    rp = search.RerankExactParams(top_k=TOP_K, top_n=case["top_n"], rank_tile_size=case["tile"],
                                  use_pq2_bound_filter=case["pq2"], use_early_stop=case["stop"] == "early")
    ix = k["nbr"] if case["neighbor_codes"] else k["plain"]
    st = dict(case=case, k=k, ix=ix, tp=tp, rp=rp)
    if case["way"] == "staged":
        st["q"] = q[0]
        if not case["entries"]:
            st["offsets"] = torch.arange(batch + 1, dtype=torch.int32, device="cuda")
            st["ids"] = torch.full((batch,), k["medoid"], dtype=torch.int32, device="cuda")
        return st
    st["searchers"] = []
    for _ in range(lanes):
        sr = search.Searcher(ix, batch, tp.capacity(rp.top_n), rp.top_n, max(case["entries"], 1))
        if case["entries"]:
            sr.set_rvq(k["rvq"], case["entries"])
        if case["pq2"]:
            sr.set_pq2(k["pq2"], case["top_l"])
        if case["stop"] == "learned":
            sr.set_rerank_learned_stop(_rerank_stop(rp.top_n))
        st["searchers"].append(sr)
    if case["way"] == "device":
        st["q"] = q[0]
        if not case["entries"]:
            st["offsets"] = torch.arange(batch + 1, dtype=torch.int32, device="cuda")
            st["ids"] = torch.full((batch,), k["medoid"], dtype=torch.int32, device="cuda")
        return st
    host = q.cpu().numpy()
    st["fixed"] = None if case["entries"] else np.array([k["medoid"]], np.uint32)
    st["q"], st["out_ids"], st["out_dists"] = [], [], []
    for i in range(lanes):
        a = _host_array(host[i].shape, host.dtype, case["pinned"])
        a[...] = host[i]
        st["q"].append(a)
        st["out_ids"].append(_host_array((batch, TOP_K), np.uint32, case["pinned"]))
        st["out_dists"].append(_host_array((batch, TOP_K), np.float32, case["pinned"]))
    if lanes > 1:
        st["streams"] = [torch.cuda.Stream() for _ in range(lanes)]
        if st["fixed"] is not None:
            # submit_host takes its entries from an RVQ model; without one the blocking calls are made in turn
            st["streams"] = None
    torch.cuda.synchronize()
    return st


def run(st):
    case, tp, rp = st["case"], st["tp"], st["rp"]
    if case["way"] == "staged":
        return _run_staged(st)
    if case["way"] == "device":
        sr = st["searchers"][0]
        ids, dists, stats = sr.run_device(st["q"], tp, rp, st.get("offsets"), st.get("ids"))
        n = case["batch"]
        return [torch.as_tensor(_DeviceArray(sr, ids, (n, TOP_K), "<i4"), device="cuda"),
                torch.as_tensor(_DeviceArray(sr, dists, (n, TOP_K), "<f4"), device="cuda"),
                torch.as_tensor(_DeviceArray(sr, stats, (n, 8), "<i4"), device="cuda")]
    if case["way"] == "pipelined" and st["streams"] is not None:
        for i, sr in enumerate(st["searchers"]):
            sr.submit_host(st["q"][i], tp, rp, st["out_ids"][i], st["out_dists"][i], stream=st["streams"][i])
        for sr in st["searchers"]:
            sr.wait()
        return st["out_ids"] + st["out_dists"]
    out = []
    for i, sr in enumerate(st["searchers"]):
        if case["pinned"]:   # a program that keeps page-locked buffers for its results
            out += sr.run_host(st["q"][i], tp, rp, st["fixed"], out_ids=st["out_ids"][i], out_dists=st["out_dists"][i])[:2]
        else:                # a program that takes the arrays the call makes
            out += [x for x in sr.run_host(st["q"][i], tp, rp, st["fixed"], want_stats=True)]
    return out


def _run_staged(st):
    case, k, ix, tp, rp, q = st["case"], st["k"], st["ix"], st["tp"], st["rp"], st["q"]
    out = []
    if case["entries"]:
        offsets, ids, clusters = k["rvq"].device_entry_batch(q, case["entries"])
        out += [ids, clusters]
    else:
        offsets, ids = st["offsets"], st["ids"]
    lut = search.lut_build(ix, q)
    cand, stats = search.beam_search(ix, tp, offsets, ids, lut=lut, capacity=tp.capacity(rp.top_n))
    out += [lut, stats]
    bounds = None
    if case["pq2"]:
        p2 = k["pq2"]
        lut2 = search.lut_build(ix, q, tables_col_major=p2.tables_col_major, centroid=p2.centroid)
        cand = search.pq2_refine(cand, stats, case["top_l"], p2.codes, lut2, base_codes=ix.codes, cross_terms=p2.cross_terms)
        bounds = p2.error_bounds
    dists, found, n_exact, n_filtered = search.rerank_exact(ix, rp, cand, q, bounds)
    top_d, top_i = search.topk_pack(dists, found, TOP_K)
    return out + [cand[..., 1].contiguous(), cand[..., 0].contiguous().view(torch.float32), top_d, top_i, n_exact, n_filtered]


def work(case):
    """Bytes: the adjacency row of every expanded node, the code row of every node that passes the visited filter, the vectors
    of the reranked ranks, the queries and the results; rows that a batch is bound to share (a small index) count once.
    Expanded and visited nodes per query are taken from the list size: top_l + 2, and 0.65 of the slots they open."""
    _, cfg = _config(case["index"])
    n, m, d = cfg.num_nodes, cfg.pq_chunks, cfg.dim
    q = _passes(case)
    vb = d * (1 if cfg.kind == "uint8" else 4)
    qb = d * (1 if case["queries"] == "uint8" else 4)
    e, v = _expanded(case), _visited(case)
    scored = case["top_n"] * (0.5 if case["pq2"] else 1.0)   # the bound filter passes about half
    rows = min(q * e, n) * 4.0 * cfg.degree + min(q * v, n * (1.0 if not case["neighbor_codes"] else cfg.degree)) * m
    vectors = min(q * scored, n) * vb
    extra = q * (qb + case["entries"] * 4.0 + TOP_K * 8.0 + 32.0)
    flops = q * (v * m + 3.0 * 256 * d + 3.0 * d * scored)
    if case["entries"]:
        flops += q * 2.0 * 512 * d
        extra += 2.0 * 256 * d * 4
    if case["pq2"]:
        rows += min(q * case["top_l"], n) * 2.0 * m
        extra += m * 65536.0 * 4
        flops += q * case["top_l"] * m * 3.0
    if case["way"] == "staged":   # the tables and lists are results here
        extra += q * (m * 1024.0 + case["top_l"] * 8.0 + case["top_n"] * 8.0) * (2 if case["pq2"] else 1)
    return {"bytes": rows + vectors + extra, "flops": flops}


def tolerance(case):
    """uint8 vectors: distances are integers and the order is decided by them, so ids and distances are exact. Float vectors:
    32-bit sums; two candidates whose distances differ in the last bits may change places."""
    return {"rel": 1e-5, "differ": 1e-3} if case["index"] in FLOATS else "exact"
