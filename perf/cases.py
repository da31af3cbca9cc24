"""The calls whose speed is watched, over the range of sizes that users bring.

Every case goes through the public Python API (reset_b200.api), as a user's
program would call it, on seeded synthetic inputs: R-MAT graphs, Zipf token
sets, a Zipf inverted index and uniform key sets, the shapes of bench.py's
workloads.  listed() are fixed cases; draw() gives others of the same ranges.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from reset_b200 import api


def listed():
    return [
        # Triangle counting: table build, rows in bucket order and count of a
        # graph that has just arrived.  A small graph (latency) ...
        {"name": "tc-s10", "kind": "tc", "scale": 10, "edge_factor": 16, "alpha": 0.2,
         "bucket": 5, "hier": True},
        # ... the plain single-graph workload, with the other hash ...
        {"name": "tc-s16", "kind": "tc", "scale": 16, "edge_factor": 16, "alpha": 0.2,
         "bucket": 5, "hier": False},
        # ... and the largest graph, with the parameters the autotuner picks for it.
        {"name": "tc-s24", "kind": "tc", "scale": 24, "edge_factor": 16, "alpha": 0.25,
         "bucket": 1, "hier": True},
        # Many small graphs at once: one build and one batched count.
        {"name": "tc-batch-96", "kind": "tc_batch", "graphs": 96, "scale_lo": 8, "scale_hi": 12,
         "edge_factor": 16, "alpha": 0.2, "bucket": 5, "hier": True},
        # Indexing a corpus: the table over an inverted index whose longest
        # lists hold hundreds of thousands of postings.
        {"name": "index-build", "kind": "build", "docs": 2_000_000, "terms": 100_000,
         "alpha": 0.2, "bucket": 5, "hier": False, "hash_order": True},
        # Similarity search, one query set against its candidates (latency).
        {"name": "sss-query", "kind": "sss", "sets": 100_000, "size_hi": 512, "pairs": 501,
         "one_query": True, "rule": "float", "inter": True, "hier": False},
        # A block of candidate pairs of uneven sizes, exact rule, sizes returned.
        {"name": "sss-pairs", "kind": "sss", "sets": 200_000, "size_hi": 1024, "pairs": 1_000_003,
         "one_query": False, "rule": "int", "inter": True, "hier": True},
        # The whole self-join over a resident index: prefix-filter candidates,
        # then every candidate decided by one batch replay.
        {"name": "sss-join", "kind": "join", "sets": 400_000, "size_hi": 1024},
        # Conjunctive retrieval over 20M documents, a block of queries per call.
        {"name": "ir-512", "kind": "ir", "docs": 20_000_000, "terms": 1_000_000,
         "queries": 512, "hier": True},
        # Two raw sets, small and large.
        {"name": "raw-1k", "kind": "raw", "na": 1_000, "nb": 1_500, "alpha": 0.2, "bucket": 5},
        # 5-cliques of an oriented graph (pattern Q5), table resident.
        {"name": "clique5-s16", "kind": "pattern", "pattern": "Q5", "scale": 16,
         "edge_factor": 16, "hier": True},
        # A general pattern with restrictions (Q6) on a symmetric graph.
        {"name": "pattern-q6-s11", "kind": "pattern", "pattern": "Q6", "scale": 11,
         "edge_factor": 16, "hier": True},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


_PARAMS = [(0.2, 5), (0.25, 1), (0.4, 2), (0.5, 4), (0.1, 9), (0.2, 1), (0.3, 5)]


def draw(rng):
    kind = rng.choice(["tc", "tc", "tc_batch", "build", "sss", "sss", "join", "ir", "raw", "raw",
                       "pattern", "pattern"])
    alpha, bucket = rng.choice(_PARAMS)
    hier = rng.random() < 0.5
    if kind == "tc":
        return {"kind": kind, "scale": rng.randint(8, 22), "edge_factor": rng.randint(4, 24),
                "alpha": alpha, "bucket": bucket, "hier": hier}
    if kind == "tc_batch":
        lo = rng.randint(7, 10)
        return {"kind": kind, "graphs": _log(rng, 5, 120), "scale_lo": lo,
                "scale_hi": lo + rng.randint(0, 2), "edge_factor": rng.randint(4, 20),
                "alpha": alpha, "bucket": bucket, "hier": hier}
    if kind == "build":
        return {"kind": kind, "docs": _log(rng, 10_000, 5_000_000),
                "terms": _log(rng, 1_000, 300_000), "alpha": alpha, "bucket": bucket,
                "hier": hier, "hash_order": rng.random() < 0.5}
    if kind == "sss":
        return {"kind": kind, "sets": _log(rng, 2_000, 300_000),
                "size_hi": rng.choice([64, 300, 1024]), "pairs": _log(rng, 33, 2_000_000),
                "one_query": rng.random() < 0.3, "rule": rng.choice(["int", "float"]),
                "inter": rng.random() < 0.6, "hier": hier}
    if kind == "join":
        return {"kind": kind, "sets": _log(rng, 3_000, 400_000),
                "size_hi": rng.choice([64, 300, 1024])}
    if kind == "ir":
        docs = _log(rng, 100_000, 20_000_000)
        return {"kind": kind, "docs": docs, "terms": max(1000, docs // rng.randint(15, 40)),
                "queries": _log(rng, 1, 512), "hier": hier}
    if kind == "raw":
        return {"kind": kind, "na": _log(rng, 16, 1 << 20), "nb": _log(rng, 16, 1 << 20),
                "alpha": alpha, "bucket": bucket}
    q = rng.choice(["Q0", "Q1", "Q2", "Q3", "Q4", "Q5", "Q6", "Q7", "Q8"])
    top = {"Q6": 11, "Q4": 13, "Q8": 13, "Q1": 14, "Q2": 14, "Q7": 15}.get(q, 16)
    return {"kind": "pattern", "pattern": q, "scale": rng.randint(7, top),
            "edge_factor": rng.randint(4, 16), "hier": hier}


def _np_rng(seed):
    return np.random.default_rng(0x5EED0000 + seed)


def _queries(df, nq, rng):
    """Queries of 2-6 terms drawn by document frequency, rarest term first."""
    p = df / df.sum()
    ks = rng.integers(2, 7, nq)
    draws = rng.choice(df.size, size=int(ks.sum()), p=p)
    out, i = [], 0
    for k in ks:
        ts = np.unique(draws[i:i + k])
        i += k
        out.append(ts[np.lexsort((ts, df[ts]))].astype(np.int32))
    return out


def _key_set(n, universe, gen):
    """n distinct keys of [0, universe), ascending."""
    got = torch.randperm(universe, generator=gen, device="cuda", dtype=torch.int64)[:n]
    return got.sort().values.to(torch.int32)


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _graph(case, seed):
    """The seed's oriented R-MAT graph, cut to as many edges for every seed:
    the last rows lose the few above six deviations below the mean."""
    off, cols = api.gen_rmat(case["scale"], case["edge_factor"], 0x5EED0000 + seed)
    mean = _rmat_edges(case["scale"], case["edge_factor"])
    m = int(mean - 6 * math.sqrt(mean))
    if cols.numel() < m:
        raise RuntimeError(f"seed {seed} drew only {cols.numel()} edges")
    return off.clamp(max=m), cols[:m].clone()


def _token_sets(case, seed):
    """Token sets of one collection, in an order of the seed's: every seed has
    as many candidate pairs."""
    off, tok = api.gen_token_sets(case["sets"], 24, 1.2, 8, case["size_hi"], dup_frac=0.2,
                                  keep_min=0.75)
    perm = torch.randperm(case["sets"], generator=_gen(seed), device="cuda")
    size = (off[1:] - off[:-1]).long()[perm]
    new = torch.zeros(case["sets"] + 1, dtype=torch.int64, device="cuda")
    new[1:] = torch.cumsum(size, 0)
    shift = torch.repeat_interleave(off[:-1].long()[perm] - new[:-1], size)
    return new.int(), tok[torch.arange(tok.numel(), device="cuda") + shift]


def _ir_index(case, seed):
    """An inverted index with the seed's document numbers: every seed has the
    same document frequencies."""
    toff, docs = api.gen_inverted_index(case["terms"], case["docs"], 1.1, case["docs"] // 2)
    perm = torch.randperm(case["docs"], generator=_gen(seed), device="cuda")
    df = (toff[1:] - toff[:-1]).long()
    key = torch.repeat_interleave(torch.arange(df.numel(), device="cuda") << 32, df)
    key += perm[docs]
    return toff, (key.sort().values & 0xFFFFFFFF).int()


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case)
    if kind == "tc":
        s["off"], s["cols"] = _graph(case, seed)
    elif kind == "tc_batch":
        rng = _np_rng(seed)
        offs, cols, starts, nv, ne = [], [], [0], 0, 0
        for _ in range(case["graphs"]):
            scale = int(rng.integers(case["scale_lo"], case["scale_hi"] + 1))
            o, c = api.gen_rmat(scale, case["edge_factor"], int(rng.integers(1 << 40)))
            offs.append(o[:-1] + ne)
            cols.append(c + nv)
            nv += o.numel() - 1
            ne += c.numel()
            starts.append(nv)
        offs.append(torch.tensor([ne], dtype=torch.int32, device="cuda"))
        s["off"], s["cols"] = torch.cat(offs), torch.cat(cols)
        s["graph_off"] = torch.tensor(starts, dtype=torch.int32, device="cuda")
    elif kind == "build":
        s["off"], s["elems"] = _ir_index(case, seed)
        s["table"] = None
    elif kind == "sss":
        n, P = case["sets"], case["pairs"]
        s["off"], s["tok"] = api.gen_token_sets(n, 24, 1.2, 8, case["size_hi"],
                                                seed=0x5EED0033 + seed, dup_frac=0.2,
                                                keep_min=0.75)
        s["table"] = api.Table(s["off"], s["tok"], hierarchical=case["hier"])
        kw = {"generator": _gen(seed), "device": "cuda", "dtype": torch.int32}
        s["pb"] = torch.randint(0, n, (P,), **kw)
        if case["one_query"]:
            s["pa"] = torch.randint(0, n, (1,), **kw).expand(P).contiguous()
        else:  # near-duplicates of a set lie within 256 places of it
            s["pa"] = torch.clamp(s["pb"] + torch.randint(1, 257, (P,), **kw), max=n - 1)
    elif kind == "join":
        s["off"], s["tok"] = _token_sets(case, seed)
        s["table"] = api.Table(s["off"], s["tok"], alpha=0.2, bucket=1)
        pa, _ = api.prefix_candidates(s["off"], s["tok"], 24)
        s["batch"] = api.Batch(s["table"], s["tok"], capacity=max(1, pa.numel()),
                               decisions_only=True)
    elif kind == "ir":
        s["toff"], s["docs"] = _ir_index(case, seed)
        s["table"] = api.Table(s["toff"], s["docs"], hierarchical=case["hier"])
        df = np.diff(s["toff"].cpu().numpy()).astype(np.int64)
        qs = _queries(df, case["queries"], _np_rng(0))
        qoff = np.zeros(len(qs) + 1, np.int32)
        qoff[1:] = np.cumsum([q.size for q in qs])
        s["query"] = torch.from_numpy(np.concatenate(qs)).cuda()
        s["qoff"] = torch.from_numpy(qoff).cuda()
    elif kind == "raw":
        g = _gen(seed)
        universe = 3 * max(case["na"], case["nb"])
        s["a"] = _key_set(case["na"], universe, g)
        s["b"] = _key_set(case["nb"], universe, g)
    elif kind == "pattern":
        oriented = api.PATTERNS[case["pattern"]].graph == "oriented"
        s["off"], s["cols"] = api.gen_rmat(case["scale"], case["edge_factor"], 0x5EED0000 + seed,
                                           oriented=oriented)
        s["table"] = api.Table(s["off"], s["cols"], hierarchical=case["hier"])
    else:
        raise ValueError(f"unknown kind {kind}")
    return s


def run(s):
    kind = s["kind"]
    if kind == "tc":
        t = api.Table(s["off"], s["cols"], alpha=s["alpha"], bucket=s["bucket"],
                      hierarchical=s["hier"], hash_order=True)
        count = api.tc_count_async(t, s["off"], t.hash_order)
        t.free_async()
        return {"count": count, "rows": t.hash_order}
    if kind == "tc_batch":
        t = api.Table(s["off"], s["cols"], alpha=s["alpha"], bucket=s["bucket"],
                      hierarchical=s["hier"])
        counts = api.tc_count_batch(t, s["off"], s["cols"], s["graph_off"])
        t.free_async()
        return counts
    if kind == "build":
        if s["table"] is not None:
            s["table"].free_async()
        t = s["table"] = api.Table(s["off"], s["elems"], alpha=s["alpha"], bucket=s["bucket"],
                                   hierarchical=s["hier"], hash_order=s["hash_order"])
        slots, length, offsets = t.tensors()
        for view in (slots, length, offsets):
            view.table = t  # the views are valid while the table lives
        return {"slots": slots, "len": length, "off": offsets, "rows": t.hash_order}
    if kind == "sss":
        if s["rule"] == "float":
            flags, inter = api.sss_float(s["table"], s["off"], s["tok"], s["pa"], s["pb"], 0.7,
                                         with_inter=s["inter"])
        else:
            flags, inter = api.sss(s["table"], s["off"], s["tok"], s["pa"], s["pb"],
                                   with_inter=s["inter"])
        return {"flags": flags, "inter": inter}
    if kind == "join":
        pa, pb = api.prefix_candidates(s["off"], s["tok"], 24)
        flags, _ = s["batch"](pa, pb)
        flags.batch = s["batch"]  # the flags are the batch's own buffer
        return {"pa": pa, "pb": pb, "flags": flags}
    if kind == "ir":
        roff, res, cnt = api.ir(s["table"], s["toff"], s["docs"], s["query"], s["qoff"])
        return {"off": roff, "docs": res, "count": cnt}
    if kind == "raw":
        return api.intersect_count(s["a"], s["b"], alpha=s["alpha"], bucket=s["bucket"])
    return api.pattern_count(s["table"], s["off"], s["cols"], s["pattern"])


# ---- what a pass cannot do without: inputs read once, outputs written once --

def _rmat_edges(scale, edge_factor):
    """Expected undirected edges of the R-MAT law after self-loops and
    duplicates are removed (a, b, c, d = 0.57, 0.19, 0.19, 0.05)."""
    a, b, d = 0.57, 0.19, 0.05
    e = edge_factor << scale
    tot = 0.0
    for j in range(1, scale + 1):  # levels in quadrant b or c
        for i in range(scale - j + 1):
            cells = math.comb(scale, j) * math.comb(scale - j, i) * 2.0 ** (j - 1)
            p = 2 * a ** i * b ** j * d ** (scale - j - i)
            tot += cells * -math.expm1(e * math.log1p(-p))
    return tot


def _df(case):
    df = np.round(case["docs"] // 2 * np.arange(1, case["terms"] + 1, dtype=np.float64) ** -1.1)
    # draws that repeat a document are dropped
    return case["docs"] * -np.expm1(-np.clip(df, 1, case["docs"]) / case["docs"])


def _mean_size(size_hi):
    k = np.arange(8, size_hi + 1, dtype=np.float64)
    return float((k * k ** -1.2).sum() / (k ** -1.2).sum())


def work(case):
    kind = case["kind"]
    if kind == "tc":  # CSR in; rows in bucket order and the count out
        m = _rmat_edges(case["scale"], case["edge_factor"])
        return {"bytes": 4 * ((1 << case["scale"]) + 1) + 8 * m + 8, "flops": 0}
    if kind == "tc_batch":
        sc = range(case["scale_lo"], case["scale_hi"] + 1)
        m = sum(_rmat_edges(x, case["edge_factor"]) for x in sc) / len(sc) * case["graphs"]
        n = sum(1 << x for x in sc) / len(sc) * case["graphs"]
        return {"bytes": 4 * n + 4 * m + 8 * case["graphs"], "flops": 0}
    if kind == "build":  # postings in; table, lengths, offsets (and rows) out
        df = _df(case)
        q = np.maximum(1, df / case["alpha"] // case["bucket"])
        length = np.maximum(8, 2 ** (np.floor(np.log2(q)) + 1))
        per = 8 if case["hash_order"] else 4
        return {"bytes": per * df.sum() + 4 * case["bucket"] * length.sum() + 16 * case["terms"],
                "flops": 0}
    if kind == "sss":  # the pairs, each set named by one (at most all), the results
        named = min(case["sets"], case["pairs"] * (1 if case["one_query"] else 2))
        out = 5 if case["inter"] else 1
        return {"bytes": 4 * named * _mean_size(case["size_hi"]) + case["pairs"] * (8 + out),
                "flops": 0}
    if kind == "join":  # token sets in; the candidates (measured share of n^2) and flags out
        n = case["sets"]
        share = 3.4e-5 if case["size_hi"] > 500 else 2e-5 if case["size_hi"] > 100 else 5e-6
        return {"bytes": 4 * n * _mean_size(case["size_hi"]) + 9 * share * n * n, "flops": 0}
    if kind == "ir":  # the rarest term's list of every query in, a result region of its size out
        df = _df(case)
        first = sum(df[q[0]] for q in _queries(df, 512, _np_rng(0))) / 512
        return {"bytes": 8 * first * case["queries"] + 40 * case["queries"], "flops": 0}
    if kind == "raw":
        return {"bytes": 4 * (case["na"] + case["nb"]) + 8, "flops": 0}
    oriented = api.PATTERNS[case["pattern"]].graph == "oriented"
    m = _rmat_edges(case["scale"], case["edge_factor"]) * (1 if oriented else 2)
    return {"bytes": 4 * ((1 << case["scale"]) + 1) + 4 * m + 8, "flops": 0}


def exact(case, seed):
    """The results that plain torch gives quickly (all are whole numbers)."""
    kind = case["kind"]
    if kind == "raw":
        s = prepare(case, seed)
        return int(torch.isin(s["a"], s["b"]).sum().item())
    if kind == "sss" and case["pairs"] <= 100_000:
        s = prepare(case, seed)
        off, size = s["off"].long(), (s["off"][1:] - s["off"][:-1]).long()
        a, b = s["pa"].long(), s["pb"].long()
        own = torch.repeat_interleave(torch.arange(size.numel(), device="cuda"), size)
        members = own * (1 << 24) + s["tok"].long()  # ascending: sets in order, rows sorted
        p = torch.repeat_interleave(torch.arange(a.numel(), device="cuda"), size[a])
        first = torch.cumsum(size[a], 0) - size[a]
        j = torch.arange(p.numel(), device="cuda") - first[p]
        want = b[p] * (1 << 24) + s["tok"].long()[off[a][p] + j]
        at = torch.searchsorted(members, want).clamp(max=members.numel() - 1)
        inter = torch.zeros_like(a).index_add_(0, p, (members[at] == want).long())
        union = size[a] + size[b] - inter
        if case["rule"] == "int":
            flags = 10 * inter >= 7 * union
        else:  # the reference compares in 32 bits
            flags = inter.float() / union.float() >= np.float32(0.7)
        return {"flags": flags.to(torch.uint8),
                "inter": inter.to(torch.int32) if case["inter"] else None}
    return None
