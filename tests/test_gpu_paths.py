"""Kernel paths at the sizes where they change: edges of tiles, packed words
and work bins, remainders, and inputs that must take the general path.
Whole-number results, compared exactly."""
from math import comb

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def R(cuda, libreset):
    from reset_b200 import api
    return api


def dev(x, torch):
    return torch.from_numpy(np.ascontiguousarray(x)).cuda()


def csr(rows):
    off = np.zeros(len(rows) + 1, np.int32)
    off[1:] = np.cumsum([len(r) for r in rows])
    return off, np.array([x for r in rows for x in r], np.int32)


# ------------------------------------------------------------- k-cliques --

@pytest.mark.parametrize("n,k", [
    (33, 4), (34, 5), (35, 6), (35, 9), (66, 5), (67, 6), (68, 7), (130, 5), (131, 6), (132, 5),
    (258, 5), (260, 6), (513, 5), (515, 5), (769, 4), (1217, 4), (1219, 4)])
def test_clique_bit_rows_at_size_limits(R, cuda, n, k):
    """Complete graphs around every width of the packed rows (32, 64, 128, 256,
    512 common neighbours), the longest row held as bits, and past both."""
    off = np.zeros(n + 1, np.int32)
    off[1:] = np.cumsum(np.arange(n - 1, -1, -1))
    cols = np.concatenate([np.arange(u + 1, n, dtype=np.int32) for u in range(n)])
    d_off, d_cols = dev(off, cuda), dev(cols, cuda)
    t = R.Table(d_off, d_cols, hierarchical=bool(n % 2))
    assert R.clique_count(t, d_off, d_cols, k) == comb(n, k)
    t.check()


@pytest.mark.parametrize("bucket", [1, 5])
@pytest.mark.parametrize("kind", ["symmetric", "loops", "shuffled", "repeated"])
def test_clique_rows_of_every_kind(R, cuda, oracle_mod, kind, bucket):
    """Dense random digraphs (rows on both sides of 32 keys) whose rows are
    sets, hold the vertex itself, are out of order, or repeat keys."""
    rng = np.random.default_rng(0x5EED7C00 + bucket)
    n = 90
    rows = []
    for u in range(n):
        p = 0.1 if u % 3 else 0.6
        keep = np.flatnonzero(rng.random(n) < p)
        keep = keep[keep != u] if kind != "loops" else np.union1d(keep, [u])
        rows.append(keep)
    if kind == "repeated":
        rows = [np.sort(np.concatenate([r, r[::3]])) for r in rows]
    off, cols = csr(rows)
    want = {k: oracle_mod.clique_k(off, cols, k) for k in (4, 5, 6)} if kind != "repeated" else None
    if kind == "shuffled":
        for u in range(n):
            rng.shuffle(cols[off[u]:off[u + 1]])
    d_off, d_cols = dev(off, cuda), dev(cols, cuda)
    t = R.Table(d_off, d_cols, alpha=0.4, bucket=bucket)
    if want is None:  # keys of the shorter row count as often as they occur there
        want = {k: _clique_multiset(rows, k) for k in (4, 5)}
    for k, w in want.items():
        assert R.clique_count(t, d_off, d_cols, k) == w, k
    t.check()


def _clique_multiset(rows, k):
    sets = [set(r.tolist()) for r in rows]

    def below(c, left):
        if left == 1:
            return sum(sum(x in sets[w] for x in c) for w in c)
        return sum(below([x for x in c if x in sets[w]], left - 1) for w in c)

    total = 0
    for u, r in enumerate(rows):
        for v in r:
            a, b = (v, u) if len(r) > len(rows[v]) else (u, v)
            total += below([x for x in rows[a].tolist() if x in sets[b]], k - 3)
    return total


# -------------------------------------------------------------- patterns --

def _patterns(R):
    P = R.PatternSpec
    out = dict(R.PATTERNS)
    out["tail_bound"] = P(4, (0, 1, 3, 4), (0, 0, 1, 2), (-1, 0, -1, 2), None, 3)
    out["tail_distinct"] = P(4, (0, 1, 3, 4), (0, 0, 1, 2), (-1, 0, -1, -1), None, 3)
    out["pair_distinct"] = P(4, (0, 1, 2, 4), (0, 0, 1, 2), (-1, -1, -1, -1), None, 2)
    out["pair_own_bound"] = P(4, (0, 1, 2, 4), (0, 0, 1, 2), (-1, -1, -1, 2), None, 1)
    out["triangle_bound"] = P(3, (0, 1, 3), (0, 0, 1), (-1, 0, 1), None, 1)
    return out


def _oracle_pattern(oracle_mod, off, cols, p):
    return oracle_mod.pattern_count(off, cols, p.k, p.flags, p.offsets, p.backward,
                                    p.restriction, p.reuse)


@pytest.mark.parametrize("n,density,loops", [(61, 0.3, True), (128, 0.2, False), (201, 0.35, True)])
def test_patterns_on_digraphs(R, cuda, oracle_mod, n, density, loops):
    """Rows that are not symmetric and may hold their own vertex; vertex
    counts around whole words of the bit rows; first sets cut into parts."""
    rng = np.random.default_rng(0x5EED7D00 + n)
    rows = []
    for u in range(n):
        keep = np.flatnonzero(rng.random(n) < density * (2 if u % 9 == 0 else 0.5))
        rows.append(keep if loops else keep[keep != u])
    off, cols = csr(rows)
    d_off, d_cols = dev(off, cuda), dev(cols, cuda)
    t = R.Table(d_off, d_cols, hierarchical=bool(n % 2))
    for name, p in _patterns(R).items():
        assert R.pattern_count(t, d_off, d_cols, p) == _oracle_pattern(oracle_mod, off, cols, p), name
    t.check()


@pytest.mark.parametrize("n", [63, 64, 65, 127, 129, 1030])
def test_codegree_tiles(R, cuda, oracle_mod, n):
    """Vertex counts around the tiles of the co-degree matrix and the words
    staged at a time; a dense core among vertices that have few neighbours."""
    rng = np.random.default_rng(n)
    core = rng.random((n, n)) < np.where(np.arange(n) < (60 if n < 200 else 12), 0.5, 2 / n)[:, None]
    core[-1, : n // 2] = True
    adj = np.triu(core, 1)
    adj |= adj.T
    off, cols = csr([np.flatnonzero(r) for r in adj])
    d_off, d_cols = dev(off, cuda), dev(cols, cuda)
    t = R.Table(d_off, d_cols)
    for name in ("Q6", "pair_distinct"):
        p = _patterns(R)[name]
        assert R.pattern_count(t, d_off, d_cols, p) == _oracle_pattern(oracle_mod, off, cols, p), name
    t.check()


def test_patterns_with_bit_rows_for_hubs_only(R, cuda, oracle_mod):
    """More vertices than a whole bit matrix takes: the long rows have bit
    rows, the others are probed in their tables."""
    off, cols = oracle_mod.rmat_graph(17, 1, 0x5EED7D17, oriented=False)
    assert (np.diff(off) >= 64).any()
    d_off, d_cols = dev(off, cuda), dev(cols, cuda)
    t = R.Table(d_off, d_cols)
    for name, p in _patterns(R).items():
        if p.graph == "symmetric" and not name.startswith("pair") and name != "tail_distinct":
            assert R.pattern_count(t, d_off, d_cols, p) == \
                _oracle_pattern(oracle_mod, off, cols, p), name
    t.check()


# ----------------------------------------------------- owner-grouped count --

def _random_symmetric(rng, n, edges, hub):
    """`edges` random edges and one vertex with `hub` neighbours."""
    e = rng.integers(0, n, (edges, 2))
    e = np.concatenate([e, np.stack([np.full(hub, 7), rng.choice(np.arange(8, n), hub, False)], 1)])
    e = np.unique(np.concatenate([e, e[:, ::-1]]), axis=0)
    e = e[e[:, 0] != e[:, 1]]
    off = np.zeros(n + 1, np.int32)
    off[1:] = np.cumsum(np.bincount(e[:, 0], minlength=n))
    return off, e[:, 1].astype(np.int32)


@pytest.mark.parametrize("n,edges,hub", [
    (300, 3000, 0), (500, 1500, 29), (500, 1500, 40), (3000, 4000, 400), (40000, 300, 31),
    (40000, 300, 200), (47000, 50000, 300)])
def test_patterns_of_sparse_graphs(R, cuda, oracle_mod, n, edges, hub):
    """Rows of at most 32 keys (no bit rows, no parts) and just more; few edges
    on many vertices, whose bit matrix would be large."""
    off, cols = _random_symmetric(np.random.default_rng(0x5EED8400 + n + hub), n, edges, hub)
    d_off, d_cols = dev(off, cuda), dev(cols, cuda)
    t = R.Table(d_off, d_cols, hierarchical=bool(hub % 2))
    for name, p in _patterns(R).items():
        assert R.pattern_count(t, d_off, d_cols, p) == _oracle_pattern(oracle_mod, off, cols, p), name
    t.check()


def test_patterns_do_not_pay_for_vertices_without_edges(R, cuda):
    times = []
    for n in (400, 40000):
        off, cols = _random_symmetric(np.random.default_rng(0x5EED8500), n, 100, 0)
        d_off, d_cols = dev(off, cuda), dev(cols, cuda)
        t = R.Table(d_off, d_cols)
        times.append(_best_ms(cuda, lambda: R.pattern_count(t, d_off, d_cols, "Q6"), 20))
    assert times[1] <= 1.5 * times[0] + 0.02


def _multiset_tc(off, cols):
    """The reference's count: every key of the shorter row (ties: the edge's
    source) looked up in the other row's set."""
    rows = [cols[off[u]:off[u + 1]] for u in range(off.size - 1)]
    sets = [np.unique(r) for r in rows]
    total = 0
    for u, r in enumerate(rows):
        for v in r:
            a, b = (v, u) if r.size > rows[v].size else (u, v)
            total += int(np.isin(rows[a], sets[b]).sum())
    return total


@pytest.mark.parametrize("alpha,bucket", [(0.2, 5), (0.25, 1), (0.9, 2), (1.0, 1)])
@pytest.mark.parametrize("kind", ["oriented", "symmetric", "repeated", "shuffled"])
def test_owner_grouped_rows_of_every_kind(R, cuda, oracle_mod, kind, alpha, bucket):
    """Groups of one to thousands of probers, rows of one chunk and less, rows
    with repeated keys, tables at the highest load."""
    off, cols = oracle_mod.rmat_graph(11, 16, 0x5EED7E00, oriented=kind != "symmetric")
    rng = np.random.default_rng(0x5EED7E00)
    if kind == "repeated":
        rows = [np.concatenate([r, r[::3]]) for r in np.split(cols, off[1:-1])]
        off, cols = csr(rows)
    if kind == "shuffled":
        for u in range(off.size - 1):
            rng.shuffle(cols[off[u]:off[u + 1]])
    want = _multiset_tc(off, cols)
    d_off, d_cols = dev(off, cuda), dev(cols, cuda)
    t = R.Table(d_off, d_cols, alpha=alpha, bucket=bucket, hash_order=True)
    for c in (d_cols, t.hash_order):
        for method in (0, 1, 3):
            assert R.tc_count(t, d_off, c, method=method) == want, method
    t.check()


@pytest.mark.parametrize("d", [7, 8, 9, 255, 256, 257, 2040, 2041, 4095, 4096, 4097, 5000])
def test_owner_grouped_set_sizes(R, cuda, d):
    """Complete graphs on the last d of n vertices: sets around a warp's and a
    CTA's staged table, and past both (probed in HBM)."""
    n = d + 1
    deg = np.arange(n - 1, -1, -1, dtype=np.int64)
    deg[200:max(200, n - 200)] = 0  # the ends of the range are enough
    off = np.zeros(n + 1, np.int64)
    off[1:] = np.cumsum(deg)
    cols = np.concatenate([np.arange(u + 1, n, dtype=np.int32) for u in range(n) if deg[u]])
    d_off, d_cols = dev(off.astype(np.int32), cuda), dev(cols, cuda)
    # sum over edges (u, v) of |N(u) n N(v)| = the keys above v, where v has a row
    u_rows = np.flatnonzero(deg)
    want = sum(int(deg[v]) * int((u_rows < v).sum()) for v in u_rows)
    for bucket, alpha in ((5, 0.2), (1, 0.25)):
        t = R.Table(d_off, d_cols, alpha=alpha, bucket=bucket, hierarchical=bucket == 1)
        assert R.tc_count(t, d_off, d_cols, method=3) == want
        t.check()
        t.free()


@pytest.mark.parametrize("alpha,bucket", [(0.2, 5), (0.5, 4), (0.9, 2), (1.0, 5), (0.25, 1)])
def test_owner_grouped_large_sets(R, cuda, oracle_mod, alpha, bucket):
    """Sets around 4096 keys, the largest staged by five CTAs per SM, up to
    20480, the largest staged at all, and past it; one more prober than a unit
    takes; in one graph and in a batch of two."""
    rng = np.random.default_rng(0x5EED7E60 + bucket)
    n = 22000
    sizes = [4095, 4096, 4097, 5000, 8192, 10000, 16384, 20479, 20480, 20481, 21900]
    rows = [np.sort(rng.choice(n, d, replace=False)) for d in sizes]
    rows += [np.sort(rng.choice(len(sizes), 3, replace=False)) for _ in range(2049)]
    rows += [np.sort(rng.choice(n, 40, replace=False)) for _ in range(n - len(rows))]
    off, cols = csr(rows)
    d_off, d_cols = dev(off, cuda), dev(cols, cuda)
    t = R.Table(d_off, d_cols, alpha=alpha, bucket=bucket)
    want = oracle_mod.tc_merge(off, cols)
    assert R.tc_count(t, d_off, d_cols, method=3) == want
    t.check()
    two_off = cuda.cat([d_off, d_off[1:] + d_cols.numel()])
    two_cols = cuda.cat([d_cols, d_cols + n])
    t2 = R.Table(two_off, two_cols, alpha=alpha, bucket=bucket, hierarchical=False)
    counts = R.tc_count_batch(t2, two_off, two_cols, dev(np.array([0, n, 2 * n], np.int32), cuda))
    assert counts.tolist() == [want, want]
    t2.check()


def test_owner_grouped_large_sets_are_staged(R, cuda):
    """Many probers of large sets: faster in shared memory than from HBM."""
    rng = np.random.default_rng(0x5EED7E70)
    n = 20000
    off, cols = csr([np.sort(rng.choice(n, 8000 if u < 300 else 60, replace=False))
                     for u in range(n)])
    d_off, d_cols = dev(off, cuda), dev(cols, cuda)
    for alpha, bucket in [(0.5, 4), (0.9, 2)]:
        t = R.Table(d_off, d_cols, alpha=alpha, bucket=bucket)
        ms = {k: _best_ms(cuda, lambda: R.tc_count_async(t, d_off, d_cols, method=k), 3)
              for k in (1, 3)}
        assert ms[3] < ms[1]


@pytest.mark.parametrize("d", [2040, 2041, 8192, 8193, 300_000])
def test_owner_grouped_long_rows(R, cuda, oracle_mod, d):
    """Rows padded in parts, at their limits; hubs whose units are many."""
    rng = np.random.default_rng(0x5EED7E90 + d)
    n = max(3000, d + 500)
    rows = [np.sort(rng.choice(n, d, replace=False)) for _ in range(3)]
    rows += [np.sort(rng.choice(n, 4, replace=False)) for _ in range(200)]
    rows += [np.array([0, 1])] * 1000 + [np.zeros(0, np.int64)] * (n - 1203)
    off, cols = csr(rows)
    d_off, d_cols = dev(off, cuda), dev(cols, cuda)
    want = oracle_mod.tc_merge(off, cols)
    for alpha, bucket in ((0.2, 5), (0.25, 1)):
        t = R.Table(d_off, d_cols, alpha=alpha, bucket=bucket)
        assert R.tc_count(t, d_off, d_cols, method=3) == want
        t.check()


def test_owner_grouped_one_hub(R, cuda):
    """One row of 900,000 keys, which 8 lanes took 4 ms and more to pad."""
    n = 1_000_000
    hub = np.arange(1, 900_001, dtype=np.int32)
    rest = (np.arange(1, n)[:, None] * np.array([3, 5, 7]) + 11) % n
    off = np.concatenate([[0], hub.size + 3 * np.arange(n)]).astype(np.int32)
    d_off, d_cols = dev(off, cuda), dev(np.concatenate([hub, rest.ravel()]).astype(np.int32), cuda)
    t = R.Table(d_off, d_cols)
    assert R.tc_count(t, d_off, d_cols, method=3) == R.tc_count(t, d_off, d_cols, method=1)
    assert _best_ms(cuda, lambda: R.tc_count_async(t, d_off, d_cols, method=3)) < 2
    t.check()


@pytest.mark.parametrize("n", [130, 600, 690, 700, 20000])
def test_owner_grouped_room_for_rows(R, cuda, n):
    """As many keys in more and more rows: a chunk per 8 keys and row, then a
    chunk per key (from 7/8 of a row per key on)."""
    rng = np.random.default_rng(n)
    adj = [[] for _ in range(n)]
    pairs = [(u, v) for u in range(40) for v in range(u + 1, 40)]  # (a core with triangles)
    for u, v in rng.permutation(pairs)[:500].tolist():
        adj[u].append(v)
    for u in rng.permutation(np.arange(40, n))[:289].tolist() if n > 400 else [40] * 80:
        adj[u].append(len(adj[u]) + 41 if n <= 400 else 0)
    rows = [sorted(set(r)) for r in adj]
    off, cols = csr(rows)
    d_off, d_cols = dev(off, cuda), dev(cols, cuda)
    t = R.Table(d_off, d_cols)
    want = sum(len(np.intersect1d(rows[u], rows[v])) for u in range(n) for v in rows[u])
    assert want > 0 and R.tc_count(t, d_off, d_cols, method=3) == want
    t.check()


def test_owner_grouped_classes_and_single_chunk_rows(R, cuda):
    """2^24 keys and more: rows in class order; long runs of rows of one chunk
    between long ones (the rings that follow the rows fill with short rows)."""
    off, cols = R.gen_rmat(21, 10, 0x5EED7E21)
    assert cols.numel() >= 1 << 24
    t = R.Table(off, cols, alpha=0.25, bucket=1)
    want = R.tc_count(t, off, cols, method=1)
    for _ in range(3):
        assert R.tc_count(t, off, cols, method=3) == want
    t.check()


@pytest.mark.parametrize("alpha,bucket", [(0.2, 5), (0.25, 1)])
def test_sparse_graphs_edge_by_edge(R, cuda, oracle_mod, alpha, bucket):
    """Graphs without long rows: whole and in a batch (every graph's own count)
    edge by edge, and grouped on demand."""
    rng = np.random.default_rng(0x5EED7E80)
    graphs = []
    for n, d in [(40000, 20), (700, 3), (1, 0), (33, 9), (90000, 5)]:
        e = np.unique(rng.integers(0, n, (n * d, 2)), axis=0)
        e = e[e[:, 0] < e[:, 1]]
        off = np.zeros(n + 1, np.int32)
        off[1:] = np.cumsum(np.bincount(e[:, 0], minlength=n))
        graphs.append((off, e[:, 1].astype(np.int32)))
    want = [oracle_mod.tc_merge(o, c) for o, c in graphs]
    assert min(want[0], want[3]) > 0
    starts = np.cumsum([0] + [o.size - 1 for o, _ in graphs]).astype(np.int32)
    ends = np.cumsum([0] + [c.size for _, c in graphs])
    off = np.concatenate([o[:-1] + z for (o, _), z in zip(graphs, ends)] + [ends[-1:]])
    cols = np.concatenate([c + v for (_, c), v in zip(graphs, starts)])
    d_off, d_cols = dev(off.astype(np.int32), cuda), dev(cols.astype(np.int32), cuda)
    t = R.Table(d_off, d_cols, alpha=alpha, bucket=bucket, hierarchical=bucket == 1)
    before = R._lib().reset_kernel_launches()
    assert R.tc_count_batch(t, d_off, d_cols, dev(starts, cuda)).tolist() == want
    assert R._lib().reset_kernel_launches() - before == 1  # (a grouped count takes five)
    assert R.tc_count(t, d_off, d_cols) == R.tc_count(t, d_off, d_cols, method=3) == sum(want)
    t.check()


@pytest.mark.parametrize("kind", ["symmetric", "shuffled", "repeated", "batch"])
def test_owner_grouped_classes_of_every_kind(R, cuda, kind):
    """2^24 keys and more, rows in class order: rows that hold lower classes
    than their own, out of order, with repeated keys, and a batch of graphs."""
    gen = cuda.Generator(device="cuda")
    gen.manual_seed(0x5EED7E24)
    scale = 20 if kind in ("symmetric", "shuffled", "repeated") else 19
    off, cols = R.gen_rmat(scale, 9, 0x5EED7E24, oriented=False)
    n = off.numel() - 1
    row = cuda.repeat_interleave(cuda.arange(n, device="cuda"), (off[1:] - off[:-1]).long())
    if kind == "shuffled":
        order = cuda.randperm(cols.numel(), generator=gen, device="cuda")
        cols = cols[order[row[order].argsort(stable=True)]].contiguous()
    if kind == "repeated":
        twice = cuda.arange(cols.numel(), device="cuda") % 5 == 0
        cols = cuda.repeat_interleave(cols, 1 + twice.long())
        off = cuda.cat([cuda.zeros(1, device="cuda", dtype=cuda.int64),
                        cuda.cumsum(cuda.bincount(cuda.repeat_interleave(row, 1 + twice.long()),
                                                  minlength=n), 0)]).int()
    if kind == "batch":
        g = 3
        cols = cuda.cat([cols + k * n for k in range(g)])
        off = cuda.cat([off[:-1] + k * (cols.numel() // g) for k in range(g)] +
                       [cuda.tensor([cols.numel()], dtype=cuda.int32, device="cuda")])
    assert cols.numel() >= 1 << 24
    t = R.Table(off, cols, alpha=0.25, bucket=1)
    want = R.tc_count(t, off, cols, method=1)
    if kind == "batch":
        starts = cuda.arange(g + 1, dtype=cuda.int32, device="cuda") * n
        assert R.tc_count_batch(t, off, cols, starts).tolist() == [want // g] * g
    assert R.tc_count(t, off, cols, method=3) == want
    t.check()


# ------------------------------------------------------------ table build --

def _check_build(R, cuda, oracle_mod, rows, alpha, bucket, hier):
    off, elems = csr(rows)
    d_off, d_el = dev(off, cuda), dev(elems, cuda)
    t = R.Table(d_off, d_el, alpha=alpha, bucket=bucket, hierarchical=hier, hash_order=True)
    t.check()
    want = oracle_mod.Table(off, elems, alpha=alpha, bucket=bucket, hier=hier)
    slots, length, offsets = (x.cpu().numpy() for x in t.tensors())
    assert np.array_equal(length, want.len) and np.array_equal(offsets, want.off64)
    assert np.array_equal(slots, want.table)
    assert np.array_equal(t.hash_order.cpu().numpy(), want.hash_order())


@pytest.mark.parametrize("alpha,bucket", [(0.2, 5), (0.25, 1), (1.0, 1), (0.9, 2), (0.3, 16)])
@pytest.mark.parametrize("hier", [True, False])
def test_long_sets_runs_and_crowding(R, cuda, oracle_mod, alpha, bucket, hier):
    """Sets past a tile: lengths around the items of 2048 keys and buckets, a
    key repeated 95, 96, 97 and 3000 times (runs at and past their limit), keys
    of the last buckets (a run that wraps), short sets between them."""
    rng = np.random.default_rng(0x5EED7F00 + bucket)
    rows = [np.arange(5)]
    for i, d in enumerate((4095, 4096, 4097, 6143, 9000, 20011)):
        x = rng.choice(1 << 24, d, replace=False)
        if i:
            rep = (95, 96, 97, 3000, 1)[i - 1]
            x[rng.choice(d, rep, replace=False)] = x[0]
        x[-40:] = (1 << 24) - 1 - np.arange(40)
        rows += [x, rng.choice(1 << 24, 3 * i, replace=False), np.zeros(0, np.int64)]
    _check_build(R, cuda, oracle_mod, rows, alpha, bucket, hier)


@pytest.mark.parametrize("bucket,keys", [(1, 14500), (2, 14500), (16, 30000)])
def test_builds_near_full_load(R, cuda, oracle_mod, bucket, keys):
    """Sets that nearly fill their tables, whose runs are long: a warp per set
    inserts them, a key in well below 0.1 us, and nothing else is tried first
    (which took another 0.1)."""
    rng = np.random.default_rng(0x5EED7E40 + bucket)
    rows = [np.sort(rng.choice(1 << 27, keys, replace=False)) for _ in range(60)]
    _check_build(R, cuda, oracle_mod, rows[:3], 1.0, bucket, True)
    off, elems = (dev(x, cuda) for x in csr(rows))

    def build():
        R.Table(off, elems, alpha=1.0, bucket=bucket, hash_order=True).free_async()

    assert _best_ms(cuda, build) < 1.25e-4 * keys


@pytest.mark.parametrize("alpha,bucket", [(0.2, 5), (0.25, 1)])
def test_builds_of_many_long_sets(R, cuda, oracle_mod, alpha, bucket):
    """So many sets just past a tile that a warp each inserts them, longer ones
    among them key-parallel."""
    rng = np.random.default_rng(0x5EED7E60)
    rows = [rng.choice(1 << 26, 1300 + i % 700, replace=False) for i in range(2200)]
    _check_build(R, cuda, oracle_mod, rows, alpha, bucket, False)
    rows[100:2200:700] = [rng.choice(1 << 26, 9000, replace=False) for _ in range(3)]
    _check_build(R, cuda, oracle_mod, rows, alpha, bucket, True)


@pytest.mark.parametrize("n,edges,hub", [(300, 3000, 0), (500, 1500, 40), (2000, 30000, 300)])
def test_path_patterns(R, cuda, oracle_mod, n, edges, hub):
    """A last level that is the row of the vertex before it, less the earlier
    vertices; rows with and without loops, with and without bit rows."""
    off, cols = _random_symmetric(np.random.default_rng(0x5EED8600 + n), n, edges, hub)
    rows = [cols[off[u]:off[u + 1]] for u in range(n)]
    for loops in (False, True):
        if loops:
            rows = [np.union1d(r, [u]) if u % 3 == 0 else r for u, r in enumerate(rows)]
        o, c = csr(rows)
        d_off, d_cols = dev(o, cuda), dev(c, cuda)
        t = R.Table(d_off, d_cols)
        for p in (R.PatternSpec(4, (0, 1, 2, 3), (0, 1, 2), None, None, 2),
                  R.PatternSpec(4, (0, 1, 3, 4), (0, 0, 1, 2), (-1, 0, -1, -1), None, 3)):
            assert R.pattern_count(t, d_off, d_cols, p) == _oracle_pattern(oracle_mod, o, c, p)
        t.check()


@pytest.mark.parametrize("alpha,bucket", [(0.2, 5), (1.0, 1), (0.95, 16)])
def test_builds_of_several_crowded_long_sets(R, cuda, oracle_mod, alpha, bucket):
    """Sets of 2^16 keys and more, crowded by a repeated key or by their load,
    among others that are not: the crowded ones are listed in any order."""
    rng = np.random.default_rng(0x5EED7E50)
    rows = []
    for i, d in enumerate((65536, 65535, 124000, 70000, 66000, 124000)):
        x = rng.choice(1 << 27, d, replace=False)
        if i % 2 == 0:
            x[rng.choice(d, 400, replace=False)] = x[0]
        rows += [x, np.arange(i)]
    _check_build(R, cuda, oracle_mod, rows, alpha, bucket, False)


def test_builds_of_all_bucket_sizes_from_several_threads(R, cuda):
    """Each thread builds tables of its own bucket size on its own stream: the
    shared memory that a tile takes differs by bucket size."""
    import threading
    rng = np.random.default_rng(0x5EED7E30)
    off, elems = csr([np.sort(rng.choice(5000, 40, replace=False)) for _ in range(50)])
    d_off, d_el = dev(off, cuda), dev(elems, cuda)
    sizes = (1, 5, 3, 7, 1, 5)
    tables = {b: R.Table(d_off, d_el, bucket=b) for b in sizes}
    want = {b: t.tensors()[0].clone() for b, t in tables.items()}
    cuda.cuda.synchronize()
    errors = []

    def work(b):
        try:
            stream = cuda.cuda.Stream()
            for i in range(300):
                t = R.Table(d_off, d_el, bucket=b, stream=stream)
                if i % 50 == 0:
                    stream.synchronize()
                    assert cuda.equal(t.tensors()[0], want[b]), b
                    cuda.cuda.current_stream().synchronize()
                t.free_async(stream)
            stream.synchronize()
        except Exception as e:
            errors.append(e)

    threads = [threading.Thread(target=work, args=(b,)) for b in sizes]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    assert not errors, errors[0]


def test_chunk_rows_of_long_rows(R, cuda, oracle_mod):
    """Chunk rows and tile starts of rows that span many chunks and tiles
    (written by a whole warp), beside empty ones."""
    rng = np.random.default_rng(0x5EED7F77)
    n = 100000
    sizes = [0, 1, 33, 0, 0, 300, 50000, 31, 32, 70000, 0, 2]
    rows = [np.sort(rng.choice(n, d, replace=False)) for d in sizes]
    rows += [np.zeros(0, np.int64)] * (n - len(rows))
    rows[n - 1] = np.arange(1, 40)  # edges into the long rows
    off, cols = csr(rows)
    want = oracle_mod.tc_merge(off, cols)
    assert want > 0
    d_off, d_cols = dev(off, cuda), dev(cols, cuda)
    for bucket in (1, 5):
        t = R.Table(d_off, d_cols, bucket=bucket)
        copy = d_off.clone()  # other offsets: chunk rows found again
        for o in (d_off, copy):
            for method in (1, 3):
                assert R.tc_count(t, o, d_cols, method=method) == want
        t.check()


# -------------------------------------------------------------- raw pair --

@pytest.mark.parametrize("nb", [0, 1, 2, 31, 33, 511, 4095, 4096, 4097, 8193, 70001])
@pytest.mark.parametrize("na", [0, 1, 513, 20011])
def test_raw_pair_sizes(R, cuda, na, nb):
    """Around the largest set held in shared memory; both unsorted, with
    repeats; keys at the ends of the range."""
    rng = np.random.default_rng(na * 7 + nb)
    hi = max(4, (na + nb) // 2)
    a = rng.integers(0, hi, na).astype(np.int32)
    b = rng.integers(0, hi, nb).astype(np.int32)
    ends = np.array([0, 2**31 - 1, 2**31 - 2, 1 << 30], np.int32)
    a[: min(na, 4)] = ends[: min(na, 4)]
    b[max(nb - 3, 0):] = ends[:nb][-3:][: len(b[max(nb - 3, 0):])]
    assert R.intersect_count(dev(a, cuda), dev(b, cuda)) == int(np.isin(a, b).sum())


@pytest.mark.parametrize("nb", [1, 100, 1025, 4096])
def test_raw_pair_of_many_keys_and_few(R, cuda, nb):
    """Several blocks per SM, each with the whole set of B."""
    rng = np.random.default_rng(nb)
    a = rng.integers(0, 6 * nb, 3_000_001).astype(np.int32)
    b = rng.integers(0, 6 * nb, nb).astype(np.int32)
    assert R.intersect_count(dev(a, cuda), dev(b, cuda)) == int(np.isin(a, b).sum())


def test_raw_pair_of_more_than_2_to_the_30_keys(R, cuda):
    """The set of 2^32 slots, the largest: its index takes all 32 bits."""
    n = (1 << 30) + 5
    b = cuda.arange(n, dtype=cuda.int32, device="cuda")
    a = cuda.tensor([0, 7, n - 1, n, n + 1, (1 << 31) - 1] * 50, dtype=cuda.int32, device="cuda")
    assert R.intersect_count(a, b) == 150
    del b
    cuda.cuda.empty_cache()
    R._lib().reset_release_cached_memory()


@pytest.mark.parametrize("pairs", [1, 33, 300, 4800, 40000])
def test_pairs_per_warp(R, cuda, pairs):
    """Few pairs are spread over the warps, one to a warp at the fewest."""
    rng = np.random.default_rng(pairs)
    rows = [np.sort(rng.choice(900, rng.integers(0, 200), replace=False)) for _ in range(400)]
    off, cols = csr(rows)
    t = R.Table(dev(off, cuda), dev(cols, cuda))
    pa, pb = (rng.integers(0, 400, pairs).astype(np.int32) for _ in range(2))
    _, inter = R.sss(t, dev(off, cuda), dev(cols, cuda), dev(pa, cuda), dev(pb, cuda), 1, 10)
    want = [len(np.intersect1d(rows[u], rows[v])) for u, v in zip(pa, pb)]
    assert inter.cpu().tolist() == want


# -------------------------------------------------------- decisions only --

@pytest.mark.parametrize("num,den", [(1, 20), (1, 2), (7, 10), (19, 20), (1, 1)])
@pytest.mark.parametrize("kind", ["ascending", "shuffled", "repeated"])
def test_decisions_only_like_full(R, cuda, kind, num, den):
    """Runs of pairs of every length with the same first set, sets of up to
    more keys than the run's bitmap takes, equal, near and unlike ones, against
    the decisions of full intersections."""
    rng = np.random.default_rng(num * 31 + den)
    rows = []
    for size in [0, 1, 2, 7, 8, 31, 33, 100, 257, 1000, 4096, 4097, 5000]:
        base = np.sort(rng.choice(20000, size, replace=False))
        rows.append(base)
        for keep in [1.0, 0.97, 0.8, 0.6, 0.1]:
            r = base[rng.random(size) < keep]
            rows.append(np.unique(np.concatenate([r, rng.choice(20000, size - len(r))])))
    if kind == "shuffled":
        rows = [rng.permutation(r) for r in rows]
    if kind == "repeated":
        rows = [np.sort(np.concatenate([r, r[: len(r) // 3]])) if i % 3 else r
                for i, r in enumerate(rows)]
    n = len(rows)
    pa, pb = [], []
    for u in range(n):  # runs of 1, 2, 3, ... and all of them
        for v in [*rng.integers(0, n, u % 37), *range(u - u % 6, u + 6 - u % 6)]:
            pa.append(u)
            pb.append(v)
    off, cols = csr(rows)
    d_off, d_cols = dev(off, cuda), dev(cols, cuda)
    t = R.Table(d_off, d_cols)
    pa, pb = dev(np.array(pa, np.int32), cuda), dev(np.array(pb, np.int32), cuda)
    for x, y in [(pa, pb), (pb, pa)]:
        full, _ = R.sss(t, d_off, d_cols, x, y, num, den)
        dec, none = R.sss(t, d_off, d_cols, x, y, num, den, with_inter=False)
        assert none is None and 0 < int(full.sum()) < full.numel()
        assert cuda.equal(full, dec)


# -------------------------------------------------------- prefix filter --

def _best_ms(cuda, f, n=5):
    f()
    best = float("inf")
    for _ in range(n):
        a, z = (cuda.cuda.Event(enable_timing=True) for _ in range(2))
        a.record()
        f()
        z.record()
        z.synchronize()
        best = min(best, a.elapsed_time(z))
    return best


@pytest.mark.parametrize("size,differ", [(63, 2), (255, 6), (300, 100), (5000, 0), (5000, 20)])
def test_decisions_only_of_like_sets(R, cuda, size, differ):
    """Sets that share most of their keys: as with sizes, at most twice the
    time (a pair's lookups are all the work, whichever way they are cut)."""
    rng = np.random.default_rng(0x5EED8100 + size + differ)
    base = rng.choice(1 << 20, size + differ, replace=False)
    rows = [np.sort(np.delete(base, rng.choice(base.size, differ, replace=False)))
            for _ in range(40)]
    off, elems = csr(rows)
    d_off, d_elems = dev(off, cuda), dev(elems, cuda)
    t = R.Table(d_off, d_elems)
    pairs = rng.integers(0, 40, (2, 3000)).astype(np.int32)
    pa, pb = dev(pairs[0], cuda), dev(pairs[1], cuda)
    for num, den in [(1, 2), (7, 10), (19, 20), (99, 100), (1, 1)]:
        full = R.sss(t, d_off, d_elems, pa, pb, num, den)[0]
        only = R.sss(t, d_off, d_elems, pa, pb, num, den, with_inter=False)[0]
        assert cuda.equal(only, full), (num, den)
        fast = _best_ms(cuda, lambda: R.sss(t, d_off, d_elems, pa, pb, num, den,
                                            with_inter=False))
        assert fast <= 2 * _best_ms(cuda, lambda: R.sss(t, d_off, d_elems, pa, pb, num, den)) + 0.02
    t.check()


@pytest.mark.parametrize("size,other,universe", [
    (100, 5000, 100_000), (2000, 2000, 6000), (64, 300, 3000), (300, 300, 1 << 20), (30, 30, 80)])
def test_decisions_only_of_one_set(R, cuda, size, other, universe):
    """Runs of pairs with one first set, at thresholds where its bitmap settles
    all, some or none of them: as with sizes, at most twice the time."""
    rng = np.random.default_rng(0x5EED8200 + size)
    rows = [np.sort(rng.choice(universe, size, replace=False))]
    rows += [np.sort(rng.choice(universe, other, replace=False)) for _ in range(400)]
    for r in rows[1::5]:  # near-duplicates among them
        k = min(size, other) * 9 // 10
        r[:k] = rng.choice(rows[0], k, replace=False)
    rows = [np.unique(r) for r in rows]
    off, elems = csr(rows)
    d_off, d_elems = dev(off, cuda), dev(elems, cuda)
    t = R.Table(d_off, d_elems)
    n = 200_000
    pa = cuda.zeros(n, dtype=cuda.int32, device="cuda")
    pb = dev(rng.integers(1, 401, n).astype(np.int32), cuda)
    for num, den in [(1, 100), (1, 20), (1, 10), (1, 2), (7, 10), (1, 1)]:
        full = R.sss(t, d_off, d_elems, pa, pb, num, den)[0]
        only = R.sss(t, d_off, d_elems, pa, pb, num, den, with_inter=False)[0]
        assert cuda.equal(only, full), (num, den)
        fast = _best_ms(cuda, lambda: R.sss(t, d_off, d_elems, pa, pb, num, den,
                                            with_inter=False))
        assert fast <= 2 * _best_ms(cuda, lambda: R.sss(t, d_off, d_elems, pa, pb, num, den)) + 0.02
    t.check()


def test_decisions_only_of_very_large_sets(R, cuda):
    """Runs of pairs of one set whose other sets' keys together exceed 2^31."""
    big = 70_000_000
    held = cuda.arange(4096, dtype=cuda.int32, device="cuda") * 17000
    few = cuda.cat([held[:1400], held[1400:] + big])
    elems = cuda.cat([held, few, cuda.arange(big, dtype=cuda.int32, device="cuda")])
    off = cuda.tensor([0, 4096, 8192, 8192 + big], dtype=cuda.int32, device="cuda")
    # two slots a bucket, at most one of them taken: no lookup walks on
    t = R.Table(off, elems, alpha=0.5, bucket=2, hierarchical=False)
    # 1401 common keys are needed: 4096 in pairs (0, 2), 1400 in pairs (1, 2)
    assert -(-(4096 + big) // 50001) == 1401
    pa = cuda.arange(64, device="cuda").div(32, rounding_mode="floor").int()
    pb = cuda.full_like(pa, 2)
    # (a batch gives a warp 32 pairs, however few there are)
    batch = R.Batch(t, elems, capacity=64, num=1, den=50000, decisions_only=True)
    flags, _ = batch(pa, pb)
    assert cuda.equal(flags, (pa == 0).to(cuda.uint8))
    batch.close()
    t.check()


@pytest.mark.parametrize("num,den", [(1, 2), (7, 10), (1, 1)])
@pytest.mark.parametrize("freq", ["skewed", "level", "repeated", "shuffled"])
def test_prefix_selection_at_set_sizes(R, cuda, freq, num, den):
    """Sets around the sizes of a row of lanes, of vectors and of the shared
    buffer and past it; frequencies that differ and tie, tokens repeated in a
    set, rows that do not ascend ("level": all tie and the row wraps)."""
    rng = np.random.default_rng(num + 10 * den)
    rows = []
    for size in [0, 1, 2, 31, 63, 64, 65, 255, 256, 257, 511, 512, 513, 1023, 1024, 1025, 1500]:
        for _ in range(3):
            if freq == "level":  # runs of a cycle: every token equally often, nearly
                r = (np.arange(size) + rng.integers(0, 4096)) % 4096
            else:
                r = (4096 * rng.random(2 * size) ** 2).astype(int)
                r = np.sort(r[:size]) if freq == "repeated" else np.unique(r)[:size]
                r = rng.permutation(r) if freq == "shuffled" else r
            rows.append(r.astype(np.int32))
    off, tok = csr(rows)
    pa, pb = R.prefix_candidates(dev(off, cuda), dev(tok, cuda), 12, num, den)
    f = np.bincount(tok, minlength=4096)
    by_token, want = {}, set()
    for i, r in enumerate(rows):
        p = len(r) - -(-num * len(r) // den) + 1 if len(r) else 0
        for t in sorted(r.tolist(), key=lambda t: (f[t], t))[:p]:
            by_token.setdefault(t, []).append((len(r), i))
    for e in by_token.values():
        e.sort()
        for k, (size, i) in enumerate(e):
            for other, j in e[k + 1:]:
                if other <= den * size // num:
                    want.add((min(i, j), max(i, j)))
    got = list(zip(pa.cpu().tolist(), pb.cpu().tolist()))
    assert got == sorted(want)


def test_prefix_outputs_in_either_memory(R, cuda, libreset):
    """Pairs in memory of the library's and of the caller's; memory refused."""
    import ctypes as C
    from reset_b200._lib import AllocFn
    off, tok = R.gen_token_sets(3000, 12, size_lo=4, size_hi=60, seed=3)
    pa, pb = R.prefix_candidates(off, tok, 12)
    args = (C.c_void_p(off.data_ptr()), C.c_void_p(tok.data_ptr()), off.numel() - 1, tok.numel(),
            12, 7, 10)
    p, q, k = C.c_void_p(), C.c_void_p(), C.c_int64()
    outs = (C.byref(p), C.byref(q), C.byref(k), C.c_void_p(0))
    cuda.cuda.synchronize()
    assert libreset.reset_prefix_candidates(*args, *outs) == 0 and k.value == pa.numel() > 0
    assert cuda.equal(R._view(p.value, k.value, cuda.int32), pa)
    assert cuda.equal(R._view(q.value, k.value, cuda.int32), pb)
    libreset.reset_free(p)
    libreset.reset_free(q)
    calls = []
    for _ in range(2):  # none, then the first alone
        mem = cuda.empty(pa.numel(), dtype=cuda.int32, device="cuda")
        fn = AllocFn(lambda n, _: calls.append(n) or (mem.data_ptr() if len(calls) == 2 else None))
        assert libreset.reset_prefix_candidates_alloc(*args, fn, None, *outs) != 0
    assert calls == [4 * pa.numel()] * 3
    a2, b2 = R.prefix_candidates(off, tok, 12, stream=cuda.cuda.Stream())
    assert cuda.equal(a2, pa) and cuda.equal(b2, pb)


# -------------------------------------------------------------- retrieval --

@pytest.mark.parametrize("hier,bucket", [(True, 5), (False, 1)])
@pytest.mark.parametrize("ascending", [True, False])
def test_retrieval_list_and_query_sizes(R, cuda, hier, bucket, ascending):
    """Lists around a row of lanes, the keys of a warp's step and a slice;
    queries of one term up to more than a warp's lanes hold."""
    rng = np.random.default_rng(bucket)
    dfs = [0, 1, 31, 32, 33, 255, 256, 257, 511, 512, 513, 1024, 1025, 2900, 2999, 3000]
    rows = [rng.choice(3000, d, replace=False) for d in dfs]
    rows = [np.sort(r) if ascending else r for r in rows]
    off, docs = csr(rows)
    d_off, d_docs = dev(off, cuda), dev(docs, cuda)
    t = R.Table(d_off, d_docs, hierarchical=hier, bucket=bucket)
    queries = [[]]
    for first in range(len(rows)):
        for more in [0, 1, 2, 5]:
            queries.append([first, *rng.integers(0, len(rows), more)])
        for more in [31, 32, 33, 40]:  # long ones that leave something over
            queries.append([first, *rng.integers(13, len(rows), more)])
    qoff, query = csr(queries)
    roff, res, cnt = R.ir(t, d_off, d_docs, dev(query, cuda), dev(qoff, cuda))
    roff, res, cnt = (x.cpu().numpy() for x in (roff, res, cnt))
    for q, terms in enumerate(queries):
        want = rows[terms[0]] if terms else np.empty(0, int)
        for term in terms[1:]:
            want = want[np.isin(want, rows[term])]
        got = res[roff[q]:roff[q + 1]]
        assert cnt[q] == len(want) and np.array_equal(got[: len(want)], want)
        assert (got[len(want):] == -1).all()


def test_retrieval_of_many_slices(R, cuda):
    """More slices than one block's share of the scan, the last one partial."""
    n = 3 * 16384 * 512 // 2 + 77
    rows = [cuda.arange(0, n, dtype=cuda.int32), cuda.arange(0, n, 3, dtype=cuda.int32),
            cuda.arange(0, n, 1000, dtype=cuda.int32)]
    off = cuda.tensor(np.cumsum([0] + [r.numel() for r in rows]), dtype=cuda.int32)
    rows = [r.cuda() for r in rows]
    off, docs = off.cuda(), cuda.cat(rows)
    t = R.Table(off, docs)
    query = cuda.tensor([0, 1, 0, 1, 0, 2, 0, 2], dtype=cuda.int32).cuda()
    qoff = cuda.tensor([0, 2, 3, 5, 7, 8], dtype=cuda.int32).cuda()
    roff, res, cnt = R.ir(t, off, docs, query, qoff)
    for q, want in enumerate([rows[1], rows[0], rows[1], rows[2], rows[2]]):
        got = res[int(roff[q]):int(roff[q + 1])]
        assert int(cnt[q]) == want.numel() and cuda.equal(got[: want.numel()], want)
        assert bool((got[want.numel():] == -1).all())


def test_served_retrieval_of_many_slices(R, cuda):
    """A request above the cost cap: a block per so many slices, the last one
    with one of them."""
    from reset_b200 import server
    n = 512 * 64 * 150 + 5
    rows = [cuda.arange(0, n, dtype=cuda.int32), cuda.arange(0, n, 7, dtype=cuda.int32)]
    off = cuda.tensor(np.cumsum([0] + [r.numel() for r in rows]), dtype=cuda.int32).cuda()
    t = R.Table(off, cuda.cat(rows).cuda())
    with server.Server(max_batch_cost=100_000) as s:
        ix = s.add_index(t)
        for terms, want in (([0], rows[0]), ([0, 1], rows[1]), ([1, 0], rows[1])):
            r = s.wait(s.submit_ir(ix, terms))
            assert r.status == 0 and np.array_equal(r.docs, want.numpy())


# ---------------------------------------------------------- scarce memory --

@pytest.mark.parametrize("call", ["tc", "tc_batch", "tc_shard", "clique", "pattern"])
def test_calls_where_memory_is_scarce(R, cuda, libreset, call):
    """Calls whose larger scratch does not fit run without it: 8 M vertices,
    with 400 MB (groups) or 80 MB (work lists, bit rows) left on the device."""
    from reset_b200 import shard
    rng = np.random.default_rng(0x5EED8300)
    n = 8_000_000
    core = [np.sort(rng.choice(np.arange(u + 1, 1200), 300, replace=False)) for u in range(200)]
    core += [np.sort(rng.choice(np.arange(u + 1, 2101), 20, replace=False)) for u in range(200, 2000)]
    deg = np.ones(n, np.int64)
    deg[:2000] = [r.size for r in core]
    off = np.concatenate([[0], np.cumsum(deg)])
    cols = np.concatenate(core + [np.arange(2000, n) * 7 % 2000])
    d_off, d_cols = dev(off.astype(np.int32), cuda), dev(cols.astype(np.int32), cuda)
    if call == "tc_shard":
        d_koff, d_kcols = shard.shard_csr(d_off, d_cols, 1, 0)
    else:
        d_koff, d_kcols = d_off, d_cols
    t = R.Table(d_koff, d_kcols, alpha=0.25, bucket=1)
    graphs = dev(np.array([0, 2000, 5_000_000, n], np.int32), cuda)
    out = cuda.zeros(1, dtype=cuda.int64, device="cuda")
    out3 = cuda.zeros(3, dtype=cuda.int64, device="cuda")

    def run():
        if call == "tc":
            return R.tc_count_async(t, d_off, d_cols, out, method=3).tolist()
        if call == "tc_batch":
            return R.tc_count_batch(t, d_off, d_cols, graphs, out3).tolist()
        if call == "tc_shard":
            s = libreset.reset_tc_count_shard(
                t.handle, d_koff.data_ptr(), d_kcols.data_ptr(), d_kcols.numel(),
                d_off.data_ptr(), d_cols.data_ptr(), d_cols.numel(), out.data_ptr(),
                cuda.cuda.current_stream().cuda_stream)
            return s, out.tolist()
        if call == "clique":
            return R.clique_count(t, d_off, d_cols, 5)
        return R.pattern_count(t, d_off, d_cols, R.PatternSpec(4, (0, 1, 2, 4), (0, 0, 1, 2), None,
                                                               None, 2))

    want = run()
    assert sum(np.atleast_1d(want[-1] if isinstance(want, tuple) else want)) > 0
    cuda.cuda.synchronize()
    libreset.reset_release_cached_memory()
    cuda.cuda.empty_cache()
    left = (80 if call in ("clique", "pattern") else 400) << 20
    ballast = cuda.empty(cuda.cuda.mem_get_info()[0] - left, dtype=cuda.uint8, device="cuda")
    try:
        got = run()
        cuda.cuda.synchronize()
    finally:
        del ballast
        cuda.cuda.empty_cache()
    assert got == want
    t.check()
