"""Stress tests of what orders a subset-DP table's writes before its reads in
the kernels of the default path: the release counts per level of the level
kernel (single graphs and batches) and the barriers of the cluster kernel; the
tile kernel's flags have theirs in test_dp_publication.py.

Before a solve the table holds something else: 0xFF bytes (FAULT_POISON: both
residue planes and the connected plane set, which no solve writes) or the table
of another graph of the same size (an edgeless, a complete, a random one: the
handle's buffer keeps it). A word of 32 subsets read too early would take its
children from there. The CPU test below reads every word of small tables with
one child word replaced by each of these: at least one of them changes the word
above it. 0xFF alone does so for connected graphs; where most subsets are
disconnected many words take it without a change."""
import numpy as np
import pytest

from gisbdw_gb300 import _lib
from gisbdw_gb300 import graphs as G

M32 = 0xFFFFFFFF


def _word(planes, adj, n, W, stale=None):
    """The planes of word W (gtd_dp.cu's arithmetic), child W - v read as what
    `stale` = (v, planes) holds."""
    from test_dp_planes import ANY, resolve_quad, small_masks
    o, c1, c2 = [0, 0, 0], 0, 0
    verts = [v for v in range(n - 5) if W >> v & 1]
    for v in verts:
        p0, p1, c = (stale[1] if stale and stale[0] == v else planes)[W ^ (1 << v)]
        o = [o[0] | p0, o[1] | p1, o[2] | (~(p0 | p1) & M32)]
        c2 |= c1 & c
        c1 |= c
    small = small_masks(adj, n, [v + 5 for v in verts]) if len(verts) <= 2 else ANY
    return resolve_quad([(o, c1, c2, small)] * 4)[0]


@pytest.mark.parametrize("g", [G.gnp_connected(10, 0.3, 1), G.gnp_connected(11, 0.2, 2), G.grid(2, 5), G.path(10),
                               G.complete(10), G.Graph(10, [(0, 9), (3, 4)], name="sparse10")], ids=lambda g: g.name)
def test_an_early_read_changes_the_word_above_with_one_of_the_fills(g):
    from test_dp_planes import plane_dp
    adj, (planes, n) = g.adjacency_masks(), plane_dp(g, 8)
    fills = [{W: (M32, M32, M32) for W in planes}] + [plane_dp(f, 8)[0] for f in _fills(n)[1:]]
    for W in planes:
        assert _word(planes, adj, n, W) == planes[W]
        for v in range(n - 5):
            if W >> v & 1:
                seen = [_word(planes, adj, n, W, (v, f)) != planes[W] for f in fills]
                assert any(seen) and (seen[0] or not g.is_connected()), (W, v, seen)


# ---------------------------------------------------------------------------


def _natural(raw, n, lb):
    S = np.arange(1 << n, dtype=np.int64)
    tile = np.array([_lib.table_index(n, lb, h << lb) >> lb for h in range(1 << (n - lb))], dtype=np.int64)
    return raw[(tile[S >> lb] << lb) | (S & ((1 << lb) - 1))]


def _connected(g):
    """Of every subset, whether it is connected (the empty one is not)."""
    S = np.arange(1 << g.n, dtype=np.int32)
    reach = S & -S
    adj = g.adjacency_masks()
    while True:
        grown = reach.copy()
        for v in range(g.n):
            grown |= np.where(grown >> v & 1, np.int32(adj[v]), np.int32(0)) & S
        if np.array_equal(grown, reach):
            return (reach == S) & (S != 0)
        reach = grown


def _solve_over(handle, fill, g):
    """`g` solved over a table that holds `fill` (None: 0xFF bytes)."""
    if fill is None:
        _lib.inject_fault(_lib.FAULT_POISON, 1)
    else:
        handle.dp_solve(fill.adj64(), fill.n)
    try:
        return handle.dp_solve(g.adj64(), g.n)
    finally:
        _lib.inject_fault(_lib.FAULT_NONE, 0)


def _fills(n):
    return [None, G.Graph(n, []), G.complete(n), G.gnp_connected(n, 0.4, 1000 + n)]


@pytest.mark.gpu
@pytest.mark.parametrize("n", [22, 23, 24])
def test_level_kernel_over_other_tables_matches_oracle(handle, port, n):
    for k in range(2):
        g = G.gnp_connected(n, (0.2, 0.35)[k], 30 * n + k)
        T = port.dp_table(g, nthreads=8)
        otd, opar = port.tree_from_table(g, T)
        conn = _connected(g) if n == 22 else None
        for fill in _fills(n):
            td, parent, _, _ = _solve_over(handle, fill, g)
            raw, tn, lb = handle.dp_read_table()
            tab = _natural(raw, tn, lb)
            assert np.array_equal(tab >> 1, T), (g.name, fill and fill.name)
            assert conn is None or np.array_equal(tab[1:] & 1, conn[1:])
            assert td == otd and parent.tolist() == list(opar)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [17, 18, 19, 20, 21])
def test_cluster_kernel_over_other_tables_matches_oracle(handle, port, n):
    """Its table is in shared memory, which keeps what the launch before left."""
    for k in range(6):
        g = G.gnp_connected(n, (0.15, 0.25, 0.4)[k % 3], 40 * n + k) if k % 2 else G.grid_deleted(n, 0.1, 40 * n + k)
        T = port.dp_table(g, nthreads=8)
        otd, opar = port.tree_from_table(g, T)
        conn = _connected(g) if k < 2 else None
        for fill in _fills(n):
            td, parent, _, _ = _solve_over(handle, fill, g)
            raw, tn, lb = handle.dp_read_table()
            tab = _natural(raw, tn, lb)
            assert np.array_equal(tab >> 1, T), (g.name, fill and fill.name)
            assert conn is None or np.array_equal(tab[1:] & 1, conn[1:])
            assert td == otd and parent.tolist() == list(opar)


@pytest.mark.gpu
@pytest.mark.parametrize("use_cuda_graph", [True, False])
@pytest.mark.parametrize("sizes", [[17, 18, 19, 20, 21] * 16, [12, 16, 17, 22, 23]])
def test_batches_by_level_over_other_tables_match_oracle(handle, port, sizes, use_cuda_graph):
    """Every batch over 0xFF bytes, then over the tables of edgeless and of
    complete graphs: a first call, and replays of it where there is a graph."""
    gs = [G.gnp_connected(n, (0.2, 0.3)[i % 2], 700 + i % 10) for i, n in enumerate(sizes)]
    known = {}
    for g in gs:
        if g.name not in known:
            known[g.name] = port.dp_solve(g, nthreads=8)
    for call, fill in enumerate([None, None, lambda n: G.Graph(n, []), G.complete]):
        if fill is None:
            _lib.inject_fault(_lib.FAULT_POISON, 1)
        else:
            handle.dp_solve_batch([fill(n) for n in sizes], use_cuda_graph=use_cuda_graph)
        try:
            td, parents, stats = handle.dp_solve_batch(gs, use_cuda_graph=use_cuda_graph)
        finally:
            _lib.inject_fault(_lib.FAULT_NONE, 0)
        assert stats["graph_replayed"] == int(use_cuda_graph and call > 0)
        for g, t, par in zip(gs, td, parents):
            otd, opar = known[g.name]
            assert t == otd and par.tolist() == list(opar), (call, g.name)
