"""Incumbent heuristics of the library (gtd_heuristic, host code) against
the oracle's restatement of the reference heuristics and the reference's own
outputs (golden fixtures) on CPU; the batched GPU restatement against the
host code."""
import numpy as np
import pytest

from gisbdw_gb300 import _lib
from gisbdw_gb300 import graphs as G


def test_heuristics_match_reference_fixtures(golden):
    for e in golden("ref_solvers.json"):
        g = G.Graph(e["n"], [tuple(x) for x in e["edges"]])
        if not g.is_connected():
            continue
        for ref_kind, our_kind in (("0", 0), ("2", 1), ("3", 2)):
            td, par = _lib.heuristic(g, our_kind)
            ref = e["heuristics"][ref_kind]
            assert td == ref["td"], (e["name"], ref_kind)
            assert par.tolist() == ref["parent"], (e["name"], ref_kind)


def test_heuristics_match_oracle_on_large_sparse(port):
    for g in G.config4_graphs(count=6) + G.config5_graphs(count=6):
        for kind, okind in ((0, 0), (1, 2), (2, 3)):
            td, par = _lib.heuristic(g, kind)
            otd, opar = port.heuristic(g, okind)
            assert td == otd and par.tolist() == opar.tolist(), (g.name, kind)


def test_score_greedy_is_valid(port):
    g = G.config4_graphs(count=1)[0]
    scores = np.random.default_rng(0).random(g.n).astype(np.float32)
    td, par = _lib.heuristic(g, 3, scores)
    assert port.check_valid(g, td, par) if g.n <= 64 else True


@pytest.mark.gpu
@pytest.mark.parametrize("kind", [0, 1, 2, 3])
def test_gpu_batch_heuristics_equal_host(handle, kind):
    """gtd_heuristic_batch (one warp per graph) gives exactly the host's
    trees: same picks, same floating-point variance scores."""
    gs = (G.config3_graphs(count=60, seed=31) + G.config4_graphs(count=24, seed=32)
          + [g for g in G.config5_graphs(count=24, seed=33)]
          + [G.path(100), G.tree_plus_edges(104, 6, 2), G.Graph(9, [(0, 1), (2, 3), (3, 4)])])
    rng = np.random.default_rng(kind)
    scores = [rng.random(g.n).astype(np.float32) for g in gs] if kind == 3 else None
    td, pars = handle.heuristic_batch(gs, kind, scores)
    for i, g in enumerate(gs):
        htd, hpar = _lib.heuristic(g, kind, scores[i] if scores is not None else None)
        assert td[i] == htd, (g.name, kind)
        assert pars[i].tolist() == hpar.tolist(), (g.name, kind)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", [0, 1, 2])
def test_gpu_rounds_at_the_word_and_warp_edges(handle, kind):
    """A thread per vertex: vertex counts around 32, 64, 96 and 128, in one
    launch with single vertices, a clique, a star and separate components."""
    gs = [G.Graph(1, []), G.path(2), G.star(33), G.complete(32), G.cycle(64), G.tree_plus_edges(65, 9, 1),
          G.random_geometric(96, 4.0, 2), G.tree_plus_edges(97, 40, 3), G.path(104), G.Graph(70, [(0, 69), (64, 1)])]
    td, pars = handle.heuristic_batch(gs, kind)
    for i, g in enumerate(gs):
        htd, hpar = _lib.heuristic(g, kind)
        assert td[i] == htd and pars[i].tolist() == hpar.tolist(), (i, g.name)


def _ary_tree(n, k):
    return G.Graph(n, [(v, (v - 1) // k) for v in range(1, n)])


@pytest.mark.gpu
@pytest.mark.parametrize("kind", [0, 2])
@pytest.mark.parametrize("n", [31, 32, 64, 104])
def test_gpu_variance_scores_that_tie_and_leave_many_parts(handle, kind, n):
    """Parts in numbers that are powers of two (integer order) and not (double
    order), more of them than a thread keeps, equal ones under other labels."""
    rng = np.random.default_rng(n)
    gs = [_ary_tree(n, k) for k in (2, 3, 4, 5, 7, 8)]
    gs += [G.Graph(n, [(v, v // 3 * 3) for v in range(n) if v % 3] + [(v, v + 3) for v in range(0, n - 3, 3)])]
    gs += [G.relabel(g, rng.permutation(n).tolist()) for g in list(gs) for _ in range(3)]
    gs += [G.tree_plus_edges(n, k, k) for k in (0, 1, 3)]
    td, pars = handle.heuristic_batch(gs, kind)
    for i, g in enumerate(gs):
        htd, hpar = _lib.heuristic(g, kind)
        assert td[i] == htd and pars[i].tolist() == hpar.tolist(), i


@pytest.mark.gpu
@pytest.mark.parametrize("kind", [0, 1, 2, 3])
@pytest.mark.parametrize("n", [7, 32, 33, 70, 128])
def test_gpu_heuristics_on_masks_that_are_not_symmetric_equal_host(handle, kind, n):
    """Edges kept in one of the two masks, next to ordinary graphs: the batch
    takes them as the host function does, with the same trees."""
    import ctypes
    rng = np.random.default_rng(100 * kind + n)
    masks = []
    for k in range(12):
        a = rng.random((n, n)) < (2.0 + k % 3) / n
        np.fill_diagonal(a, False)
        if k % 4 == 0:
            a |= a.T
        elif k % 4 == 1:  # a single edge of an ordinary graph lacks its other direction
            a |= a.T
            u, v = np.argwhere(a)[rng.integers(int(a.sum()))] if a.any() else (0, 1)
            a[u, v], a[v, u] = True, False
        masks.append([sum(1 << int(u) for u in np.flatnonzero(row)) for row in a])
    pool = np.array([w for m in masks for x in m for w in (x & (1 << 64) - 1, x >> 64)], dtype=np.uint64)
    scores = rng.random(n * len(masks)).astype(np.float32)
    descs = (_lib.GraphDesc * len(masks))()
    for i in range(len(masks)):
        descs[i].n, descs[i].offset = n, i * n
    td = np.zeros(len(masks), dtype=np.int32)
    par = np.zeros(n * len(masks), dtype=np.int32)
    handle.heuristic_batch([G.path(3)], 1)  # binds the entry point
    L, p = handle.L, _lib._ptr
    sc = p(scores) if kind == 3 else None
    assert L.gtd_heuristic_batch(handle._h, ctypes.cast(descs, ctypes.c_void_p), len(masks), p(pool), n * len(masks),
                                 kind, sc, p(td), p(par)) == 0
    _lib.heuristic(G.path(3))
    for i in range(len(masks)):
        t, q = ctypes.c_int32(), np.zeros(n, dtype=np.int32)
        own, s = pool[2 * n * i:2 * n * (i + 1)].copy(), scores[n * i:n * (i + 1)].copy()
        assert L.gtd_heuristic(p(own), n, kind, p(s), ctypes.byref(t), p(q)) == 0
        assert td[i] == t.value and par[n * i:n * (i + 1)].tolist() == q.tolist(), i
