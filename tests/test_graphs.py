"""Generators and the reference's text format."""
import numpy as np
import pytest

from gisbdw_gb300 import graphs as G


def test_generators_deterministic():
    a = G.config1_graph()
    b = G.config1_graph()
    assert a.edges == b.edges and a.n == 20 and a.is_connected()
    c4a = G.config4_graphs(count=6)
    c4b = G.config4_graphs(count=6)
    assert [g.edges for g in c4a] == [g.edges for g in c4b]
    for g in c4a:
        assert 40 <= g.n <= 64 and g.is_connected()
        assert 2.5 <= 2 * g.m / g.n <= 5.5


def test_config_families_connected():
    for g in G.config3_graphs(count=30):
        assert 10 <= g.n <= 24 and g.is_connected()
    for g in G.config2_graphs():
        assert g.n in (28, 30, 32) and g.is_connected()
    for g in G.config5_graphs(count=12):
        assert 20 <= g.n <= 80 and g.is_connected()


def test_text_roundtrip():
    g = G.chordal_cycle(12)
    h = G.from_text(G.to_text(g))
    assert h.n == g.n and h.edges == g.edges


def test_text_vertex_count_grows_with_edges():
    # the reference's vecS graph grows on add_edge (main.cpp:138-143)
    h = G.from_text("graph G {\n0;\n1;\n0 -- 1;\n1 -- 4;\n}\n")
    assert h.n == 5 and h.edges == [(0, 1), (1, 4)]


def test_masks():
    g = G.grid(3, 3)
    adj = g.adj64()
    assert all(((int(adj[v]) >> v) & 1) == 0 for v in range(9))
    a2 = g.adj128()
    assert np.all(a2[0::2] == adj) and np.all(a2[1::2] == 0)


def test_adjacency_pool_equals_the_per_graph_masks():
    """The native packer against adj64 / adj128, and its way out: anything but
    pairs of plain integers in range takes the per-graph path."""
    from gisbdw_gb300 import _lib
    gs = [G.Graph(1, []), G.path(2), G.complete(64), G.grid(4, 5), G.Graph(3, [])]
    assert np.array_equal(_lib.adjacency_pool(gs, 1), np.concatenate([g.adj64() for g in gs]))
    wide = gs + [G.cycle(65), G.complete(128), G.star(127)]
    assert np.array_equal(_lib.adjacency_pool(wide, 2), np.concatenate([g.adj128() for g in wide]))
    assert _lib.adjacency_pool([], 2).size == 0
    odd = G.path(5)
    odd.edges = [(np.int64(0), 1), [2, 3]]  # not tuples of int
    assert np.array_equal(_lib.adjacency_pool([G.path(3), odd], 1),
                          np.concatenate([G.path(3).adj64(), odd.adj64()]))
    bad = G.path(4)
    bad.edges = [(0, 7)]
    with pytest.raises(IndexError):
        _lib.adjacency_pool([bad], 1)
    with pytest.raises(ValueError):
        _lib.adjacency_pool([G.path(65)], 1)


@pytest.mark.parametrize("words", [1, 2])
def test_small_batches_are_packed_as_fast_as_graph_by_graph(words):
    """The native pass costs several times what a few small graphs take; the
    masks are the same on either side of the rule."""
    import timeit

    from gisbdw_gb300 import _lib

    def per_graph(gs):
        return np.concatenate([g.adj64() if words == 1 else g.adj128() for g in gs])
    for n in range(1, 40):
        for gs in ([G.path(n)], [G.complete(n)], [G.path(n), G.Graph(1, []), G.cycle(max(n, 3))]):
            assert np.array_equal(_lib.adjacency_pool(gs, words), per_graph(gs))

    def best(f):
        return min(timeit.repeat(f, number=200, repeat=9))
    for gs in ([G.path(5)], [G.Graph(1, []), G.path(4)]):
        assert best(lambda: _lib.adjacency_pool(gs, words)) < 2.5 * best(lambda: per_graph(gs))
