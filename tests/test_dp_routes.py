"""Which kernel a subset-DP call takes, by the number of CTAs that its
statistics report, and each of them against the oracle. A poisoned solve
(gtd_inject_fault) whose caller names tile bits runs the tile kernel whatever
the sizes, so the tile kernel's edges are tested that way."""
import numpy as np
import pytest

from gisbdw_gb300 import Handle, _lib
from gisbdw_gb300 import graphs as G

pytestmark = pytest.mark.gpu


class poisoned:
    def __init__(self, count=1):
        self.count = count

    def __enter__(self):
        _lib.inject_fault(_lib.FAULT_POISON, self.count)

    def __exit__(self, *exc):
        _lib.inject_fault(_lib.FAULT_NONE, 0)


def natural_order(raw, n, lb):
    """The byte table by subset mask."""
    S = np.arange(1 << n, dtype=np.int64)
    tile = np.array([_lib.table_index(n, lb, h << lb) >> lb for h in range(1 << (n - lb))], dtype=np.int64)
    return raw[(tile[S >> lb] << lb) | (S & ((1 << lb) - 1))]


def same(got, want):
    (td, parents), gs = got, want
    for g, t, par in zip(gs, td, parents):
        otd, opar = ORACLE(g)
        assert t == otd and par.tolist() == list(opar), g.name


ORACLE = None


@pytest.fixture(autouse=True)
def _oracle(port):
    global ORACLE
    known = {}

    def solve(g):
        key = (g.n, tuple(g.edges))
        if key not in known:
            known[key] = port.dp_solve(g)
        return known[key]
    ORACLE = solve


@pytest.mark.parametrize("n", [9, 16, 18, 20, 22, 24])
@pytest.mark.parametrize("tile_bits", [8, 9, 10, 12])
def test_given_tile_bits_take_the_kernels_of_the_default(handle, port, n, tile_bits):
    g = G.gnp_connected(n, 0.3, n)
    ctas = handle.dp_solve(g.adj64(), n)[3]["ctas"]
    td, parent, _, stats = handle.dp_solve(g.adj64(), n, tile_bits=tile_bits)
    assert stats["ctas"] == ctas and stats["tile_bits"] == min(n, tile_bits)
    raw, tn, lb = handle.dp_read_table()
    assert (tn, lb) == (n, min(n, tile_bits))
    if n <= 20:
        T = port.dp_table(g)
        assert np.array_equal(natural_order(raw, n, lb) >> 1, T)
        otd, opar = port.tree_from_table(g, T)
        assert (td, parent.tolist()) == (otd, opar.tolist())


@pytest.mark.parametrize("tile_bits", [8, 9, 10, 11, 12])
@pytest.mark.parametrize("n", [2, 4, 7, 8, 9, 12, 13, 16, 18])
def test_tile_kernel_at_tile_edges_matches_oracle(handle, port, tile_bits, n):
    """Padded tiles (n < 8), one tile, one to a few tiles per level, levels of
    just under and over a group: every byte, the tree, the order."""
    for g in (G.gnp(n, 0.35, 40 + n), G.path(n), G.complete(n)):
        with poisoned():
            td, parent, order, _ = handle.dp_solve(g.adj64(), n, tile_bits=tile_bits)
        T = port.dp_table(g)
        otd, opar = port.tree_from_table(g, T)
        assert (td, parent.tolist()) == (otd, opar.tolist()), g.name
        assert sorted(order.tolist()) == list(range(n))
        raw, tn, lb = handle.dp_read_table()
        assert tn == n and lb == min(n, tile_bits)
        assert np.array_equal(natural_order(raw, n, lb) >> 1, T), g.name


@pytest.mark.parametrize("n", [17, 20, 21, 22, 24])
def test_cluster_and_level_kernels_equal_the_tile_kernel(handle, n):
    """Whole tables, trees, orders and queries."""
    for g in (G.gnp_connected(n, 0.25, n), G.grid(2, n // 2), G.Graph(n, [(v, v + 3) for v in range(n - 3)])):
        adj = np.zeros(n, dtype=np.uint64)
        adj[:g.n] = g.adj64()
        with poisoned():
            a = handle.dp_solve(adj, n, tile_bits=10)
        table, query = handle.dp_read_table()[0], handle.dp_query((1 << n) - 6)
        b = handle.dp_solve(adj, n)
        assert a[3]["ctas"] != b[3]["ctas"]
        assert a[0] == b[0] and a[1].tolist() == b[1].tolist() and a[2].tolist() == b[2].tolist()
        assert np.array_equal(table, handle.dp_read_table()[0]) and query == handle.dp_query((1 << n) - 6)


@pytest.mark.parametrize("tile_bits", [8, 10, 12])
@pytest.mark.parametrize("sizes", [[20, 20], [17, 24, 3, 16, 20, 1, 18], [9, 12, 16] * 20])
def test_batches_with_given_tile_bits_take_the_kernels_of_the_default(handle, tile_bits, sizes):
    gs = [G.gnp_connected(n, 0.3, 10 + n) if n > 1 else G.Graph(1, []) for n in sizes]
    ctas = handle.dp_solve_batch(gs)[2]["ctas"]
    td, parents, stats = handle.dp_solve_batch(gs, tile_bits=tile_bits)
    assert stats["ctas"] == ctas and stats["tile_bits"] == tile_bits
    same((td, parents), gs)


@pytest.mark.parametrize("tile_bits", [8, 9, 10, 11, 12])
def test_tile_kernel_batches_match_oracle(handle, tile_bits):
    """Graphs of every size, smaller than a tile as well, in the tile kernel:
    a first call, a replay with other contents and a call without a graph."""
    sizes = [1, 2, 5, 8, 9, 10, 11, 13, 16, 17, 18, 20, 21] * 2
    default = handle.dp_solve_batch([G.gnp(n, 0.3, n) for n in sizes])[2]["ctas"]
    for call, (seed, use_graph) in enumerate(((1, True), (2, True), (3, False))):
        gs = [G.gnp(n, 0.3, 100 * seed + i % 13) for i, n in enumerate(sizes)]
        with poisoned():
            td, parents, stats = handle.dp_solve_batch(gs, tile_bits=tile_bits, use_cuda_graph=use_graph)
        assert stats["graph_replayed"] == int(call == 1) and stats["ctas"] != default
        same((td, parents), gs)


def _rated(choice, n_min=2, n_max=28, eff=1.0):
    """A handle with rates that favour choice(n) tile bits."""
    h = Handle(0)
    r = np.ones((n_max - n_min + 1, 5), dtype=np.float32)
    for n in range(n_min, n_max + 1):
        r[n - n_min, choice(n) - 8] = 1e4
    h.dp_set_rates(n_min, r, mixed_eff=np.full(5, eff))
    return h


@pytest.mark.parametrize("sizes", [[20, 20], [17, 24, 3, 16, 20, 18], [17, 18, 19, 20, 21] * 8, [9, 12, 16] * 20])
def test_rated_handles_take_the_kernels_of_the_others(handle, sizes):
    """Batches of few subsets: with rates as without them."""
    gs = [G.gnp_connected(n, 0.3, 30 + n) for n in sizes]
    ctas = handle.dp_solve_batch(gs)[2]["ctas"]
    with _rated(lambda n: 9 + n % 3) as h:
        td, parents, stats = h.dp_solve_batch(gs)
        assert stats["ctas"] == ctas
        assert stats["tile_bits_by_n"] == {n: 9 + n % 3 for n in set(sizes)} or len(set(sizes)) == 1
        same((td, parents), gs)


@pytest.mark.parametrize("choice", [lambda n: 8 if n <= 16 else 12, lambda n: 9 + n % 3, lambda n: 11 if n >= 20 else 10])
def test_mixed_tile_kernel_matches_oracle(handle, choice):
    """The mixed-size tile kernel on graphs of every size: a first call and a
    replay with other contents."""
    sizes = [2, 5, 8, 9, 10, 11, 13, 16, 17, 18, 20, 21] * 2
    default = handle.dp_solve_batch([G.gnp(n, 0.3, n) for n in sizes])[2]["ctas"]
    with _rated(choice) as h:
        for call in range(2):
            gs = [G.gnp(n, 0.3, 100 * call + i % 12) for i, n in enumerate(sizes)]
            with poisoned():
                td, parents, stats = h.dp_solve_batch(gs)
            assert stats["tile_bits_by_n"] == {n: choice(n) for n in sizes}
            assert stats["graph_replayed"] == call and stats["ctas"] != default
            same((td, parents), gs)


def test_rates_of_small_graphs_are_not_asked_for(handle):
    """More subsets than the level kernel takes: the rates of the graphs in the
    tile kernel choose its tile size, with or without rates of the others."""
    gs = [G.gnp_connected(24, 0.2, i % 3) for i in range(40)] + [G.gnp_connected(10, 0.3, 1)]

    def solve(h, **kw):  # treedepths, least device time of eight
        runs = [h.dp_solve_batch(gs, **kw) for _ in range(8)]
        return runs[0][0].tolist(), min(r[2]["dp_ms"] for r in runs)
    td8, t8 = solve(handle, tile_bits=8)
    td10, t10 = solve(handle)
    with _rated(lambda n: 8, n_min=17) as h:
        td, t = solve(h)
    assert td == td8 == td10
    # 8-bit tiles take a quarter more time here: which of the two sizes ran
    assert t8 > 1.1 * t10 and t > (t8 + t10) / 2, (t8, t10, t)


@pytest.mark.parametrize("n,tile_bits", [(2, 0), (8, 0), (20, 10), (26, 0), (27, 8), (28, 12)])
def test_table_is_read_in_pieces_where_there_is_no_room_for_it(n, tile_bits):
    """The allocation of the byte table fails: gtd_dp_read_table still gives
    every byte (27 and 28 vertices: two and four pieces), gtd_dp_table GTD_OOM."""
    g = G.gnp(n, 0.2, n)
    with Handle(0) as h:
        h.dp_solve(g.adj64(), n, tile_bits=tile_bits)
        _lib.inject_fault(_lib.FAULT_ALLOC, 1)
        try:
            with pytest.raises(_lib.GtdError) as e:
                h.dp_table_info()
            assert e.value.status == 3
            _lib.inject_fault(_lib.FAULT_ALLOC, 1)
            pieces = h.dp_read_table()
        finally:
            _lib.inject_fault(_lib.FAULT_NONE, 0)
        whole = h.dp_read_table()
        assert pieces[1:] == whole[1:] and np.array_equal(pieces[0], whole[0])
