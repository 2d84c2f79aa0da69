"""CPU checks of the bit-sliced subset DP (gtd_dp.cu): treedepths kept modulo
3 in two bit planes and connectivity in a third, 32 subsets per word.

* A subset's children S - v have treedepth td(S) - 1 or td(S), so the
  residues present among them name both values, and
  td(S) = 1 + min (connected) or max (disconnected) follows modulo 3.
* Four tiles are resolved together: a byte transpose leaves the three lowest
  vertices inside a byte, resolved by subset size in four rounds (position 0,
  its broadcast, one shift per vertex, position 7), and the four bytes of a
  word one after another.
* Treedepths are read back along a chain of vertex deletions.
* A tile's child tiles are ranked while its high part is unranked.

The kernel's word arithmetic is restated here and checked against the
oracle's tables (dynamic_cpu.hpp / dynamic_gpu.cu:68-111); the GPU test runs
the kernel at the edges of its tiles and groups."""
from math import comb

import numpy as np
import pytest

from gisbdw_gb300 import graphs as G
from gisbdw_gb300.validate import check_tree

M32 = 0xFFFFFFFF
SINGLES = 0x10116            # positions with one of the five bits
ONES, PAIRS, TOP = 0x01010101, 0x68686868, 0x80808080
HAS = [0xAAAAAAAA, 0xCCCCCCCC, 0xF0F0F0F0]


def resolve(o, conn):
    """Residue planes from the residues present among the children."""
    def plane(k):
        prev, nxt = o[(k + 2) % 3], o[(k + 1) % 3]
        return ~nxt & ((conn & prev) | (~conn & o[k])) & M32
    return plane(0), plane(1)


def spread(a):
    return (a & 1) << 1 | (a & 2) << 1 | (a & 4) << 2 | (a & 8) << 5 | (a & 16) << 12


def small_masks(adj, n, verts):
    """(keep, set, zero) of a word whose position 0 is the set `verts` of at
    most two vertices >= 5: connectivity of its subsets of size <= 2."""
    at = lambda v: adj[v] if v < n else 0  # noqa: E731
    if len(verts) == 2:
        return M32 ^ 1, at(verts[0]) >> verts[1] & 1, 0
    if len(verts) == 1:
        return M32 ^ (1 | SINGLES), 1 | spread(at(verts[0]) & 31), 0
    pairs = sum(1 << x for x in range(32) if bin(x).count("1") == 2)
    s = SINGLES
    for i in range(1, 5):
        s |= spread(at(i) & ((1 << i) - 1)) << (1 << i)
    return M32 ^ (1 | SINGLES | pairs), s, 1


def maj(x, y, z):
    return (x & y) | (x & z) | (y & z)


def resolve_octets(o, c1, c2, keep, forced, zero):
    """Planes (td % 3 == 0, td % 3 == 1, connected) of four sets of 8 subsets
    from what their other children have: residues o[0..2], at least one
    connected child c1, at least two c2."""
    def finish(acc, two):
        conn = (two & keep) | forced
        p0, p1 = resolve(acc, conn)
        return p0 | zero, p1, conn

    def three(p0, p1):
        return p0, p1, ~(p0 | p1) & M32
    p0, p1, c = finish(o, c2)
    b = lambda x: (x & ONES) * 0x16  # noqa: E731
    p0, p1, c = finish([o[k] | b(x) for k, x in enumerate(three(p0, p1))], c2 | (c1 & b(c)))
    acc = list(o)
    for k, x in enumerate(three(p0, p1)):
        for i in range(3):
            acc[k] |= (x << (1 << i)) & HAS[i]
    x, y, z = ((c << (1 << i)) & HAS[i] for i in range(3))
    p0, p1, c = finish(acc, c2 | maj(x, y, z) | (c1 & (x | y | z)))
    acc = [o[k] | (((x & PAIRS) + 0x78787878) & TOP) for k, x in enumerate(three(p0, p1))]
    x, y, z = c << 4, c << 2, c << 1
    q0, q1, qc = finish(acc, c2 | ((maj(x, y, z) | (c1 & (x | y | z))) & TOP))
    return [(u & ~TOP & M32) | (v & TOP) for u, v in ((p0, q0), (p1, q1), (c, qc))]


def byte_perm(x, y, sel):
    b = [(x >> (8 * i)) & 0xFF for i in range(4)] + [(y >> (8 * i)) & 0xFF for i in range(4)]
    return sum(b[(sel >> (4 * i)) & 7] << (8 * i) for i in range(4))


def transpose_bytes(x):
    a, b = byte_perm(x[0], x[1], 0x5140), byte_perm(x[2], x[3], 0x5140)
    c, d = byte_perm(x[0], x[1], 0x7362), byte_perm(x[2], x[3], 0x7362)
    return [byte_perm(a, b, 0x5410), byte_perm(a, b, 0x7632), byte_perm(c, d, 0x5410), byte_perm(c, d, 0x7632)]


def resolve_quad(words):
    """Planes of the words of four tiles, each given as (o, c1, c2, small)."""
    cols = [transpose_bytes(list(col)) for col in
            zip(*([*o, c1, c2, *small] for o, c1, c2, small in words))]
    r = []
    for t in range(4):
        o, c1, c2, small = [cols[k][t] for k in range(3)], cols[3][t], cols[4][t], [cols[k][t] for k in (5, 6, 7)]
        for child in [x for x in (t & 1, t & 2) if x]:
            p0, p1, c = r[t ^ child]
            o = [o[0] | p0, o[1] | p1, o[2] | (~(p0 | p1) & M32)]
            c2 |= c1 & c
            c1 |= c
        r.append(resolve_octets(o, c1, c2, *small))
    return list(zip(*(transpose_bytes(list(col)) for col in zip(*r))))


ANY = (M32, 0, 0)


def plane_dp(g, lb):
    """Planes of every word (S >> 5): tiles of 2^lb subsets, four tiles of a
    level at a time."""
    n = max(g.n, lb)
    adj = g.adjacency_masks()
    planes = {}
    words = 1 << (lb - 5)
    for j in range(n - lb + 1):
        level = [H for H in range(1 << (n - lb)) if bin(H).count("1") == j]
        for quad in (level[i:i + 4] for i in range(0, len(level), 4)):
            for w in sorted(range(words), key=lambda x: (bin(x).count("1"), x)):
                given = []
                for H in quad:
                    W = H * words | w
                    o, c1, c2 = [0, 0, 0], 0, 0
                    verts = [v for v in range(n - 5) if W >> v & 1]
                    for v in verts:
                        p0, p1, c = planes[W ^ (1 << v)]
                        o = [o[0] | p0, o[1] | p1, o[2] | (~(p0 | p1) & M32)]
                        c2 |= c1 & c
                        c1 |= c
                    small = small_masks(adj, g.n, [v + 5 for v in verts]) if len(verts) <= 2 else ANY
                    given.append((o, c1, c2, small))
                given += [given[0]] * (4 - len(given))
                for H, r in zip(quad, resolve_quad(given)):
                    planes[H * words | w] = r
    return planes, n


def residue(planes, S):
    p0, p1, _ = planes[S >> 5]
    return 0 if p0 >> (S & 31) & 1 else 1 if p1 >> (S & 31) & 1 else 2


def treedepth(planes, S):
    td = 0
    while S:
        td += (residue(planes, S) - residue(planes, S & (S - 1))) % 3
        S &= S - 1
    return td


def connected(g, S):
    adj, reach, front = g.adjacency_masks(), S & -S, S & -S
    while front:
        nb = 0
        for v in range(g.n):
            if front >> v & 1:
                nb |= adj[v]
        front = nb & S & ~reach
        reach |= front
    return reach == S


GRAPHS = [G.gnp_connected(9, 0.3, 1), G.gnp_connected(10, 0.5, 2), G.grid(2, 5), G.complete(9), G.path(10),
          G.star(7), G.path(3), G.Graph(10, [(0, 1), (2, 3), (3, 4), (6, 7), (7, 8), (8, 6)], name="forest10"),
          G.Graph(8, [], name="empty8")]


@pytest.mark.parametrize("g", GRAPHS, ids=lambda g: g.name)
def test_planes_match_oracle(port, g):
    planes, n = plane_dp(g, 8)
    T = port.dp_table(g)
    for S in range(1 << g.n):
        assert treedepth(planes, S) == T[S], (g.name, S)
        if S:
            assert planes[S >> 5][2] >> (S & 31) & 1 == connected(g, S), (g.name, S)


def test_child_ranks_while_unranking():
    def rank(H):
        return sum(comb(v, i + 1) for i, v in enumerate(v for v in range(12) if H >> v & 1))
    for nh in range(0, 10):
        for j in range(nh + 1):
            for r in range(comb(nh, j)):
                rest, k, shifted, H, kids = r, j, 0, 0, {}
                for a in range(nh - 1, -1, -1):
                    if k > 0 and rest >= comb(a, k):
                        rest -= comb(a, k)
                        H |= 1 << a
                        kids[a] = rest + shifted
                        shifted += comb(a, k - 1)
                        k -= 1
                assert rest == 0 and bin(H).count("1") == j and rank(H) == r
                assert kids == {a: rank(H ^ (1 << a)) for a in kids}


@pytest.mark.gpu
@pytest.mark.parametrize("tile_bits", [0, 8, 9, 10, 11, 12])  # 0: the level kernel
@pytest.mark.parametrize("n", [2, 4, 7, 8, 9, 12, 13, 16, 18])
def test_kernel_at_tile_edges_matches_oracle(handle, port, tile_bits, n):
    """Padded tiles (n < 8), one tile, one to a few tiles per level, levels of
    just under and over a group or chunk: every byte of the table, the tree,
    the order."""
    from gisbdw_gb300 import _lib
    for g in (G.gnp(n, 0.35, 40 + n), G.path(n), G.complete(n)):
        td, parent, order, _ = handle.dp_solve(g.adj64(), n, tile_bits=tile_bits)
        T = port.dp_table(g)
        otd, opar = port.tree_from_table(g, T)
        assert (td, parent.tolist()) == (otd, opar.tolist()), g.name
        assert sorted(order.tolist()) == list(range(n))
        raw, tn, lb = handle.dp_read_table()
        assert tn == n and lb == min(n, tile_bits or 10)
        S = np.arange(1 << n, dtype=np.int64)
        tile = np.array([_lib.table_index(n, lb, int(h) << lb) >> lb for h in range(1 << (n - lb))], dtype=np.int64)
        tab = raw[(tile[S >> lb] << lb) | (S & ((1 << lb) - 1))]
        assert np.array_equal(tab >> 1, T), g.name
        for s in (1, (1 << n) - 1, 3, 5 % (1 << n), (1 << n) - 2):
            assert tab[s] & 1 == connected(g, s), (g.name, s)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [2, 3, 12, 18, 19, 31, 32])
def test_tree_of_deep_wide_and_forest_shaped_graphs(handle, port, n):
    # one warp, a vertex per lane: all lanes in use, one component per depth
    # (complete), many (path, star), none but single vertices, and a forest
    gs = [G.path(n), G.star(n), G.Graph(n, [])]
    gs += [G.complete(n)] if n <= 19 else []
    gs += [G.Graph(n, [(v, v + 2) for v in range(n - 2)]), G.relabel(G.path(n), list(reversed(range(n))))]
    for g in gs:
        otd, oparent = (port.dp_solve(g) if n <= 19 else (None, None))
        td, parent, order, _ = handle.dp_solve(g.adj64(), n)
        if otd is not None:
            assert td == otd and parent.tolist() == oparent.tolist(), (n, g.edges[:3])
        assert check_tree(g, td, parent, allow_forest=True) and sorted(order.tolist()) == list(range(n))
        # the order removes a root only after every vertex above it
        place = {v: i for i, v in enumerate(order.tolist())}
        assert all(parent[v] < 0 or place[parent[v]] < place[v] for v in range(n))


@pytest.mark.gpu
@pytest.mark.parametrize("n", [16, 17, 18, 20, 21, 22])
def test_cluster_kernel_equals_the_tile_kernel(handle, n):
    # 17..21: words over 16 CTAs by their top bits; one vertex less and more on
    # either side. Whole tables, trees, orders and queries.
    for g in (G.gnp_connected(n, 0.25, n), G.grid(2, n // 2), G.Graph(n, [(v, v + 3) for v in range(n - 3)])):
        adj = np.zeros(n, dtype=np.uint64)
        adj[:g.n] = g.adj64()
        a = handle.dp_solve(adj, n, tile_bits=10)
        table, query = handle.dp_read_table()[0], handle.dp_query((1 << n) - 6)
        b = handle.dp_solve(adj, n)
        assert a[0] == b[0] and a[1].tolist() == b[1].tolist() and a[2].tolist() == b[2].tolist()
        assert np.array_equal(table, handle.dp_read_table()[0]) and query == handle.dp_query((1 << n) - 6)
