"""The learned ordering: the numpy FP64 reference network (CPU), the GPU
forward / backward kernels against it (gradient check), training on DP
labels, and what the trained network gains over branching without it."""
import numpy as np
import pytest

from gisbdw_gb300 import gnn
from gisbdw_gb300 import graphs as G
from gisbdw_gb300.validate import check_tree


def _toy_batch(seed=0):
    rng = np.random.default_rng(seed)
    gs = [G.gnp_connected(n, 0.35, s) for n, s in ((7, 1), (9, 2), (6, 3))] + [G.path(5), G.star(6)]
    roots = [(rng.random(g.n) < 0.3).astype(np.float32) for g in gs]
    return gs, gnn.make_batch(gs, roots=roots, tds=[3, 4, 3, 3, 2])


def test_reference_gradient_matches_finite_differences():
    _, b = _toy_batch()
    shape = (gnn.IN_FEATURES, 8, 2)
    npar = shape[0] * 8 + 8 + 2 * (2 * 64 + 8) + 2 * 8 + 2
    rng = np.random.default_rng(1)
    # parameters exactly representable in BF16, so rounding does not move them
    p = gnn.bf16_round((rng.standard_normal(npar) * 0.3).astype(np.float32)).astype(np.float32)
    loss, grad = gnn.reference_loss(p, b, shape)
    for i in rng.choice(npar, 25, replace=False):
        e = np.zeros(npar)
        e[i] = 2.0 ** -6
        lp = gnn.reference_loss((p + e).astype(np.float32), b, shape, want_grad=True)[0]
        lm = gnn.reference_loss((p - e).astype(np.float32), b, shape, want_grad=True)[0]
        assert abs((lp - lm) / (2 * e[i]) - grad[i]) < 2e-3 + 0.02 * abs(grad[i]), i


def test_features_shape_and_values():
    g = G.star(5)
    f = gnn.features(g)
    assert f.shape == (5, gnn.IN_FEATURES)
    assert f[0, 0] == 1.0 and f[1, 0] == 0.25  # degree / 4
    assert f[1, 4] == 1.0 and f[0, 4] == 0.0   # pendant flag


def test_native_features_and_pack_match_python():
    gs = [G.gnp(n, 0.3, s) for n, s in ((12, 1), (20, 2), (9, 3))] + [G.grid(4, 5), G.random_regular3(70, 4)]
    for g in gs:
        np.testing.assert_allclose(gnn.native_features(g), gnn.features(g), rtol=1e-6, atol=1e-7)
    b = gnn.make_batch(gs)
    assert b.graph_start.tolist() == np.cumsum([0] + [g.n for g in gs]).tolist()
    base = 0
    for g in gs:
        adj = g.adjacency_masks()
        for v in range(g.n):
            got = b.nbr[b.nbr_start[base + v]:b.nbr_start[base + v + 1]].tolist()
            assert got == [base + u for u in range(g.n) if adj[v] >> u & 1]
        base += g.n


def test_label_set_batch_gather_matches_pack():
    gs = [G.gnp_connected(n, 0.3, s) for n, s in ((8, 1), (12, 2), (10, 3), (15, 4))]
    ns = np.array([g.n for g in gs])
    offs = np.concatenate([[0], np.cumsum(ns)[:-1]])
    adj2 = np.concatenate([g.adj128() for g in gs]).astype(np.uint64)
    data = gnn.LabelSet(adj2, ns, offs, np.array([5, 3, 9, 1], dtype=np.uint64), np.array([3, 4, 4, 5], dtype=np.int32))
    for idx in ([2, 0], [3, 1, 2], [1]):
        b, ref = data.batch(idx), gnn.make_batch([gs[i] for i in idx])
        for name in ("x", "graph_start", "nbr_start", "nbr"):
            assert np.array_equal(getattr(b, name), getattr(ref, name)), name
        y = np.concatenate([[(int(data.roots[i]) >> v) & 1 for v in range(gs[i].n)] for i in idx])
        assert np.array_equal(b.root_label, y.astype(np.float32))
        assert b.td_label.tolist() == [float(data.td[i]) for i in idx]


@pytest.mark.gpu
def test_gpu_forward_and_gradients_match_reference(handle):
    _, b = _toy_batch(3)
    net = gnn.GNN(handle, seed=7)
    p = net.params()
    logits, td = net.forward(b)
    rl, rtd = gnn.reference_loss(p, b, want_grad=False)
    np.testing.assert_allclose(logits, rl, rtol=1e-4, atol=1e-4)
    np.testing.assert_allclose(td, rtd, rtol=1e-4, atol=1e-4)
    grad, loss = net.gradients(b)
    rloss, rgrad = gnn.reference_loss(p, b)
    assert abs(loss - rloss) < 1e-4 * max(1.0, abs(rloss))
    # FP32 accumulation in a different order than the FP64 reference
    np.testing.assert_allclose(grad, rgrad, rtol=2e-3, atol=2e-5)


@pytest.mark.gpu
def test_training_is_deterministic(handle):
    """Weight gradients are summed in a fixed order (no float atomics), so
    the same seed and batches give bit-identical parameters."""
    gs, b = _toy_batch(4)
    big = gnn.make_batch(G.config3_graphs(count=300, seed=4))  # > 64 nodes: several gradient chunks
    big.root_label = (np.arange(len(big.x)) % 3 == 0).astype(np.float32)
    big.node_mask = np.ones(len(big.x), dtype=np.float32)
    big.td_label = np.full(len(big.graph_start) - 1, 5.0, dtype=np.float32)
    nets = [gnn.GNN(handle, seed=11) for _ in range(2)]
    for net in nets:
        for _ in range(3):
            net.train_step(b)
            net.train_step(big)
    assert np.array_equal(nets[0].params(), nets[1].params())


@pytest.mark.gpu
def test_label_set_matches_oracle(handle, port):
    base = G.config3_graphs(count=6, seed=23)
    data = gnn.label_set(handle, base, per_graph=12, seed=3)
    assert len(data) >= 6 and np.all(data.ns >= 2)
    for i in range(len(data)):
        g = data.graph(i)
        assert g.is_connected()
        T = port.dp_table(g)
        full = (1 << g.n) - 1
        td = int(T[full])  # the oracle's table holds td per subset
        assert data.td[i] == td
        roots = sum(1 << v for v in range(g.n) if int(T[full & ~(1 << v)]) == td - 1)
        assert int(data.roots[i]) == roots


@pytest.mark.gpu
def test_family_label_set_matches_oracle(handle, port):
    """The larger in-family labels (gnn.family_label_set): every relabelled
    subgraph is connected, and its treedepth and optimal-root mask are the
    oracle's."""
    graphs = gnn.family_graphs(8, seed=5, n_min=14, n_max=18)
    data = gnn.family_label_set(handle, graphs, per_graph=6, seed=4, drop=6)
    assert len(data) == 8 * 7
    for i in range(len(data)):
        g = data.graph(i)
        assert g.is_connected()
        T = port.dp_table(g)
        full = (1 << g.n) - 1
        td = int(T[full])
        assert data.td[i] == td
        assert int(data.roots[i]) == sum(1 << v for v in range(g.n) if int(T[full & ~(1 << v)]) == td - 1)


@pytest.mark.gpu
def test_training_on_dp_labels_learns_roots(handle):
    base = G.config3_graphs(count=60, seed=21)
    samples = gnn.label_set(handle, base, per_graph=20, seed=1)
    assert len(samples) > 600
    train_s, test_s = samples.split(0.8)
    net = gnn.GNN(handle, seed=3)
    before = gnn.root_accuracy(net, test_s)
    losses = gnn.train(net, train_s, epochs=6, batch_graphs=128, lr=3e-3)
    after = gnn.root_accuracy(net, test_s)
    assert np.mean(losses[-5:]) < np.mean(losses[:5])
    assert after["top1_root"] > after["uniform_root"] + 0.05
    assert after["top1_root"] >= before["top1_root"]


@pytest.mark.gpu
def test_learned_order_keeps_treedepth_and_cuts_search(handle):
    base = G.config3_graphs(count=80, seed=22)
    samples = gnn.label_set(handle, base, per_graph=15, seed=2)
    net = gnn.GNN(handle, seed=5)
    gnn.train(net, samples, epochs=6, batch_graphs=128, lr=3e-3)
    gs = [g for g in G.config5_graphs(count=40, seed=9) if g.n <= 36][:16]
    plain = handle.bnb_solve_batch(gs, deadline_ns=20 * 10**9)
    orders, seeds = gnn.orders_and_seeds(net, gs)
    learned = handle.bnb_solve_batch(gs, orders=orders, seeds=seeds, deadline_ns=20 * 10**9)
    both = (plain["status"] == 0) & (learned["status"] == 0)
    print("solved plain", int((plain["status"] == 0).sum()), "learned", int((learned["status"] == 0).sum()),
          "both", int(both.sum()), "of", len(gs))
    assert both.sum() >= len(gs) // 3
    assert np.array_equal(plain["td"][both], learned["td"][both])
    for g, t, par in zip(gs, learned["td"], learned["parents"]):
        assert check_tree(g, t, par), g.name
    # per graph: the search's refutation part does not depend on the order,
    # so compare the typical graph, not the total (dominated by a few hard ones)
    ratio = (learned["nodes"][both] + 1.0) / (plain["nodes"][both] + 1.0)
    assert np.median(ratio) < 1.0


def _layerwise(b):
    """The same nodes, neighbours and labels with an empty graph at the end:
    batches with one take the layer-by-layer kernels."""
    return gnn.Batch(b.x, np.append(b.graph_start, b.graph_start[-1]).astype(np.int32), b.nbr_start, b.nbr,
                     b.root_label, b.node_mask, np.append(b.td_label, np.float32(1.0)))


@pytest.mark.gpu
@pytest.mark.parametrize("sizes", [(1,), (32,) * 3, (33, 31, 1), (64, 64), (65, 2, 60), (128, 5), (24,) * 40])
def test_tile_kernels_equal_the_layerwise_kernels(handle, sizes):
    """Tiles just filled, overfull and with padding rows: logits bit for bit,
    estimates and gradients (whose mean over graphs counts the empty graph)
    against float64."""
    rng = np.random.default_rng(len(sizes))
    gs = [G.gnp_connected(n, min(1.0, 3.0 / max(1, n - 1) + 0.1), 7 + i) if n > 1 else G.Graph(1, [])
          for i, n in enumerate(sizes)]
    b = gnn.make_batch(gs, roots=[(rng.random(g.n) < 0.4).astype(np.float32) for g in gs],
                       tds=[3.0] * len(gs))
    net = gnn.GNN(handle, seed=9)
    logits, td = net.forward(b)
    logits2, td2 = net.forward(_layerwise(b))
    assert np.array_equal(logits, logits2) and np.array_equal(td, td2[:-1])
    rlogits, rtd = gnn.reference_loss(net.params(), b, want_grad=False)
    # float32 sums of at most 128 terms per layer, four layers
    np.testing.assert_allclose(logits, rlogits, rtol=2e-4, atol=2e-5)
    np.testing.assert_allclose(td, rtd, rtol=2e-4, atol=2e-5)
    grad, loss = net.gradients(b)
    rloss, rgrad = gnn.reference_loss(net.params(), b)
    assert abs(loss - rloss) < 1e-4 * max(1.0, abs(rloss))
    assert np.linalg.norm(grad - rgrad) < 1e-4 * np.linalg.norm(rgrad)


@pytest.mark.gpu
def test_neighbours_outside_their_graph_take_the_layerwise_kernels(handle):
    """Two graphs joined by an edge of the neighbour lists: one network over
    all nodes, as the reference computes it."""
    _, b = _toy_batch(3)
    n = int(b.graph_start[-1])
    lists = [b.nbr[b.nbr_start[v]:b.nbr_start[v + 1]].tolist() for v in range(n)]
    lists[0].append(n - 1)
    lists[n - 1].append(0)
    c = gnn.Batch(b.x, b.graph_start, np.concatenate([[0], np.cumsum([len(x) for x in lists])]).astype(np.int32),
                  np.array(sum(lists, []), dtype=np.int32), b.root_label, b.node_mask, b.td_label)
    net = gnn.GNN(handle, seed=4)
    logits, td = net.forward(c)
    rlogits, rtd = gnn.reference_loss(net.params(), c, want_grad=False)
    np.testing.assert_allclose(logits, rlogits, rtol=2e-4, atol=2e-5)
    np.testing.assert_allclose(td, rtd, rtol=2e-4, atol=2e-5)


def _joined_singles(count, n, seed, across):
    """A training batch of `count` graphs of n vertices between two single
    vertices of the same features and labels. These are each other's neighbours
    (`across`: the batch takes the layer-by-layer kernels) or each its own (the
    tile kernels), which makes the same network: every sum has the same terms."""
    rng = np.random.default_rng(seed)
    kinds = [G.tree_plus_edges(n, n // 4, seed + i) for i in range(16)]
    one = G.Graph(1, [])
    gs = [one] + [kinds[i % 16] for i in range(count)] + [one]
    roots = [(rng.random(g.n) < 0.4).astype(np.float32) for g in gs]
    roots[-1] = roots[0]
    b = gnn.make_batch(gs, roots=roots, tds=[2.0 + i % 5 for i in range(count + 1)] + [2.0])
    last = int(b.graph_start[-1]) - 1
    ends = (last, 0) if across else (0, last)
    nbr = np.concatenate([[ends[0]], b.nbr[:b.nbr_start[-1]], [ends[1]]]).astype(np.int32)
    start = b.nbr_start + 1
    start[0], start[-1] = 0, len(nbr)
    return gnn.Batch(b.x, b.graph_start, start.astype(np.int32), nbr, b.root_label, b.node_mask, b.td_label)


@pytest.mark.gpu
@pytest.mark.parametrize("count", [1600, 1700, 3400])  # 500, 532 and 1063 chunks of 64 nodes
def test_weight_gradients_of_many_chunks_equal_the_layerwise_kernels(handle, count):
    """Runs of 512 chunks, one to three of them: the sums go on where the run
    before ended, so the bits are those of the layer-by-layer kernels."""
    net = gnn.GNN(handle, seed=2)
    tiles, layers = (net.gradients(_joined_singles(count, 20, 5, across))[0] for across in (False, True))
    assert np.array_equal(tiles, layers)


@pytest.mark.gpu
def test_a_large_training_batch_takes_no_more_memory_than_layer_by_layer():
    import torch

    from gisbdw_gb300 import Handle
    layers, hid = 8, 64
    b = _joined_singles(9000, 24, 1, False)  # 216,002 nodes
    nodes = len(b.x)
    with Handle(0) as h:
        net = gnn.GNN(h, seed=1, layers=layers)
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        net.gradients(b)
        used = before - torch.cuda.mem_get_info()[0]
        net.close()
    # features; Z and h of every layer and the input, the means; dh, dz, da and one more
    assert used < 4 * nodes * (gnn.IN_FEATURES + hid * (2 * (layers + 1) + layers + 4)), used


@pytest.mark.gpu
@pytest.mark.parametrize("where", [0, 2, 5])
@pytest.mark.parametrize("empties", [1, 70])
def test_graphs_without_nodes_count_in_loss_and_gradients(handle, where, empties):
    """Their estimate is the graph head's bias: its gradient and the loss have
    their terms, at the start, between others and at the end (more of them than
    nodes as well), whatever the buffers held before."""
    _, b = _toy_batch(5)
    net = gnn.GNN(handle, seed=6)
    noise = gnn.Batch(b.x * 50, b.graph_start, b.nbr_start, b.nbr, b.root_label, b.node_mask, b.td_label + 500)
    net.gradients(_layerwise(noise))  # other values in the buffers
    c = gnn.Batch(b.x, np.insert(b.graph_start, where, [b.graph_start[where]] * empties).astype(np.int32), b.nbr_start,
                  b.nbr, b.root_label, b.node_mask, np.insert(b.td_label, where, [7.0] * empties).astype(np.float32))
    grad, loss = net.gradients(c)
    with np.errstate(divide="ignore"):
        rloss, rgrad = gnn.reference_loss(net.params(), c)
    assert abs(loss - rloss) < 1e-4 * max(1.0, abs(rloss))
    np.testing.assert_allclose(grad, rgrad, rtol=2e-3, atol=2e-5)


@pytest.mark.gpu
def test_gradients_that_cannot_be_had_leave_the_output_untouched():
    """A batch with a neighbour outside its graph, taken up again layer by
    layer, without room for that: GTD_OOM, and neither array written."""
    import ctypes

    from gisbdw_gb300 import Handle, _lib
    b = _joined_singles(40, 20, 3, True)
    with Handle(0) as h:
        net = gnn.GNN(h, seed=1, layers=1)  # with one layer the second buffer is the larger one
        grad, loss = np.full(net.nparams, 7.0, dtype=np.float32), np.full(1, 7.0, dtype=np.float32)
        cb, p = b.c(), _lib._ptr
        _lib.inject_fault(_lib.FAULT_ALLOC, 2)  # the tile kernels' buffer, then the other's
        try:
            st = h.L.gtd_gnn_gradients(net._g, ctypes.byref(cb), 0.05, p(grad), p(loss))
        finally:
            _lib.inject_fault(_lib.FAULT_NONE, 0)
        assert st == 3 and np.all(grad == 7.0) and loss[0] == 7.0
        assert h.L.gtd_gnn_gradients(net._g, ctypes.byref(cb), 0.05, p(grad), p(loss)) == 0
        assert np.array_equal(grad, net.gradients(b)[0])
        net.close()


@pytest.mark.gpu
def test_a_network_may_outlive_its_handle():
    """Closed in either order, also by the garbage collector: nothing is left
    for a later call to trip over."""
    from gisbdw_gb300 import Handle
    _, b = _toy_batch(2)
    for _ in range(3):
        h = Handle(0)
        net = gnn.GNN(h, seed=1)
        want = net.forward(b)[0]
        h.close()
        others = [Handle(0) for _ in range(4)]  # take the freed memory
        net.close()
        with Handle(0) as h2:
            again = gnn.GNN(h2, seed=1)
            assert np.array_equal(again.forward(b)[0], want)
            again.close()
        for o in others:
            o.close()


@pytest.mark.gpu
@pytest.mark.parametrize("hidden", [8, 32, 63, 64])
def test_layerwise_gradients_match_reference(handle, hidden):
    """The layer-by-layer kernels, which other widths than 64 and neighbours
    outside their graph take."""
    c = _joined_singles(3, 14, 8, True)
    net = gnn.GNN(handle, seed=7, hidden=hidden)
    shape = (gnn.IN_FEATURES, hidden, gnn.LAYERS)
    logits, td = net.forward(c)
    rl, rtd = gnn.reference_loss(net.params(), c, shape, want_grad=False)
    np.testing.assert_allclose(logits, rl, rtol=2e-4, atol=2e-5)
    np.testing.assert_allclose(td, rtd, rtol=2e-4, atol=2e-5)
    grad, loss = net.gradients(c)
    rloss, rgrad = gnn.reference_loss(net.params(), c, shape)
    assert abs(loss - rloss) < 1e-4 * max(1.0, abs(rloss))
    # FP32 accumulation in a different order than the FP64 reference
    np.testing.assert_allclose(grad, rgrad, rtol=2e-3, atol=2e-5)


@pytest.mark.gpu
@pytest.mark.parametrize("count,n", [(1, 2), (5, 32), (3, 64), (4, 128), (70, 20)])
def test_tile_gradients_and_steps_equal_the_layerwise_ones(handle, count, n):
    """The same network by either kernels, bit for bit: gradients, and the
    parameters after three steps. The loss is summed in another order."""
    tiles, layers = (_joined_singles(count, n, 11, across) for across in (False, True))
    nets = [gnn.GNN(handle, seed=12) for _ in range(2)]
    (g0, l0), (g1, l1) = nets[0].gradients(tiles), nets[1].gradients(layers)
    assert np.array_equal(g0, g1) and abs(l0 - l1) < 1e-5 * max(1.0, abs(l0))
    for _ in range(3):
        a, b = nets[0].train_step(tiles), nets[1].train_step(layers)
        assert abs(a - b) < 1e-5 * max(1.0, abs(a))
    assert np.array_equal(nets[0].params(), nets[1].params())


@pytest.mark.gpu
@pytest.mark.parametrize("repeat", [1, 43, 300])
def test_neighbour_lists_that_repeat_entries(handle, repeat):
    """Degrees far above the number of nodes (43 and 300 times every entry, in
    lists that no longer fit the tile's shared memory): means and gradients as
    layer by layer, bit for bit, and against float64."""
    pair = []
    for across in (False, True):
        b = _joined_singles(3, 14, 8, across)
        deg = np.diff(b.nbr_start)
        nbr = np.concatenate([np.tile(b.nbr[s:s + d], repeat) for s, d in zip(b.nbr_start, deg)]).astype(np.int32)
        start = np.concatenate([[0], np.cumsum(deg * repeat)]).astype(np.int32)
        pair.append(gnn.Batch(b.x, b.graph_start, start, nbr, b.root_label, b.node_mask, b.td_label))
    net = gnn.GNN(handle, seed=13)
    (logits, td), (logits2, td2) = net.forward(pair[0]), net.forward(_layerwise(pair[0]))
    assert np.array_equal(logits, logits2) and np.array_equal(td, td2[:-1])
    rl, rtd = gnn.reference_loss(net.params(), pair[0], want_grad=False)
    np.testing.assert_allclose(logits, rl, rtol=2e-3, atol=2e-4)  # sums of up to 2000 terms
    np.testing.assert_allclose(td, rtd, rtol=2e-3, atol=2e-4)
    tiles, layers = (net.gradients(b)[0] for b in pair)
    assert np.array_equal(tiles, layers)
