"""The work that a user of this package has it do, as cases that can be timed.

Each case is one call (or one short sequence) of the public entry points of
``gisbdw_gb300``, over the sizes that the package's own configurations, tests
and benchmark use: the subset DP on one graph from the smallest call to tables
beyond the L2 cache, the batched DP from a handful of small graphs to the 4096
mixed graphs of its batch workload, the bottom-up heuristic DP, the greedy
incumbents of a graph stream, the branch and bound, and the network that
orders it (inference on a stream, gradients of a training batch).

``exact`` gives the network's outputs in float64; every other output is a
whole number (treedepths, parents, orders, bounds).
"""
from __future__ import annotations

import numpy as np
import torch

from gisbdw_gb300 import Handle, _lib, gnn
from gisbdw_gb300 import graphs as G

IN_FEATURES, HIDDEN, LAYERS = 8, 64, 3
TD_WEIGHT = 0.05
DEADLINE_NS = 20 * 10**9


def listed():
    return [
        # The smallest exact solve: a 12-vertex graph, all latency (the tests' usual size).
        {"name": "dp_n12", "kind": "dp", "n": 12, "p": 0.3, "device": False},
        # The plain DP configuration: one connected G(20, 0.25), host arrays in and out.
        {"name": "dp_n20", "kind": "dp", "n": 20, "p": 0.25, "device": False},
        # An odd size between the small and the large tables.
        {"name": "dp_n25", "kind": "dp", "n": 25, "p": 0.2, "device": False},
        # The single-graph configuration at n = 30, enqueued on device arrays as a pipeline does.
        {"name": "dp_n30_device", "kind": "dp", "n": 30, "p": 0.2, "device": True},
        # The largest single table: odd, far beyond the L2 cache.
        {"name": "dp_n33", "kind": "dp", "n": 33, "p": 0.1, "device": False},
        # A small request of a few dozen small graphs.
        {"name": "batch_48_small", "kind": "batch", "count": 48, "n_min": 5, "n_max": 16, "device": False},
        # The batched workload: 4096 graphs, n in [10, 24], three families.
        {"name": "batch_4096", "kind": "batch", "count": 4096, "n_min": 10, "n_max": 24, "device": True},
        # The bottom-up heuristic, the innermost incumbent of the reference's chain (n <= 32).
        {"name": "bottom_up_n26", "kind": "bottom_up", "n": 26, "p": 0.2},
        # Incumbents of a graph stream: 1024 sparse graphs, n in [20, 80] (the reference's chain).
        {"name": "heuristic_1024", "kind": "heuristic", "count": 1024, "n_min": 20, "n_max": 80},
        # Exact search on a batch of sparse graphs, every one proven well within the cap.
        {"name": "bnb_48", "kind": "bnb", "count": 48, "n_min": 24, "n_max": 36},
        # Network inference for a graph stream.
        {"name": "gnn_forward_1024", "kind": "gnn", "count": 1024, "n_min": 20, "n_max": 80, "grad": False},
        # Loss and gradients of one training batch: 256 labelled subgraphs, n <= 24.
        {"name": "gnn_gradients_256", "kind": "gnn", "count": 256, "n_min": 5, "n_max": 24, "grad": True},
    ]


def _log_int(rng, lo, hi):
    """An integer in [lo, hi], uniform in its logarithm."""
    return min(hi, max(lo, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    kind = rng.choice(["dp", "dp", "dp", "batch", "batch", "bottom_up", "heuristic", "bnb", "gnn", "gnn"])
    if kind == "dp":
        # a table doubles with every vertex: n itself is already a logarithm
        n = rng.randint(8, 33)
        return {"kind": kind, "n": n, "p": round(rng.uniform(0.3 if n < 16 else 0.15, 0.5), 3),
                "device": rng.random() < 0.5}
    if kind == "batch":
        n_min = rng.randint(4, 14)
        return {"kind": kind, "count": _log_int(rng, 4, 4000), "n_min": n_min, "n_max": rng.randint(n_min, 24),
                "device": rng.random() < 0.5}
    if kind == "bottom_up":
        return {"kind": kind, "n": rng.randint(10, 25), "p": round(rng.uniform(0.15, 0.5), 3)}
    if kind == "heuristic":
        n_min = rng.randint(6, 60)
        return {"kind": kind, "count": _log_int(rng, 4, 1000), "n_min": n_min, "n_max": rng.randint(n_min, 80)}
    if kind == "bnb":
        n_min = rng.randint(16, 30)
        return {"kind": kind, "count": _log_int(rng, 4, 64), "n_min": n_min, "n_max": rng.randint(n_min, 34)}
    grad = rng.random() < 0.5
    n_min = rng.randint(3, 20)
    return {"kind": "gnn", "count": _log_int(rng, 4, 1000), "n_min": n_min,
            "n_max": rng.randint(n_min, 24 if grad else 80), "grad": grad}


# ---------------------------------------------------------------------------
# Inputs.
# ---------------------------------------------------------------------------

def _sizes(case, rng):
    """Vertex counts of a many-graph case. Their multiset is fixed by the case
    (spread evenly over its range), their order by the seed."""
    span = case["n_max"] - case["n_min"] + 1
    return rng.permutation(case["n_min"] + np.arange(case["count"]) * 7919 % span)


def _dense(ns, rng, sparse=False):
    """Connected random graphs as one (count, N, N) boolean array: a random
    tree plus up to n extra edges, unless `sparse` every third graph with
    G(n, p) density (p in [0.1, 0.5]) instead; labels shuffled."""
    count, N = len(ns), int(ns.max())
    a = np.zeros((count, N, N), dtype=bool)
    g = np.arange(count)
    for v in range(1, N):
        has = ns > v
        a[g[has], v, (rng.random(int(has.sum())) * v).astype(np.int64)] = True
    extra = rng.uniform(0.0, 2.0, count) / np.maximum(2, ns)
    if not sparse:
        extra = np.where(g % 3 == 0, rng.uniform(0.1, 0.5, count), extra)
    a |= rng.random((count, N, N), dtype=np.float32) < extra[:, None, None]
    ids = np.arange(N)
    inside = ids[None, :] < ns[:, None]
    a &= np.tril(np.ones((N, N), dtype=bool), -1) & inside[:, :, None] & inside[:, None, :]
    a |= a.transpose(0, 2, 1)
    # shuffle the labels 0..n-1 of every graph; the unused labels stay last
    perm = np.argsort(np.where(inside, rng.random((count, N)), 2.0 + ids), axis=1)
    a = np.take_along_axis(a, perm[:, :, None], axis=1)
    return np.take_along_axis(a, perm[:, None, :], axis=2)


def _pool(ns, rng):
    """Descriptors and 64-bit adjacency pool of a batch of random graphs."""
    a = _dense(ns, rng)
    masks = (a * (np.uint64(1) << np.arange(a.shape[2], dtype=np.uint64))).sum(axis=2, dtype=np.uint64)
    descs = (_lib.GraphDesc * len(ns))()
    off = np.concatenate([[0], np.cumsum(ns)])
    for i, n in enumerate(ns):
        descs[i].n, descs[i].offset = int(n), int(off[i])
    return descs, np.concatenate([masks[i, :n] for i, n in enumerate(ns)])


def _sparse_graphs(ns, rng):
    """Connected sparse graphs of the search families: random geometric
    graphs, grids with deleted edges, trees plus a few edges."""
    out = []
    for i, n in enumerate(ns.tolist()):
        v = np.arange(1, n)
        label = rng.permutation(n)
        if i % 3 == 0:  # mean degree about 3; every vertex is joined to the nearest one before it
            xy = rng.random((n, 2))
            d2 = ((xy[:, None, :] - xy[None, :, :]) ** 2).sum(-1)
            d2[np.triu_indices(n)] = np.inf
            u, w = np.nonzero(d2 <= 3.0 / (np.pi * (n - 1)))
            u, w = np.concatenate([u, v]), np.concatenate([w, d2[1:].argmin(1)])
        elif i % 3 == 1:  # a row-major grid that keeps one edge back from every vertex and most of the others
            cols = -(-n // int(n ** 0.5))
            left, up = v % cols > 0, v >= cols
            both = left & up
            drop = both & (rng.random(n - 1) < 0.4)
            side = rng.random(n - 1) < 0.5
            left, up = left & ~(drop & side), up & ~(drop & ~side)
            u, w = np.concatenate([v[left], v[up]]), np.concatenate([v[left] - 1, v[up] - cols])
            label = np.arange(n)
        else:  # a random tree plus n / 6 edges
            k = max(1, n // 6)
            u = np.concatenate([v, rng.integers(1, n, k)])
            w = np.concatenate([(rng.random(n - 1) * v).astype(np.int64), rng.integers(0, n, k)])
        keep = u != w
        out.append(G.Graph(n, list(zip(label[u[keep]].tolist(), label[w[keep]].tolist()))))
    return out


def _gnn_inputs(case, seed):
    """Parameters, features, neighbour lists and labels of a network batch."""
    rng = np.random.default_rng([seed, case["count"], case["n_max"]])
    ns = _sizes(case, rng)
    a = torch.from_numpy(_dense(ns, rng, sparse=not case["grad"]))
    if torch.cuda.is_available():
        a = a.cuda()
    count, N = a.shape[0], a.shape[1]
    f = a.float()
    inside = (torch.arange(N, device=a.device)[None, :] < torch.from_numpy(ns).to(a.device)[:, None])
    deg = f.sum(2)
    # core numbers: peel the vertices of degree < k, k = 1, 2, ...
    core = torch.zeros_like(deg)
    alive = inside.float()
    for k in range(1, N):
        if not bool(alive.any()):
            break
        while True:
            d = torch.bmm(f, alive[:, :, None])[:, :, 0]
            stay = alive * (d >= k)
            if torch.equal(stay, alive):
                break
            alive = stay
        core = torch.where(alive > 0, torch.full_like(core, float(k)), core)
    # eccentricities: breadth-first layers of every vertex at once
    seen = torch.eye(N, device=a.device).expand(count, N, N).clone()
    ecc = torch.zeros_like(deg)
    for d in range(1, N):
        grown = ((torch.bmm(f, seen) + seen) > 0).float()
        new = (grown.sum(1) > seen.sum(1))
        if not bool(new.any()):
            break
        ecc = torch.where(new, torch.full_like(ecc, float(d)), ecc)
        seen = grown
    nbr_deg = torch.bmm(f, deg[:, :, None])[:, :, 0] / deg.clamp(min=1)
    size = torch.from_numpy(ns).to(a.device).float()[:, None].expand(count, N)
    x = torch.stack([deg / 4, core / 4, ecc / 8, nbr_deg / 4, (deg == 1).float(), 1 / (1 + deg), size / 64,
                     torch.ones_like(deg)], dim=2)
    x = x[inside].cpu().numpy().astype(np.float32)
    a = a.cpu().numpy()
    start = np.concatenate([[0], np.cumsum(ns)]).astype(np.int32)
    gi, u, v = np.nonzero(a)
    nbr = (start[gi] + v).astype(np.int32)
    per = a.sum(2)[np.arange(N)[None, :] < ns[:, None]]
    total = int(ns.sum())
    lim = [(IN_FEATURES, HIDDEN)] + [(HIDDEN, HIDDEN), (HIDDEN, HIDDEN)] * LAYERS
    parts = []
    for i, (k, h) in enumerate(lim):
        parts.append(rng.uniform(-1, 1, k * h) * np.sqrt(6.0 / (k + h)))
        if i % 2 == 0:  # the bias follows the input weights and every layer's second matrix
            parts.append(rng.uniform(-0.1, 0.1, h))
    for _ in range(2):
        parts += [rng.uniform(-1, 1, HIDDEN) * np.sqrt(6.0 / (HIDDEN + 1)), rng.uniform(-0.1, 0.1, 1)]
    b = {"x": x, "graph_start": start, "nbr": nbr if len(nbr) else np.zeros(1, dtype=np.int32),
         "nbr_start": np.concatenate([[0], np.cumsum(per)]).astype(np.int32),
         "root_label": (rng.random(total) < 0.5).astype(np.float32),
         "node_mask": np.ones(total, dtype=np.float32),
         "td_label": (2 + rng.integers(0, 8, count)).astype(np.float32)}
    return np.concatenate(parts).astype(np.float32), b


def prepare(case, seed):
    kind = case["kind"]
    h = Handle(0)
    rng = np.random.default_rng([seed, len(kind), case["n" if "n" in case else "count"]])
    if kind == "dp":
        adj = G.gnp_connected(case["n"], case["p"], int(rng.integers(1, 1 << 30))).adj64()
        st = {"h": h, "n": case["n"], "adj": adj}
        if case["device"]:
            st["d_adj"] = torch.from_numpy(adj.view(np.int64)).cuda()
            st["out"] = [torch.zeros(k, dtype=torch.int32, device="cuda") for k in (1, case["n"], case["n"])]
    elif kind == "batch":
        descs, pool = _pool(_sizes(case, rng), rng)
        st = {"h": h, "descs": descs, "pool": pool, "count": len(descs)}
        if case["device"]:
            st["d_pool"] = torch.from_numpy(pool.view(np.int64)).cuda()
            st["out"] = [torch.zeros(k, dtype=torch.int32, device="cuda") for k in (len(descs), len(pool))]
    elif kind == "bottom_up":
        st = {"h": h, "g": G.gnp_connected(case["n"], case["p"], int(rng.integers(1, 1 << 30)))}
    elif kind in ("heuristic", "bnb"):
        st = {"h": h, "graphs": _sparse_graphs(_sizes(case, rng), rng)}
    else:
        params, b = _gnn_inputs(case, seed)
        net = gnn.GNN(h, seed=1)
        net.set_params(params)
        st = {"h": h, "net": net, "batch": gnn.Batch(**b), "grad": case["grad"]}
    st["kind"] = kind
    return st


def run(st):
    kind, h = st["kind"], st["h"]
    if kind == "dp":
        if "d_adj" in st:
            td, parent, order = st["out"]
            h.dp_solve_device(st["d_adj"].data_ptr(), st["n"], td.data_ptr(), parent.data_ptr(), order.data_ptr())
            return td, parent, order
        td, parent, order, _ = h.dp_solve(st["adj"], st["n"])
        return td, parent, order
    if kind == "batch":
        if "d_pool" in st:
            td, parent = st["out"]
            h.dp_solve_batch_device(st["descs"], st["count"], st["d_pool"].data_ptr(), len(st["pool"]),
                                    td.data_ptr(), parent.data_ptr())
            return td, parent
        td, parents, _ = h.dp_solve_batch(None, packed=(st["descs"], st["pool"]))
        return td, np.concatenate(parents[:])
    if kind == "bottom_up":
        return h.bottom_up(st["g"])
    if kind == "heuristic":
        td, parents = h.heuristic_batch(st["graphs"], 0)
        return td, np.concatenate(parents)
    if kind == "bnb":
        # which of several optimal trees comes back depends on the search's timing: the values that do not are returned
        r = h.bnb_solve_batch(st["graphs"], deadline_ns=DEADLINE_NS)
        return r["td"], r["status"], r["lower_bound"]
    if st["grad"]:
        return st["net"].gradients(st["batch"], TD_WEIGHT)
    return st["net"].forward(st["batch"])


def work(case):
    """Bytes in and out once; operations: one per (subset, deleted vertex) of
    a subset DP, times n for the forests of the bottom-up heuristic, n^2 per
    graph for the greedy ones, the products of the network."""
    kind = case["kind"]
    if kind in ("dp", "bottom_up"):
        n = case["n"]
        return {"bytes": 16 * n + 4, "flops": n * 2 ** (n - 1) * (n if kind == "bottom_up" else 1)}
    ns = _sizes(case, np.random.default_rng(0)).astype(np.int64)
    total = int(ns.sum())
    if kind == "batch":
        return {"bytes": 12 * total + 12 * len(ns), "flops": int((ns << (ns - 1)).sum())}
    if kind in ("heuristic", "bnb"):
        return {"bytes": 20 * total + 12 * len(ns), "flops": int((ns**2).sum())}
    macs = total * (IN_FEATURES * HIDDEN + 2 * LAYERS * HIDDEN * HIDDEN + 2 * HIDDEN)
    params = HIDDEN * (IN_FEATURES + 1 + LAYERS * (2 * HIDDEN + 1) + 2) + 2
    nbytes = total * (4 * IN_FEATURES + 4 * 4 + 4) + 2 * params
    if case["grad"]:
        return {"bytes": nbytes + 8 * total + 4 * params, "flops": 6 * macs}
    return {"bytes": nbytes, "flops": 2 * macs}


# ---------------------------------------------------------------------------
# The network in float64.
# ---------------------------------------------------------------------------

def exact(case, seed):
    if case["kind"] != "gnn":
        return None
    params, b = _gnn_inputs(case, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    # the kernels keep their weights in bfloat16
    p = torch.from_numpy(params).to(dev).bfloat16().double()
    at = 0

    def take(*shape):
        nonlocal at
        k = int(np.prod(shape))
        at += k
        return p[at - k:at].reshape(shape)

    w_in, b_in = take(IN_FEATURES, HIDDEN), take(HIDDEN)
    layers = [(take(HIDDEN, HIDDEN), take(HIDDEN, HIDDEN), take(HIDDEN)) for _ in range(LAYERS)]
    w_out, b_out, w_g, b_g = take(HIDDEN), take(1), take(HIDDEN), take(1)
    t = {k: torch.from_numpy(v).to(dev) for k, v in b.items()}
    ns = (t["graph_start"][1:] - t["graph_start"][:-1]).long()
    deg = (t["nbr_start"][1:] - t["nbr_start"][:-1]).long()
    total, count = int(ns.sum()), len(ns)
    row = torch.repeat_interleave(torch.arange(total, device=dev), deg)
    col = t["nbr"].long()[:len(row)]
    of = torch.repeat_interleave(torch.arange(count, device=dev), ns)
    inv_deg = (1.0 / deg.clamp(min=1).double())[:, None]

    def sums(values, to, k):
        return torch.zeros(k, HIDDEN, dtype=torch.float64, device=dev).index_add_(0, to, values)

    z = t["x"].double() @ w_in + b_in
    zs, hs, means = [z], [z.clamp(min=0)], []
    for ws, wn, bias in layers:
        means.append(sums(hs[-1][col], row, total) * inv_deg)
        z = hs[-1] @ ws + means[-1] @ wn + bias
        zs.append(z)
        hs.append(z.clamp(min=0))
    logits = hs[-1] @ w_out + b_out
    pooled = sums(hs[-1], of, count) / ns.double()[:, None]
    td = pooled @ w_g + b_g
    if not case["grad"]:
        return logits.cpu().numpy(), td.cpu().numpy()
    y, m, tl = (t[k].double() for k in ("root_label", "node_mask", "td_label"))
    inv = 1.0 / m.sum()
    loss = (m * (logits.clamp(min=0) - logits * y + torch.log1p(torch.exp(-logits.abs())))).sum() * inv
    loss = loss + TD_WEIGHT * ((td - tl) ** 2).mean()
    dl = m * (torch.sigmoid(logits) - y) * inv
    dt = 2 * TD_WEIGHT * (td - tl) / count
    head = [hs[-1].T @ dl, dl.sum()[None], pooled.T @ dt, dt.sum()[None]]
    dh = dl[:, None] * w_out + (dt / ns.double())[of][:, None] * w_g
    back = []
    for i in range(LAYERS - 1, -1, -1):
        dz = dh * (zs[i + 1] > 0)
        back.insert(0, [hs[i].T @ dz, means[i].T @ dz, dz.sum(0)])
        dm = (dz @ layers[i][1].T) * inv_deg
        dh = dz @ layers[i][0].T + sums(dm[row], col, total)
    dz = dh * (zs[0] > 0)
    flat = [t["x"].double().T @ dz, dz.sum(0)] + [g for layer in back for g in layer] + head
    return torch.cat([g.reshape(-1) for g in flat]).cpu().numpy(), float(loss)
