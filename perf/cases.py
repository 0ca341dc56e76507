"""Performance cases: the work users of this package have it do, through its public entry points.

A case names an entry point (``call``), a graph family with its sizes, and the SCAN parameters.
``prepare`` builds the graph from the seed and the handle a program keeps; ``run`` is one pass.

Entry points: ``Graph.run`` on a resident graph, the drop-in ``GPUScan`` on host arrays,
``Graph.common_neighbors``, ``Batch.run``, a ``Server`` answering a burst of queries, and
``Graph.run`` on a streamed graph.  Families: R-MAT (a/b/c/d = .57/.19/.19/.05), Chung-Lu power
laws, planted communities, and stochastic block models (the batched small graphs).

Graphs are generated with torch from counter-based hashes, on the GPU where there is one: the
same seed gives the same graph on every device.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import efficientstructuralgraphclusteringongpus_gb300 as scan

REF, EXACT = "ref-f64", "exact"
_COUNTS = ("num_cores", "num_clusters", "num_hubs", "num_outliers", "num_borders", "num_similar_edges",
           "pred_disagreements", "multi_cluster_borders")
_MODES = {REF: scan.PRED_REF_F64, EXACT: scan.PRED_EXACT}


def listed() -> list[dict]:
    return [
        # The smallest call: a graph of a few thousand edges, clustered again and again by an
        # interactive user.  Launches and host work are all there is.
        _rmat("run_rmat10", "run", 1 << 10, 16, "0.5", 5, REF),
        # The small plain configuration (R-MAT scale 16, edge factor 16), exact predicate.
        _rmat("run_rmat16", "run", 1 << 16, 16, "0.5", 5, EXACT),
        # The benchmark configuration, graph resident: R-MAT scale 22, eps 0.5, mu 5.
        _rmat("run_rmat22", "run", 1 << 22, 16, "0.5", 5, REF),
        # The low end of the benchmark's parameter sweep, where little is pruned, on a vertex
        # count that is no power of two.
        _rmat("run_rmat21_low_eps", "run", 1_500_007, 16, "0.2", 2, EXACT),
        # The drop-in call on a small odd-sized graph: one upload, one run, one free per call.
        _rmat("dropin_rmat13", "dropin", 6_007, 16, "0.3", 2, REF),
        # The drop-in call on the benchmark's graph (host arrays in, labels out); mu 2, the
        # sweep's lowest, gives labels where mu 5 finds no core.
        _rmat("dropin_rmat22", "dropin", 1 << 22, 16, "0.5", 2, REF),
        # Hub-heavy: a power law of exponent 2.1 whose largest hubs hold several percent of the
        # vertices, a sixteenth of the billion-edge configuration.
        {"name": "run_chunglu", "call": "run", "family": "chunglu", "n": 3_125_001, "avg_degree": 40,
         "max_degree": 131_072, "eps": "0.4", "mu": 5, "predicate": REF},
        # A graph with real communities: most edges inside them are similar and most vertices
        # end up in clusters, so counts have to be settled one way or the other near eps.
        {"name": "run_communities", "call": "run", "family": "communities", "n": 400_009, "avg_degree": 40,
         "community": 48, "eps": "0.4", "mu": 5, "predicate": EXACT},
        # Every common-neighbour count, returned to the host: the input of a serving cache or of
        # a caller's own similarity measure.
        _rmat("count_rmat19", "count", 500_009, 16, "0.5", 5, REF),
        # Many small graphs, each with its own parameters, in one call.
        {"name": "batch_sbm", "call": "batch", "family": "sbm", "graphs": 512, "n_min": 100, "n_max": 20_000,
         "avg_degree": 64, "predicate": REF},
        # A burst of mixed queries on a resident pool with cached counts.
        {"name": "serve_pool", "call": "serve", "family": "rmat", "graphs": 8, "scale_min": 12, "scale_max": 19,
         "edge_factor": 16, "queries": 30},
        # A graph whose adjacency stays in host memory (device budget below its size).
        _rmat("stream_rmat19", "stream", 400_003, 16, "0.5", 5, REF),
    ]


def _rmat(name, call, n, edge_factor, eps, mu, predicate) -> dict:
    return {"name": name, "call": call, "family": "rmat", "n": n, "edge_factor": edge_factor, "eps": eps, "mu": mu,
            "predicate": predicate}


def draw(rng) -> dict:
    """One more case of the listed ranges; none costs more than the largest listed one."""
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    eps = rng.choice(["0.2", "0.3", "0.35", "0.4", "0.5", "0.6", "0.7", "0.8"])
    mu = rng.randint(2, 10)
    predicate = rng.choice([REF, EXACT])
    kind = rng.choice(["run", "run", "run", "dropin", "chunglu", "communities", "count", "batch", "serve", "stream"])
    if kind == "chunglu":
        n = log_int(50_000, 3_125_001)
        return {"call": "run", "family": "chunglu", "n": n, "avg_degree": rng.randint(12, 40),
                "max_degree": max(64, int(n * rng.uniform(0.01, 0.04))), "eps": rng.choice(["0.3", "0.4", "0.5"]),
                "mu": mu, "predicate": predicate}
    if kind == "communities":
        call = rng.choice(["run", "dropin"])
        if call == "dropin":
            eps = rng.choice(["0.3", "0.4", "0.5"])
        return {"call": call, "family": "communities", "n": log_int(3_000, 400_009),
                "avg_degree": rng.randint(12, 40), "community": rng.randint(20, 80), "eps": eps, "mu": mu,
                "predicate": predicate}
    if kind == "batch":
        return {"call": "batch", "family": "sbm", "graphs": log_int(16, 512), "n_min": 100,
                "n_max": log_int(1_000, 20_000), "avg_degree": 64, "predicate": predicate}
    if kind == "serve":
        return {"call": "serve", "family": "rmat", "graphs": rng.randint(2, 8), "scale_min": 12,
                "scale_max": rng.randint(13, 19), "edge_factor": 16, "queries": rng.randint(8, 30)}
    top = {"run": 1 << 22, "dropin": 1 << 22, "count": 500_009, "stream": 400_003}[kind]
    n = log_int(1 << 14 if kind == "count" else 1 << 10, top)
    if kind == "dropin":   # labels alone come back: parameters at which R-MAT graphs have clusters
        eps, mu = rng.choice(["0.2", "0.3", "0.4"]), rng.randint(2, 3)
    if kind in ("run", "dropin") and eps in ("0.2", "0.3"):
        n = min(n, 1_500_007)
    return {"call": kind, "family": "rmat", "n": n, "edge_factor": rng.choice([8, 13, 16]), "eps": eps, "mu": mu,
            "predicate": predicate}


# ---- what a program has in hand before the call --------------------------------------------


def prepare(case: dict, seed: int) -> dict:
    call = case["call"]
    state = {"call": call}
    if call == "batch":
        offsets, adj, cuts = _sbm_union(case, seed)
        graphs = []
        for lo, hi in zip(cuts[:-1], cuts[1:]):
            o = offsets[lo:hi + 1]
            graphs.append(scan.Graph.from_csr(o - o[0], adj[int(o[0]):int(o[-1])] - lo))
        r = np.random.RandomState(case["graphs"])
        state.update(batch=scan.Batch(graphs), graphs=graphs, mode=_MODES[case["predicate"]],
                     eps=[("0.3", "0.5", "0.7")[i] for i in r.randint(0, 3, len(graphs))],
                     mus=r.randint(2, 9, len(graphs)))
        return state
    if call == "serve":
        server = scan.Server(memory_budget_bytes=1 << 30, max_in_flight=8)
        r = np.random.RandomState(case["queries"])   # the same mix of queries for every seed
        span = case["scale_max"] - case["scale_min"]
        for i in range(case["graphs"]):   # scales evenly over the range
            scale = case["scale_min"] + round(span * i / max(case["graphs"] - 1, 1))
            g = scan.Graph.from_csr(*_rmat_csr(1 << scale, case["edge_factor"], seed + 7919 * i))
            server.add_graph(g)
            g.close()
        state["server"] = server
        state["queries"] = [(int(r.randint(case["graphs"])), "0.%d" % r.randint(1, 10), int(r.randint(2, 21)),
                             int(r.randint(2))) for _ in range(case["queries"])]
        return state
    offsets, adj = _csr(case, seed)
    state.update(eps=case["eps"], mu=case["mu"], mode=_MODES[case["predicate"]])
    if call == "dropin":
        # the reference's graph_t arrays, in pinned memory as a caller that uploads would keep them
        state.update(offsets=_pinned(offsets.astype(np.uint32)), adj=_pinned(adj.astype(np.int32)))
        return state
    g = scan.Graph.from_csr(offsets, adj)
    if call == "stream":
        g.upload_streamed()
    else:
        g.upload()
    state["graph"] = g
    return state


def run(state: dict):
    call = state["call"]
    if call in ("run", "stream"):
        r = state["graph"].run(state["eps"], state["mu"], state["mode"])
        return {"label": r.label, "role": r.role, "counts": [r.stats[k] for k in _COUNTS]}
    if call == "dropin":
        return {"label": scan.GPUScan(state["offsets"], state["adj"], float(state["eps"]), state["mu"])}
    if call == "count":
        return {"cn": state["graph"].common_neighbors()[0].view(np.int32)}
    if call == "batch":
        labels, roles, _ = state["batch"].run(state["eps"], state["mus"], state["mode"])
        return {"label": np.concatenate(labels), "role": np.concatenate(roles)}
    server = state["server"]
    tickets = [server.submit(g, eps, mu, mode) for g, eps, mu, mode in state["queries"]]
    results = [server.wait(t) for t in tickets]
    return {"label": [r[0] for r in results], "role": [r[1] for r in results]}


def work(case: dict) -> dict:
    """Bytes of the CSR in and of the results out (sizes before repeated pairs are merged)."""
    call = case["call"]
    if call == "batch":
        n = case["graphs"] * (case["n_max"] - case["n_min"]) / math.log(case["n_max"] / case["n_min"])
        m = n * case["avg_degree"] * 0.7
        return {"bytes": 4 * m + 4 * n + 5 * n, "flops": 4 * m}
    if call == "serve":   # per query: the cached count and both endpoints of each edge
        span = case["scale_max"] - case["scale_min"]
        n = sum(2 ** (case["scale_min"] + round(span * i / max(case["graphs"] - 1, 1))) for i in range(case["graphs"]))
        n = n / case["graphs"] * case["queries"]
        return {"bytes": 12 * n * case["edge_factor"] + 5 * n, "flops": 8 * n * case["edge_factor"]}
    n = case["n"]
    m = n * (2 * case["edge_factor"] if case["family"] == "rmat" else case["avg_degree"])
    out = 2 * m if call == "count" else 5 * n
    return {"bytes": 4 * m + 4 * n + out, "flops": 4 * m}


# ---- graphs ---------------------------------------------------------------------------------


def _device() -> torch.device:
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _pinned(a: np.ndarray) -> np.ndarray:
    t = torch.from_numpy(a)
    return t.pin_memory().numpy() if torch.cuda.is_available() else a


def _i64(x: int) -> int:
    x &= (1 << 64) - 1
    return x - (1 << 64) if x >> 63 else x


def _hash(idx: torch.Tensor, seed: int, stream: int) -> torch.Tensor:
    """splitmix64 of a counter: 53 random bits per index, the same on every device."""
    key = _i64((seed * 0x9E3779B97F4A7C15) ^ ((stream + 1) * 0xD1B54A32D192ED03))
    x = (idx ^ key) * _i64(0x9E3779B97F4A7C15)
    x = (x ^ ((x >> 30) & ((1 << 34) - 1))) * _i64(0xBF58476D1CE4E5B9)
    x = (x ^ ((x >> 27) & ((1 << 37) - 1))) * _i64(0x94D049BB133111EB)
    x = x ^ ((x >> 31) & ((1 << 33) - 1))
    return (x >> 11) & ((1 << 53) - 1)


def _unit(idx: torch.Tensor, seed: int, stream: int) -> torch.Tensor:
    return _hash(idx, seed, stream).double() * (1.0 / (1 << 53))


def _csr_of_pairs(u: torch.Tensor, v: torch.Tensor, n: int, most: int | None = None):
    """Pairs -> symmetric CSR without loops or repeats, lists ascending: (uint64[n+1], uint32[m]).
    most: keep that many edges, chosen by a hash."""
    lo, hi = torch.minimum(u, v), torch.maximum(u, v)
    key = torch.unique((lo * n + hi)[lo != hi])
    if most is not None and most < key.numel():
        key = torch.sort(key[torch.argsort(_hash(key, 1, 99))[:most]]).values
    lo, hi = key // n, key % n
    key = torch.sort(torch.cat([key, hi * n + lo])).values
    offsets = torch.zeros(n + 1, dtype=torch.int64, device=u.device)
    offsets[1:] = torch.cumsum(torch.bincount(key // n, minlength=n), 0)
    adj = (key % n).to(torch.int32)
    return offsets.cpu().numpy().astype(np.uint64), adj.cpu().numpy().view(np.uint32)


def _rmat_csr(n: int, edge_factor: int, seed: int, most: int | None = None):
    """R-MAT of the scale that holds n vertices; ids >= n wrap to the low ones."""
    scale = max(1, (n - 1).bit_length())
    idx = torch.arange(n * edge_factor, dtype=torch.int64, device=_device())
    u, v = torch.zeros_like(idx), torch.zeros_like(idx)
    for level in range(scale):
        r = _unit(idx, seed, level)
        u = 2 * u + (r >= 0.76).long()
        v = 2 * v + (((r >= 0.57) & (r < 0.76)) | (r >= 0.95)).long()
    return _csr_of_pairs(u % n, v % n, n, most)


def _chunglu_csr(n: int, avg_degree: int, max_degree: int, seed: int):
    """Weights (i + 1)^(-1 / 1.1) (exponent 2.1), capped so that no expected degree exceeds max_degree."""
    dev = _device()
    pairs = n * avg_degree // 2
    w = torch.arange(1, n + 1, dtype=torch.float64, device=dev) ** (-1.0 / 1.1)
    for _ in range(40):
        w = torch.minimum(w, w.sum() * (max_degree / (2.0 * pairs)))
    cdf = torch.cumsum(w, 0)
    idx = torch.arange(pairs, dtype=torch.int64, device=dev)
    u, v = (torch.searchsorted(cdf, _unit(idx, seed, s) * cdf[-1], right=True).clamp_(max=n - 1) for s in (0, 1))
    return _csr_of_pairs(u, v, n)


def _communities_csr(n: int, avg_degree: int, community: int, seed: int):
    """Communities of `community` consecutive vertices on average (half to one and a half times
    that), 85% of each vertex's pairs inside its own."""
    dev = _device()
    count = max(1, n // community)
    sizes = 0.5 + _unit(torch.arange(count, dtype=torch.int64, device=dev), seed, 3)
    ends = torch.round(torch.cumsum(sizes, 0) * (n / sizes.sum())).long().clamp_(max=n)
    ends[-1] = n
    starts = torch.cat([ends.new_zeros(1), ends[:-1]])
    idx = torch.arange(n * avg_degree // 2, dtype=torch.int64, device=dev)
    u = (_unit(idx, seed, 0) * n).long().clamp_(max=n - 1)
    c = torch.searchsorted(ends, u, right=True)
    r = _unit(idx, seed, 1)
    inside = starts[c] + (r * (ends - starts)[c]).long()
    v = torch.where(_unit(idx, seed, 2) < 0.85, inside, (r * n).long()).clamp_(max=n - 1)
    return _csr_of_pairs(u, v, n)


def _sbm_union(case: dict, seed: int):
    """`graphs` block models as one union CSR with the vertex cuts between them: vertex counts
    log-uniform, 2-64 blocks, p_in 0.1, p_out 0.001, expected degree capped at avg_degree."""
    dev = _device()
    r = np.random.RandomState(case["n_max"])   # the same sizes for every seed
    n = np.exp(r.uniform(math.log(case["n_min"]), math.log(case["n_max"]), case["graphs"])).astype(np.int64)
    blocks = np.minimum(r.randint(2, 65, case["graphs"]), n // 2)
    d_in, d_out = 0.1 * n / blocks, 0.001 * n * (1 - 1 / blocks)
    pairs = np.maximum((n * np.minimum(d_in + d_out, case["avg_degree"]) / 2).astype(np.int64), 1)
    cuts = np.concatenate([[0], np.cumsum(n)])
    total = int(cuts[-1])
    tensor = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)  # noqa: E731
    g = torch.repeat_interleave(torch.arange(case["graphs"], device=dev), tensor(pairs))
    idx = torch.arange(int(pairs.sum()), dtype=torch.int64, device=dev)
    size, k, base = tensor(n)[g], tensor(blocks)[g], tensor(cuts[:-1])[g]
    u = torch.minimum((_unit(idx, seed, 0) * size).long(), size - 1)
    b = u * k // size
    lo, hi = (b * size + k - 1) // k, ((b + 1) * size + k - 1) // k   # block b's vertices
    x = _unit(idx, seed, 1)
    inside = lo + (x * (hi - lo)).long()
    p_in = tensor(d_in / (d_in + d_out))[g]
    v = torch.minimum(torch.where(_unit(idx, seed, 2) < p_in, inside, (x * size).long()), size - 1)
    offsets, adj = _csr_of_pairs(base + u, base + v, total)
    return offsets, adj, cuts.tolist()


def _csr(case: dict, seed: int):
    if case["family"] == "rmat":
        # one count per edge comes back: the same number of edges for every seed
        most = case["n"] * case["edge_factor"] * 3 // 4 if case["call"] == "count" else None
        return _rmat_csr(case["n"], case["edge_factor"], seed, most)
    if case["family"] == "chunglu":
        return _chunglu_csr(case["n"], case["avg_degree"], case["max_degree"], seed)
    return _communities_csr(case["n"], case["avg_degree"], case["community"], seed)


# ---- the same answers from plain torch ------------------------------------------------------

_EXACT_PROBES = 4 << 30   # list entries looked up at most


def exact(case: dict, seed: int):
    """SCAN in 64-bit integers and floats, without this package; None where it would take long."""
    if case["call"] in ("batch", "serve") or case["n"] > 500_009:
        return None
    offsets, adj = (torch.from_numpy(a.astype(np.int64)).to(_device()) for a in _csr(case, seed))
    n = offsets.numel() - 1
    deg = offsets[1:] - offsets[:-1]
    src = torch.repeat_interleave(torch.arange(n, device=adj.device), deg)
    # lower endpoint u, higher endpoint v in (degree, id) order; edges by (u, v)
    low = (deg[src] < deg[adj]) | ((deg[src] == deg[adj]) & (src < adj))
    u, v = src[low], adj[low]
    if int(deg[u].sum()) > _EXACT_PROBES:
        return None
    t = _common(offsets, adj, src * n + adj, u, v, n)
    if case["call"] == "count":
        return {"cn": t.to(torch.int32).cpu().numpy()}
    label, role = _scan(case, n, deg, u, v, t)
    if case["call"] == "dropin":
        return {"label": label}
    return {"label": label, "role": role, "counts": [None] * len(_COUNTS)}


def _common(offsets, adj, keys, u, v, n):
    """|N(u) & N(v)| of every edge: each entry of u's list looked up among v's entries."""
    deg = offsets[1:] - offsets[:-1]
    ends = torch.cumsum(deg[u], 0)
    out = torch.zeros_like(u)
    step, first = 1 << 26, 0
    while first < u.numel():
        done = int(ends[first - 1]) if first else 0
        last = max(first + 1, int(torch.searchsorted(ends, done + step, right=True)))
        e = torch.arange(first, min(last, u.numel()), device=u.device)
        d = deg[u[e]]
        owner = torch.repeat_interleave(e, d)
        pos = torch.arange(owner.numel(), device=u.device) - torch.repeat_interleave(torch.cumsum(d, 0) - d, d)
        want = v[owner] * n + adj[offsets[u[owner]] + pos]
        at = torch.searchsorted(keys, want).clamp_(max=keys.numel() - 1)
        out.index_add_(0, owner, (keys[at] == want).long())
        first = int(e[-1]) + 1
    return out


def _scan(case, n, deg, u, v, t):
    dev = u.device
    du, dv = deg[u] + 1, deg[v] + 1
    if case["predicate"] == REF or case["call"] == "dropin":
        eps = float(case["eps"])
        fu, fv = du.double(), dv.double()
        square = ((t + 2) * (t + 2)).to(torch.int32).double()
        sim = ((eps * eps * fu * fv <= 4.0) | ~(square < eps * eps * fu * fv)) & ~(fu < fv * eps * eps)
    else:
        q = 10 ** len(case["eps"].split(".")[1])
        p = int(round(float(case["eps"]) * q))
        sim = (t + 2) ** 2 * q * q >= p * p * du * dv
    su, sv = u[sim], v[sim]
    core = torch.bincount(torch.cat([su, sv]), minlength=n) >= case["mu"]
    big = torch.iinfo(torch.int64).max
    cluster = torch.where(core, torch.arange(n, device=dev), big)
    both = core[su] & core[sv]
    cu, cv = su[both], sv[both]
    while True:   # smallest core id of each component: neighbours' minima, then pointer jumps
        new = cluster.clone()
        new.scatter_reduce_(0, cu, cluster[cv], "amin")
        new.scatter_reduce_(0, cv, cluster[cu], "amin")
        new[core] = torch.minimum(new[core], new[new[core]])
        if torch.equal(new, cluster):
            break
        cluster = new
    label = cluster.clone()
    for a, b in ((su, sv), (sv, su)):   # borders: the smallest cluster among similar cores
        m = core[a] & ~core[b]
        label.scatter_reduce_(0, b[m], cluster[a[m]], "amin")
    role = torch.where(core, 3, torch.where(label < big, 2, 0))
    lo, hi = torch.full_like(label, big), torch.full_like(label, -1)
    for a, b in ((u, v), (v, u)):       # hubs: two clusters among an unlabelled vertex's neighbours
        m = (label[a] < big) & (label[b] == big)
        lo.scatter_reduce_(0, b[m], label[a[m]], "amin")
        hi.scatter_reduce_(0, b[m], label[a[m]], "amax")
    free = label == big
    hub = free & (lo < hi)
    label = torch.where(hub, -1, torch.where(free, -2, label))
    role = torch.where(hub, 1, role)
    return label.to(torch.int32).cpu().numpy(), role.to(torch.uint8).cpu().numpy()
