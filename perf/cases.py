"""What a user of this framework has it do, as cases that can be timed.

Every case is one pass through the public entry points of ``silvan_b200``, as
a program calls them: an estimation (``Probabilistic`` on a resident graph,
``run``, ``get_centrality`` and in top-k mode ``topk``), several of them in one
call (``run_batched``), a stream of requests through ``Server``, an upload of
host rows followed by an estimation, the ingest of an edge-list file
(``Graph.load``) and the exact centralities (``Graph.exact_betweenness``).

The graphs are the families of the benchmark and the tests: Barabasi-Albert,
Erdos-Renyi with mean degree 8, R-MAT with edge factor 16 (0.57, 0.19, 0.19,
0.05), and the road-like grid with 5 % of its edges deleted and 0.1 %
shortcuts.  A case holds plain values:

  job      what is called: estimate, batch, serve, upload, ingest or exact
  family   ba, er, rmat, grid or mixed (ba and er in turn)
  size     nodes; for rmat the scale, for grid the side, for mixed the largest
  degree   edges per new node (ba)
  count    graphs (batch) or requests (serve)
  directed, eps, k, sigma, ...  the estimator's options

The seed of ``prepare`` gives the graph and the sample stream.
"""
import os
import tempfile

import numpy as np
import torch

import silvan_b200 as sb

DELTA = 0.05


def _case(name, job, family, size, degree=0, directed=False, eps=0.01, k=0, sigma=False, count=1):
    return {"name": name, "job": job, "family": family, "size": size, "degree": degree,
            "directed": directed, "eps": eps, "k": k, "sigma": sigma, "count": count}


def listed():
    return [
        # the smallest call: a few hundred nodes, a loose bound; launches and
        # round trips are all there is
        _case("ba_600", "estimate", "ba", 600, 3, eps=0.05),
        # an ordinary undirected graph, all nodes, eps 0.01
        _case("ba_10k", "estimate", "ba", 10000, 5),
        # the headline: a directed power-law graph of a million nodes
        _case("rmat20_directed", "estimate", "rmat", 20, directed=True, eps=0.005),
        # a mid-size undirected power-law graph at a tight bound
        _case("rmat16_tight", "estimate", "rmat", 16, eps=0.0025),
        # the ten most central nodes of a power-law graph
        _case("rmat14_top10", "estimate", "rmat", 14, eps=0.1, k=10),
        # the ten most central crossings of a road-like graph: deep, narrow
        # searches, one path a sample
        _case("grid384_top10", "estimate", "grid", 384, eps=0.1, k=10),
        # all nodes of a larger, odd-sided one with uniformly chosen paths
        _case("grid511_sigma", "estimate", "grid", 511, eps=0.02, sigma=True),
        # graphs of uneven size estimated together in shared launches
        _case("batch_16_mixed", "batch", "mixed", 200000, count=16),
        # a burst of requests of different sizes and bounds on a server
        _case("serve_24", "serve", "rmat", 14, count=24),
        # rows in host memory, seen once: upload, estimate, read the result
        _case("upload_rmat19", "upload", "rmat", 19, directed=True, eps=0.005),
        # an edge-list file of a road-like graph, as the command line reads it
        _case("ingest_grid700", "ingest", "grid", 700),
        # exact centralities, to check estimates against
        _case("exact_ba_10k", "exact", "ba", 10000, 5),
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    job = rng.choice(["estimate"] * 7 + ["batch", "serve", "upload", "ingest", "exact"])
    if job == "estimate":
        kind = rng.choice(["ba", "er", "rmat", "directed", "top", "grid", "grid_top"])
        if kind == "ba":
            return _drawn(job, "ba", _log(rng, 500, 200000), rng.randint(2, 8),
                          eps=rng.choice([0.05, 0.02, 0.01, 0.005]))
        if kind == "er":
            return _drawn(job, "er", _log(rng, 700, 200000), eps=rng.choice([0.02, 0.01, 0.005]))
        if kind == "rmat":
            return _drawn(job, "rmat", rng.randint(10, 18), eps=rng.choice([0.01, 0.005, 0.0025]))
        if kind == "directed":
            return _drawn(job, "rmat", rng.randint(10, 20), directed=True,
                          eps=rng.choice([0.01, 0.005]))
        if kind == "top":
            return _drawn(job, "rmat", rng.randint(10, 14), directed=rng.random() < 0.5,
                          eps=round(rng.uniform(0.1, 0.25), 3), k=rng.randint(5, 10))
        if kind == "grid":
            return _drawn(job, "grid", _log(rng, 48, 600), eps=rng.choice([0.05, 0.03, 0.02]),
                          sigma=rng.random() < 0.5)
        return _drawn(job, "grid", _log(rng, 40, 300), eps=round(rng.uniform(0.1, 0.3), 3),
                      k=rng.randint(3, 10))
    if job == "batch":
        return _drawn(job, "mixed", _log(rng, 2000, 200000), count=rng.randint(3, 16))
    if job == "serve":
        return _drawn(job, "rmat", rng.randint(11, 14), count=rng.randint(4, 24))
    if job == "upload":
        return _drawn(job, "rmat", rng.randint(12, 19), directed=rng.random() < 0.7,
                      eps=rng.choice([0.01, 0.005]))
    if job == "ingest":
        if rng.random() < 0.5:
            return _drawn(job, "grid", _log(rng, 50, 700))
        return _drawn(job, "rmat", rng.randint(10, 17), directed=rng.random() < 0.5)
    return _drawn(job, "ba", _log(rng, 300, 10000), rng.randint(2, 6))


def _drawn(*args, **kw):
    c = _case("", *args, **kw)
    del c["name"]
    return c


# ---- inputs ----------------------------------------------------------------


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _rmat_pairs(scale, directed, seed):
    """R-MAT edges (edge factor 16) without self-loops and duplicates."""
    dev = _device()
    gen = torch.Generator(dev).manual_seed(seed)
    m = 16 << scale
    u = torch.zeros(m, dtype=torch.int64, device=dev)
    v = torch.zeros_like(u)
    for _ in range(scale):
        r = torch.rand(m, generator=gen, device=dev)
        u = u * 2 + (r >= 0.76)
        v = v * 2 + (((r >= 0.57) & (r < 0.76)) | (r >= 0.95))
    if not directed:
        u, v = torch.minimum(u, v), torch.maximum(u, v)
    u[0], v[0] = 0, (1 << scale) - 1  # the last node is there
    key = torch.unique((u << 32) | v)
    u, v = key >> 32, key & 0xffffffff
    return torch.stack([u, v], 1)[u != v]


def _er_pairs(n, seed):
    """Random pairs at mean degree 8 (the few duplicates are the loader's to
    remove)."""
    dev = _device()
    gen = torch.Generator(dev).manual_seed(seed)
    p = torch.randint(0, n, (4 * n, 2), generator=gen, device=dev)
    p[0, 0], p[0, 1] = 0, n - 1  # the last node is there
    return p[p[:, 0] != p[:, 1]]


def _pairs(family, size, degree, directed, seed):
    if family == "rmat":
        return _rmat_pairs(size, directed, seed)
    if family == "er":
        return _er_pairs(size, seed)
    made = (sb.barabasi_albert(size, degree, seed) if family == "ba"
            else sb.grid(size, 0.05, 0.001, seed))
    return torch.from_numpy(made.astype(np.int64)).to(_device())


def _text(pairs):
    """The edge list as the bytes of a "u v" file."""
    p = pairs.to(torch.int32)
    tens = torch.tensor([10 ** k for k in range(7, -1, -1)], dtype=torch.int32, device=p.device)
    digits = (p[:, :, None] // tens % 10 + 48).to(torch.uint8)
    shown = (p[:, :, None] >= tens) | (tens == 1)
    end = torch.tensor([32, 10], dtype=torch.uint8, device=p.device).expand(len(p), 2)[:, :, None]
    text = torch.cat([digits, end], 2)
    return text[torch.cat([shown, torch.ones_like(end, dtype=torch.bool)], 2)].cpu().numpy()


def _write(pairs):
    """The edge-list file, in a folder that goes when the returned object does."""
    folder = tempfile.TemporaryDirectory(prefix="silvan_")
    path = os.path.join(folder.name, "graph.txt")
    _text(pairs).tofile(path)
    return folder, path


def _graph(family, size, degree, directed, seed):
    folder, path = _write(_pairs(family, size, degree, directed, seed))
    g = sb.Graph.load(path, directed)
    folder.cleanup()
    return g


def _host_graph(scale, directed, seed):
    p = _pairs("rmat", scale, 0, directed, seed).to(torch.int32).cpu().numpy()
    return sb.HostGraph.from_pairs(p.astype(np.uint32), directed)


def _sizes(case):
    """The sizes of a batch, from 1000 nodes up, spread over their logarithm."""
    c = case["count"]
    return [int(round(1000 * (case["size"] / 1000) ** (i / max(1, c - 1)))) | 1 for i in range(c)]


def _options(case, seed):
    """Estimator options of a case; road-like graphs are sampled one path at
    a time (-s 0), the others at the default rate."""
    o = dict(eps=case["eps"], delta=DELTA, k=case["k"], seed=seed)
    if case["family"] == "grid":
        o.update(alpha=0.0, alpha_given=True)
    if case["sigma"]:
        o.update(backtrack="sigma")
    return o


def prepare(case, seed):
    job, directed = case["job"], case["directed"]
    family, size, degree = case["family"], case["size"], case["degree"]
    if job == "batch":
        graphs = [_graph("er" if i % 2 else "ba", s, 4, False, seed * 64 + i)
                  for i, s in enumerate(_sizes(case))]
        return {"case": case, "graphs": graphs, "seed": seed}
    if job == "serve":
        # requests of scale 10 up to the case's, directed or not, at two bounds
        reqs = []
        for i in range(case["count"]):
            scale = 10 + i % (size - 9)
            o = dict(eps=(0.01, 0.005)[i % 3 == 0], delta=DELTA, seed=seed + i)
            reqs.append((_host_graph(scale, i % 2 == 1, seed * 64 + i), o))
        return {"case": case, "requests": reqs, "server": sb.Server(1 << size, budget=8 << 30)}
    if job == "ingest":
        pairs = _pairs(family, size, degree, directed, seed)
        if family == "rmat":  # in random order, the same number for every seed
            gen = torch.Generator(pairs.device).manual_seed(seed)
            mix = torch.randperm(len(pairs), generator=gen, device=pairs.device)
            last = pairs[pairs.max(1).values == (1 << size) - 1][:1]
            rest = pairs[mix][pairs[mix].max(1).values < (1 << size) - 1]
            pairs = torch.cat([rest[: (8 << size) - 1], last])
        folder, path = _write(pairs)
        return {"case": case, "folder": folder, "path": path}
    g = _graph(family, size, degree, directed, seed)
    if job == "upload":
        csr = g.csr()
        for f in ("out_off", "out_adj", "in_off", "in_adj", "cc"):
            a = torch.from_numpy(np.ascontiguousarray(getattr(csr, f)))
            setattr(csr, f, (a.pin_memory() if torch.cuda.is_available() else a).numpy())
        return {"case": case, "csr": csr, "options": _options(case, seed)}
    return {"case": case, "graph": g, "options": _options(case, seed)}


# ---- one pass ----------------------------------------------------------------

_COUNTS = ("first_pass_samples", "num_samples", "vis_edges", "void_samples", "backtracked_paths",
           "checks")


def _outputs(result, centrality):
    out = {f: int(result[f]) for f in _COUNTS}
    out["centrality"] = centrality
    return out


def _estimate(graph, options):
    est = sb.Probabilistic(graph, **options)
    out = _outputs(est.run(), est.get_centrality())
    if options["k"]:
        nodes, values = est.topk()
        # the count varies with the graph: room for any
        out["top_nodes"] = np.zeros(4096, np.int64)
        out["top_values"] = np.zeros(4096)
        out["top_nodes"][:len(nodes)] = nodes
        out["top_values"][:len(nodes)] = values
    return out


def run(state):
    case = state["case"]
    job = case["job"]
    if job == "estimate":
        return _estimate(state["graph"], state["options"])
    if job == "upload":
        return _estimate(sb.Graph.upload(state["csr"]), state["options"])
    if job == "batch":
        jobs = [sb.Probabilistic(g, eps=case["eps"], delta=DELTA, seed=state["seed"] + i)
                for i, g in enumerate(state["graphs"])]
        results = sb.run_batched(jobs)
        return {"num_samples": np.array([r["num_samples"] for r in results]),
                "vis_edges": np.array([r["vis_edges"] for r in results]),
                "centrality": [j.get_centrality() for j in jobs]}
    if job == "serve":
        server = state["server"]
        ids = [server.submit(hg, **o) for hg, o in state["requests"]]
        results = [server.wait(i) for i in ids]
        return {"num_samples": np.array([r["num_samples"] for r in results]),
                "vis_edges": np.array([r["vis_edges"] for r in results]),
                "centrality": [server.estimates(i, hg.info().n)
                               for i, (hg, _) in zip(ids, state["requests"])]}
    if job == "ingest":
        c = sb.Graph.load(state["path"], case["directed"]).csr()
        return {"out_off": c.out_off.view(np.int64), "out_adj": c.out_adj.view(np.int32),
                "in_off": c.in_off.view(np.int64), "in_adj": c.in_adj.view(np.int32),
                "cc": c.cc.view(np.int32), "n_components": c.n_components, "diameter": c.diameter}
    return state["graph"].exact_betweenness()


# ---- what a pass cannot do without -----------------------------------------


def _shape(family, size, degree):
    """(nodes, adjacency entries) of a graph, about."""
    if family == "rmat":
        return 1 << size, 16 << size
    if family == "grid":
        return size * size, int(3.8 * size * size)
    return size, (8 if family == "er" else 2 * degree) * size


def _estimate_bytes(family, size, degree, directed, eps, k):
    """Bytes of an estimation, about: per scanned entry the neighbour's id and
    its state, per sample the entries that two searches from both ends scan
    until they meet; the centralities written once."""
    n, m = _shape(family, size, degree)
    if family == "grid":
        scanned = 35.0 * m ** 0.5
        samples = (9000.0 if k else 72.0) / eps
    else:
        scanned = 1.5 * m ** 0.5 * (0.4 if directed else 1.0)
        samples = 120.0 / eps if not k else 20000.0 / eps
    return samples * scanned * 8 + 8 * n


def work(case):
    family, size, degree = case["family"], case["size"], case["degree"]
    directed = case["directed"]
    n, m = _shape("er" if family == "mixed" else family, size, degree)
    rows = 2 if directed else 1
    if case["job"] == "exact":
        # every source: its search reads each entry and each node's state
        # twice (forward, backward)
        return {"bytes": 2.0 * n * (4 * m + 16 * n), "flops": 3.0 * n * m}
    if case["job"] == "ingest":
        text = 13.0 * m / (1 if directed else 2)
        return {"bytes": text + rows * (4 * m + 8 * n) * 2 + 4 * n, "flops": 0}
    if case["job"] == "batch":
        return {"bytes": sum(_estimate_bytes("er", s, 4, False, case["eps"], 0)
                             for s in _sizes(case)), "flops": 0}
    if case["job"] == "serve":
        total = 0.0
        for i in range(case["count"]):
            scale = 10 + i % (size - 9)
            total += (16 << scale) * 8 + _estimate_bytes("rmat", scale, 0, i % 2 == 1, 0.0075, 0)
        return {"bytes": total, "flops": 0}
    total = _estimate_bytes(family, size, degree, directed, case["eps"], case["k"])
    if case["job"] == "upload":
        total += rows * (4 * m + 8 * n) + 4 * n
    return {"bytes": total, "flops": 0}


# ---- values in 64 bits ----------------------------------------------------------


def exact(case, seed):
    """The exact centralities of the graph of an ``exact`` case, from dense
    64-bit path counts.  An estimate is a sum over a stream of sampled paths,
    one search after another, whose length the stopping rule sets: replayed
    without this library it takes minutes; an ingest gives whole numbers."""
    if case["job"] != "exact" or case["size"] > 12000:
        return None
    dev = _device()
    n = case["size"]
    pairs = _pairs(case["family"], n, case["degree"], False, seed)
    n = int(pairs.max()) + 1
    adj = torch.zeros(n, n, dtype=torch.float64, device=dev)
    adj[pairs[:, 0], pairs[:, 1]] = 1
    adj[pairs[:, 1], pairs[:, 0]] = 1
    # row s: the searches from s, one level a step
    dist = torch.full((n, n), -1, dtype=torch.int64, device=dev)
    sigma = torch.eye(n, dtype=torch.float64, device=dev)
    dist.fill_diagonal_(0)
    level, front = 0, sigma.clone()
    while True:
        reached = front @ adj
        new = (dist < 0) & (reached > 0)
        if not bool(new.any()):
            break
        level += 1
        dist[new] = level
        front = torch.where(new, reached, 0.0)
        sigma += front
    dep = torch.zeros_like(sigma)
    for d in range(level, 0, -1):
        share = torch.where(dist == d, (1 + dep) / sigma.clamp(min=1), 0.0)
        dep += torch.where(dist == d - 1, sigma * (share @ adj), 0.0)
    dep.fill_diagonal_(0)
    return (dep.sum(0) / (n * (n - 1))).cpu().numpy()
