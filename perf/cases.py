"""The work a user of the engine has it do, as cases that can be timed and checked one by one.

Every case is a graph of the R-MAT family (a, b, c, d = 0.57, 0.19, 0.19, 0.05; n need not be a
power of two) made from its seed on the GPU, and one pass through the public entry points on it:

  solve    one whole solve on the device loop, with the command line's automatic settings, and
           the results read into pinned host memory (measure pr, katz, ev or all)
  host     the same solve by the host-driven pass loop (snapshot, plan, push, wait), the
           command line's default
  pinned   a solve whose later chunks stay in pinned host memory, read in place over the link
  query    one personalized PageRank query, seeded into the engine and resumed
  batch    B personalized PageRank (or Katz) queries at once, and every lane read back
  adjoint  weighted PageRank or Katz through torch.autograd: x, and the gradients of the
           edge weights and of the teleport (beta) vector
  params   the given constants of a graph (lambda1, alpha, means) and its unit eigenvector

eps: PageRank 0.01 unless given; "given" takes Katz and the eigenvector to 1 % of their means, the
rule of the given constants, with alpha = 0.85 / lambda1; a number is an absolute threshold with
alpha = 0.9 / lambda1, FP64 eigenvector start and the FP64 normalisation step, as the benchmark.
An eigenvector has no scale of its own: it is compared, as everywhere here, as a unit vector.
"""
import math
import random

import numpy as np
import torch

import excent_b200 as X
from excent_b200.autograd import WeightedGraph, centrality

A, B, C = 0.57, 0.19, 0.19
DAMP = 0.85


def listed():
    return [
        # the shipped sample's size with its own constants: every pass is launches and latency
        {"name": "sample_all", "path": "solve", "measure": "all", "n": 2000, "ef": 8, "eps": "given"},
        # the smallest benchmark graph, plain PageRank to the default threshold
        {"name": "pr_s16", "path": "solve", "measure": "pr", "n": 1 << 16, "ef": 16, "eps": 0.01},
        # Katz of a mid-sized graph of a ragged size, to 1 % of its mean
        {"name": "katz_mid", "path": "solve", "measure": "katz", "n": 300007, "ef": 24, "eps": "given"},
        # the eigenvector of a sparse graph of several chunks, to the benchmark's threshold
        {"name": "ev_1m", "path": "solve", "measure": "ev", "n": 1200001, "ef": 8, "eps": 1e-6},
        # plain PageRank on the largest cached benchmark graph
        {"name": "pr_s24", "path": "solve", "measure": "pr", "n": 1 << 24, "ef": 16, "eps": 0.01},
        # the benchmark's default workload: all three measures over one stream of that graph
        {"name": "all_s24", "path": "solve", "measure": "all", "n": 1 << 24, "ef": 16, "eps": 1e-6},
        # the command line's own loop: the host plans every pass
        {"name": "host_all", "path": "host", "measure": "all", "n": 700001, "ef": 16, "eps": "given"},
        # a graph that does not fit the edge cache: half its chunks read over the host link
        {"name": "pinned_pr", "path": "pinned", "measure": "pr", "n": 1 << 20, "ef": 16, "eps": 0.01},
        # a single personalized query against a loaded graph
        {"name": "query_s20", "path": "query", "n": 1 << 20, "ef": 16, "eps": 1e-6, "size": 64},
        # a batch of queries of uneven seed sets, to an accuracy that a ranking can use
        {"name": "batch_s17", "path": "batch", "kind": "ppr", "n": 1 << 17, "ef": 16, "lanes": 64, "eps": 1e-6},
        # training through the centrality: forward, adjoint and the gradient of every edge weight
        {"name": "adjoint_s20", "path": "adjoint", "kind": "pr", "n": 1 << 20, "ef": 16, "eps": 1e-7},
        # the constants that Katz, the eigenvector and `all` need of any new graph
        {"name": "params_s20", "path": "params", "n": 1 << 20, "ef": 16},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["solve", "solve", "solve", "solve", "host", "pinned", "query", "batch", "adjoint", "params"])
    ef = rng.choice([8, 12, 16, 24, 32])
    c = {"path": path, "ef": ef}
    if path in ("solve", "host", "pinned"):
        c["measure"] = rng.choice(["pr", "katz", "ev", "all"]) if path != "pinned" else rng.choice(["pr", "all"])
        top = {"solve": 1 << 26, "host": 1 << 24, "pinned": 1 << 24}[path] // ef
        low = 2000 if path != "pinned" else (10 << 20) // ef   # a graph of several chunks
        c["n"] = _log_int(rng, low, top)
        c["eps"] = rng.choice([0.01, 0.01, 1e-3, 1e-4]) if c["measure"] == "pr" else rng.choice(["given", "given", 1e-6])
    elif path == "query":
        c["n"] = _log_int(rng, 2000, (1 << 24) // ef)
        c["eps"] = rng.choice([1e-6, 1e-7])
        c["size"] = _log_int(rng, 1, min(4096, c["n"] // 4))
    elif path == "batch":
        c["lanes"] = rng.choice([32, 64, 128, 256])
        c["n"] = _log_int(rng, 2000, (1 << 22) // ef)
        c["kind"] = rng.choice(["ppr", "ppr", "katz"])
        c["eps"] = rng.choice([1e-6, 1e-7])
    elif path == "adjoint":
        c["n"] = _log_int(rng, 2000, (1 << 24) // ef)
        c["kind"] = rng.choice(["pr", "katz"])
        c["eps"] = rng.choice([1e-6, 1e-7])
    else:
        c["n"] = _log_int(rng, 2000, (1 << 24) // ef)
    return c


def _rmat_pairs(n, count, gen):
    """`count` (source, target) pairs below n: quadrant by quadrant, those outside n or on the diagonal drawn again."""
    got, have = [], 0
    scale = max(1, (n - 1).bit_length())
    while have < count:
        k = min(max(2 * (count - have), 1024), 1 << 24)
        s = torch.zeros(k, dtype=torch.int64, device="cuda")
        t = torch.zeros(k, dtype=torch.int64, device="cuda")
        for _ in range(scale):
            u = torch.rand(k, generator=gen, device="cuda")
            s = 2 * s + (u >= A + B)
            t = 2 * t + (((u >= A) & (u < A + B)) | (u >= A + B + C))
        keep = (s < n) & (t < n) & (s != t)
        s, t = s[keep][: count - have], t[keep][: count - have]
        got.append((s, t))
        have += len(s)
    return torch.cat([p[0] for p in got]), torch.cat([p[1] for p in got])


def graph(n, ef, seed, symmetric=True):
    """CSR on the GPU, sorted lists without duplicates: offsets int64 [n + 1], targets int32 [m].
    A directed graph has n * ef entries exactly (so have its weights), a symmetric one at most that many."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    if symmetric:
        s, t = _rmat_pairs(n, n * ef // 2, gen)
        keys = torch.unique(torch.cat([s * n + t, t * n + s]))
    else:
        keys, count = torch.empty(0, dtype=torch.int64, device="cuda"), n * ef
        while len(keys) < n * ef:
            count += count // 4
            s, t = _rmat_pairs(n, count, gen)
            keys = torch.unique(s * n + t)
        keys = keys[torch.randperm(len(keys), generator=gen, device="cuda")[: n * ef].sort().values]
    del s, t
    idx = torch.searchsorted(keys, torch.arange(n + 1, device="cuda") * n)
    return idx, (keys % n).to(torch.int32)


def _weights(m, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed + 7)
    return torch.rand(m, generator=gen, device="cuda") + 0.5


def _targets(n, seed):
    """Which vertices the loss of the adjoint case sums over."""
    r = np.random.RandomState(seed)
    return torch.from_numpy(np.sort(r.choice(n, min(1000, n // 4), replace=False))).cuda()


def _queries(n, count, seed, size=None):
    """Seed sets, log-uniform in [1, 4096] unless the size is given."""
    r = np.random.RandomState(seed)
    top = min(4096, n // 4)
    sizes = [size or max(1, int(math.exp(r.uniform(0, math.log(top))))) for _ in range(count)]
    return [np.sort(r.choice(n, k, replace=False)).astype(np.int32) for k in sizes]


def _kinds(case):
    return ["pr", "katz", "ev"] if case["measure"] == "all" else [case["measure"]]


def _engine(case, idx, adj):
    """An engine with the settings that the command line picks by itself; the cache is left to the caller."""
    n, m = case["n"], adj.numel()
    m_kind, kw, v1 = case["measure"], {}, None
    if m_kind == "pr":
        kw["eps_pr"] = case["eps"]
    else:
        given = case["eps"] == "given"
        v1 = torch.empty(n, dtype=torch.float32, device="cuda")
        p = X.params_fp64(n, idx, adj, 0.85 if given else 0.9, v1_out=v1)
        kw = {"alpha": p["alpha"], "lam": p["lambda"],
              "eps_katz": 0.01 * p["mean_katz"] if given else case["eps"],
              "eps_ev": 0.01 * p["mean_ev"] if given else case["eps"], "ev_init_fp64": not given}
        if given or m_kind == "katz":
            v1 = None
    meas = X.measures(m_kind, **kw)
    v0, e = X.plan_chunks(idx.cpu().numpy().view(np.uint64), X.chunk_cap(m))
    return X.Engine(n, m, meas, v0, e), v1


def _hub_targets(eng):
    k = (2048 if eng.nc > 1 else 16384) if eng.meas.nm == 1 else 4096
    return min(k, eng.n)


def prepare(case, seed):
    path, n = case["path"], case["n"]
    st = {"case": case}
    idx, adj = graph(n, case["ef"], seed, symmetric=path != "adjoint")
    m = adj.numel()
    torch.cuda.synchronize()
    if path in ("solve", "host", "pinned"):
        eng, v1 = _engine(case, idx, adj)
        if path == "pinned":
            eng.upload_offsets(idx.cpu())
            first = int(eng.chunk_e[max(1, eng.nc // 2)])
            host = adj.cpu()
            eng.reserve_cache(first)
            eng.load_cache(0, first, host[:first])
            eng.set_hub_targets(_hub_targets(eng))
            buf, at = eng.host_cache()
            buf[:] = host[at:].numpy()
        else:
            eng.upload_device(idx, adj)
            eng.set_hub_targets(_hub_targets(eng))
        if v1 is not None:
            eng.ev_project(v1)
        st["eng"] = eng
        st["out"] = {k: torch.empty(n, dtype=torch.float32, pin_memory=True) for k in _kinds(case)}
    elif path == "query":
        meas = X.measures("pr", eps_pr=case["eps"] * (1 - DAMP))
        v0, e = X.plan_chunks(idx.cpu().numpy().view(np.uint64), X.chunk_cap(m))
        eng = X.Engine(n, m, meas, v0, e)
        eng.upload_device(idx, adj)
        st["eng"] = eng
        st["query"] = _queries(n, 1, seed, case["size"])[0]
        st["out"] = torch.empty(n, dtype=torch.float32, pin_memory=True)
    elif path == "batch":
        alpha = DAMP if case["kind"] == "ppr" else 0.5 / X.params_fp64(n, idx, adj)["lambda"]
        st["graph"] = (idx, adj)   # the batch reads the caller's arrays
        st["batch"] = X.Batch(n, m, idx, adj, case["lanes"], case["kind"], alpha)
        st["queries"] = _queries(n, case["lanes"], seed)
        st["values"] = [_mass(case) / len(q) for q in st["queries"]]
        st["out"] = torch.empty(case["lanes"], n, dtype=torch.float32, pin_memory=True)
    elif path == "adjoint":
        w = _weights(m, seed)
        st["graph"] = WeightedGraph(n, idx, adj, w)
        st["w"] = w.requires_grad_()
        st["t"] = torch.ones(n, device="cuda", requires_grad=True)
        st["targets"] = _targets(n, seed)
    else:
        st["graph"] = (idx, adj)
        st["v1"] = torch.empty(n, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    return st


def _mass(case):
    return 1 - DAMP if case["kind"] == "ppr" else 1.0


def _read(eng, outs):
    """Every measure into the caller's pinned memory; the eigenvector as a unit vector."""
    got = {}
    for i, (k, o) in enumerate(outs.items()):
        eng.read(i, out=o)
        got[k] = o
        if k == "ev":
            x = o.cuda(non_blocking=True)
            got[k] = x / torch.linalg.vector_norm(x, dtype=torch.float64)
    return got


def run(st):
    case = st["case"]
    path = case["path"]
    if path in ("solve", "pinned"):
        st["eng"].solve()
        return _read(st["eng"], st["out"])
    if path == "host":
        eng = st["eng"]
        eng.init()
        while True:
            cnt, _, _ = eng.snapshot()
            pending = cnt[0::2] > 0
            if not pending.any():
                break
            eng.push_cached(pending.astype(np.uint8), cnt)
            eng.sync()
        return _read(eng, st["out"])
    if path == "query":
        eng = st["eng"]
        X.seed_engine(eng, st["query"], (1 - DAMP) / len(st["query"]))
        X.resume(eng)
        eng.read(0, out=st["out"])
        return st["out"]
    if path == "batch":
        b = st["batch"]
        b.seed(st["queries"], st["values"], case["eps"] * _mass(case))
        b.solve()
        for lane in range(case["lanes"]):
            b.read(lane, out=st["out"][lane])
        return st["out"]
    if path == "adjoint":
        st["w"].grad = st["t"].grad = None
        x = centrality(st["graph"], st["w"], st["t"], case["kind"], _strength(case), eps=case["eps"])
        x[st["targets"]].sum().backward()
        return {"x": x.detach(), "w": st["w"].grad, "t": st["t"].grad}
    idx, adj = st["graph"]
    p = X.params_fp64(case["n"], idx, adj, v1_out=st["v1"])
    return {"v1": st["v1"], **{k: float(p[k]) for k in ("lambda", "alpha", "mean_ev", "mean_katz")}}


def _strength(case):
    return DAMP if case["kind"] == "pr" else 0.6


def work(case):
    """The graph read once and the results written once; an add (and a multiply) per entry and result column."""
    n, path = case["n"], case["path"]
    m = n * case["ef"]
    if path in ("solve", "host", "pinned"):
        cols = len(_kinds(case))
    else:
        cols = case.get("lanes", 1)
    by, fl = 8 * (n + 1) + 4 * m + 4 * n * cols, 2 * m * cols
    if path == "adjoint":   # weights and targets read, x, both gradients written; forward, adjoint and gradient
        by, fl = 8 * (n + 1) + 8 * m + 4 * n * 3 + 4 * m, 6 * m
    return {"bytes": by, "flops": fl}


# ---------------------------------------------------------------- 64-bit values

def _matrix(n, idx, adj, values=None):
    values = torch.ones(adj.numel(), dtype=torch.float64, device="cuda") if values is None else values
    return torch.sparse_csr_tensor(idx.to(torch.int32), adj, values, size=(n, n), check_invariants=False)


def _fixed(apply, c, tol=1e-14, most=2000):
    """x = c + apply(x) by iteration, to a change of tol of the largest value."""
    x = c.clone()
    for i in range(most):
        y = c + apply(x)
        if i % 8 == 7 and float((y - x).abs().max()) <= tol * float(y.abs().max()):
            return y
        x = y
    return x


def _dominant(n, a, sweeps=3000):
    x = torch.full((n,), 1 / math.sqrt(n), dtype=torch.float64, device="cuda")
    lam = 0.0
    for i in range(sweeps):
        y = a @ x
        lam = float(torch.linalg.vector_norm(y)) if i % 8 == 7 else lam
        y /= torch.linalg.vector_norm(y)
        if i % 8 == 7 and float((y - x).abs().max()) < 1e-13:
            break
        x = y
    return y, lam


def exact(case, seed):
    path, n = case["path"], case["n"]
    idx, adj = graph(n, case["ef"], seed, symmetric=path != "adjoint")
    if path == "adjoint":
        return _exact_adjoint(case, seed, idx, adj)
    a = _matrix(n, idx, adj)
    deg = (idx[1:] - idx[:-1]).clamp(min=1).to(torch.float64)

    def ppr(x):
        return DAMP * (a @ (x / (deg[:, None] if x.dim() == 2 else deg)))

    one = torch.ones(n, dtype=torch.float64, device="cuda")
    if path in ("solve", "host", "pinned"):
        out, v, lam = {}, None, 0.0
        if case["measure"] != "pr":
            v, lam = _dominant(n, a)
        alpha = (0.85 if case["eps"] == "given" else 0.9) / lam if lam else 0.0
        for k in _kinds(case):
            out[k] = (_fixed(ppr, (1 - DAMP) * one) if k == "pr" else
                      _fixed(lambda x: alpha * (a @ x), one) if k == "katz" else v)
        return out
    if path in ("query", "batch"):
        qs = _queries(n, 1, seed, case["size"]) if path == "query" else _queries(n, case["lanes"], seed)
        mass = 1 - DAMP if path == "query" else _mass(case)
        c = torch.zeros(n, len(qs), dtype=torch.float64, device="cuda")
        for j, q in enumerate(qs):
            c[torch.from_numpy(q.astype(np.int64)).cuda(), j] = float(np.float32(mass / len(q)))
        if path == "query":
            return _fixed(ppr, c[:, 0])
        alpha = 0.5 / _dominant(n, a)[1] if case["kind"] == "katz" else 0.0
        return _fixed(ppr if case["kind"] == "ppr" else lambda x: alpha * (a @ x), c).t()
    v, lam = _dominant(n, a)
    katz = _fixed(lambda x: 0.85 / lam * (a @ x), one)
    return {"v1": v, "lambda": lam, "alpha": 0.85 / lam, "mean_ev": float(v.sum()) ** 2 / n,
            "mean_katz": float(katz.mean())}


def _exact_adjoint(case, seed, idx, adj):
    n, s = case["n"], _strength(case)
    m = adj.numel()
    w = _weights(m, seed).double()
    row = torch.repeat_interleave(torch.arange(n, device="cuda"), idx[1:] - idx[:-1])
    total = torch.zeros(n, dtype=torch.float64, device="cuda").index_add_(0, row, w)
    wn = w / total[row]
    order = torch.argsort(adj.long() * n + row)
    t_idx = torch.searchsorted(adj.long()[order], torch.arange(n + 1, device="cuda"))
    fwd, back = _matrix(n, t_idx, row[order].to(torch.int32), wn[order]), _matrix(n, idx, adj, wn)
    c0 = 1 - s if case["kind"] == "pr" else 1.0
    x = _fixed(lambda v: s * (fwd @ v), torch.full((n,), c0, dtype=torch.float64, device="cuda"))
    c = torch.zeros(n, dtype=torch.float64, device="cuda")
    c[_targets(n, seed)] = 1.0
    lam = _fixed(lambda v: s * (back @ v), c)
    g = s * x[row] * lam[adj.long()]
    dot = torch.zeros(n, dtype=torch.float64, device="cuda").index_add_(0, row, wn * g)
    return {"x": x, "w": (g - dot[row]) / total[row], "t": c0 * lam}


if __name__ == "__main__":
    print([c["name"] for c in listed()], draw(random.Random(1)))
