"""The solve that runs its passes in one launch, against the host-driven loop
and the FP64 oracle: edges of the tiles, waves, chunk tables and orders."""
import numpy as np
import pytest

import oracle as O
from test_long_lists_gpu import edged_graph

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a GPU", allow_module_level=True)

import excent_b200 as X  # noqa: E402

EPS = 1e-6


def engine(n, idx, adj, measure, cap, **kw):
    meas = X.measures(measure, eps_pr=EPS, eps_katz=EPS, eps_ev=EPS, **kw)
    v0, e = X.plan_chunks(idx, cap)
    eng = X.Engine(n, len(adj), meas, v0, e)
    eng.upload_graph(idx, adj)
    return eng


def close_enough(kind, n, x, ref):
    """What residuals of at most EPS leave: PageRank in the 1-norm (factor 1 / 0.15), Katz at alpha =
    0.5 / lambda1 in the 2-norm (factor 2); FP32 sums beside it."""
    d = np.abs(x.astype(np.float64) - ref)
    if kind == "pr":
        return d.sum() <= n * EPS / 0.15 + 1e-5 * ref.sum()
    return np.linalg.norm(d) <= 2 * np.sqrt(n) * EPS + 1e-5 * np.linalg.norm(ref)


@pytest.mark.parametrize("n", [1, 2, 33, 2500, 70001, 300007])
@pytest.mark.parametrize("hubs", [0, 300])
def test_pagerank_sizes(n, hubs):
    if n < 100:
        idx = np.arange(n + 1, dtype=np.uint64)          # a directed ring
        adj = ((np.arange(n) + 1) % n).astype(np.int32)
        ref = np.ones(n)
    else:
        idx, adj = edged_graph(n, n, symmetric=True)
        ref = O.reference_solution(n, idx, adj, "pr")
    for use_graph in (True, False):
        eng = engine(n, idx, adj, "pr", len(adj))
        eng.set_hub_targets(min(hubs, n))
        st = eng.solve(use_graph=use_graph)
        assert np.all(np.abs(eng.read(0, residual=True)) <= np.float32(EPS))
        assert close_enough("pr", n, eng.read(0), ref), use_graph
        s2, log = eng.stats(with_log=True)
        assert sum(int(p.pushed) for p in log) == st.pushed and len(log) == st.passes
        eng.close()


@pytest.mark.parametrize("order", ["table", "first", "last", "launch-first"])
@pytest.mark.parametrize("sweep", [False, True])
@pytest.mark.parametrize("cap", [1, 900, 10 ** 9])
def test_orders_and_chunk_tables(order, sweep, cap):
    """cap 1: one vertex a chunk, more chunks than a block plans for; 10^9: a single chunk."""
    n = 2500
    idx, adj = edged_graph(n, 3, symmetric=True)
    lam = float(O.params(n, idx, adj)["_lambda"])
    kw = dict(alpha=0.5 / lam, lam=lam, ev_init_fp64=True)
    eng = engine(n, idx, adj, "all", cap, **kw)
    assert eng.nc == (1 if cap > n * n else eng.nc) and (cap != 1 or eng.nc > 1024)
    eng.set_hub_order(order)
    eng.set_chunk_sweep(sweep)
    eng.set_sweep_demand(0.25)
    # (the eigenvector keeps a component above 1e-6 in FP32 in the order "last", with any loop: it only
    # runs beside the other two here)
    st = eng.solve(max_passes=300)
    assert st.passes > 0
    for i, k in enumerate(("pr", "katz")):
        assert np.all(np.abs(eng.read(i, residual=True)) <= np.float32(EPS))
        ref = O.reference_solution(n, idx, adj, k, alpha=0.5 / lam)
        assert close_enough(k, n, eng.read(i), ref), k
    eng.close()


@pytest.mark.parametrize("passes", [0, 1, 5])
def test_pass_limit(passes):
    """The passes themselves, step by step in FP64: the lists longer than 256 entries are taken
    together and scattered, then the others (a few thousand vertices are one wave)."""
    n = 2500
    idx, adj = edged_graph(n, 5, symmetric=True)
    deg = np.diff(idx.astype(np.int64))
    src = np.repeat(np.arange(n), deg)
    r, x = np.full(n, float(np.float32(1) - np.float32(0.85))), np.zeros(n)
    for _ in range(passes):
        for phase in (deg > 256, deg <= 256):
            d = np.where(phase & (np.abs(r) > EPS), r, 0.0)
            x += d
            r -= d
            np.add.at(r, adj, (0.85 * d / np.maximum(deg, 1))[src])
    eng = engine(n, idx, adj, "pr", len(adj))
    st = eng.solve(max_passes=passes)
    assert st.passes == passes
    # FP32 sums of up to 2049 terms
    assert np.allclose(eng.read(0), x, rtol=1e-5, atol=1e-6)
    assert np.allclose(eng.read(0, residual=True), r, rtol=1e-5, atol=1e-6)
    eng.close()


@pytest.mark.parametrize("kind", ["directed", "one entry turned", "symmetric", "reloaded"])
@pytest.mark.parametrize("n", [2500, 70001])
def test_swept_passes_gather_only_on_symmetric_graphs(n, kind):
    """A swept pass gathers along a vertex's own list, which holds what points to it only on a
    symmetric graph: with lists that are not, and with lists loaded anew, the solve agrees with the
    host-driven loop (two residuals of at most EPS per vertex apart in the 1-norm)."""
    idx, adj = edged_graph(n, 7, symmetric=kind != "directed")
    if kind == "one entry turned":
        v = int(np.nonzero(np.diff(idx.astype(np.int64)) == 2)[0][0])
        lst = adj[int(idx[v]):int(idx[v + 1])]
        lst[0] = next(u for u in range(n) if u not in lst and u != v)
    got = []
    for use_graph in (True, False):
        eng = engine(n, idx, adj, "pr", len(adj) // 6 + 1)
        assert eng.nc > 4
        eng.set_hub_targets(100)
        eng.set_sweep_demand(0.1)
        if kind == "reloaded":   # solved on other lists first
            other = np.ascontiguousarray((n - 1 - adj).astype(np.int32))
            eng.load_cache(0, len(adj), other)
            eng.solve(use_graph=use_graph)
            eng.load_cache(0, len(adj), adj)
        eng.solve(use_graph=use_graph)
        assert np.all(np.abs(eng.read(0, residual=True)) <= np.float32(EPS))
        got.append(eng.read(0).astype(np.float64))
        eng.close()
    assert np.abs(got[0] - got[1]).sum() <= 2 * n * EPS / 0.15 + 1e-5 * got[1].sum()


@pytest.mark.parametrize("measure", ["pr", "all"])
@pytest.mark.parametrize("passes", [1, 2])
def test_swept_pass_of_every_part_length(passes, measure):
    """The parts of a split list (neighbours taken before the vertex, and the others) at the edges of
    their classes, both ways: the passes step by step in FP64, chunk by chunk, lists longer than 256
    entries first; a chunk takes what is pending by then, unless the pass began with less than
    list_frac of it pending, which are then the ones taken. FP32 sums of up to some 600 terms."""
    n = 4000
    rng = np.random.default_rng(11)
    src, dst = [], []
    for i, k in enumerate([1, 7, 8, 9, 31, 32, 33, 64, 257, 600]):
        for v, lo in ((n - 1 - i, 0), (i, n // 2)):   # neighbours in the first quarter, or in the third
            src.append(np.full(k, v))
            dst.append(lo + 100 + rng.choice(n // 4, k, replace=False))
    src, dst = np.concatenate(src), np.concatenate(dst)
    keys = np.unique(np.concatenate([src * n + dst, dst * n + src]))
    src, dst = keys // n, keys % n
    idx = np.zeros(n + 1, dtype=np.uint64)
    np.cumsum(np.bincount(src, minlength=n), out=idx[1:])
    adj = dst.astype(np.int32)
    deg = np.diff(idx.astype(np.int64))
    eng = engine(n, idx, adj, measure, len(adj) // 8 + 1, alpha=0.01, lam=25.0)
    assert eng.nc > 4
    eng.set_chunk_sweep(True)
    eng.set_sweep_demand(0.01)
    assert eng.solve(max_passes=passes, list_frac=0.5).passes == passes
    chunk = np.searchsorted(np.asarray(eng.chunk_v0)[:eng.nc], np.arange(n), side="right") - 1
    r, x = np.full(n, float(np.float32(1) - np.float32(0.85))), np.zeros(n)
    for _ in range(passes):
        first = np.abs(r) > EPS
        few = np.bincount(chunk, first, eng.nc) < 0.5 * np.bincount(chunk, minlength=eng.nc)
        for c in range(eng.nc):
            for long in (True, False):
                d = np.where((chunk == c) & ((deg > 256) == long) & (np.abs(r) > EPS) & (first | ~few[chunk]), r, 0.0)
                x += d
                r -= d
                np.add.at(r, adj, (0.85 * d / np.maximum(deg, 1))[src])
    assert np.allclose(eng.read(0), x, rtol=1e-5, atol=1e-6)
    assert np.allclose(eng.read(0, residual=True), r, rtol=1e-5, atol=1e-6)
    eng.close()
