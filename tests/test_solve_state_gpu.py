"""What a solve and a host-driven push leave behind, and what engines and
streams share."""
import ctypes as C
import threading

import numpy as np
import pytest

import oracle as O
from test_long_lists_gpu import edged_graph
from test_passes_gpu import EPS, close_enough, engine

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a GPU", allow_module_level=True)

import excent_b200 as X  # noqa: E402
import excent_b200._capi as K  # noqa: E402


@pytest.mark.parametrize("sweep", [False, True])
@pytest.mark.parametrize("n,cap", [(2500, 900), (2500, 1), (70001, 20000), (300007, 10 ** 9)])
def test_pending_lists_after_a_solve(n, cap, sweep):
    """The pending list of every chunk is that of the last snapshot, whichever pass it ended: the
    vertices whose residual is above eps, none of them after convergence."""
    idx, adj = edged_graph(n, 4, symmetric=True)
    eng = engine(n, idx, adj, "pr", cap)
    assert (eng.nc == 1) == (cap > len(adj))
    eng.set_chunk_sweep(sweep)
    eng.set_sweep_demand(0.2)
    ends = np.append(eng.chunk_v0[1:], n)
    few = range(eng.nc) if eng.nc < 50 else list(range(20)) + list(range(eng.nc - 20, eng.nc))
    for passes in (0, 1, 2, 3, 4, 9, 10, 100000):
        eng.solve(max_passes=passes)
        pending = np.abs(eng.read(0, residual=True)) > np.float32(EPS)
        assert pending.any() == (passes < 100000)
        for c in few:
            lo, hi = int(eng.chunk_v0[c]), int(ends[c])
            assert np.array_equal(np.sort(eng.chunk_list(c)), lo + np.nonzero(pending[lo:hi])[0]), (passes, c)
    eng.close()


@pytest.mark.parametrize("how", ["set after a solve", "set after a solve, lists loaded anew"])
@pytest.mark.parametrize("measure,slots", [("pr", 32768), ("all", 8192)])
def test_swept_passes_follow_the_slots_set_last(measure, slots, how):
    """The phases of a swept pass follow the wave, which follows the slots: a first chunk of more
    vertices than six waves of one block to an SM is taken in one phase without slots and in two
    with all of them, whichever was set first and whether or not the lists are loaded anew (63
    chunks: the tables of the second split take more room than those of the first)."""
    n = 300007
    idx, adj = edged_graph(n, 6, symmetric=True)
    v0 = np.array([0] + [240000 + 968 * k for k in range(62)], dtype=np.int32)
    e = idx[np.append(v0, n)].astype(np.uint64)
    got = []
    for solved_before in (False, True):
        eng = X.Engine(n, len(adj), X.measures(measure, eps_pr=EPS, eps_katz=EPS, eps_ev=EPS, alpha=0.01, lam=25.0), v0, e)
        eng.upload_graph(idx, adj)
        eng.set_sweep_demand(0.01)
        if solved_before:
            eng.solve(max_passes=1)
        eng.set_hub_targets(slots)
        if solved_before and how.endswith("anew"):
            eng.load_cache(0, len(adj), adj)
        eng.solve(max_passes=1)
        got.append((eng.read(0), eng.read(0, residual=True)))
        eng.close()
    for a, b in zip(*got):   # the same takes in the same order: FP32 sums of up to 2049 terms apart
        assert np.allclose(a, b, rtol=1e-5, atol=1e-6)


def test_slots_of_another_engine_leave_an_engine_its_own(rmat16):
    """Two engines of one process: the one with more slots solves and pushes as before after the other
    has set fewer."""
    n, idx, adj = rmat16
    lam = float(O.params(n, idx, adj)["_lambda"])
    many = engine(n, idx, adj, "all", len(adj) // 5, alpha=0.5 / lam, lam=lam)
    many.set_hub_targets(8192)
    few = engine(n, idx, adj, "all", len(adj) // 5, alpha=0.5 / lam, lam=lam)
    few.set_hub_targets(64)
    for sweep in (True, False):
        many.set_chunk_sweep(sweep)
        for use_graph in (True, False):
            many.solve(max_passes=20, use_graph=use_graph)
        many.init()
        cnt, _, _ = many.snapshot()
        many.push_cached((cnt[0::2] > 0).astype(np.uint8), cnt)
        many.sync()
    assert many.scatter_peak() > 0
    many.close()
    few.close()


def test_small_solves_of_two_threads(rmat12):
    """Two threads solve small graphs with different numbers of slots at the same time."""
    n, idx, adj = rmat12
    engines = [engine(n, idx, adj, "pr", len(adj)) for _ in range(2)]
    for eng, k in zip(engines, (n, 8)):
        eng.set_hub_targets(k)
    bad = []

    def solves(eng):
        try:
            for _ in range(300):
                eng.solve(max_passes=3)
        except Exception as ex:   # noqa: BLE001
            bad.append(ex)
    threads = [threading.Thread(target=solves, args=(eng,)) for eng in engines]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, bad[0]
    for eng in engines:
        eng.close()


@pytest.mark.parametrize("use_graph", [True, False])
def test_one_chunk_of_lists_in_host_memory_goes_as_a_range(use_graph):
    """A chunk read over the host link is pushed as a range in every pass, also by the solve of a
    graph whose vertices fit the GPU's threads: one that turns pending in a pass is pushed in it."""
    n = 2500
    idx, adj = edged_graph(n, 8, symmetric=True)
    meas = X.measures("pr", eps_pr=EPS)
    eng = X.Engine(n, len(adj), meas, *X.plan_chunks(idx, len(adj)))
    assert eng.nc == 1
    eng.upload_offsets(idx)
    eng.reserve_cache(0)
    buf, first = eng.host_cache()
    assert first == 0
    buf[:] = adj
    st = eng.solve(use_graph=use_graph)
    assert (st.n_list, st.n_range) == (0, st.passes) and eng.host_pushed() == st.pushed
    assert close_enough("pr", n, eng.read(0), O.reference_solution(n, idx, adj, "pr"))
    eng.close()


@pytest.mark.parametrize("kind,s", [("pr", 0.85), ("katz", 0.6)])
def test_a_residual_that_is_not_a_number_stays_where_it_is(kind, s):
    """A row whose weights are all 0 has no normalised weights. Its targets' residuals are no numbers
    from its first push on: they are taken no more, and nothing of them reaches other vertices."""
    from excent_b200.autograd import WeightedGraph
    n, k = 2000, 4
    rng = np.random.default_rng(3)
    adj = np.concatenate([np.sort(rng.choice(n, k, replace=False)) for _ in range(n)]).astype(np.int32)
    idx = (np.arange(n + 1) * k).astype(np.uint64)
    w = rng.uniform(0.5, 1.5, len(adj)).astype(np.float32)
    u = 77
    w[u * k:(u + 1) * k] = 0
    dev = torch.device("cuda")
    G = WeightedGraph(n, torch.from_numpy(idx.view(np.int64)).to(dev), torch.from_numpy(adj).to(dev),
                      torch.from_numpy(w).to(dev))
    src = np.repeat(np.arange(n), k)
    with np.errstate(all="ignore"):
        wn = w / np.bincount(src, w, n)[src]

    def push(frm, to, r):
        x = np.zeros(n)
        for _ in range(400):
            d = np.where(np.abs(r) > 1e-12, r, 0.0)   # (no number is above nothing)
            x += d
            r = np.where(d != 0, 0.0, r)
            np.add.at(r, to, np.where(d[frm] != 0, s * wn * d[frm], 0.0))
        return x

    c0 = 1 - s if kind == "pr" else 1.0
    x, _, _ = G.forward(kind, s, None, 1e-7)
    assert np.allclose(x.cpu().numpy(), push(src, adj, np.full(n, c0)), rtol=1e-4, atol=1e-5)
    c = np.zeros(n)
    c[rng.choice(n, 300, replace=False)] = 1
    c[adj[u * k]] = 1
    gt, gw = G.vjp(torch.from_numpy(c.astype(np.float32)).to(dev), 1e-7)
    lam = push(adj, src, c)
    assert np.allclose(gt.cpu().numpy(), c0 * lam, rtol=1e-4, atol=1e-5)
    finite = np.isfinite(gw.cpu().numpy())
    assert finite[src != u].all()
    G.close()


@pytest.mark.parametrize("order", ["first", "last", "launch-first"])
@pytest.mark.parametrize("sweep,degree_cache", [(False, False), (True, False), (False, True)])
def test_a_push_of_some_chunks_leaves_the_others_alone(order, sweep, degree_cache):
    """Chunks without pending vertices at the snapshot are in no push: their vertices, high-degree
    and without entries alike, keep what reaches them, also where their lists are not loaded."""
    n = 2500
    idx, adj = edged_graph(n, 9, symmetric=True)
    deg = np.diff(idx.astype(np.int64))
    eng = engine(n, idx, adj, "pr", 900)
    ends = np.append(eng.chunk_v0[1:], n)
    chunk = np.searchsorted(eng.chunk_v0, np.arange(n), side="right") - 1
    asked = np.arange(eng.nc) >= eng.nc // 2
    hubs = np.nonzero(deg > 256)[0]
    assert eng.nc > 4 and len(hubs) > 5 and not asked[chunk[hubs]].all()
    eng.set_hub_order(order)
    eng.set_chunk_sweep(sweep)
    eng.set_sweep_demand(0.0)
    for c in np.nonzero(~asked)[0]:
        eng.set_loaded(int(c), False)
    eng.init()
    x0 = np.zeros(n, dtype=np.float32)
    r0 = np.where(asked[chunk], np.float32(0.5), np.float32(0)).astype(np.float32)
    eng.write(0, x0, r0)
    if degree_cache:   # one vertex in it: the pushes go chunk by chunk as launches of their own
        v = int(np.nonzero((deg > 0) & (deg < 9) & ~asked[chunk])[0][0])
        ids, off, bits = np.array([v], np.int32), np.array([0, deg[v]], np.uint64), np.zeros((n + 31) // 32, np.uint32)
        bits[v >> 5] = 1 << (v & 31)
        K.call("excent_engine_hot_setup", eng.h, 1, ids.ctypes.data_as(K.i32p), off.ctypes.data_as(K.u64p),
               bits.ctypes.data_as(K.u32p))
    cnt, _, _ = eng.snapshot(use_hot=degree_cache)
    assert np.array_equal(cnt[0::2] > 0, asked)
    eng.push_cached(asked.astype(np.uint8), cnt)
    eng.sync()
    x, r = eng.read(0), eng.read(0, residual=True)
    rest = ~asked[chunk]
    assert not x[rest].any()
    assert r[hubs[rest[hubs]]].min() > EPS   # (something did reach them)
    # what was taken is delivered: sum r + (1 - 0.85) sum x (vertices without entries keep all they take)
    lost = np.where(deg == 0, 1.0, 0.15)
    assert abs(r.astype(np.float64).sum() + (lost * x).sum() - r0.astype(np.float64).sum()) <= 1e-5 * r0.sum()
    eng.close()


def test_slots_and_one_launch_pushes_do_not_run_side_by_side():
    """Gathered lists in the slots and cached pushes in one launch, in turn and without a wait of
    the host between them: nothing of a residual is lost. What is taken is delivered, so sum r +
    (1 - 0.85) sum x stays as it was (a vertex without entries keeps all that it takes)."""
    n = 70001
    idx, adj = edged_graph(n, 12, symmetric=True)
    deg = np.diff(idx.astype(np.int64))
    for cap, sweep in ((len(adj), False), (len(adj) // 5, True), (len(adj) // 5, False)):
        eng = engine(n, idx, adj, "pr", cap)
        eng.set_chunk_sweep(sweep)
        eng.set_sweep_demand(0.0)
        k = int(np.diff(np.append(eng.chunk_v0, n)).max())   # (a gather is of one chunk's size at most)
        K.call("excent_engine_slots_create", eng.h, len(adj), k, 0)
        for s in (0, 1):
            ed, vi, of = C.POINTER(C.c_int32)(), C.POINTER(C.c_int32)(), C.POINTER(C.c_uint64)()
            K.call("excent_engine_slot_buffers", eng.h, s, C.byref(ed), C.byref(vi), C.byref(of))
            np.ctypeslib.as_array(ed, shape=(len(adj),))[:] = adj
            np.ctypeslib.as_array(vi, shape=(k,))[:] = np.arange(k)
            np.ctypeslib.as_array(of, shape=(k + 1,))[:] = idx[:k + 1]
        eng.init()
        cnt, _, _ = eng.snapshot()
        mode = np.ones(eng.nc, dtype=np.uint8)
        before = float(np.float32(1) - np.float32(0.85)) * n
        for turn in range(12):
            s = turn % 2
            K.call("excent_engine_slot_wait", eng.h, s)
            K.call("excent_engine_push_gather", eng.h, s, k, int(idx[k]))
            eng.push_cached(mode, cnt)
        eng.sync()
        x, r = eng.read(0).astype(np.float64), eng.read(0, residual=True).astype(np.float64)
        now = r.sum() + (np.where(deg == 0, 1.0, 0.15) * x).sum()
        assert abs(now - before) <= 1e-5 * before, (cap, sweep, now / before)
        eng.close()


@pytest.mark.parametrize("measure,scale,ef", [("pr", 21, 17), ("pr", 22, 2), ("all", 20, 8)])
def test_unswept_solves_of_large_graphs_ask_the_host_nothing(measure, scale, ef):
    """Where the passes of a solve are launches of their own they still run in one submission, and a
    pass limit ends them all: no high-degree list is pushed past it, and nothing is lost (what is taken
    is delivered: sum r + (1 - 0.85) sum x of PageRank stays as it was)."""
    from torch.profiler import ProfilerActivity, profile
    g = X.DeviceGraph(scale, ef, 5)
    di, da, _ = g.device_ptrs()
    idx = np.empty(g.n + 1, dtype=np.uint64)
    adj = np.empty(g.m, dtype=np.int32)
    g.download(idx, adj)
    deg = np.diff(idx.astype(np.int64))
    assert (deg > 256).any()
    meas = X.measures(measure, eps_pr=0.01, eps_katz=0.01, eps_ev=0.01, alpha=1e-4, lam=1e3)
    eng = X.Engine(g.n, g.m, meas, *X.plan_chunks(idx, g.m))
    eng.upload_device(di, da)
    eng.solve(max_passes=1)
    with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA], acc_events=True) as prof:
        st = eng.solve(max_passes=40)
    waits = sum(ev.name == "cudaStreamSynchronize" for ev in prof.events())
    assert st.passes > 10 and waits <= 2, (st.passes, waits)
    for passes in (1, 2, 5, 100000):
        st, log = (eng.solve(max_passes=passes), eng.stats(with_log=True)[1])
        assert st.passes == passes or passes == 100000
        assert sum(int(p.pushed) for p in log) == st.pushed
        res = [eng.read(i, residual=True) for i in range(meas.nm)]
        pending = np.any([np.abs(r) > np.float32(0.01) for r in res], axis=0)
        assert np.array_equal(np.sort(eng.chunk_list(0)), np.nonzero(pending)[0])
        total = res[0].astype(np.float64).sum() + (np.where(deg == 0, 1.0, 0.15) * eng.read(0)).sum()
        assert abs(total - 0.15 * g.n) <= 1e-5 * 0.15 * g.n
    eng.close()
    g.close()
