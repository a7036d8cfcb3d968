"""The kernels of a device solve that a rule on sizes picks, each at a size that picks it: two
vertices a thread, waves smaller than a pass, chunks of several phases; and the split lists with
self-loops, repeated entries and pushes by the host."""
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

R0 = float(np.float32(1) - np.float32(0.85))


def launches(eng, **kw):
    before = eng.launches()
    eng.solve(**kw)
    return eng.launches() - before


# vertices and slots at which 148 SMs take: two vertices a thread; a wave of one block of 256 threads to an
# SM, smaller than the items of a pass
@pytest.mark.parametrize("measure", ["pr", "all"])
@pytest.mark.parametrize("n,slots", [(150001, 300), (70001, "all")])
def test_one_launch_variants(n, slots, measure):
    idx, adj = edged_graph(n, 21, symmetric=True)
    lam = float(O.params(n, idx, adj)["_lambda"])
    eng = engine(n, idx, adj, measure, len(adj), alpha=0.5 / lam, lam=lam, ev_init_fp64=True)
    assert eng.nc == 1
    eng.set_hub_targets(slots if slots != "all" else 32768 if measure == "pr" else 8192)
    for use_graph in (True, False):
        st = eng.solve(max_passes=400, use_graph=use_graph)
        s2, log = eng.stats(with_log=True)
        assert sum(int(p.pushed) for p in log) == st.pushed and len(log) == st.passes
        for i, k in enumerate(("pr", "katz")[:eng.meas.nm]):
            assert np.all(np.abs(eng.read(i, residual=True)) <= np.float32(EPS))
            assert close_enough(k, n, eng.read(i), O.reference_solution(n, idx, adj, k, alpha=0.5 / lam)), (k, use_graph)
    eng.close()


def swept_pass(idx, adj, chunk, v0, per_phase, r, x, list_frac=0.5):
    """One pass chunk by chunk in FP64: the lists longer than 256 entries, then the others phase by phase."""
    n, nc = len(r), len(v0)
    deg = np.diff(idx.astype(np.int64))
    src = np.repeat(np.arange(n), deg)
    phase = (np.arange(n) - v0[chunk]) // per_phase
    first = np.abs(r) > EPS
    few = np.bincount(chunk, first, nc) < list_frac * np.bincount(chunk, minlength=nc)
    for c in range(nc):
        steps = [deg > 256] + [(deg <= 256) & (phase == q) for q in range(int(phase[chunk == c].max()) + 1)]
        for now in steps:
            d = np.where((chunk == c) & now & (np.abs(r) > EPS) & (first | ~few[chunk]), r, 0.0)
            x += d
            r -= d
            r += np.bincount(adj, (0.85 * d / np.maximum(deg, 1))[src], n)


@pytest.mark.parametrize("symmetric", [True, False])
def test_chunk_of_several_phases(symmetric):
    """With all slots a wave is 256 items to an SM and a phase six waves. On a symmetric graph the
    pass gathers along split lists, made once by the first solve (four kernels more than the check
    that a directed graph fails)."""
    n = 300007
    idx, adj = edged_graph(n, 22, symmetric=symmetric)
    per_phase = 6 * 256 * torch.cuda.get_device_properties(0).multi_processor_count
    v0 = np.array([0, per_phase + 5000, per_phase + 40000], dtype=np.int32)
    chunk = np.searchsorted(v0, np.arange(n), side="right") - 1
    eng = X.Engine(n, len(adj), X.measures("pr", eps_pr=EPS), v0, idx[np.append(v0, n)])
    eng.upload_graph(idx, adj)
    eng.set_hub_targets(32768)
    eng.set_sweep_demand(0.01)
    first, again = launches(eng, max_passes=1), launches(eng, max_passes=1)
    assert first - again == 3 + (6 if symmetric else 2)   # (three list the long lists)
    if symmetric:
        r, x = np.full(n, R0), np.zeros(n)
        swept_pass(idx, adj, chunk, v0, per_phase, r, x)
        # FP32 sums of up to 2049 terms
        assert np.allclose(eng.read(0), x, rtol=1e-5, atol=1e-6)
        assert np.allclose(eng.read(0, residual=True), r, rtol=1e-5, atol=1e-6)
    eng.solve()
    assert np.all(np.abs(eng.read(0, residual=True)) <= np.float32(EPS))
    if symmetric:
        assert close_enough("pr", n, eng.read(0), O.reference_solution(n, idx, adj, "pr"))
    eng.close()


@pytest.mark.parametrize("by", ["solve", "push_cached"])
@pytest.mark.parametrize("passes", [1, 4])
def test_split_lists_with_self_loops_and_repeats(by, passes):
    """Step by step in FP64. Sums of up to some 600 terms in each pass, and a residual within their
    rounding of eps may be taken in one and not in the other."""
    n = 4000
    rng = np.random.default_rng(23)
    src = np.concatenate([np.full(k, v) for v, k in ((7, 600), (3900, 500), (2000, 300))] + [rng.integers(0, n, 9000)])
    dst = rng.integers(0, n, len(src))
    keys = np.unique(np.concatenate([src * n + dst, dst * n + src]))
    twice = keys[rng.choice(len(keys), 300, replace=False)]
    loops = np.concatenate([[7, 3900], rng.choice(n, 60, replace=False)])
    keys = np.sort(np.concatenate([keys, twice, (twice % n) * n + twice // n, loops * n + loops]))
    src, adj = keys // n, (keys % n).astype(np.int32)
    idx = np.zeros(n + 1, dtype=np.uint64)
    np.cumsum(np.bincount(src, minlength=n), out=idx[1:])
    eng = engine(n, idx, adj, "pr", len(adj) // 8 + 1)
    assert eng.nc > 4
    eng.set_sweep_demand(0.01)
    if by == "solve":
        first, again = launches(eng, max_passes=1), launches(eng, max_passes=1)
        assert first - again == 9   # (the lists are split)
        eng.solve(max_passes=passes)
    else:
        eng.init()
        for _ in range(passes):
            cnt, _, _ = eng.snapshot()
            eng.push_cached((cnt[0::2] > 0).astype(np.uint8), cnt, 0.5)
            eng.sync()
    chunk = np.searchsorted(eng.chunk_v0, np.arange(n), side="right") - 1
    r, x = np.full(n, R0), np.zeros(n)
    for _ in range(passes):
        swept_pass(idx, adj, chunk, eng.chunk_v0, n, r, x)
    assert np.allclose(eng.read(0), x, rtol=1e-5, atol=2e-6)
    assert np.allclose(eng.read(0, residual=True), r, rtol=1e-5, atol=2e-6)
    eng.close()
