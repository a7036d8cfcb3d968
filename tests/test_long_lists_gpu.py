"""Lists at the edges of the kernels' split into segments: rows of exactly the
segment thresholds and one either side, beside empty and short ones."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a GPU", allow_module_level=True)

import excent_b200 as X  # noqa: E402

DEGREES = (255, 256, 257, 511, 512, 513, 767, 1024, 1025, 2047, 2049)


def edged_graph(n, seed, symmetric=False):
    """CSR whose rows 5, 10, 15, ... have the degrees above, the others 0 to 6."""
    rng = np.random.default_rng(seed)
    deg = rng.integers(0, 7, n)
    at = np.arange(1, len(DEGREES) + 1) * 5
    deg[at] = DEGREES
    src = np.repeat(np.arange(n), deg)
    dst = np.concatenate([np.sort(rng.choice(n, k, replace=False)) for k in deg])
    if symmetric:
        keys = np.unique(np.concatenate([src * n + dst, dst * n + src]))
        keys = keys[keys // n != keys % n]
        src, dst = keys // n, keys % n
    idx = np.zeros(n + 1, dtype=np.uint64)
    np.cumsum(np.bincount(src, minlength=n), out=idx[1:])
    return idx, dst.astype(np.int32)


@pytest.mark.parametrize("kind,s", [("pr", 0.85), ("katz", 0.6)])
@pytest.mark.parametrize("n", [2500, 70001])
def test_weighted_solve_and_gradient_with_long_rows(n, kind, s):
    from excent_b200.autograd import WeightedGraph
    idx, adj = edged_graph(n, n)
    rng = np.random.default_rng(1)
    w = rng.uniform(0.5, 1.5, len(adj)).astype(np.float32)
    dev = torch.device("cuda")
    G = WeightedGraph(n, torch.from_numpy(idx.view(np.int64)).to(dev), torch.from_numpy(adj).to(dev),
                      torch.from_numpy(w).to(dev))
    eps = 1e-7
    x, passes, pushed = G.forward(kind, s, None, eps)
    assert passes > 0 and pushed > 0
    wn = O.row_normalise(idx, w)
    c0 = 1 - s if kind == "pr" else 1.0
    x_ref = O.weighted_forward(idx, adj, wn, c0, s, np.ones(n))
    # a residual of at most eps per vertex leaves an L1 error of n eps / (1 - s); FP32 sums of up to 2049 terms
    assert np.abs(x.cpu().numpy() - x_ref).sum() <= n * eps / (1 - s) + 1e-5 * np.abs(x_ref).sum()
    c = np.zeros(n)
    c[rng.choice(n, 100, replace=False)] = 1
    lam_ref = O.weighted_adjoint(idx, adj, wn, s, c)
    gw_ref = O.weighted_grad(idx, adj, w, wn, s, x_ref, lam_ref)
    gt, gw = G.vjp(torch.from_numpy(c.astype(np.float32)).to(dev), eps)
    assert np.linalg.norm(gt.cpu().numpy() - c0 * lam_ref) <= 1e-4 * np.linalg.norm(c0 * lam_ref)
    assert np.linalg.norm(gw.cpu().numpy() - gw_ref) <= 1e-3 * np.linalg.norm(gw_ref)
    G.close()
