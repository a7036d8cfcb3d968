"""Batched solves whose rows of short lists scatter over their groups (words of 32 vertices for half of
the GPU's warps, an eighth with 256 lanes) and over their entries, with lists at the edges of the 128
entries and of the 512 that go at once."""
import numpy as np
import pytest

import oracle as O
from test_batched_gpu import queries

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a GPU", allow_module_level=True)

import excent_b200 as X  # noqa: E402


def graph(n):
    rng = np.random.default_rng(n)
    src = [rng.integers(0, n, 3 * n)]
    dst = [rng.integers(0, n, 3 * n)]
    for i, k in enumerate((31, 33, 96, 127, 128, 129, 160, 255, 257, 511, 512, 513, 700)):
        src.append(np.full(k, 40 * i + 3))
        dst.append(n // 2 + rng.choice(n // 2, k, replace=False))
    src, dst = np.concatenate(src), np.concatenate(dst)
    keys = np.unique(np.concatenate([src * n + dst, dst * n + src]))
    idx = np.zeros(n + 1, dtype=np.uint64)
    np.cumsum(np.bincount(keys // n, minlength=n), out=idx[1:])
    return idx, (keys % n).astype(np.int32)


@pytest.mark.parametrize("greedy", [True, False])
@pytest.mark.parametrize("n,B", [(9000, 32), (80001, 32), (80001, 64), (80001, 128), (9000, 256), (20003, 256)])
def test_rows_over_groups_and_over_entries(n, B, greedy):
    idx, adj = graph(n)
    di, da = torch.from_numpy(idx.view(np.int64)).cuda(), torch.from_numpy(adj).cuda()
    d, nq = 0.85, B - 1
    qs = queries(n, nq, B)
    eps = 1e-6 * (1 - d)
    b = X.Batch(n, len(adj), di, da, B, "ppr", d)
    b.set_greedy(greedy)
    b.seed(qs, [(1 - d) / len(s) for s in qs], eps)
    b.solve()
    for q in (0, nq // 2, nq - 1):
        r, x = b.read(q, residual=True), b.read(q)
        assert np.all(np.abs(r) <= np.float32(eps))
        t = np.zeros(n)
        t[qs[q]] = 1.0 / len(qs[q])
        # the push conserves mass, so the L1 error is at most |r|_1 / (1 - d); 10 % and 1e-5 for FP32
        err = np.abs(x - O.ppr(n, idx, adj, t, kind=0, d=d)).sum()
        assert err <= 1.1 * np.abs(r.astype(np.float64)).sum() / (1 - d) + 1e-5, (q, err)
    assert not b.read(nq).any()
    b.close()
