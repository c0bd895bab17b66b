"""Batches with matrices whose sketch and Qs'Qs are large enough for tensor-core products of their own beside
small ones: the results of the single solves, repeatably, with the same iteration counts."""
import numpy as np
import pytest

from test_gpu_batched import run_batch, single

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("x", ["s", "d"])
def test_large_and_small_in_one_batch(lib, oracle, x):
    dt = torch.float32 if x == "s" else torch.float64
    N, mats = 8, []
    g = torch.Generator(device="cuda").manual_seed(3)
    for m, n, k in ((700, 300, 8), (9000, 2001, 32), (1500, 400, 16), (6501, 1500, 64), (300, 200, 4)):
        r = 2 * k
        u, v = (torch.linalg.qr(torch.randn(q, r, device="cuda", generator=g, dtype=torch.float64))[0] for q in (m, n))
        w = torch.logspace(0, -2, r, device="cuda", dtype=torch.float64)
        a = (u * w) @ v.T + 1e-5 * torch.randn(m, n, device="cuda", generator=g, dtype=torch.float64)
        mats.append(dict(m=m, n=n, k=k, p=k // 2, a=a.to(dt).contiguous()))
    seeds = [11 + i for i in range(len(mats))]
    first, again = run_batch(lib, x, mats, N, seeds, solves=2)
    tol_s, tol_a = (1e-5, 1e-3) if x == "s" else (1e-10, 1e-8)  # as for small matrices
    for i, d in enumerate(mats):
        s, u, v, it = single(lib, x, d, N, seeds[i])
        k = d["k"]
        assert abs(first[3][i] - it) <= (1 if x == "s" else 0)
        assert np.abs(first[0][i] - s).max() <= tol_s * s.max()
        assert oracle.column_angles(first[1][i][:, :k].astype(np.float64), u[:, :k].astype(np.float64)).max() < tol_a
        assert oracle.column_angles(first[2][i][:, :k].astype(np.float64), v[:, :k].astype(np.float64)).max() < tol_a
        for p in range(4):
            assert np.array_equal(first[p][i], again[p][i])
