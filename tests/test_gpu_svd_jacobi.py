"""The one-sided Jacobi SVD of the hierarchical reduction at the edges of its lane groups (16 lanes per
column pair, 2, 4, 8 or 11 elements each) and of its shared-memory layouts (V beside B up to l = 120)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("l", [1, 2, 15, 16, 17, 31, 32, 33, 64, 65, 96, 119, 120, 121, 128, 129, 160])
def test_hierarchical_reduction_sizes(lib, oracle, l):
    rng = np.random.default_rng(l)
    N, m = 3, 2 * l + 30
    base = np.linalg.qr(rng.standard_normal((m, l)))[0]
    qs = np.concatenate([np.linalg.qr(base + 0.3 * rng.standard_normal((m, l)) / np.sqrt(m))[0] for _ in range(N)], 1)
    ref = oracle.integrate_hierarchical_reduction(qs.copy(), l, N)[0]
    qt, y = np.zeros((m, l)), qs.copy()
    lib.integrate("d", "HR", lib.create_param(m, m, l, 0, N), y, N * l, qt, l, retc=0)
    assert lib.last_error()[0] == 0
    tol = 64 * l * 2.0 ** -53  # two levels of products and factors of l x l and m x l matrices of norm 1
    assert np.abs(qt.T @ qt - np.eye(l)).max() <= tol
    assert np.abs(qt @ qt.T - ref @ ref.T).max() <= tol
