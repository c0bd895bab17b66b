"""The one-sided Jacobi SVD with NaN or infinities in its matrix (hierarchical reduction, tall-skinny
postprocessing): an error status or non-finite results, and the library works on afterwards."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _bases(m, l, N, dt):
    rng = np.random.default_rng(l)
    return np.concatenate([np.linalg.qr(rng.standard_normal((m, l)))[0] for _ in range(N)], 1).astype(dt)


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("x", ["s", "d"])
@pytest.mark.parametrize("l", [5, 48, 100, 130])
def test_hierarchical_reduction(lib, l, x, bad):
    m, N = 600, 4
    good = _bases(m, l, N, np.float32 if x == "s" else np.float64)
    prm = lib.create_param(m, m, l, 0, N)
    for entry in ([(3, 1)], [(i, l + 2) for i in range(m)]):  # one entry, a whole column
        qs = good.copy()
        for e in entry:
            qs[e] = bad
        qt = np.zeros((m, l), good.dtype)
        lib.integrate(x, "HR", prm, qs, N * l, qt, l)
        assert lib.last_error()[0] != 0 or not np.isfinite(qt).all()
        lib.clear_error()
    qs, qt = good.copy(), np.zeros((m, l), good.dtype)
    lib.integrate(x, "HR", prm, qs, N * l, qt, l)
    assert lib.last_error()[0] == 0
    assert np.abs(qt.T.astype(float) @ qt - np.eye(l)).max() <= 100 * np.finfo(good.dtype).eps


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("x", ["s", "d"])
@pytest.mark.parametrize("l", [8, 64, 140])
def test_tall_skinny_postprocessing(lib, l, x, bad):
    m, n = 500, 400
    q = _bases(m, l, 1, np.float32 if x == "s" else np.float64)
    a = np.random.default_rng(1).standard_normal((m, n)).astype(q.dtype)
    a[10, 20] = bad
    s, u, v = np.zeros(l, q.dtype), np.zeros((m, l), q.dtype), np.zeros((n, l), q.dtype)
    lib.postprocess(x, "TS", lib.create_param(m, n, l, 0, 1), a, n, q, l, s, u, l, v, l)
    assert lib.last_error()[0] != 0 or not all(np.isfinite(t).all() for t in (s, u, v))
    lib.clear_error()
