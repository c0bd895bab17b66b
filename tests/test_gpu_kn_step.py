"""The l x l Kolmogorov-Nagumo step at the edges of its row-cut form (8-row tiles, l = 128 the largest)
and in each of its evaluations of C and C^-1: the chain of powers, Horner steps in Z^4 and Z^8, and
Newton-Schulz.  One iteration of the FP64 integration stage against the NumPy restatement."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _blocks(l, N, t, seed):
    """N blocks spanning nearly the same l-dimensional space U; the first is sqrt(1-t) U + sqrt(t) W
    with W orthogonal to U, which puts the eigenvalues of 4 Z near 3 t for small t (N = 8: 0.77 at
    t = 0.5, where ||Z^4||_F^(1/4) bounds it by more than 0.9 for l >= 8)."""
    rng = np.random.default_rng(seed)
    m = 3 * l + 40
    uw = np.linalg.qr(rng.standard_normal((m, 2 * l)))[0]
    u, w = uw[:, :l], uw[:, l:]
    qs = np.empty((m, N * l))
    for i in range(N):
        r = np.linalg.qr(rng.standard_normal((l, l)))[0]
        b = u @ r if i else np.sqrt(1 - t) * u + np.sqrt(t) * w
        qs[:, i * l:(i + 1) * l] = np.linalg.qr(b + 1e-4 * rng.standard_normal((m, l)) / np.sqrt(m))[0]
    return m, qs


@pytest.mark.parametrize("t", [1e-5, 0.02, 0.1, 0.5], ids=["chain", "z4", "z8", "newton"])
@pytest.mark.parametrize("l", [1, 2, 7, 8, 9, 31, 32, 33, 63, 65, 96, 97, 127, 128, 129])
def test_kn_step_matches_oracle(lib, oracle, l, t):
    N = 8
    m, qs = _blocks(l, N, t, seed=100 * l + int(1000 * t))
    prm = lib.create_param(m, m, l, 0, N)
    qt = np.zeros((m, l))
    r = lib.integrate("d", "KN", prm, qs, N * l, qt, l, argv=[1, 1e-30])
    assert lib.last_error()[0] == 0
    q_ref, it, err = oracle.integrate_kolmogorov_nagumo(qs, l, N, maxit=1, tol=1e-30)
    assert int(r[0]) == it == 2
    # each of the step's at most about forty dependent products leaves l u ~ 3e-14 of its norm (<= 2);
    # the square roots at lambda <= 0.24 amplify it by at most 1 / (2 sqrt(1/4 - lambda)) = 5
    assert np.abs(qt - q_ref).max() < 1e-11
    assert abs(r[1] - err) < 1e-11 * max(1.0, np.sqrt(l))
