"""The l x l symmetric eigensolver (FP32 one-sided Jacobi, FP64 refinement, two-sided Jacobi for what
does not settle) at the edges of its column blocks and clusters, through the two postprocessing stages
that call it: symmetric (indefinite, ascending) and Gramian (positive semidefinite, descending)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SPECTRA = {
    "spread": lambda l, rng: np.linspace(1.0, 0.1, l),
    "graded": lambda l, rng: np.geomspace(1.0, 1e-6, l),
    "multiple": lambda l, rng: np.concatenate([np.ones(l // 2), np.zeros(l - l // 2)]),
    "cluster": lambda l, rng: 1.0 + 1e-9 * rng.standard_normal(l),
    "pairs": lambda l, rng: np.concatenate([np.linspace(1, 2, l // 2), np.linspace(1, 2, l - l // 2) * (1 + 1e-11)]),
    "signs": lambda l, rng: rng.standard_normal(l) * 1e80,
}


@pytest.mark.parametrize("kind", list(SPECTRA))
@pytest.mark.parametrize("l", [1, 2, 3, 4, 5, 8, 9, 31, 32, 33, 47, 64, 65, 72, 96, 97, 127, 128, 129])
def test_symmetric_eigensolver(lib, l, kind):
    rng = np.random.default_rng(1000 + l)
    lam = SPECTRA[kind](l, rng)
    big = np.abs(lam).max()
    m = l + 40
    q = np.linalg.qr(rng.standard_normal((m, l)))[0]
    o = np.linalg.qr(rng.standard_normal((l, l)))[0]
    w = (o * lam) @ o.T
    # Backward stable solvers leave a small multiple of l u ||W|| (l u <= 1.5e-14); 64 l u bounds the
    # constants of A's formation, the products on both sides and the solver's thresholds together
    tol = 64 * l * 2.0 ** -53
    a = q @ (0.5 * (w + w.T)) @ q.T
    a = 0.5 * (a + a.T)
    s, u = np.zeros(l), np.zeros((m, l))
    lib.postprocess("d", "SY", lib.create_param(m, m, l, 0, 1), a, m, np.ascontiguousarray(q), l, s, u, l, None, l,
                    vt_root=-2)
    assert lib.last_error()[0] == 0
    assert np.abs(s - np.sort(lam)).max() <= tol * big
    assert np.abs(a @ u - u * s).max() <= tol * big
    # orthogonality of the eigenvectors, and of q
    assert np.abs(u.T @ u - np.eye(l)).max() <= 2 * tol
    if kind == "signs":
        return
    n = l + 9
    v = np.linalg.qr(rng.standard_normal((n, l)))[0]
    a = np.ascontiguousarray((q @ o * np.abs(lam)) @ v.T)
    s, u, vt = np.zeros(l), np.zeros((m, l)), np.zeros((n, l))
    lib.postprocess("d", "GR", lib.create_param(m, n, l, 0, 1), a, n, np.ascontiguousarray(q), l, s, u, l, vt, l)
    assert lib.last_error()[0] == 0
    # the squares are exact to tol: singular values to sqrt(tol) where they are small
    assert np.abs(s ** 2 - np.sort(np.abs(lam))[::-1] ** 2).max() <= tol * big ** 2
    assert np.abs(u.T @ u - np.eye(l)).max() <= 2 * tol
    if kind != "multiple":  # V = Z W / sigma of a zero sigma is undefined
        assert np.abs((u * s) @ vt.T - a).max() <= tol * big
