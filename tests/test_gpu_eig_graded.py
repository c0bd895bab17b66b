"""Graded matrices in the l x l eigensolver: the singular values of a postprocessing whose Z'Z is D H D keep their
accuracy relative to themselves, not to the largest."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _one_sided(z):
    """Singular values of z (rows) by one-sided Jacobi on the rows, to a few u each (Demmel & Veselic)."""
    z = z.copy()
    l = len(z)
    for _ in range(30):
        big = 0.0
        for i in range(l - 1):
            for j in range(i + 1, l):
                a, b, g = z[i] @ z[i], z[j] @ z[j], z[i] @ z[j]
                big = max(big, abs(g) / np.sqrt(a * b))
                if abs(g) > 1e-16 * np.sqrt(a * b):
                    t = (b - a) / (2 * g)
                    t = np.copysign(1.0, t) / (abs(t) + np.hypot(1.0, t))
                    c = 1.0 / np.sqrt(1.0 + t * t)
                    z[i], z[j] = c * (z[i] - t * z[j]), c * (t * z[i] + z[j])
        if big < 1e-15:
            break
    return np.sort(np.linalg.norm(z, axis=1))[::-1]


@pytest.mark.parametrize("order", [b"R", b"C"])
@pytest.mark.parametrize("lo", [1.0, 0.3, 1e-2, 1e-3, 1e-4, 1e-5, 1e-6])
@pytest.mark.parametrize("l", [5, 32, 48, 100])
def test_gramian_postprocessing(lib, l, lo, order):
    m, n = 150, 400
    rng = np.random.default_rng(l)
    a = rng.standard_normal((m, n))
    a[:l] *= rng.permutation(np.geomspace(1.0, lo, l))[:, None]
    q = np.eye(m, l)  # Z' = Qbar' A: the graded rows of A
    s, u, v = np.zeros(l), np.zeros((m, l)), np.zeros((n, l))
    lib.postprocess("d", "GR", lib.create_param(m, n, l, 0, 1), a if order == b"R" else np.ascontiguousarray(a.T),
                    n if order == b"R" else m, q, l, s, u, l, v, l, ordera=order)
    assert lib.last_error()[0] == 0
    ref = _one_sided(a[:l])
    # H = D^-1 W D^-1 has unit diagonal up to sqrt(2 / n) and condition (1 + sqrt(l / n))^2 / (1 - sqrt(l / n))^2 <= 9;
    # its entries round by sqrt(n) u, Jacobi by l u, both times the condition, halved by the root
    assert np.abs(s / ref - 1.0).max() <= 9 * (n ** 0.5 + l) * 2.0 ** -53
    assert np.abs(u.T @ u - np.eye(l)).max() <= 1e-13
