"""The hierarchical reduction's SVD started from the eigenvectors of B'B: graded and scaled spectra, and
inputs whose B'B does not settle or does not exist (rank-deficient, zero, equal bases)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


def _reduce(lib, q1, q2):
    m, l = q1.shape
    y, qt = np.concatenate([q1, q2], 1), np.zeros((m, l))
    lib.integrate("d", "HR", lib.create_param(m, m, l, 0, 2), y, 2 * l, qt, l, retc=0)
    assert lib.last_error()[0] == 0
    return qt


@pytest.mark.parametrize("scale", [1.0, 2.0 ** -100, 2.0 ** 100])
@pytest.mark.parametrize("l", [31, 32, 33, 48, 64, 100, 128, 129])
def test_graded_spectra(lib, oracle, l, scale):
    rng = np.random.default_rng(l)
    m = 2 * l + 10
    q1, w, t = (np.linalg.qr(rng.standard_normal((k, l)))[0] for k in (m, l, l))
    q2 = scale * ((q1 @ w) * np.logspace(0, -6, l)) @ t.T
    qt = _reduce(lib, q1, q2)
    ref = oracle.integrate_hierarchical_reduction(np.concatenate([q1, q2], 1), l, 2)[0]
    # the projector's error: rounding of B relative to its norm over the smallest gap of the vectors that
    # Q1 and Q2 share is absorbed by W and T together; l products of norm max(1, scale) each
    nrm = np.linalg.norm(ref, 2)
    assert np.abs(qt @ qt.T - ref @ ref.T).max() <= 64 * l * U * nrm ** 2


@pytest.mark.parametrize("l", [32, 48, 128])
def test_degenerate(lib, l):
    rng = np.random.default_rng(l)
    m = 2 * l + 10
    q = np.linalg.qr(rng.standard_normal((m, 2 * l)))[0]
    q1, q2 = q[:, :l], q[:, l:]
    tol = 64 * l * U
    qt = _reduce(lib, q1, q1)  # all singular values 1
    assert np.abs(qt @ qt.T - q1 @ q1.T).max() <= tol
    h = l // 2
    mixed = np.concatenate([q1[:, :h], q2[:, h:]], 1)  # half of them 1, half 0
    qt = _reduce(lib, q1, mixed)
    assert np.abs(qt[:, :h] @ qt[:, :h].T - q1[:, :h] @ q1[:, :h].T).max() <= tol
    assert np.isfinite(_reduce(lib, q1, np.zeros_like(q1))).all()
