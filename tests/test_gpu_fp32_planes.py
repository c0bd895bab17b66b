"""NATIVE FP32 products on the bf16 tensor cores (three planes per operand): accuracy against FP64 at
tile edges, odd block widths and both storage orders, infinities and NaN, and the products that the
planes leave to the CUDA cores."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

U = 2.0 ** -24


def _lib_sketch(lib, a, m, n, nl, order, seed=3):
    y = torch.zeros(m, nl, device="cuda")
    src = a if order == b"R" else a.t().contiguous()
    lib.sketch("s", lib.create_param(m, n, nl, 0, 1), src, n if order == b"R" else m, y, nl, seed, ordera=order)
    assert lib.last_error()[0] == 0
    return y


def _omega(lib, n, nl, seed=3):
    """Omega of a seed, through the FP64 sketch of the identity (exact)."""
    y = torch.zeros(n, nl, device="cuda", dtype=torch.float64)
    eye = torch.eye(n, device="cuda", dtype=torch.float64)
    lib.sketch("d", lib.create_param(n, n, nl, 0, 1), eye, n, y, nl, seed)
    return y


@pytest.mark.parametrize("order", [b"R", b"C"])
@pytest.mark.parametrize("shape", [(1025, 1999, 1040), (4097, 801, 770), (3001, 1500, 255), (20011, 257, 512), (129, 9000, 1024)])
def test_sketch_accuracy(lib, shape, order):
    """Per output, chunks of 32 or 64 terms: at most 3 x 4 truncations at 2^-23 of a chunk's partial sum
    (their mean half of that: under 6 x 2 u), then n / 64 roundings of the running sum that add up
    like a random walk, u sqrt(n / 64) / 2: relative to the norm, under 12 u + u sqrt(n / 64)."""
    m, n, nl = shape
    g = torch.Generator(device="cuda").manual_seed(m)
    a = torch.randn(m, n, device="cuda", generator=g) * torch.exp(2 * torch.randn(m, n, device="cuda", generator=g))
    y = _lib_sketch(lib, a, m, n, nl, order)
    ref = a.double() @ _omega(lib, n, nl)
    err = float((y.double() - ref).norm() / ref.norm())
    assert err <= (12 + (n / 64) ** 0.5) * U


def test_sketch_non_finite_and_largest_values(lib):
    m, n, nl = 2000, 1500, 512
    g = torch.Generator(device="cuda").manual_seed(1)
    a = torch.randn(m, n, device="cuda", generator=g)
    a[3, 7], a[5, 1499], a[700, 0] = float("inf"), float("-inf"), float("nan")
    a[11, :] = 0.0
    a[11, 40] = torch.finfo(torch.float32).max  # rounds to infinity as bf16
    om = _omega(lib, n, nl)
    y = _lib_sketch(lib, a, m, n, nl, b"R")
    assert bool((y[3] == torch.sign(om[7]).float() * float("inf")).all())
    assert bool((y[5] == -torch.sign(om[1499]).float() * float("inf")).all())
    assert bool(torch.isnan(y[700]).all())
    keep = om[40].abs() < 0.99
    ref = 3.4028234663852886e38 * om[40]
    assert float(((y[11].double() - ref).abs() / ref.abs())[keep].max()) <= 4 * U
    rest = torch.ones(m, dtype=torch.bool, device="cuda")
    rest[[3, 5, 11, 700]] = False
    assert bool(torch.isfinite(y[rest]).all())


@pytest.mark.parametrize("l", [31, 48, 63, 64, 65, 96, 100, 128, 129])
def test_tall_skinny_qr_blocks(lib, l):
    """Block Grams and applies of padded blocks: orthonormal to FP32 and the span of Y's blocks."""
    m, N = 40000, 8
    g = torch.Generator(device="cuda").manual_seed(l)
    y = torch.randn(m, N * l, device="cuda", generator=g)
    q = y.clone()
    lib.orthogonalize("s", "TS", lib.create_param(m, m, l, 0, N), q, N * l)
    assert lib.last_error()[0] == 0
    for i in (0, 1, N - 1):
        qi, yi = (t[:, i * l:(i + 1) * l].double() for t in (q, y))
        # W and R^-1 carry FP32 rounding of sums of m terms (chunks of 64, split sums in FP64), the
        # products l terms: a few tens of u in norm, with the margin of a factor four
        assert float((qi.t() @ qi - torch.eye(l, device="cuda")).abs().max()) <= 100 * U
        assert float((yi - qi @ (qi.t() @ yi)).norm() / yi.norm()) <= 100 * U


@pytest.mark.parametrize("l,N", [(33, 16), (64, 16), (65, 12), (128, 9)])
def test_kn_and_postprocess(lib, oracle, l, N):
    """G = Qs'Qs and Qbar = Qs M from one split, Z = A' Qbar and the outer products."""
    m, n = 12001, 2003
    rng = np.random.default_rng(l)
    base = np.linalg.qr(rng.standard_normal((m, l)))[0]
    qs = np.concatenate([np.linalg.qr(base + 0.2 * rng.standard_normal((m, l)) / np.sqrt(m))[0] for _ in range(N)], 1)
    qs = qs.astype(np.float32)
    prm = lib.create_param(m, n, l, 0, N)
    qt = np.zeros((m, l), np.float32)
    r = lib.integrate("s", "KN", prm, qs, N * l, qt, l, argv=[3, 1e-9])
    assert lib.last_error()[0] == 0
    ref, it, _ = oracle.integrate_kolmogorov_nagumo(qs.astype(np.float64), l, N, maxit=3, tol=1e-9)
    assert int(r[0]) == it
    # G to a few u and Qbar's own sums; columns of norm 1, so entries are far below the norm bound
    assert np.linalg.norm(qt - ref) / np.linalg.norm(ref) <= 32 * U
    a = (base * np.linspace(1, 0.5, l)) @ rng.standard_normal((l, n)) + 1e-3 * rng.standard_normal((m, n))
    a = a.astype(np.float32)
    for order, store in ((b"R", a), (b"C", np.ascontiguousarray(a.T))):
        s, u, v = np.zeros(l, np.float32), np.zeros((m, l), np.float32), np.zeros((n, l), np.float32)
        lib.postprocess("s", "GR", prm, store, n if order == b"R" else m, qt, l, s, u, l, v, l, ordera=order)
        assert lib.last_error()[0] == 0
        q64 = qt.astype(np.float64)
        z = a.astype(np.float64).T @ q64
        sv = np.linalg.svd(z, compute_uv=False)
        assert np.abs(s - sv).max() <= 32 * U * sv[0]
        assert np.linalg.norm((u.astype(np.float64) * s) @ v.T - q64 @ z.T) <= 64 * U * np.linalg.norm(z)
