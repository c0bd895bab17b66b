"""FP64 products of few output tiles, by clusters that split K: the coefficient products of the
Kolmogorov-Nagumo loop at widths around the tiles' edges, and short and ragged K, through the stages."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

U = 2.0 ** -53


@pytest.mark.parametrize("order", [b"R", b"C"])
@pytest.mark.parametrize("shape", [(1, 1, 1), (33, 17, 5), (64, 15, 64), (65, 16, 65), (31, 129, 97), (500, 127, 33),
                                   (1000, 600, 40), (97, 1333, 63), (2000, 255, 128), (300, 4097, 30)])
def test_integers_are_exact(lib, shape, order):
    """A Omega with 19-bit integers: every partial sum is below 2^53, in any order."""
    m, n, nl = shape
    g = torch.Generator(device="cuda").manual_seed(n)
    a = torch.randint(-2 ** 18, 2 ** 18 + 1, (m, n), device="cuda", generator=g).double()
    om = torch.randint(-2 ** 18, 2 ** 18 + 1, (n, nl), device="cuda", generator=g).double()
    y = torch.full((m, nl + 3), 7.0, device="cuda", dtype=torch.float64)
    src = a if order == b"R" else a.t().contiguous()
    lib.sketch_omega("d", lib.create_param(m, n, 1, 0, nl), src, n if order == b"R" else m, om, nl, y, nl + 3, ordera=order)
    assert lib.last_error()[0] == 0
    assert torch.equal(y[:, :nl], a @ om)
    assert bool((y[:, nl:] == 7.0).all())


@pytest.mark.parametrize("l,N", [(1, 2), (3, 5), (8, 4), (31, 3), (32, 8), (33, 7), (63, 16), (64, 16), (65, 16), (96, 16), (127, 9), (128, 16)])
def test_kn_coefficient_products(lib, oracle, l, N):
    m = 2500
    rng = np.random.default_rng(l)
    base = np.linalg.qr(rng.standard_normal((m, l)))[0]
    qs = np.concatenate([np.linalg.qr(base + 0.2 * rng.standard_normal((m, l)) / np.sqrt(m))[0] for _ in range(N)], 1)
    qt = np.zeros((m, l))
    r = lib.integrate("d", "KN", lib.create_param(m, m, l, 0, N), qs, N * l, qt, l, argv=[4, 1e-12])
    assert lib.last_error()[0] == 0
    ref, it, _ = oracle.integrate_kolmogorov_nagumo(qs, l, N, maxit=4, tol=1e-12)
    assert int(r[0]) == it
    # orthonormal columns; a few tens of u for G and each of the products of up to four iterations
    assert np.linalg.norm(qt - ref) / np.linalg.norm(ref) <= 1000 * U
