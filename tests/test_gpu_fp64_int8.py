"""Large FP64 products on the int8 tensor cores: exact for integer operands in every layout and at ragged
sizes, FP64-accurate for random ones, and rows that do not split (outliers, infinities, NaN, zeros, extreme
exponents) computed as before."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

U = 2.0 ** -53


def _sketch(lib, a, om, order):
    m, n = a.shape
    nl = om.shape[1]
    y = torch.full((m, nl), 7.0, device="cuda", dtype=torch.float64)
    src = a if order == b"R" else a.t().contiguous()
    lib.sketch_omega("d", lib.create_param(m, n, nl, 0, 1), src, n if order == b"R" else m, om, nl, y, nl, ordera=order)
    assert lib.last_error()[0] == 0
    return y


# tile edges (128), digit-block edges (64) and chunk edges (16384) of the three sizes; few tiles (split K)
SHAPES = [(20011, 1501, 384), (20000, 1536, 1024), (12001, 1473, 1000), (4097, 2047, 1153), (2300, 16449, 1000), (640, 40001, 512)]


@pytest.mark.parametrize("order", [b"R", b"C"])
@pytest.mark.parametrize("shape", SHAPES)
def test_integers_are_exact(lib, shape, order):
    """19-bit integers: every partial sum is below 2^53, so any correct FP64 product is exact."""
    m, n, nl = shape
    g = torch.Generator(device="cuda").manual_seed(n)
    bits = 18  # products of 2^36, at most 2^16 of them
    a = torch.randint(-2 ** bits, 2 ** bits + 1, (m, n), device="cuda", generator=g).double()
    om = torch.randint(-2 ** bits, 2 ** bits + 1, (n, nl), device="cuda", generator=g).double()
    assert torch.equal(_sketch(lib, a, om, order), a @ om)


@pytest.mark.parametrize("order", [b"R", b"C"])
def test_random_and_rows_that_do_not_split(lib, order):
    m, n, nl = 20011, 1501, 640
    g = torch.Generator(device="cuda").manual_seed(5)
    a = torch.randn(m, n, device="cuda", generator=g, dtype=torch.float64)
    om = torch.randn(n, nl, device="cuda", generator=g, dtype=torch.float64)
    a *= torch.exp(3 * torch.randn(m, 1, device="cuda", generator=g, dtype=torch.float64))
    a[200] = 0.0
    a[1000] *= torch.exp(8 * torch.randn(n, device="cuda", generator=g, dtype=torch.float64))  # outliers
    a[3000, 5], a[5000, 1500], a[7000, 0] = float("inf"), float("nan"), float("-inf")
    a[9000] *= 2.0 ** 500
    a[11000] *= 2.0 ** -500
    a[20010] *= 2.0 ** 390
    y, ref = _sketch(lib, a, om, order), a @ om
    assert bool((y[200] == 0).all())
    for r, k in ((3000, 5), (7000, 0)):
        assert bool((y[r] == torch.sign(om[k]) * a[r, k]).all())
    assert bool(torch.isnan(y[5000]).all())
    rows = torch.ones(m, dtype=torch.bool, device="cuda")
    rows[[200, 3000, 5000, 7000]] = False
    # row by row, relative to |a_i| (om has unit variance): a running sum of n terms rounds like a random
    # walk, under u sqrt(n) / 2 per output for either side (the margin is a factor two)
    scale = a[rows].abs().amax(1, keepdim=True)  # the largest exponents square out of range
    err = ((y[rows] - ref[rows]) / scale).norm(dim=1) / (a[rows] / scale).norm(dim=1) / nl ** 0.5
    assert float(err.max()) <= 2 * U * n ** 0.5


@pytest.mark.parametrize("l,N", [(96, 16), (65, 20)])
def test_gram_of_the_bases(lib, oracle, l, N):
    """G = Qs'Qs (the upper tiles, one set of digits) through the KN integration."""
    m = 30011
    rng = np.random.default_rng(l)
    base = np.linalg.qr(rng.standard_normal((m, l)))[0]
    qs = np.concatenate([np.linalg.qr(base + 0.2 * rng.standard_normal((m, l)) / np.sqrt(m))[0] for _ in range(N)], 1)
    qt = np.zeros((m, l))
    r = lib.integrate("d", "KN", lib.create_param(m, m, l, 0, N), qs, N * l, qt, l, argv=[3, 1e-9])
    assert lib.last_error()[0] == 0
    ref, it, _ = oracle.integrate_kolmogorov_nagumo(qs, l, N, maxit=3, tol=1e-9)
    assert int(r[0]) == it
    # columns of norm 1; G and the products to a few tens of u each over three iterations
    assert np.linalg.norm(qt - ref) / np.linalg.norm(ref) <= 1000 * U
