"""Large FP64 products of operands graded against each other (large entries of a row meet small ones of a
column): every entry keeps the error bound of an FP64 inner product, relative to sum |a_ik| |b_kj|."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

U = 2.0 ** -53


def _bound(a, om):
    # any order of n multiply-adds: n u sum |a| |b|; as much again for the product it is compared with
    return 2 * a.shape[1] * U * (a.abs() @ om.abs())


def _check(lib, a, om, order):
    m, n = a.shape
    nl = om.shape[1]
    y = torch.full((m, nl), 7.0, device="cuda", dtype=torch.float64)
    src = a if order == b"R" else a.t().contiguous()
    lib.sketch_omega("d", lib.create_param(m, n, nl, 0, 1), src, n if order == b"R" else m, om, nl, y, nl, ordera=order)
    assert lib.last_error()[0] == 0
    assert bool(((y - a @ om).abs() <= _bound(a, om)).all())


@pytest.mark.parametrize("order", [b"R", b"C"])
@pytest.mark.parametrize("m,n,nl", [(12001, 2000, 640), (2300, 17000, 1000), (640, 40001, 512)])
@pytest.mark.parametrize("scale", [1e-3, 1e-10])
def test_opposed_halves(lib, m, n, nl, order, scale):
    g = torch.Generator(device="cuda").manual_seed(n)
    a = torch.randn(m, n, device="cuda", generator=g, dtype=torch.float64)
    om = torch.randn(n, nl, device="cuda", generator=g, dtype=torch.float64)
    a[:, : n // 2] *= scale
    om[n // 2:] *= scale
    _check(lib, a, om, order)
    # one row and one column of a kind among ordinary ones, and zero rows and columns
    a[:, : n // 2] /= scale
    om[n // 2:] /= scale
    a[m // 3, : n // 2] *= scale
    om[n // 2:, nl // 5] *= scale
    a[m // 2] = 0.0
    om[:, nl // 2] = 0.0
    _check(lib, a, om, order)


def test_opposed_columns_of_a_gram(lib):
    """G = Qs'Qs whose columns live on different rows: through the KN integration's first iterate."""
    m, l, N = 30011, 32, 12
    g = torch.Generator(device="cuda").manual_seed(1)
    qs = torch.randn(m, N * l, device="cuda", generator=g, dtype=torch.float64)
    w = torch.full((m, N * l), 1e-9, device="cuda", dtype=torch.float64)
    for i in range(N):
        w[i * 2500:(i + 1) * 2500, i * l:(i + 1) * l] = 1.0
    w[N * 2500:] = 1.0
    qs *= w
    qs = torch.cat([torch.linalg.qr(qs[:, i * l:(i + 1) * l])[0] for i in range(N)], 1).contiguous()
    qt = torch.zeros(m, l, device="cuda", dtype=torch.float64)
    lib.integrate("d", "KN", lib.create_param(m, m, l, 0, N), qs, N * l, qt, l, argv=[1, 1e-12])
    assert lib.last_error()[0] == 0
    # one step (reference @x@_integrate_kolmogorov_nagumo.c): Qbar = Q0 F + Qs (G E0) / N C^-1, in the span of Q0
    # and Qs Qs'Q0; its component beside them is rounding
    c = qs.t() @ qs[:, :l]
    basis = torch.linalg.qr(torch.cat([qs[:, :l], qs @ c], 1))[0]
    assert float((qt - basis @ (basis.t() @ qt)).norm() / qt.norm()) <= 1000 * U
