"""A NaN or an infinity in an operand of the NATIVE FP32 plane products is seen in the results or reported:
through block Grams and applies, Qs'Qs and Qs M, A'Qbar, whole solves and the adjoint, with the 32- and the
64-deep accumulation chunks."""
import pytest

from test_gpu_adjoint_sizes import _adjoint

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

BAD = [float("nan"), float("inf"), float("-inf")]


def _randn(*shape, seed=1):
    return torch.randn(*shape, device="cuda", generator=torch.Generator(device="cuda").manual_seed(seed))


def _bases(m, l, N):
    return torch.cat([torch.linalg.qr(_randn(m, l, seed=7 + i))[0] for i in range(N)], 1).contiguous()


def _noticed(lib, *outputs):
    status = lib.last_error()[0]
    lib.clear_error()
    return status != 0 or any(not bool(torch.isfinite(t).all()) for t in outputs)


@pytest.mark.parametrize("bad", BAD)
@pytest.mark.parametrize("order", [b"R", b"C"])
@pytest.mark.parametrize("nl", [64, 256])
def test_sketch_of_a_given_omega(lib, nl, order, bad):
    m, n = 9000, 1500
    a, om = _randn(m, n), _randn(n, nl, seed=2)
    a[700, 40] = bad
    y = torch.zeros(m, nl, device="cuda")
    src = a if order == b"R" else a.t().contiguous()
    lib.sketch_omega("s", lib.create_param(m, n, nl, 0, 1), src, n if order == b"R" else m, om, nl, y, nl, ordera=order)
    assert lib.last_error()[0] == 0
    fin = torch.isfinite(y)
    assert not bool(fin[700].any())
    fin[700] = True
    assert bool(fin.all())


@pytest.mark.parametrize("bad", BAD)
@pytest.mark.parametrize("alg", ["GR", "TS"])
@pytest.mark.parametrize("l", [64, 65, 100, 128])
def test_orthogonalization(lib, l, alg, bad):
    m, N = 20000, 8
    y = _randn(m, N * l)
    y[12345, 2 * l + 3] = bad
    lib.orthogonalize("s", alg, lib.create_param(m, m, l, 0, N), y, N * l)
    assert _noticed(lib, y)


@pytest.mark.parametrize("bad", BAD)
@pytest.mark.parametrize("alg", ["KN", "WY", "HR"])
@pytest.mark.parametrize("l", [48, 100])
def test_integration(lib, l, alg, bad):
    m, N = 12000, 8
    qs = _bases(m, l, N)
    qs[777, 3 * l] = bad
    qt = torch.zeros(m, l, device="cuda")
    lib.integrate("s", alg, lib.create_param(m, m, l, 0, N), qs, N * l, qt, l, argv=[3, 1e-9] if alg != "HR" else None)
    assert _noticed(lib, qt)


@pytest.mark.parametrize("bad", BAD)
@pytest.mark.parametrize("alg", ["GR", "TS"])
@pytest.mark.parametrize("where", ["a", "q"])
@pytest.mark.parametrize("n,l", [(1001, 40), (4000, 100)])
def test_postprocessing(lib, n, l, where, alg, bad):
    m = 12000
    a, q = _randn(m, n), _bases(m, l, 1)
    (a if where == "a" else q)[5000, 17] = bad
    s, u, v = (torch.zeros(*sh, device="cuda") for sh in ((l,), (m, l), (n, l)))
    lib.postprocess("s", alg, lib.create_param(m, n, l, 0, 1), a, n, q, l, s, u, l, v, l)
    assert _noticed(lib, s, u, v)


@pytest.mark.parametrize("bad", BAD)
@pytest.mark.parametrize("order", [b"R", b"C"])
@pytest.mark.parametrize("algs", [("GP", "GR", "KN", "GR"), ("GP", "TS", "WY", "GR"), ("GP", "TS", "HR", "TS")])
def test_whole_solve(lib, algs, order, bad):
    m, n, k, p, N = 20000, 1501, 40, 16, 8
    l = k + p
    a = _randn(m, 2 * l) @ _randn(2 * l, n, seed=3) + 0.01 * _randn(m, n, seed=4)
    a[19999, 1500] = bad
    src = a if order == b"R" else a.t().contiguous()
    s, u, v = (torch.zeros(*sh, device="cuda") for sh in ((l,), (m, l), (n, l)))
    _, _, status = lib.isvd("s", lib.create_param(m, n, k, p, N), algs, src, n if order == b"R" else m, s, u, l, v, l,
                            seed=3, ordera=order, retc=(0, 0, 0, 0), precision=0)
    assert status != 0 or _noticed(lib, s, u[:, :k], v[:, :k])
    lib.clear_error()


@pytest.mark.parametrize("bad", BAD)
def test_native_adjoint(lib, bad):
    m, n, k = 9519, 3069, 48
    u, v = torch.linalg.qr(_randn(m, k))[0], torch.linalg.qr(_randn(n, k))[0]
    s = torch.linspace(2.0, 1.0, k, device="cuda")
    a = (u * s) @ v.t()
    a[100, 200] = bad
    da, _ = _adjoint(lib, "s", a.contiguous(), s, u.contiguous(), v.contiguous(), _randn(k), _randn(m, k), _randn(n, k), 20,
                     1e-7)
    assert not bool(torch.isfinite(da).all())
