"""NATIVE FP32 work on a device that is nearly full: what has no room for planes runs on the CUDA cores, as it did
before planes, with the same results to FP32 rounding.  isvd_gpu_alloc_limit stands for the full device."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

U = 2.0 ** -24
MB = 1 << 20


@pytest.fixture
def room(lib):
    var = ctypes.c_size_t.in_dll(lib.lib, "isvd_gpu_alloc_limit")

    def leave(megabytes):
        var.value = int(megabytes * MB)
    yield leave
    var.value = 0


def _rel(x, y):
    return float((x.double() - y.double()).norm() / y.double().norm())


@pytest.mark.parametrize("order", [b"R", b"C"])
@pytest.mark.parametrize("megabytes", [400, 60, 13, 9])
def test_sketch(lib, room, order, megabytes):
    """All of A's planes are 480 MB; Omega' is 5 MB as a plane and 8 MB in FP32, 256 rows of planes are 6 MB."""
    m, n, nl = 20000, 4000, 512
    a = torch.randn(m, n, device="cuda", generator=torch.Generator(device="cuda").manual_seed(1))
    src = a if order == b"R" else a.t().contiguous()
    prm, lda = lib.create_param(m, n, nl, 0, 1), n if order == b"R" else m
    y, ref = torch.zeros(m, nl, device="cuda"), torch.zeros(m, nl, device="cuda")
    lib.sketch("s", prm, src, lda, ref, nl, 3, ordera=order)
    assert lib.last_error()[0] == 0
    room(megabytes)
    lib.sketch("s", prm, src, lda, y, nl, 3, ordera=order)
    assert lib.last_error()[0] == 0, lib.last_error()
    # a chain of n FP32 multiply-adds rounds like a random walk: under u sqrt(n) / 2, twice that for the margin
    assert _rel(y, ref) <= U * n ** 0.5


def _blocks(m, l, N):
    g = torch.Generator(device="cuda").manual_seed(l)
    return torch.randn(m, N * l, device="cuda", generator=g)


@pytest.mark.parametrize("alg", ["GR", "TS"])
@pytest.mark.parametrize("megabytes", [85, 119, 121, 300])
def test_orthogonalization(lib, room, alg, megabytes):
    """The blocks' planes are 118 MB; the temporary of the CUDA-core product is 78 MB."""
    m, l, N = 40000, 64, 8
    y = _blocks(m, l, N)
    q = y.clone()
    room(megabytes)
    lib.orthogonalize("s", alg, lib.create_param(m, m, l, 0, N), q, N * l)
    assert lib.last_error()[0] == 0, lib.last_error()
    for i in (0, N - 1):
        qi, yi = (t[:, i * l:(i + 1) * l].double() for t in (q, y))
        # as test_gpu_fp32_planes.py, with the CUDA cores' chains of m / 16 terms: u sqrt(2500) / 2 = 25 u, times four
        assert float((qi.t() @ qi - torch.eye(l, device="cuda")).abs().max()) <= 100 * U
        assert float((yi - qi @ (qi.t() @ yi)).norm() / yi.norm()) <= 100 * U


@pytest.mark.parametrize("alg", ["KN", "WY"])
@pytest.mark.parametrize("megabytes", [60, 119, 123, 300])
def test_integration(lib, room, alg, megabytes):
    m, l, N = 40000, 64, 8
    g = torch.Generator(device="cuda").manual_seed(2)
    base = torch.randn(m, l, device="cuda", generator=g)
    y = _blocks(m, l, N)
    qs = torch.cat([torch.linalg.qr(base + 0.2 * y[:, i * l:(i + 1) * l])[0] for i in range(N)], 1).contiguous()
    prm = lib.create_param(m, m, l, 0, N)
    qt, ref = torch.zeros(m, l, device="cuda"), torch.zeros(m, l, device="cuda")
    lib.integrate("s", alg, prm, qs, N * l, ref, l, argv=[3, 1e-9])
    assert lib.last_error()[0] == 0
    room(megabytes)
    lib.integrate("s", alg, prm, qs, N * l, qt, l, argv=[3, 1e-9])
    assert lib.last_error()[0] == 0, lib.last_error()
    assert _rel(qt, ref) <= 200 * U


@pytest.mark.parametrize("algs", [("GP", "GR", "KN", "GR"), ("GP", "TS", "WY", "TS"), ("GP", "TS", "HR", "GR")])
@pytest.mark.parametrize("megabytes", [260, 1015, 1030, 1100, 4000])
def test_solve(lib, room, algs, megabytes):
    """The planes of A that the sketch keeps for the projection are 927 MB, Y, Qbar and Omega 92 MB, the rest of the
    solve up to 160 MB."""
    m, n, k, p, N = 40000, 4000, 48, 16, 8
    l = k + p
    g = torch.Generator(device="cuda").manual_seed(5)
    x, w = (torch.randn(q, 2 * l, device="cuda", generator=g) for q in (m, n))
    a = (x * torch.linspace(1, 0.1, 2 * l, device="cuda")) @ w.t() + 0.01 * torch.randn(m, n, device="cuda", generator=g)
    prm = lib.create_param(m, n, k, p, N)

    def solve():
        s, u, v = (torch.zeros(*sh, device="cuda") for sh in ((l,), (m, l), (n, l)))
        _, _, status = lib.isvd("s", prm, algs, a, n, s, u, l, v, l, seed=3, retc=(0, 0, 0, 0), precision=0)
        assert status == 0, lib.last_error()
        return s, (u[:, :k].double() * s[:k]) @ v[:, :k].double().t()

    s0, a0 = solve()
    room(megabytes)
    s1, a1 = solve()
    # FP32 solves of the same sketch by other roundings: a few tens of u sqrt(n) at most
    assert float((s1 - s0).abs().max()) <= 20 * U * n ** 0.5 * float(s0[0])
    assert _rel(a1, a0) <= 100 * U * n ** 0.5


@pytest.mark.parametrize("megabytes", [40, 176, 180, 184, 188, 192, 196, 200, 208, 400])
def test_native_adjoint(lib, room, megabytes):
    """The planes of A are 171 MB, everything else up to 40 MB."""
    from test_gpu_adjoint_sizes import _adjoint
    m, n, k = 9519, 3069, 48
    g = torch.Generator(device="cuda").manual_seed(m)
    rn = lambda *sh: torch.randn(*sh, device="cuda", dtype=torch.float64, generator=g)  # noqa: E731
    r = 4 * k
    uu, vv = torch.linalg.qr(rn(m, r))[0], torch.linalg.qr(rn(n, r))[0]
    sig = torch.cat([torch.arange(2 * k, k, -1), torch.linspace(0.3 * k, 0.1, r - k)]).to("cuda", torch.float64)
    f = lambda t: t.to(torch.float32).contiguous()  # noqa: E731
    args = f((uu * sig) @ vv.t()), f(sig[:k]), f(uu[:, :k]), f(vv[:, :k]), f(rn(k)), f(rn(m, k)), f(rn(n, k)), 200, 1e-9
    ref, _ = _adjoint(lib, "s", *args)
    room(megabytes)
    da, _ = _adjoint(lib, "s", *args)
    assert _rel(da, ref) <= 20 * U  # either within 10 u of the FP64 adjoint (test_gpu_adjoint_native.py)
