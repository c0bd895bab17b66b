"""The MIXED adjoint with more columns than a CTA's default shared memory holds sums for (both systems side by
side: 2 k > 6144), against the FP64 adjoint."""
import pytest

from test_gpu_adjoint_sizes import _adjoint

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def test_gram_cg_of_a_nearly_full_factorization(lib):
    m, n, k = 3088, 3080, 3073
    g = torch.Generator(device="cuda").manual_seed(k)
    rn = lambda *sh: torch.randn(*sh, device="cuda", dtype=torch.float64, generator=g)  # noqa: E731
    uu, vv = torch.linalg.qr(rn(m, n))[0], torch.linalg.qr(rn(n, n))[0]
    # gaps of 1 between neighbours, a wide one below s_k
    sig = torch.cat([torch.arange(2 * k, k, -1), torch.linspace(0.3 * k, 0.1, n - k)]).to("cuda", torch.float64)
    f = lambda t: t.to(torch.float32).contiguous()  # noqa: E731
    a, s, u, v = f((uu * sig) @ vv.t()), f(sig[:k]), f(uu[:, :k]), f(vv[:, :k])
    ds, du, dv = f(rn(k)), f(rn(m, k)), f(rn(n, k))
    d = lambda t: t.double()  # noqa: E731
    ref, _ = _adjoint(lib, "d", d(a), d(s), d(u), d(v), d(ds), d(du), d(dv), 400, 1e-13)
    lib.lib.isvd_gpu_set_precision(1)
    try:
        da, its = _adjoint(lib, "s", a, s, u, v, ds, du, dv, 200, 1e-6)
    finally:
        lib.lib.isvd_gpu_set_precision(0)
    # the residual tolerance times the systems' condition (under 2), and A to 2^-17 in two planes
    assert float((da.double() - ref).norm() / ref.norm()) <= 4e-6 + 2.0 ** -15
    assert 0 < its < 400
