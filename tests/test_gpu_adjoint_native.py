"""The NATIVE FP32 adjoint, its operator on bf16 planes where that pays, keeps FP32 accuracy: against the FP64
adjoint of the same factors, in both storage orders of the complement systems."""
import pytest

from test_gpu_adjoint_sizes import _adjoint

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

U = 2.0 ** -24


@pytest.mark.parametrize("m,n,k", [(9519, 3069, 48), (4001, 2001, 64), (13000, 1277, 16), (2000, 3000, 32), (600, 500, 8)])
def test_native_fp32_accuracy(lib, m, n, k):
    g = torch.Generator(device="cuda").manual_seed(m + k)
    rn = lambda *sh: torch.randn(*sh, device="cuda", dtype=torch.float64, generator=g)  # noqa: E731
    r = 4 * k
    uu, vv = torch.linalg.qr(rn(m, r))[0], torch.linalg.qr(rn(n, r))[0]
    # a wide gap below s_k and gaps of 1 between neighbours: the systems' conditions and the factor F add
    # little to the rounding of the products
    sig = torch.cat([torch.arange(2 * k, k, -1), torch.linspace(0.3 * k, 0.1, r - k)]).to("cuda", torch.float64)
    f = lambda t: t.to(torch.float32).contiguous()  # noqa: E731
    a, s, u, v = f((uu * sig) @ vv.t()), f(sig[:k]), f(uu[:, :k]), f(vv[:, :k])
    ds, du, dv = f(rn(k)), f(rn(m, k)), f(rn(n, k))
    d = lambda t: t.double()  # noqa: E731
    ref, _ = _adjoint(lib, "d", d(a), d(s), d(u), d(v), d(ds), d(du), d(dv), 400, 1e-13)
    lib.lib.isvd_gpu_set_precision(0)
    da, _ = _adjoint(lib, "s", a, s, u, v, ds, du, dv, 200, 1e-9)
    # FP32 inputs and outputs (u), the systems' operator and right-hand sides to a few u: under 10 u (CUDA-core
    # products give 2 to 5 u)
    assert float((da.double() - ref).norm() / ref.norm()) <= 10 * U
