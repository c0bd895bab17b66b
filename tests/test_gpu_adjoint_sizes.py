"""The conjugate-gradient launches of the MIXED adjoint (one system or both side by side) at column counts
around a warp and a CTA's width and row counts that leave remainders, against the FP64 adjoint."""
import ctypes

import numpy as np
import pytest

from isvd_b200.capi import c_int_t, ptr

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _adjoint(lib, x, a, s, u, v, ds, du, dv, iters, tol):
    m, n, k = u.shape[0], v.shape[0], u.shape[1]
    vp = ctypes.c_void_p
    fn = getattr(lib.lib, "isvd_%sSvdAdjoint" % x)
    fn.argtypes = [c_int_t, c_int_t, c_int_t, ctypes.c_char, vp, c_int_t, vp, vp, c_int_t, vp, c_int_t, vp, vp,
                   c_int_t, vp, c_int_t, vp, c_int_t, ctypes.c_int, ctypes.c_double, ctypes.POINTER(ctypes.c_int)]
    fn.restype = ctypes.c_int
    da, its = torch.zeros_like(a), ctypes.c_int(0)
    st = fn(m, n, k, b"R", ptr(a), n, ptr(s), ptr(u), k, ptr(v), k, ptr(ds), ptr(du), k, ptr(dv), k, ptr(da), n, iters,
            tol, ctypes.byref(its))
    assert st == 0, lib.last_error()
    return da, its.value


@pytest.mark.parametrize("both", [False, True], ids=["u", "uv"])
@pytest.mark.parametrize("m,n,k", [(1200, 520, 5), (1000, 1000, 16), (2050, 1048, 31), (3001, 2000, 33), (2500, 1304, 129),
                                   (2600, 1600, 160)])
def test_gram_cg_sizes(lib, m, n, k, both):
    g = torch.Generator(device="cuda").manual_seed(m + k)
    rn = lambda *sh: torch.randn(*sh, device="cuda", dtype=torch.float64, generator=g)  # noqa: E731
    r = 2 * k + 20
    uu, vv = torch.linalg.qr(rn(m, r))[0], torch.linalg.qr(rn(n, r))[0]
    sig = torch.cat([torch.linspace(2.0, 1.0, k), torch.linspace(0.5, 0.1, r - k)]).to("cuda", torch.float64)
    f = lambda t: t.to(torch.float32).contiguous()  # noqa: E731
    a32, s32, u32, v32 = f((uu * sig) @ vv.t()), f(sig[:k]), f(uu[:, :k]), f(vv[:, :k])
    ds, du, dv = f(rn(k)), f(rn(m, k)), f(rn(n, k)) if both else None
    d = lambda t: None if t is None else t.double()  # noqa: E731
    ref, _ = _adjoint(lib, "d", d(a32), d(s32), d(u32), d(v32), d(ds), d(du), d(dv), 400, 1e-13)
    lib.lib.isvd_gpu_set_precision(1)
    try:
        da, its = _adjoint(lib, "s", a32, s32, u32, v32, ds, du, dv, 200, 1e-6)
        stop, cap = _adjoint(lib, "s", a32, s32, u32, v32, ds, du, dv, 3, 1e-30)
    finally:
        lib.lib.isvd_gpu_set_precision(0)
    # the residual tolerance times the systems' condition (s_k^2 / (s_k^2 - 0.25) < 2), and A to 2^-17 in two planes
    # with 1 / (s_i^2 - s_j^2) up to k / 2 between neighbours
    assert float((da.double() - ref).norm() / ref.norm()) <= 4e-6 + 2.0 ** -17 * k / 2
    assert 0 < its < 200 * (1 + both)
    assert cap == 3 * (1 + both)
    assert bool(torch.isfinite(stop).all())
