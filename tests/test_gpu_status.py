"""A wait that ran out inside a tensor-core product is reported by every entry point that ran it.  The status is
injected from the host (ISVD_GPU_INJECT_TIMEOUT names the product); the kernels run as always."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

TIMEOUT = 4  # ISVD_GPU_ERROR_TIMEOUT


@pytest.fixture
def inject(monkeypatch):
    def arm(tag):
        monkeypatch.setenv("ISVD_GPU_INJECT_TIMEOUT", tag)
    yield arm
    monkeypatch.delenv("ISVD_GPU_INJECT_TIMEOUT", raising=False)


@pytest.mark.parametrize("x,given,tag", [("s", False, "sketch"), ("s", True, "fp32"), ("d", False, "int8"), ("d", True, "int8")])
@pytest.mark.parametrize("order", [b"R", b"C"])
def test_sketch(lib, inject, monkeypatch, x, given, tag, order):
    m, n, nl = 9000, 1500, 512
    dt = torch.float32 if x == "s" else torch.float64
    a, om = torch.randn(m, n, device="cuda", dtype=dt), torch.randn(n, nl, device="cuda", dtype=dt)
    y = torch.zeros(m, nl, device="cuda", dtype=dt)
    prm, lda = lib.create_param(m, n, nl, 0, 1), n if order == b"R" else m

    def run():
        if given:
            lib.sketch_omega(x, prm, a, lda, om, nl, y, nl, ordera=order)
        else:
            lib.sketch(x, prm, a, lda, y, nl, 3, ordera=order)
        code = lib.last_error()[0]
        lib.clear_error()
        return code

    inject(tag)
    assert run() == TIMEOUT
    monkeypatch.delenv("ISVD_GPU_INJECT_TIMEOUT")
    assert run() == 0


@pytest.mark.parametrize("x,tag", [("s", "fp32"), ("d", "int8")])
def test_batch(lib, inject, monkeypatch, x, tag):
    """The products of a matrix of its own (its sketch, Qs'Qs)."""
    from test_gpu_batched import run_batch
    dt = torch.float32 if x == "s" else torch.float64
    g = torch.Generator(device="cuda").manual_seed(1)
    mats = [dict(m=m, n=n, k=k, p=k // 2, a=torch.randn(m, n, device="cuda", generator=g, dtype=dt))
            for m, n, k in ((300, 200, 4), (9000, 2001, 32))]
    inject(tag)
    with pytest.raises(AssertionError):
        run_batch(lib, x, mats, 8, [1, 2])
    assert lib.last_error()[0] == TIMEOUT
    lib.clear_error()
    monkeypatch.delenv("ISVD_GPU_INJECT_TIMEOUT")
    run_batch(lib, x, mats, 8, [1, 2])


@pytest.mark.parametrize("mixed,tag", [(1, "adjoint_a"), (1, "adjoint_gram_op"), (0, "adjoint_a2"), (0, "adjoint_a"),
                                       (0, "fp32")])
def test_adjoint(lib, inject, monkeypatch, mixed, tag):
    from test_gpu_adjoint_sizes import _adjoint
    x, dt = "s", torch.float32
    m, n, k = 9519, 3072, 64
    g = torch.Generator(device="cuda").manual_seed(1)
    rn = lambda *sh: torch.randn(*sh, device="cuda", dtype=dt, generator=g)  # noqa: E731
    u, v = torch.linalg.qr(rn(m, k))[0].contiguous(), torch.linalg.qr(rn(n, k))[0].contiguous()
    s = torch.linspace(2.0, 1.0, k, device="cuda", dtype=dt)
    args = ((u * s) @ v.t()).contiguous(), s, u, v, rn(k), rn(m, k), rn(n, k), 20, 1e-6
    lib.lib.isvd_gpu_set_precision(mixed)
    try:
        inject(tag)
        with pytest.raises(AssertionError):
            _adjoint(lib, x, *args)
        assert lib.last_error()[0] == TIMEOUT
        lib.clear_error()
        monkeypatch.delenv("ISVD_GPU_INJECT_TIMEOUT")
        _adjoint(lib, x, *args)
    finally:
        lib.lib.isvd_gpu_set_precision(0)
