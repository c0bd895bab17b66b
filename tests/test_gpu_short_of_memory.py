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
