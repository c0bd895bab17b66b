"""A sketch with a given Omega that selects or copies columns of A returns them to the last bit, up to the
largest value: products of one term are exact in FP32, whichever path computes them."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("order", [b"R", b"C"])
@pytest.mark.parametrize("m,n,nl", [(9000, 1500, 64), (9000, 1500, 256), (30011, 700, 100), (300, 200, 16)])
def test_selected_columns(lib, m, n, nl, order):
    g = torch.Generator(device="cuda").manual_seed(n)
    a = torch.randn(m, n, device="cuda", generator=g)
    sel = torch.randperm(n, device="cuda", generator=g)[:nl]
    a[5, sel[0]] = torch.finfo(torch.float32).max
    om = torch.zeros(n, nl, device="cuda")
    om[sel, torch.arange(nl, device="cuda")] = 1.0
    y = torch.zeros(m, nl, device="cuda")
    src = a if order == b"R" else a.t().contiguous()
    lib.sketch_omega("s", lib.create_param(m, n, nl, 0, 1), src, n if order == b"R" else m, om, nl, y, nl, ordera=order)
    assert lib.last_error()[0] == 0
    assert torch.equal(y, a[:, sel])
