"""Planes of FP32 rows: vector and general reads at ragged widths, with row strides beyond the width whose
gap is never read into the product (it holds NaN)."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

U = 2.0 ** -24


@pytest.mark.parametrize("lda_mod", [0, 1])
@pytest.mark.parametrize("m,n", [(2001, 1996), (2048, 2001), (2050, 2047), (1999, 2050), (2001, 4095)])
def test_sketch_of_strided_rows(lib, m, n, lda_mod):
    nl = 512
    lda = (n + 7) // 4 * 4 + lda_mod  # 16-byte aligned rows or not
    g = torch.Generator(device="cuda").manual_seed(n)
    a = torch.full((m, lda), float("nan"), device="cuda")
    a[:, :n] = torch.randn(m, n, device="cuda", generator=g)
    om = torch.randn(n, nl, device="cuda", generator=g)
    y = torch.zeros(m, nl, device="cuda")
    lib.sketch_omega("s", lib.create_param(m, n, 1, 0, nl), a, lda, om, nl, y, nl)
    assert lib.last_error()[0] == 0
    ref = a[:, :n].double() @ om.double()
    # chunks of 32 or 64 terms truncate at 2^-23 of their partial sums, n / 64 roundings of the running sum:
    # under 12 u + u sqrt(n / 64) relative to the norm
    err = float((y.double() - ref).norm() / ref.norm())
    assert err <= (12 + (n / 64) ** 0.5) * U
