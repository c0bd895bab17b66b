"""Bases with a few rows of high leverage: the tiles of G = Qs'Qs that fall back to the FP64 tensor cores, in
K splits, beside those of the int8 products."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

U = 2.0 ** -53


@pytest.mark.parametrize("blocks", ["one", "all"])
@pytest.mark.parametrize("m,l,N", [(40000, 64, 16), (20011, 48, 9), (30011, 65, 12)])
def test_gram_with_outlier_rows(lib, oracle, m, l, N, blocks):
    g = torch.Generator(device="cuda").manual_seed(l)
    base = torch.randn(m, l, device="cuda", generator=g, dtype=torch.float64)
    parts = []
    for i in range(N):
        q = base + 0.2 * torch.randn(m, l, device="cuda", generator=g, dtype=torch.float64)
        if blocks == "all" or i == 3:
            q[:10] *= 100.0
        parts.append(torch.linalg.qr(q)[0])
    qs = torch.cat(parts, 1).contiguous()
    qt = torch.zeros(m, l, device="cuda", dtype=torch.float64)
    r = lib.integrate("d", "KN", lib.create_param(m, m, l, 0, N), qs, N * l, qt, l, argv=[3, 1e-9])
    assert lib.last_error()[0] == 0
    ref, it, _ = oracle.integrate_kolmogorov_nagumo(qs.cpu().numpy(), l, N, maxit=3, tol=1e-9)
    assert int(r[0]) == it
    # columns of norm 1; G and the products to a few tens of u each over three iterations
    assert np.linalg.norm(qt.cpu().numpy() - ref) / np.linalg.norm(ref) <= 1000 * U
