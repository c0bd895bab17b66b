"""FP64 orthogonalizations that overwrite their blocks in place: widths around the tiles' edges, ragged row
counts, rows longer than the blocks (the gap stays untouched)."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

U = 2.0 ** -53


@pytest.mark.parametrize("alg", ["GR", "TS"])
@pytest.mark.parametrize("l", [1, 7, 31, 63, 64, 65, 96, 127, 128, 129])
def test_blocks_in_place(lib, alg, l):
    for m, N in ((l + 130, 3), (4097, 5)):
        g = torch.Generator(device="cuda").manual_seed(l)
        ld = N * l + 3
        y = torch.full((m, ld), 7.0, device="cuda", dtype=torch.float64)
        y[:, :N * l] = torch.randn(m, N * l, device="cuda", generator=g, dtype=torch.float64)
        q = y.clone()
        lib.orthogonalize("d", alg, lib.create_param(m, m, l, 0, N), q, ld)
        assert lib.last_error()[0] == 0
        assert bool((q[:, N * l:] == 7.0).all())
        # Gaussian blocks: condition at most (sqrt(m) + sqrt(l)) / (sqrt(m) - sqrt(l)), squared by GR's Gram
        cond = ((m ** 0.5 + l ** 0.5) / (m ** 0.5 - l ** 0.5)) ** 2
        for i in range(N):
            qi, yi = (t[:, i * l:(i + 1) * l] for t in (q, y))
            assert float((qi.t() @ qi - torch.eye(l, device="cuda", dtype=torch.float64)).abs().max()) <= 64 * l * U * cond
            assert float((yi - qi @ (qi.t() @ yi)).norm() / yi.norm()) <= 64 * l * U * cond
