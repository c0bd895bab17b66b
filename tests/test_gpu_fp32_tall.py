"""NATIVE FP32 with more rows than 65535 tiles of 128: sketch, orthogonalization and integration."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

U = 2.0 ** -24
M, N_COLS, L, NS = 8400001, 64, 36, 2
STEP = 1 << 20


@pytest.fixture(scope="module")
def tall():
    g = torch.Generator(device="cuda").manual_seed(1)
    yield torch.randn(M, N_COLS, device="cuda", generator=g)
    torch.cuda.empty_cache()


def _gram(x, y):
    return sum(x[r:r + STEP].double().t() @ y[r:r + STEP].double() for r in range(0, M, STEP))


def _worst(x, y, c):
    """Largest row-block error of x against y c, relative to x."""
    return max(float((x[r:r + STEP].double() - y[r:r + STEP].double() @ c).norm() / x[r:r + STEP].double().norm())
               for r in range(0, M, STEP))


def _omega(lib, n, nl, seed):
    y = torch.zeros(n, nl, device="cuda", dtype=torch.float64)
    lib.sketch("d", lib.create_param(n, n, nl, 0, 1), torch.eye(n, device="cuda", dtype=torch.float64), n, y, nl, seed)
    return y


@pytest.mark.parametrize("alg", ["GR", "TS"])
def test_stages_row_major(lib, tall, alg):
    nl = L * NS
    prm = lib.create_param(M, N_COLS, L, 0, NS)
    y = torch.zeros(M, nl, device="cuda")
    lib.sketch("s", prm, tall, N_COLS, y, nl, 3)
    assert lib.last_error()[0] == 0
    assert _worst(y, tall, _omega(lib, N_COLS, nl, 3)) <= 13 * U
    q = y.clone()
    lib.orthogonalize("s", alg, prm, q, nl)
    assert lib.last_error()[0] == 0
    # Gram entries: running sums of M / 64 chunks in up to 16 splits, a random walk of about 8000 roundings
    # (45 u), a few of them in a row; bounds with a factor four
    for i in range(NS):
        qi, yi = q[:, i * L:(i + 1) * L], y[:, i * L:(i + 1) * L]
        g = _gram(qi, qi)
        assert float((g - torch.eye(L, device="cuda")).abs().max()) <= 400 * U
        assert _worst(yi, qi, _gram(qi, yi)) <= 400 * U
    qt = torch.zeros(M, L, device="cuda")
    lib.integrate("s", "KN", prm, q, nl, qt, L, argv=[2, 1e-9])
    assert lib.last_error()[0] == 0
    assert _worst(qt, q, torch.linalg.solve(_gram(q, q), _gram(q, qt))) <= 32 * U


def test_sketch_column_major(lib, tall):
    """The columns' planes are split through tiles of 32 rows of A."""
    nl = L * NS
    y = torch.zeros(M, nl, device="cuda")
    lib.sketch("s", lib.create_param(M, N_COLS, L, 0, NS), tall.t().contiguous(), M, y, nl, 3, ordera=b"C")
    assert lib.last_error()[0] == 0
    assert _worst(y, tall, _omega(lib, N_COLS, nl, 3)) <= 13 * U
