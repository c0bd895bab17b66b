"""Host matrices copied through the pinned staging buffers: pieces of whole lines, lines longer than a
buffer, padded leading dimensions and odd sizes give the results of the same matrix on the device."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("m,n,pad,order", [(3001, 701, 0, b"R"), (3001, 701, 3, b"R"), (70001, 33, 5, b"R"),
                                           (9, 300001, 0, b"R"), (9, 300001, 7, b"R"), (600011, 5, 1, b"C"),
                                           (2047, 1025, 1, b"C")])
@pytest.mark.parametrize("x", ["s", "d"])
def test_host_sketch_equals_device_sketch(lib, x, m, n, pad, order):
    """Each element takes part in the same products on either side, so the results are equal bit for bit."""
    rng = np.random.default_rng(m + n + pad)
    dt = np.float32 if x == "s" else np.float64
    lines, inner = (m, n) if order == b"R" else (n, m)
    a = rng.standard_normal((lines, inner + pad)).astype(dt)
    ld, nl = inner + pad, 6
    prm = lib.create_param(m, n, nl, 0, 1)
    out = []
    for src in (a, torch.from_numpy(a).cuda()):
        y = torch.zeros(m, nl, device="cuda", dtype=torch.float32 if x == "s" else torch.float64)
        lib.sketch(x, prm, src, ld, y, nl, 7, ordera=order)
        assert lib.last_error()[0] == 0
        out.append(y)
    assert bool((out[0] == out[1]).all())
    assert float(out[0].abs().sum()) > 0
