"""The fp32 weight and bias gradient kernel against a float64 product, accumulating and scaled: one tile and one row, tile edges in k and n,
widths off four floats, one row slice and many with a ragged last one."""
import importlib

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,k,n", [(1, 1, 1), (31, 64, 64), (33, 65, 63), (257, 128, 4), (2048, 128, 128), (1000, 24, 683), (4097, 130, 130)])
def test_linear_gradients(rows, k, n):
    lib = importlib.import_module("neural-networks_b200._lib").lib
    g = torch.Generator(device="cuda").manual_seed(rows + k + n)
    x, dy, dw, db = (torch.randn(*s, device="cuda", generator=g) for s in ((rows, k), (rows, n), (k, n), (n,)))
    want_w, want_b = dw.double() + 0.5 * (x.double().t() @ dy.double()), db.double() + 0.5 * dy.double().sum(0)
    size = lib.xlstm_linear_grad_f32_workspace_bytes(rows, k, n)
    ws = torch.full((max(size, 1),), 255, dtype=torch.uint8, device="cuda")  # NaN patterns: every part it reads must have been written
    rc = lib.xlstm_linear_grad_f32(torch.cuda.current_stream().cuda_stream, x.data_ptr(), dy.data_ptr(), dw.data_ptr(), db.data_ptr(), rows, k, n, 0.5,
                                   ws.data_ptr(), size)
    assert rc == 0
    for got, want in ((dw, want_w), (db, want_b)):
        assert float((got.double() - want).abs().max() / want.abs().max()) <= 1e-5


@pytest.mark.parametrize("kind", ["transposed", "expanded", "sliced", "strided input", "no rows"])
def test_a_projection_takes_gradients_of_any_strides(kind):
    """The fp32 projection's backward on rows that do not lie one behind the other, and on none: as on their copies."""
    import importlib
    layers = importlib.import_module("neural-networks_b200.layers")
    g = torch.Generator(device="cuda").manual_seed(3)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)
    rows, k, n = (0 if kind == "no rows" else 96), 40, 24
    w, b, x, dy = r(k, n), r(n), r(rows, k), r(rows, n)
    if kind == "transposed":
        dy = r(n, rows).t()
    elif kind == "expanded":
        dy = r(1, n).expand(rows, n)
    elif kind == "sliced":
        dy = r(rows, 2 * n)[:, n:]
    elif kind == "strided input":
        x, dy = r(k, rows).t(), r(n, rows).t()
    lin = layers.Linear(w, b)
    lin.forward(x)
    dx = lin.backward(dy, scale=0.5)
    ref = 0.5 * dy.double()
    for got, want in ((dx, ref @ w.double().t()), (lin.w.g, x.double().t() @ ref), (lin.b.g, ref.sum(0))):
        assert got.shape == want.shape
        if want.numel():
            assert float((got.double() - want).abs().max()) <= 1e-5 * max(float(want.abs().max()), 1.0)
