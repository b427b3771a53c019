"""A projection adds the bias it holds at the call: one written in place since the last optimizer step counts, in every form of the
epilogue (the reference adds the bias tensor itself, src/gpu/linear.rs)."""
import importlib

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bf16,narrow,scale", [(True, True, 1.0), (True, True, 0.125), (True, True, 96 ** -0.5), (True, False, 1.0), (False, False, 1.0)])
def test_a_bias_written_in_place_is_the_one_added(bf16, narrow, scale):
    layers = importlib.import_module("neural-networks_b200.layers")
    g = torch.Generator(device="cuda").manual_seed(5)
    w, b, x = (torch.randn(*s, device="cuda", generator=g) for s in ((64, 32), (32,), (48, 64)))
    lin = layers.Linear(w, torch.zeros_like(b), bf16=bf16)
    lin.b.w.copy_(b)
    want = layers.Linear(w, b, bf16=bf16)
    if narrow:  # between two products the narrowed bias is read again
        assert not torch.equal(lin.forward(x, narrow=True, scale=scale), layers.Linear(w, torch.zeros_like(b), bf16=True).forward(x, narrow=True, scale=scale))
    assert torch.equal(lin.forward(x, narrow=narrow, scale=scale), want.forward(x, narrow=narrow, scale=scale))
    assert torch.equal(lin.forward(x, residual=torch.ones(48, 32, device="cuda")), want.forward(x, residual=torch.ones(48, 32, device="cuda")))


@pytest.mark.parametrize("d", [128, 256])
def test_a_cells_biases_written_in_place_are_the_ones_added(d):
    """q, k and v of a cell narrow their biases together, once a forward call: heads of 256 scale k by a power of two, of 128 not."""
    import numpy as np
    layers = importlib.import_module("neural-networks_b200.layers")
    p = layers.init_lm_params(np.random.default_rng(1), 16, d, 1, 1, d, d, 64, std=0.3)["blocks"][0]["cell"]
    t = {k: (torch.as_tensor(v) if k != "kind" else v) for k, v in p.items()}
    x = torch.randn(40, d, device="cuda", generator=torch.Generator(device="cuda").manual_seed(4))
    want = layers.MLstm(t, 1, d, d, bf16=True).forward(x, 1, 40)
    cell = layers.MLstm({k: (torch.zeros_like(v) if k in ("bq", "bk", "bv") else v) for k, v in t.items()}, 1, d, d, bf16=True)
    assert not torch.equal(cell.forward(x, 1, 40), want)
    for l, n in ((cell.lq, "bq"), (cell.lk, "bk"), (cell.lv, "bv")):
        l.b.w.copy_(t[n])
    assert torch.equal(cell.forward(x, 1, 40), want)


def test_narrowing_several_vectors_is_rounding_each():
    ops = importlib.import_module("neural-networks_b200").ops
    g = torch.Generator(device="cuda").manual_seed(6)
    v = [torch.randn(n, device="cuda", generator=g) for n in (1, 7, 256, 300001)]
    for scale in (1.0, 0.0625):
        for a, b in zip(ops.narrow_biases(v, [scale] * 4), v):
            assert torch.equal(a, (b * scale).to(torch.bfloat16))
