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
