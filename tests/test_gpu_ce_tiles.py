"""The tiled narrow-row cross-entropy and the unaligned wide-row form, at the sizes where they can go wrong: rows that fill no tile, a
last tile whose bytes are no multiple of 16, widths at the register variants' edges, one row, odd wide rows (every offset of a row
inside a 16-byte piece), arrays that start off 16 bytes. Against the same loss in float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,C,cap,masked,shift", [
    (1, 61, 0.0, False, 0), (3, 257, 30.0, True, 0), (8, 64, 30.0, False, 0), (9, 65, 0.0, True, 0), (2501, 257, 30.0, True, 0),
    (5000, 288, 0.0, False, 0), (777, 289, 30.0, True, 0), (333, 1023, 0.0, True, 0), (1001, 1024, 30.0, False, 0), (70, 513, 30.0, False, 1),
    (13, 1025, 30.0, True, 0), (9, 8191, 0.0, False, 0), (7, 50303, 30.0, True, 0), (6, 60001, 0.0, True, 0), (11, 1761, 30.0, False, 3)])
def test_cross_entropy_rows_of_any_width(rows, C, cap, masked, shift):
    from gpu_util import ops
    g = torch.Generator(device="cuda").manual_seed(rows + C)
    z = torch.randn(rows * C + 4, device="cuda", generator=g)[shift:shift + rows * C].view(rows, C)
    z.mul_(3.0)
    t = torch.randint(0, C, (rows,), device="cuda", generator=g, dtype=torch.int32)
    mask = (torch.rand(rows, device="cuda", generator=g) < 0.7).to(torch.int32) if masked else None
    inv = 0.5 / rows
    x = z.double().requires_grad_()
    y = cap * torch.tanh(x / cap) if cap else x
    per = torch.logsumexp(y, dim=1) - y.gather(1, t.long()[:, None])[:, 0]
    want = (per * (mask if masked else 1)).sum() * inv
    want.backward()
    d, loss = torch.full((rows * C + 4,), float("nan"), device="cuda")[shift:shift + rows * C].view(rows, C), torch.ones(1, device="cuda")
    for out in (d, z):  # into another array, then in place
        loss.fill_(1.0)
        if cap:
            ops.softcap_cross_entropy(z, t, out, loss, cap, mask=mask, inv=inv)
        else:
            ops.softmax_cross_entropy(z, t, out, loss, mask=mask, inv=inv)
        torch.cuda.synchronize()
        assert ops.lib.xlstm_device_status() == 0
        assert abs(loss.item() - 1.0 - want.item()) <= 1e-5 * max(1.0, abs(want.item()))
        assert float((out.double() - x.grad).abs().max()) <= 1e-5 * max(float(x.grad.abs().max()), 1e-30)


@pytest.mark.parametrize("rows,C,cap,shift", [(40, 61, 0.0, 0), (40, 257, 30.0, 0), (33, 1024, 0.0, 0), (20, 300, 30.0, 1), (9, 5001, 30.0, 0), (5, 60001, 0.0, 0)])
def test_a_target_that_is_no_symbol_touches_nothing(rows, C, cap, shift):
    """Such a row has the gradient of its softmax alone and the loss of a probability at its floor; the rows beside it, and what lies
    behind the array, are as without it."""
    import math
    from gpu_util import ops
    g = torch.Generator(device="cuda").manual_seed(C)
    buf = torch.randn(rows * C + 4, device="cuda", generator=g) * 3.0
    z = buf[shift:shift + rows * C].view(rows, C)
    t = torch.randint(0, C, (rows,), device="cuda", generator=g, dtype=torch.int32)
    bad = {1: C, 2: C + 7, 3: -1, rows - 1: 0x7fffffff}
    for r, v in bad.items():
        t[r] = v
    live = torch.ones(rows, dtype=torch.bool, device="cuda")
    live[list(bad)] = False
    x = z.double()
    y = cap * torch.tanh(x / cap) if cap else x
    p = torch.softmax(y, 1)
    one = torch.zeros_like(p)
    one[live, t[live].long()] = 1.0
    inv = 1.0 / rows
    want = (p - one) * inv * ((1 - (y / cap) ** 2) if cap else 1.0)
    loss_want = ((-(p * one).sum(1)[live].log()).sum() - len(bad) * math.log(1e-30)) * inv
    out = torch.full((rows * C + 4,), 7.0, device="cuda")
    d, loss = out[shift:shift + rows * C].view(rows, C), torch.zeros(1, device="cuda")
    if cap:
        ops.softcap_cross_entropy(z, t, d, loss, cap, inv=inv)
    else:
        ops.softmax_cross_entropy(z, t, d, loss, inv=inv)
    torch.cuda.synchronize()
    assert ops.lib.xlstm_device_status() == 0
    assert float((d.double() - want).abs().max()) <= 1e-5 * float(want.abs().max())
    assert abs(loss.item() - float(loss_want)) <= 1e-5 * float(loss_want)
    assert bool((out[:shift] == 7.0).all()) and bool((out[shift + rows * C:] == 7.0).all())
