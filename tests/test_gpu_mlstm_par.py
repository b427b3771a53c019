"""The chunk-parallel mLSTM kernels (square heads of 128 and 256, the longer sequences) against the CPU oracle, at the edges of
their tiling: a last chunk of one position, of 127 and full; every column split of the state kernel (few heads, about a wave of
them, more than a wave); states carried in and out in both directions; records saved and recomputed; both gradient widths."""
import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu
FW = ("ytil", "m", "psi", "C", "n", "mlast")
BW = ("dq", "dk", "dv", "dig", "dfg", "dC", "dn")


def _run(shape, gdtype, seed, carried, save):
    from gpu_util import ops, xl, dev, host, mlstm_inputs, bf16_round
    B, H, T, d = shape
    q, k, v, ig, fg, dy = mlstm_inputs(B, H, T, d, d, seed=seed, bf16=True)
    if gdtype == torch.bfloat16:
        dy = bf16_round(dy)
    r = np.random.default_rng(seed + 1)
    f32 = lambda a: a.astype(np.float32).astype(np.float64)
    carry = (f32(r.standard_normal((B * H, d, d))), f32(r.standard_normal((B * H, d))), f32(r.standard_normal((B * H,)))) if carried else None
    dst = (f32(r.standard_normal((B * H, d, d)) * 0.1), f32(r.standard_normal((B * H, d)) * 0.1)) if carried else None
    bf = torch.bfloat16
    st = ops.MlstmShape(B, H, T, d, d, 64, bf, gdtype)
    args = (dev(q, bf), dev(k, bf), dev(v, bf), dev(ig), dev(fg))
    cin, din = (None if x is None else tuple(dev(a) for a in x) for x in (carry, dst))
    fused = ops.mlstm_fused_fw(*args, st, carry_in=cin, save_states=save)
    g = ops.mlstm_fused_bw(fused, *args, dev(dy, gdtype), st, carry_in=cin, dstate_in=din)
    torch.cuda.synchronize()
    assert xl._lib.lib.xlstm_device_status() == 0, xl._lib.lib.xlstm_last_error()
    got = dict(ytil=host(fused.ytil), m=host(fused.msv), psi=host(fused.psiv), C=host(fused.state[0]), n=host(fused.state[1]),
               mlast=host(fused.state[2]), dq=host(g[0]), dk=host(g[1]), dv=host(g[2]), dig=host(g[3]), dfg=host(g[4]), dC=host(g[5][0]), dn=host(g[5][1]))
    c0 = dict(C0=carry[0], n0=carry[1], m0=carry[2]) if carried else dict(C0=None, n0=None, m0=None)
    d0 = dict(dC_in=dst[0], dn_in=dst[1]) if carried else dict(dC_in=None, dn_in=None)
    ref = dict(O.mlstm_core_fw(q, k, v, ig, fg, B, H, T, d, d, **c0))
    ref.update(O.mlstm_core_bw(q, k, v, ig, fg, dy, B, H, T, d, d, **c0, **d0))
    return got, ref, fused, g


@pytest.mark.parametrize("shape,gdtype,carried,save", [
    ((1, 2, 385, 128), torch.float32, False, True), ((1, 2, 511, 128), torch.bfloat16, True, True), ((2, 1, 512, 128), torch.float32, True, False),
    ((1, 1, 385, 256), torch.bfloat16, True, True), ((3, 1, 65, 256), torch.float32, False, True), ((1, 2, 128, 256), torch.bfloat16, True, False),
    ((2, 2, 511, 256), torch.float32, False, False), ((1, 2, 640, 256), torch.float32, True, True),
    ((25, 4, 400, 128), torch.bfloat16, False, True), ((40, 4, 390, 128), torch.float32, True, True), ((20, 3, 300, 256), torch.bfloat16, False, True)])
def test_chunk_parallel_kernels_match_the_oracle(shape, gdtype, carried, save):
    from gpu_util import rel_to_max
    got, ref, _, _ = _run(shape, gdtype, 71, carried, save)
    bad = ["%s %.3e" % (n, rel_to_max(got[n], ref[n])) for n in FW + BW if not rel_to_max(got[n], ref[n]) <= 2e-2]
    assert not bad, bad


def test_forgetting_inside_a_ragged_last_chunk_stays_finite():
    """Forget gates near zero drive the in-chunk decay to e^-400: positions past the end must not turn that into inf * 0."""
    from gpu_util import ops, dev, host, mlstm_inputs, rel_to_max
    B, H, T, d = 1, 2, 511, 128
    q, k, v, ig, fg, dy = mlstm_inputs(B, H, T, d, d, seed=73, fbias=-4.0, bf16=True)
    bf = torch.bfloat16
    st = ops.MlstmShape(B, H, T, d, d, 64, bf, torch.float32)
    args = (dev(q, bf), dev(k, bf), dev(v, bf), dev(ig), dev(fg))
    fused = ops.mlstm_fused_fw(*args, st)
    g = ops.mlstm_fused_bw(fused, *args, dev(dy), st)
    ref = dict(O.mlstm_core_fw(q, k, v, ig, fg, B, H, T, d, d), **O.mlstm_core_bw(q, k, v, ig, fg, dy, B, H, T, d, d))
    for n, x in (("ytil", fused.ytil), ("dq", g[0]), ("dk", g[1]), ("dv", g[2]), ("dig", g[3]), ("dfg", g[4])):
        assert rel_to_max(host(x), ref[n]) <= 2e-2, n


def test_recomputed_states_leave_the_gradients_bit_identical():
    a = _run((2, 2, 400, 128), torch.float32, 72, True, True)[3]
    b = _run((2, 2, 400, 128), torch.float32, 72, True, False)[3]
    for x, y in zip(a[:5] + a[5], b[:5] + b[5]):
        assert torch.equal(x, y)


@pytest.mark.parametrize("shape", [(1, 2, 385, 128), (1, 1, 65, 256)])
def test_states_that_start_at_any_float_are_read(shape):
    """A state cut out of a larger array starts where that array left off: on four bytes, not on sixteen."""
    from gpu_util import ops, xl, dev, mlstm_inputs
    B, H, T, d = shape
    q, k, v, ig, fg, dy = mlstm_inputs(B, H, T, d, d, seed=74, bf16=True)
    r = np.random.default_rng(75)
    f = lambda *s: dev(r.standard_normal(s))
    carry, dst = (f(B * H, d, d), f(B * H, d), f(B * H)), (f(B * H, d, d), f(B * H, d))

    def shifted(x):
        out = torch.empty(x.numel() + 1, device="cuda")[1:].view(x.shape)
        out.copy_(x)
        assert out.data_ptr() % 16 == 4
        return out

    bf = torch.bfloat16
    st = ops.MlstmShape(B, H, T, d, d, 64, bf, torch.float32)
    args = (dev(q, bf), dev(k, bf), dev(v, bf), dev(ig), dev(fg))
    res = []
    for c, ds in ((carry, dst), (tuple(map(shifted, carry)), tuple(map(shifted, dst)))):
        fused = ops.mlstm_fused_fw(*args, st, carry_in=c)
        g = ops.mlstm_fused_bw(fused, *args, dev(dy), st, carry_in=c, dstate_in=ds)
        torch.cuda.synchronize()
        res.append((fused.ytil, *fused.state, *g[:5], *g[5]))
    assert xl._lib.lib.xlstm_device_status() == 0
    assert all(torch.equal(a, b) for a, b in zip(*res))


def test_a_record_serves_a_backward_of_the_other_gradient_width():
    """64 heads of 400 positions, where the two gradient widths would be worth different kernels: a forward called with one gradient
    type leaves the record that a backward called with the other reads."""
    from gpu_util import ops, dev, mlstm_inputs
    B, H, T, d = 8, 8, 400, 128
    q, k, v, ig, fg, dy = mlstm_inputs(B, H, T, d, d, seed=76, bf16=True)
    bf = torch.bfloat16
    args, dyb = (dev(q, bf), dev(k, bf), dev(v, bf), dev(ig), dev(fg)), dev(dy, bf)
    wide, narrow = (ops.MlstmShape(B, H, T, d, d, 64, bf, t) for t in (torch.float32, bf))
    for fw, bw, g in ((wide, narrow, dyb), (narrow, wide, dyb.float())):
        got = ops.mlstm_fused_bw(ops.mlstm_fused_fw(*args, fw), *args, g, bw)
        want = ops.mlstm_fused_bw(ops.mlstm_fused_fw(*args, bw), *args, g, bw)
        for a, b in zip(got[:5] + got[5], want[:5] + want[5]):
            assert torch.equal(a, b)


@pytest.mark.parametrize("shape,carried", [((1, 4, 1500, 128), True), ((1, 2, 3000, 256), False), ((2, 2, 385, 128), True)])
def test_stabiliser_and_normaliser_keep_their_fp32_precision(shape, carried):
    """m and n are fp32 results that no product of the tensor cores enters. Each is rounded once where it is stored (6e-8) and inherits the
    fp32 logarithms, exponentials and sums behind it, a few roundings more: 2e-7 for m, 4e-7 for n, whatever the number of chunks."""
    got, ref, fused, _ = _run(shape, torch.float32, 77, carried, True)
    B, H, T, _ = shape
    for name, tol in (("m", 2e-7), ("mlast", 2e-7), ("n", 4e-7)):
        a, b = got[name].reshape(-1), np.asarray(ref[name]).reshape(-1)
        assert np.linalg.norm(a - b) <= tol * np.linalg.norm(b), (name, np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("shape", [(1, 2, 400, 128), (2, 1, 130, 256)])
def test_final_state_alone_agrees_with_a_chunk_parallel_forward(shape):
    """The states-only entry point keeps the kernels of one CTA per head: C within the bf16 products' bar, n and m to fp32 rounding."""
    from gpu_util import ops, dev, host, mlstm_inputs, rel_to_max
    B, H, T, d = shape
    q, k, v, ig, fg, _ = mlstm_inputs(B, H, T, d, d, seed=78, bf16=True)
    r = np.random.default_rng(79)
    cin = tuple(dev(a) for a in (r.standard_normal((B * H, d, d)), r.standard_normal((B * H, d)), r.standard_normal((B * H,))))
    bf = torch.bfloat16
    st = ops.MlstmShape(B, H, T, d, d, 64, bf, torch.float32)
    args = (dev(q, bf), dev(k, bf), dev(v, bf), dev(ig), dev(fg), st)
    full, alone = ops.mlstm_fused_fw(*args, carry_in=cin).state, ops.mlstm_final_state(*args, carry_in=cin)
    for a, b, tol in zip(alone, full, (2e-2, 2e-6, 2e-6)):
        assert rel_to_max(host(a), host(b)) <= tol
