"""The CUDA-core mLSTM path as a walk of the states and one CTA per chunk, against the CPU oracle: one chunk, a last chunk of one position
and full, chunks shorter than a warp, uneven head widths, states carried in and out, the record kept or rebuilt in the workspace."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,T,dqk,dhv,L,carried,save", [
    (1, 2, 64, 32, 32, 64, True, True), (2, 1, 65, 24, 24, 64, True, False), (1, 3, 128, 16, 48, 64, False, True),
    (2, 2, 130, 48, 16, 64, True, True), (1, 2, 33, 8, 8, 5, True, False), (1, 1, 200, 96, 96, 64, False, False)])
def test_walk_and_chunks_match_the_oracle(B, H, T, dqk, dhv, L, carried, save):
    import torch
    from gpu_util import ops, dev, host, mlstm_inputs, rel_to_max
    q, k, v, ig, fg, dy = mlstm_inputs(B, H, T, dqk, dhv, seed=81)
    r = np.random.default_rng(82)
    f32 = lambda a: a.astype(np.float32).astype(np.float64)
    carry = (f32(r.standard_normal((B * H, dhv, dqk))), f32(r.standard_normal((B * H, dqk))), f32(r.standard_normal((B * H,)))) if carried else None
    dst = (f32(r.standard_normal((B * H, dhv, dqk)) * 0.1), f32(r.standard_normal((B * H, dqk)) * 0.1)) if carried else None
    st = ops.MlstmShape(B, H, T, dqk, dhv, L, torch.float32, torch.float32)
    args = tuple(dev(x) for x in (q, k, v, ig, fg))
    cin, din = (None if x is None else tuple(dev(a) for a in x) for x in (carry, dst))
    fused = ops.mlstm_fused_fw(*args, st, carry_in=cin, save_states=save)
    g = ops.mlstm_fused_bw(fused, *args, dev(dy), st, carry_in=cin, dstate_in=din)
    got = dict(ytil=fused.ytil, m=fused.msv, psi=fused.psiv, C=fused.state[0], n=fused.state[1], mlast=fused.state[2], dq=g[0], dk=g[1], dv=g[2],
               dig=g[3], dfg=g[4], dC=g[5][0], dn=g[5][1])
    c0 = dict(C0=carry[0], n0=carry[1], m0=carry[2]) if carried else dict(C0=None, n0=None, m0=None)
    d0 = dict(dC_in=dst[0], dn_in=dst[1]) if carried else dict(dC_in=None, dn_in=None)
    ref = dict(O.mlstm_core_fw(q, k, v, ig, fg, B, H, T, dqk, dhv, **c0))
    ref.update(O.mlstm_core_bw(q, k, v, ig, fg, dy, B, H, T, dqk, dhv, **c0, **d0))
    for n, x in got.items():
        assert rel_to_max(host(x), ref[n]) <= 1e-4, n


@pytest.mark.parametrize("T,carried", [(64, False), (300, False), (129, True)])
def test_forget_gates_around_zero_do_not_cost_the_stabiliser_its_digits(T, carried):
    """log sigmoid(0) = -0.69 a position: the gates' sum reaches -44 over a chunk, one unit in whose last place is 3.8e-6, while m stays a
    number around 1. m_t is i_s plus the log gates of the few positions since s, each good to half a unit (3e-8) of its own, and is
    rounded once itself (6e-8 at 1): within 3e-7."""
    import torch
    from gpu_util import ops, dev, host
    B, H, d = 2, 3, 32
    r = np.random.default_rng(T)
    f32 = lambda a: a.astype(np.float32).astype(np.float64)
    q, k, v = (f32(r.standard_normal((B * T, H * d))) for _ in range(3))
    ig, fg = f32(0.5 * r.standard_normal((B * T, H))), f32(0.1 * r.standard_normal((B * T, H)))
    c0 = (f32(r.standard_normal((B * H, d, d))), f32(r.standard_normal((B * H, d))), f32(r.standard_normal(B * H))) if carried else None
    st = ops.MlstmShape(B, H, T, d, d, 64, torch.float32, torch.float32)
    fused = ops.mlstm_fused_fw(*(dev(a) for a in (q, k, v, ig, fg)), st, carry_in=None if c0 is None else tuple(dev(a) for a in c0))
    ref = O.mlstm_core_fw(q, k, v, ig, fg, B, H, T, d, d, **(dict(C0=c0[0], n0=c0[1], m0=c0[2]) if carried else {}))
    assert np.abs(host(fused.msv) - ref["m"]).max() <= 3e-7
    assert np.abs(host(fused.state[2]) - ref["mlast"]).max() <= 3e-7
