"""The sLSTM time loops with register-resident weights (heads of a multiple of 16 up to 512 units, from a few steps on) against the CPU
oracle, at the edges of their geometry: one CTA and one warp's worth of a head, heads that do not fill the row slices, both column
groupings, batches that leave a group ragged or need several passes a step, states carried in and out."""
import pytest

from test_gpu_slstm import _case, _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,NH,dh,T,carry", [
    (1, 1, 16, 14, True), (3, 2, 48, 19, False), (7, 4, 96, 16, True), (33, 1, 32, 15, True), (5, 2, 160, 17, False), (32, 4, 256, 9, True),
    (9, 4, 256, 8, False), (1, 4, 512, 10, True), (9, 4, 512, 8, True), (19, 4, 384, 9, True), (4, 1, 512, 8, False), (2, 2, 480, 11, True)])
def test_register_resident_loops_match_the_oracle(B, NH, dh, T, carry):
    _check(*_case(B, NH * dh, NH, T, seed=B + dh, carry=carry))


@pytest.mark.parametrize("B,NH,dh,T,carry", [(33, 4, 512, 8, True), (67, 4, 512, 8, False), (130, 4, 256, 8, True), (70, 4, 160, 14, True), (130, 4, 128, 14, False)])
def test_batches_of_several_launches_or_none_match_the_oracle(B, NH, dh, T, carry):
    """A backward whose words exceed what the pool holds runs as two or more launches over slices of the batch, the last one smaller; narrow
    heads that would take several passes a step run on the cluster kernels backwards, or in both directions."""
    _check(*_case(B, NH * dh, NH, T, seed=B + dh, carry=carry))


def test_slices_of_a_batch_give_the_bits_of_the_whole():
    """Sequences are independent: a batch that is cut gives what its halves give alone, in the carried state too."""
    import torch
    from gpu_util import ops
    B, NH, dh, T = 48, 4, 512, 8
    H = NH * dh
    g = torch.Generator(device="cuda").manual_seed(2)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)
    wh, pre, bc, dy = r(NH, dh, 4 * dh) / dh ** 0.5, r(B, T, 4 * H), r(4 * H), r(B, T, H)
    st, ds = (r(B, H), r(B, H).abs() + 0.5, r(B, H), torch.tanh(r(B, H))), tuple(r(B, H) * 0.1 for _ in range(3))

    def run(lo, hi):
        s, d = (tuple(t[lo:hi].clone() for t in x) for x in (st, ds))
        gg, out, slabs = pre[lo:hi].clone(), torch.empty((hi - lo, T, H), device="cuda"), ops.SlstmSlabs(hi - lo, T, H, "cuda")
        ops.slstm_fused_time(wh, gg, bc, s, out, slabs, nh=NH, carry=True)
        ops.slstm_fused_time_bwd(wh, dy[lo:hi].contiguous(), gg, d, slabs, nh=NH, carry=True)
        return [out, gg, *s, *d, *slabs.t.values()]

    whole, halves = run(0, B), [torch.cat(x) for x in zip(run(0, B // 2), run(B // 2, B))]
    assert ops.lib.xlstm_device_status() == 0
    assert all(torch.equal(a, b) for a, b in zip(whole, halves))
