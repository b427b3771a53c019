"""The sLSTM loops inside a captured graph: recorded once after a first call outside, replayed on new inputs."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,NH,dh,T", [(8, 4, 256, 24), (3, 2, 64, 6), (40, 4, 512, 8)])
def test_loops_replay_from_a_graph(B, NH, dh, T):
    from gpu_util import ops
    H = NH * dh
    g = torch.Generator(device="cuda").manual_seed(3)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)
    wh, bc = r(NH, dh, 4 * dh) / dh ** 0.5, r(4 * H)
    pre, dy, gates, out = r(B, T, 4 * H), r(B, T, H), torch.empty((B, T, 4 * H), device="cuda"), torch.empty((B, T, H), device="cuda")
    slabs = ops.SlstmSlabs(B, T, H, "cuda")
    st, ds = (tuple(torch.empty((B, H), device="cuda") for _ in range(n)) for n in (4, 3))

    def run():
        gates.copy_(pre)
        ops.slstm_fused_time(wh, gates, bc, st, out, slabs, nh=NH)
        ops.slstm_fused_time_bwd(wh, dy, gates, ds, slabs, nh=NH)

    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        run()
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        run()
    for _ in range(2):
        pre.copy_(r(B, T, 4 * H))
        dy.copy_(r(B, T, H))
        graph.replay()
        torch.cuda.synchronize()
        got = [t.clone() for t in (out, gates, *st, *ds)]
        run()
        torch.cuda.synchronize()
        assert ops.lib.xlstm_device_status() == 0
        assert all(torch.equal(a, b) for a, b in zip(got, (out, gates, *st, *ds)))
    del graph
