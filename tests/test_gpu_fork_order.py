"""The state-free backward's two kernels on their two streams.  Each holds one CTA per SM while it has tiles, so the one
that comes first decides: with chunk_dkv's few long tiles behind chunk_dq's many short ones the two run one after the
other, which a replayed graph does and eager launches happened not to.  A replay runs the same kernels without the
host, so it is no slower than the eager pass; a quarter is allowed for clocks and the graph's own launch."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _us(fn, n):
    a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    times = []
    for _ in range(5):
        a.record()
        for _ in range(n):
            fn()
        b.record()
        torch.cuda.synchronize()
        times.append(a.elapsed_time(b) * 1e3 / n)
    return sorted(times)[2]


@pytest.mark.parametrize("b,t,h,r", [(4, 1024, 2, 12), (4, 2048, 2, 12), (4, 2048, 2, 4)])
def test_replay_is_no_slower_than_eager(cuda_device, b, t, h, r):
    import retention_integration_b200 as prb

    g = torch.Generator(cuda_device).manual_seed(t + r)
    leaves = [torch.randn(b, t, n, 64, generator=g, device=cuda_device).bfloat16().requires_grad_() for n in (h * r, h, h)]
    dO = torch.randn(b, t, h * r, 64, generator=g, device=cuda_device).bfloat16()

    def step():
        return torch.autograd.grad(prb.power_retention(*leaves), leaves, dO)

    eager = step()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        kept = step()
    graph.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(x, y) for x, y in zip(eager, kept))
    for _ in range(10):
        step()
    assert _us(graph.replay, 20) <= 1.25 * _us(step, 20)
