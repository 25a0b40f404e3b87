"""Short sequences without states run in the quadratic form whatever chunk was asked for (retention.QUADRATIC_TOKENS).
The result does not depend on the blocking: the same 6e-3 between two blockings that the choice of the chunk size is
held to, from both sides of the line, for every form of the request."""
import pytest
import torch
import torch.nn.functional as F

from tests._golden import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("t", [129, 1024, 1025, 1999, 2048, 2049])
@pytest.mark.parametrize("chunk,r,gated,dtype", [(128, 1, True, torch.bfloat16), (1024, 2, False, torch.float16),
                                                 (100, 1, True, torch.bfloat16), (1536, 1, True, torch.bfloat16)])
@pytest.mark.parametrize("d", [32, 48, 64])
def test_short_sequences(cuda_device, t, chunk, r, gated, dtype, d):
    import retention_integration_b200 as prb
    from retention_integration_b200 import retention

    g = torch.Generator(cuda_device).manual_seed(t + chunk)
    h = 2
    R = lambda *s: torch.randn(*s, generator=g, device=cuda_device)
    base = [R(1, t, h * r, d).to(dtype), R(1, t, h, d).to(dtype), R(1, t, h, d).to(dtype)]
    base += [F.logsigmoid(R(1, t, h) + 2.0)] if gated else []
    dO = R(1, t, h * r, d).to(dtype)
    # queries as a view with other strides too: the native path makes them dense
    base[0] = torch.cat([base[0], base[0]], 1)[:, :t]

    def run(auto, native=True, **kw):
        retention.AUTO_CHUNK, retention.NATIVE_SEQUENCER = auto, native
        try:
            leaves = [x.detach().requires_grad_(True) for x in base]
            out = prb.power_retention(*leaves, chunk_size=chunk, **kw)
            return [out.detach(), *torch.autograd.grad(out, leaves, dO)]
        finally:
            retention.AUTO_CHUNK, retention.NATIVE_SEQUENCER = True, True

    asked, auto = run(False), run(True)
    for x, y in zip(asked, auto):
        assert x.shape == y.shape and rel_l2(y.float(), x.float()) < 6e-3
    if t <= retention.QUADRATIC_TOKENS:
        never = run(False, switch_over_seq_len=float("inf"))  # the quadratic form by request: the same kernels
        assert all(torch.equal(x, y) for x, y in zip(never, auto))
        if t % 128 == 0 and d == 64:
            assert all(torch.equal(x, y) for x, y in zip(run(True, native=False), auto))
