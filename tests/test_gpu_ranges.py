"""Values near the ends of the exponent range."""
import pytest
import torch

from oracle import power_retention_oracle as oracle
from tests._golden import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [1e-3, 1.0, 1e3, 1e6])
@pytest.mark.parametrize("deg,chunk", [(2, None), (2, 128), (4, None)])
def test_fast_gates_with_row_sums_of_any_size(cuda_device, size, deg, chunk):
    """Gates that lose e^-78 within 64 tokens: the separated factors of the gate are near the smallest normal number and
    only just not replaced by the exponential per pair, and row sums of (s q.k)^deg from 1e-24 to 1e24 go with them.
    16-bit operands give 2e-3 to 5e-3 at every size; deg 4 doubles it."""
    import retention_integration_b200 as prb

    if deg == 4:
        size = size ** 0.5
    g = torch.Generator(cuda_device).manual_seed(3)
    Q, K, V, dO = (torch.randn(1, 384, 2, 64, generator=g, device=cuda_device).to(torch.bfloat16) for _ in range(4))
    leaves = [Q * size, K * size, V, torch.full((1, 384, 2), -1.24, device=cuda_device)]

    def grads(fn, xs):
        xs = [x.detach().clone().requires_grad_(True) for x in xs]
        out = fn(*xs)
        return [out.detach(), *torch.autograd.grad(out, xs, dO.to(out.dtype))]

    got = grads(lambda *x: prb.power_retention(*x, deg=deg, chunk_size=chunk), leaves)
    want = grads(lambda *x: oracle.power_retention_quadratic(*x, deg=deg), [x.double() for x in leaves])
    for name, x, y in zip(("O", "dQ", "dK", "dV", "dlog_G"), got, want):
        assert rel_l2(x.double().cpu(), y.cpu()) < deg * 5e-3, name
