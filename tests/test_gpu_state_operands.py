"""Operands of the state kernels that the package itself never makes, or makes only at other sizes: state-path gradients that
start 16 bytes past a 32-byte boundary (a C host's buffers may), fp16 chunk states, operand heads summed over launches in
which a CTA takes several items, chunks that are no multiple of a stage."""
import pytest
import torch

from tests._golden import rel_l2
from tests.test_gpu_state_kernels import _pairs, _status

pytestmark = pytest.mark.gpu


def _at_16(x):
    """The same values 16 bytes past a 32-byte boundary."""
    room = torch.empty(x.numel() + 4, device=x.device, dtype=x.dtype)
    y = room[4:].view(x.shape).copy_(x)
    assert x.data_ptr() % 32 == 0 and y.data_ptr() % 32 == 16
    return y


@pytest.mark.parametrize("d,dtype", [(64, torch.bfloat16), (48, torch.float16), (32, torch.bfloat16), (16, torch.float16)])
@pytest.mark.parametrize("t,c", [(384, 192), (200, 200)])
def test_state_gradients_at_16_bytes(cuda_device, d, dtype, t, c):
    from retention_integration_b200 import ops

    g = torch.Generator(cuda_device).manual_seed(t + d)
    R = lambda *s: torch.randn(*s, generator=g, device=cuda_device)
    b, h, r = 2, 3, 2
    Q, dO = R(b, t, h * r, d).to(dtype), R(b, t, h * r, d).to(dtype)
    K, V = R(b, t, h, d).to(dtype), R(b, t, h, d).to(dtype)
    a = -torch.rand(b, t // c, c, h, generator=g, device=cuda_device).cumsum(2).view(b, t, h)
    dl, l = R(b, t, h * r), 1 + R(b, t, h * r).abs()
    dqs, dks = R(b, t, h * r, d), R(b, t, h, d)
    for without, at_32, at_16 in ((ops.chunk_dq(Q, dO, K, V, a, dl, l, None, c, 0.125),
                                   ops.chunk_dq(Q, dO, K, V, a, dl, l, dqs, c, 0.125),
                                   ops.chunk_dq(Q, dO, K, V, a, dl, l, _at_16(dqs), c, 0.125)),
                                  (ops.chunk_dkv(Q, dO, K, V, None, a, None, dl, l, None, c, -1, 0.125),
                                   ops.chunk_dkv(Q, dO, K, V, None, a, None, dl, l, dks, c, -1, 0.125),
                                   ops.chunk_dkv(Q, dO, K, V, None, a, None, dl, l, _at_16(dks), c, -1, 0.125))):
        assert all(torch.equal(x, y) for x, y in zip(at_32, at_16))
        # one rounding to 16 bits each side of the difference; the gradients themselves are of the state path's size
        added = dqs if at_32[0].shape == Q.shape else dks
        size = added.norm() + 2 * without[0].float().norm()
        assert (at_32[0].float() - without[0].float() - added).norm() < size * (2 ** -8 if dtype == torch.bfloat16 else 2 ** -11)
    assert _status(cuda_device) == 0


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("b,n,nh,group,c", [(1, 2, 1, 1, 64), (2, 8, 4, 3, 64), (1, 9, 4, 4, 192), (1, 33, 2, 2, 72), (1, 5, 8, 12, 200)])
def test_chunk_state(cuda_device, dtype, b, n, nh, group, c):
    from retention_integration_b200 import ops

    g = torch.Generator(cuda_device).manual_seed(n + c)
    hx, cp, dev = nh * group, (c + 63) // 64 * 64, cuda_device
    xt, xs = (torch.randn(b, n, hx, 64, cp, generator=g, device=dev).to(dtype) for _ in range(2))
    xt[..., c:], xs[..., c:] = 0, 0  # what a transposed copy holds past the end of a chunk
    v = torch.randn(b, n * c, hx, 64, generator=g, device=dev).to(dtype)
    S, G = ops.chunk_state(xt, xs, v, c, nh, key_weights=True, want_gram=True)
    S2, G2 = ops.chunk_state(xt, xs, v, c, nh, key_weights=True, want_gram=True)
    assert _status(dev) == 0
    assert torch.equal(S, S2) and torch.equal(G, G2)
    fa, fb = _pairs(dev)
    w = torch.where(fa < fb // 16 * 16, 2.0, 1.0).double()
    vc = v.view(b, n, c, nh, group, 64).double()
    for m in range(n):
        x = xt[:, m, ..., :c].view(b, nh, group, 64, c)
        phi = (x[:, :, :, fa] * x[:, :, :, fb]).double()  # the product of two 16-bit values, rounded once
        ref = torch.einsum("bhgDi,bihge->bhDe", phi, vc[:, m]) * w[:, None]
        # one rounding of the result, 1.1e-3 of the norm in bf16 and an eighth of that in fp16; fp32 sums
        assert rel_l2(S[:, m].double(), ref) < (2e-3 if dtype == torch.bfloat16 else 2.5e-4), m
        xg = xs[:, m, ..., :c].view(b, nh, group, 64, c).double()
        assert rel_l2(G[:, m].double(), torch.einsum("bhgai,bhgei->bhae", xg, x.double())) < 2e-5, m
