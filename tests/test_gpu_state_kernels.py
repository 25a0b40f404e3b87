"""The kernels of the chunk states, each at the sizes where its work is split differently: launches of few and of many
CTAs, states whose items follow one another in a CTA, Gram matrices at the end, last chunks that are shorter.

The references are the sums themselves in float64 on the operands as the kernels round them, so that what is left is
fp32 accumulation (2e-5 leaves a factor of ten over sqrt(n) 2^-24 with the n of these sizes) and one rounding of a
16-bit result (2^-9 / sqrt(3) = 1.1e-3 of the norm for bf16)."""
import pytest
import torch

from tests._golden import rel_l2

pytestmark = pytest.mark.gpu


def _pairs(dev):
    """First and second factor of every entry of the block layout at d = 64."""
    ab = [(a, 16 * y + i) for y in range(4) for a in range(16 * (y + 1)) for i in range(16)]
    return torch.tensor(ab, device=dev).T


def _status(dev):
    from retention_integration_b200 import _lib

    torch.cuda.synchronize()
    return _lib.device_status(dev.index or 0)


@pytest.mark.parametrize("b,n,nh,group,c", [(1, 1, 1, 1, 64), (1, 2, 2, 1, 192), (1, 3, 1, 3, 128), (2, 9, 4, 1, 320),
                                            (1, 40, 8, 1, 64)])
@pytest.mark.parametrize("weights,gram", [(True, True), (False, True), (True, False)])
def test_chunk_state(cuda_device, b, n, nh, group, c, weights, gram):
    from retention_integration_b200 import ops

    g = torch.Generator(cuda_device).manual_seed(n + c)
    hx = nh * group
    xt = torch.randn(b, n, hx, 64, c, generator=g, device=cuda_device).bfloat16()
    xs = torch.randn(b, n, hx, 64, c, generator=g, device=cuda_device).bfloat16()
    v = torch.randn(b, n * c, hx, 64, generator=g, device=cuda_device).bfloat16()
    S, G = ops.chunk_state(xt, xs, v, c, nh, key_weights=weights, want_gram=gram)
    S2, G2 = ops.chunk_state(xt, xs, v, c, nh, key_weights=weights, want_gram=gram)
    assert _status(cuda_device) == 0
    assert torch.equal(S, S2) and (G is None or torch.equal(G, G2))
    fa, fb = _pairs(cuda_device)
    w = torch.where(fa < fb // 16 * 16, 2.0, 1.0).double() if weights else torch.ones(fa.numel(), device=cuda_device).double()
    vc = v.view(b, n, c, nh, group, 64).double()
    for m in range(n):
        x = xt[:, m].view(b, nh, group, 64, c)
        phi = (x[:, :, :, fa] * x[:, :, :, fb]).double()  # the product of two bf16, rounded once
        ref = torch.einsum("bhgDi,bihge->bhDe", phi, vc[:, m]) * w[:, None]
        assert rel_l2(S[:, m].double(), ref) < 2e-3, m
        if gram:
            xg = xs[:, m].view(b, nh, group, 64, c).double()
            assert rel_l2(G[:, m].double(), torch.einsum("bhgai,bhgei->bhae", xg, x.double())) < 2e-5, m


@pytest.mark.parametrize("b,n,h,r,c", [(1, 2, 1, 1, 64), (1, 2, 1, 1, 512), (1, 3, 2, 2, 384), (2, 4, 4, 2, 200),
                                       (1, 12, 8, 1, 1024)])
@pytest.mark.parametrize("query_side", [True, False])
def test_expand_grad(cuda_device, b, n, h, r, c, query_side):
    from retention_integration_b200 import ops

    g = torch.Generator(cuda_device).manual_seed(n + c)
    hx, t, dev = h * r, n * c, cuda_device
    R = lambda *s: torch.randn(*s, generator=g, device=dev)
    W, X = R(b, t, hx, 64).bfloat16(), R(b, t, hx, 64).bfloat16()
    S, hi, lo = R(b, n, h, 2560, 64).bfloat16(), R(b, n, h, 64, 64).bfloat16(), (0.01 * R(b, n, h, 64, 64)).bfloat16()
    row_g = R(b, t, hx) if query_side else None
    scale, mult = (0.125, 2.0) if query_side else (1.0, 1.0)
    first, last = (1, n - 1) if query_side else (0, n - 2)
    args = (W, X, S, hi, lo, None, None, row_g, c, h, query_side, scale, mult, first, last)
    dX, gdot = ops.expand_grad(*args)
    dX2, gdot2 = ops.expand_grad(*args)
    assert _status(cuda_device) == 0
    assert torch.equal(dX, dX2) and torch.equal(gdot, gdot2)
    fa, fb = _pairs(dev)
    for m in range(n):
        rows = slice(m * c, (m + 1) * c)
        if not first <= m <= last:
            assert torch.count_nonzero(dX[:, rows]) == 0 and torch.count_nonzero(gdot[:, rows]) == 0
            continue
        for k in range(hx):
            x = (X[:, rows, k].float() * scale).bfloat16().double()
            dphi = torch.einsum("bie,bDe->biD", W[:, rows, k].double(), S[:, m, k // r].double())
            Gs = hi[:, m, k // r].double() + lo[:, m, k // r].double()
            gx = mult * torch.einsum("bae,bie->bia", Gs, x) * (row_g[:, rows, k].double()[..., None] if query_side else 1)
            gx.index_add_(2, fa, dphi * x[:, :, fb])
            gx.index_add_(2, fb, dphi * x[:, :, fa])
            assert rel_l2(dX[:, rows, k].double(), gx * scale) < 2e-5, (m, k)
            assert rel_l2(gdot[:, rows, k].double(), 0.5 * (gx * x).sum(-1)) < 2e-5, (m, k)
