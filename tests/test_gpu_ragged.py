"""Sizes where the kernels' edges lie: last chunks that are shorter than the others (down to one token), narrow heads,
and launches with more tiles than the GPU holds CTAs, where a CTA takes over the tiles of others.

The oracle is the quadratic form in float64 on the same 16-bit inputs.  16-bit operands give up to 5e-3 on every tensor
at most of these sizes, so 1e-2 bounds them with a factor of two.  On top of it comes what three roundings do that the
row sums divide: the backward takes <O, dO> from the rounded O, and the read-out's gradient from the rounded dO / l
and the rounded state.  Each puts half a unit per element on a difference that cancels, and a row whose weights all
happen to be tiny divides that by their small sum, so that one such row can carry a whole tensor's error.
_rounding_bound gives it row by row from the exact weights: rows where it is small are held to the plain 1e-2, and so
are all rows of the last chunk together, which see enough tokens."""
import pytest
import torch
import torch.nn.functional as F

from oracle import power_retention_oracle as oracle
from tests._golden import rel_l2

pytestmark = pytest.mark.gpu


def _inputs(dev, b, t, h, r, d, gated, dtype, seed):
    g = torch.Generator(dev).manual_seed(seed)
    Q, K, V, dO = (torch.randn(b, t, n, d, generator=g, device=dev).to(dtype) for n in (h * r, h, h, h * r))
    lg = F.logsigmoid(torch.randn(b, t, h, generator=g, device=dev) + 2.0) if gated else None
    return [Q, K, V] + ([lg] if gated else []), dO


def _grads(fn, leaves, dO):
    leaves = [x.detach().clone().requires_grad_(True) for x in leaves]
    out = fn(*leaves)
    return [out.detach(), *torch.autograd.grad(out, leaves, dO.to(out.dtype))]


def _rounding_bound(leaves, dO, gold):
    """dQ_i is off by e_i sum_j M_ij k_j and dK_j by sum_i e_i M_ij q_i where <O_i, dO_i> is off by e_i, with
    M_ij = 2 (q_i.k_j) e^{a_i-a_j} / l_i.  e_i is a sum of independent roundings of up to half a unit, three per
    element: three standard deviations are three half units times |O_i dO_i|.  The norm of every row, [b, t, heads]."""
    Q, K = (x.double() for x in leaves[:2])
    unit = 2.0 ** (-9 if leaves[0].dtype == torch.bfloat16 else -12)
    b, t, h, _ = K.shape
    r = Q.shape[2] // h
    Kx = K.repeat_interleave(r, dim=2)
    s = torch.einsum("bihd,bjhd->bhij", Q, Kx)
    decay = torch.ones_like(s)
    if len(leaves) == 4:
        a = leaves[3].double().cumsum(1).transpose(1, 2).repeat_interleave(r, dim=1)
        decay = torch.exp(torch.tril(a[..., :, None] - a[..., None, :]))
    decay = torch.tril(decay)
    l = (s * s * decay).sum(-1, keepdim=True)
    m = 2 * s * decay / l
    e = 3 * unit * (gold[0] * dO.double()).norm(dim=-1).transpose(1, 2)  # [b, hq, t]
    dq = torch.einsum("bhi,bhij,bjhd->bihd", e, m, Kx).norm(dim=-1)
    dk = torch.einsum("bhi,bhij,bihd->bjhd", e ** 2, m ** 2, Q ** 2).sum(-1)
    return {"dQ": dq, "dK": dk.view(b, t, h, r).sum(-1).sqrt()}


def _check(dev, b, t, h, r, d, chunk, gated, dtype=torch.bfloat16):
    import retention_integration_b200 as prb
    from retention_integration_b200 import _lib

    leaves, dO = _inputs(dev, b, t, h, r, d, gated, dtype, seed=t + d)
    ours = _grads(lambda *x: prb.power_retention(*x, deg=2, chunk_size=chunk), leaves, dO)
    gold = _grads(lambda *x: oracle.power_retention_quadratic(*x), [x.double() for x in leaves], dO)
    torch.cuda.synchronize()
    assert _lib.device_status(dev.index or 0) == 0
    last = (t - 1) // chunk * chunk if chunk else 0  # first token of the last chunk
    bound = _rounding_bound(leaves, dO, gold)
    for name, x, y in zip(("O", "dQ", "dK", "dV", "dlog_G"), ours, gold):
        x, y = (z if z.dim() == 4 else z[..., None] for z in (x.double(), y))
        err, size = (x - y).norm(dim=-1), y.norm(dim=-1)
        if name in bound:
            sure = bound[name] < 1e-2 * size
            assert sure.double().mean() > 0.75, name
            rest = 1e-2 * size[~sure].norm() + bound[name][~sure].norm()
            assert err[~sure].norm() <= rest, name
            assert err[sure].norm() < 1e-2 * size[sure].norm(), name
        else:
            assert err.norm() < 1e-2 * size.norm(), name
        # a gate's gradient is a difference of sums over the tokens; of the last few it may happen to be small
        floor = size.square().mean().sqrt() if name == "dlog_G" else 0.0
        assert err[:, last:].norm() < 1e-2 * max(size[:, last:].norm(), floor * size[:, last:].numel() ** 0.5), name


@pytest.mark.parametrize("t,chunk", [(129, 128), (191, 64), (193, 64), (255, 128), (257, 128), (300, 192), (321, 320),
                                     (1025, 1024), (1151, 1024)])
@pytest.mark.parametrize("d,r,gated,dtype", [(64, 1, True, torch.bfloat16), (64, 2, False, torch.float16),
                                             (32, 1, True, torch.bfloat16), (16, 2, True, torch.float16)])
def test_last_chunk_is_shorter(cuda_device, t, chunk, d, r, gated, dtype):
    _check(cuda_device, 2, t, 2, r, d, chunk, gated, dtype)


@pytest.mark.parametrize("b,t,h,r,d,chunk", [(8, 300, 32, 1, 64, 128), (4, 449, 16, 2, 64, 64), (8, 200, 32, 1, 32, 128),
                                             (6, 260, 32, 2, 64, None)])
def test_more_tiles_than_resident_ctas(cuda_device, b, t, h, r, d, chunk):
    _check(cuda_device, b, t, h, r, d, chunk, True)


@pytest.mark.parametrize("b,t,h,r", [(4, 1100, 24, 1), (4, 1025, 24, 2), (2, 2080, 8, 4)])
def test_runs_of_empty_tiles_are_taken_over(cuda_device, b, t, h, r):
    """A last chunk of a tile or less leaves seven tiles in a row that hold no rows, in every head of many more tiles
    than the GPU holds CTAs: each CTA takes over such runs, and its warps must not lose step in them."""
    _check(cuda_device, b, t, h, r, 64, 1024, True)


def test_final_state_of_a_ragged_sequence(cuda_device):
    """With a last chunk of 44 tokens the state after the last token is the one of any other blocking."""
    import retention_integration_b200 as prb

    (Q, K, V, lg), _ = _inputs(cuda_device, 2, 300, 2, 2, 64, True, torch.bfloat16, seed=1)
    O1, (s1, n1) = prb.power_retention(Q, K, V, lg, return_final_state=True, chunk_size=128)
    O2, (s2, n2) = prb.power_retention(Q, K, V, lg, return_final_state=True, chunk_size=320)
    # both round chunk states and operands to bf16 (2^-9 relative each)
    for x, y in ((O1, O2), (s1, s2), (n1, n2)):
        assert rel_l2(x.float().cpu(), y.float().cpu()) < 1e-2


def test_forward_mode_is_refused(cuda_device):
    """There is no forward-mode derivative; a tangent must not be dropped in silence."""
    import torch.autograd.forward_ad as fwAD

    import retention_integration_b200 as prb

    (Q, K, V, lg), _ = _inputs(cuda_device, 1, 64, 1, 1, 64, True, torch.bfloat16, seed=2)
    with fwAD.dual_level():
        Qd = fwAD.make_dual(Q, torch.ones_like(Q))
        with pytest.raises((RuntimeError, NotImplementedError)):
            prb.power_retention(Qd, K, V, lg, chunk_size=None)


@pytest.mark.parametrize("tk", [1, 63, 65, 300, 1025])
@pytest.mark.parametrize("h,gated,old,dtype", [(2, True, True, torch.bfloat16), (3, False, True, torch.float16),
                                               (40, True, False, torch.bfloat16)])
def test_compressed_cache(cuda_device, tk, h, gated, old, dtype):
    """The switch-over's new state against its float64 definition.  Operands and result are rounded to 16 bits: the
    gated key twice as a factor, the old state once more (2^-9 each in bf16, at most four in a row)."""
    import retention_integration_b200 as prb
    from retention_integration_b200 import _lib

    b, d = 2, 64
    (Q, K, V, *lg), _ = _inputs(cuda_device, b, tk, h, 1, d, gated, dtype, seed=tk + h)
    i, j = torch.triu_indices(d, d, device=cuda_device)
    w = torch.where(i == j, 1.0, 2.0).double()
    g = torch.Generator(cuda_device).manual_seed(7)
    state = torch.randn(b, h, i.numel(), d, generator=g, device=cuda_device).to(dtype) if old else None
    sok = torch.rand(b, h, i.numel(), generator=g, device=cuda_device) if old else None
    _, s1, n1 = prb.power_retention_inference(Q, K, V, lg[0] if gated else None, state, sok, switch_over_seq_len=tk)
    torch.cuda.synchronize()
    assert _lib.device_status(cuda_device.index or 0) == 0
    a = lg[0].double().cumsum(1) if gated else torch.zeros(b, tk, h, device=cuda_device, dtype=torch.float64)
    k64 = K.double() * torch.exp((a[:, -1:] - a) / 2).unsqueeze(-1)
    phi = k64[..., i] * k64[..., j] * w  # [b, tk, h, D]
    want, want_n = torch.einsum("bthp,bthe->bhpe", phi, V.double()), phi.sum(1)
    if old:
        want = want + state.double() * torch.exp(a[:, -1])[..., None, None]
        want_n = want_n + sok.double() * torch.exp(a[:, -1])[..., None]
    tol = 4 * 2.0 ** (-9 if dtype == torch.bfloat16 else -12)
    assert rel_l2(s1.double().cpu(), want.cpu()) < tol
    assert rel_l2(n1.double().cpu(), want_n.cpu()) < tol


def test_same_bits_whatever_else_is_in_the_launch(cuda_device):
    """Which tiles a persistent CTA has worked on before does not change the order of any sum."""
    import retention_integration_b200 as prb

    leaves, dO = _inputs(cuda_device, 4, 640, 48, 1, 64, True, torch.bfloat16, seed=9)
    fn = lambda *x: prb.power_retention(*x, deg=2, chunk_size=320)
    full = _grads(fn, leaves, dO)
    for lo in (0, 17, 45):
        part = _grads(fn, [x[:, :, lo:lo + 3].contiguous() for x in leaves], dO[:, :, lo:lo + 3].contiguous())
        for name, x, y in zip(("O", "dQ", "dK", "dV", "dlog_G"), part, full):
            assert torch.equal(x, y[:, :, lo:lo + 3]), (name, lo)


@pytest.mark.parametrize("t,chunk", [(200, 128), (640, 128), (100, 128)])
def test_states_that_nothing_reads_are_not_made(cuda_device, t, chunk):
    """The last chunk's state (no final state asked for) and the gradient of the first one's stay unwritten in the
    workspaces: whatever lies there, NaN here, reaches no result."""
    import retention_integration_b200 as prb

    leaves, dO = _inputs(cuda_device, 2, t, 2, 2, 64, True, torch.bfloat16, seed=t)
    want = _grads(lambda *x: prb.power_retention(*x, return_final_state=True, chunk_size=chunk)[0], leaves, dO)
    torch.cuda.empty_cache()
    for mb in (1, 2, 4, 8, 16, 32, 64):  # what the caching allocator hands out next
        torch.full((mb << 18,), float("nan"), device=cuda_device)
    got = _grads(lambda *x: prb.power_retention(*x, chunk_size=chunk, switch_over_seq_len=1), leaves, dO)
    for name, x, y in zip(("O", "dQ", "dK", "dV", "dlog_G"), got, want):
        assert torch.equal(x, y), name
