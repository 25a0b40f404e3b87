"""Short sequences without states run in the chunks that were asked for (or their multiple, retention.effective_chunk), bit for
bit: the quadratic form is the same function, but its float32 gradient of the gates rounds 1e-3 differently.  It is there
for a caller who asks for it, by chunk_size=None or by retention.QUADRATIC_TOKENS."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("native", [True, False])
@pytest.mark.parametrize("b,t,h,r,d,chunk,gated,dtype", [(1, 2000, 2, 1, 64, 128, True, torch.bfloat16),
                                                         (2, 2048, 2, 4, 64, 1024, False, torch.float16),
                                                         (1, 1100, 4, 1, 64, 128, True, torch.float16),
                                                         (1, 2048, 2, 12, 32, 512, True, torch.bfloat16),
                                                         (1, 1999, 1, 2, 16, 1536, True, torch.bfloat16),
                                                         (1, 700, 2, 1, 48, 400, True, torch.bfloat16)])
def test_short_sequences_run_as_asked(cuda_device, native, b, t, h, r, d, chunk, gated, dtype):
    import retention_integration_b200 as prb
    from retention_integration_b200 import retention

    g = torch.Generator(cuda_device).manual_seed(t + chunk)
    R = lambda *s: torch.randn(*s, generator=g, device=cuda_device)
    leaves = [R(b, t, n, d).to(dtype).requires_grad_() for n in (h * r, h, h)]
    leaves += [F.logsigmoid(R(b, t, h)).requires_grad_()] if gated else []
    dO = R(b, t, h * r, d).to(dtype)
    retention.AUTO_CHUNK = True
    c = retention.effective_chunk(t, chunk)

    def run(auto, chunk, tokens=None, **kw):
        old = retention.QUADRATIC_TOKENS
        retention.AUTO_CHUNK, retention.NATIVE_SEQUENCER = auto, native
        retention.QUADRATIC_TOKENS = old if tokens is None else tokens
        try:
            out = prb.power_retention(*leaves, chunk_size=chunk, **kw)
            return [out.detach(), *torch.autograd.grad(out, leaves, dO)]
        finally:
            retention.AUTO_CHUNK, retention.NATIVE_SEQUENCER, retention.QUADRATIC_TOKENS = False, True, old

    same = lambda x, y: all(torch.equal(p, q) for p, q in zip(x, y))
    asked, whole = run(True, chunk), run(False, chunk, switch_over_seq_len=float("inf"))
    assert same(asked, run(False, c))
    if native or t % c == 0:  # padded, the quadratic form of the other path has other tiles
        assert same(whole, run(True, chunk, tokens=t)) and same(asked, run(True, chunk, tokens=t - 1))
    if t > c:
        assert not same(asked, whole)
