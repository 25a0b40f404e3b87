"""The choice between the quadratic form and chunks for sequences without states (pr_blocking): by the heads and the width,
not by the tokens alone; the same on every path; and what runs is what it says, bit for bit."""
import ctypes
import random

import pytest
import torch
import torch.nn.functional as F


def _choice(b, t, h, hq, d, chunk, longest=2048):
    from retention_integration_b200 import _lib

    i = ctypes.c_int
    return _lib.lib().pr_blocking(i(b), ctypes.c_longlong(t), i(h), i(hq), i(d), i(chunk), i(longest))


def test_choice_by_work():
    """0: quadratic.  Every shape here was measured in both forms, more than 5 % apart (replayed; the shapes of
    retention.blocking's docstring among them)."""
    want = {(1, 2000, 2, 2, 64, 128): 0, (8, 2048, 16, 16, 64, 1024): 0, (8, 2048, 4, 32, 64, 1024): 0,
            (4, 2048, 2, 24, 64, 1024): 0, (16, 1100, 32, 32, 64, 128): 0, (1, 2048, 1, 12, 64, 1024): 1024,
            (1, 1999, 1, 16, 64, 1536): 768, (8, 2048, 16, 16, 32, 1024): 0, (1, 2048, 2, 2, 32, 128): 0,
            (1, 2048, 2, 24, 32, 1024): 1024, (16, 2048, 4, 48, 32, 1024): 1024, (1, 2048, 2, 2, 16, 128): 0,
            (16, 2048, 32, 32, 16, 1024): 1024, (8, 2048, 4, 32, 16, 1024): 1024, (16, 1100, 32, 32, 16, 128): 0}
    for args, c in want.items():
        assert _choice(*args) == c, args


def test_choice_properties():
    from retention_integration_b200 import _lib, retention

    fast = _lib.lib().pr_fast_chunk
    rng = random.Random(3)
    for _ in range(3000):
        t, chunk = rng.randint(1, 5000), rng.choice([0, rng.randint(1, 3000)])
        h, r, d, b = rng.randint(1, 32), rng.randint(1, 16), rng.choice([16, 32, 64]), rng.randint(1, 64)
        c, got = fast(ctypes.c_longlong(t), ctypes.c_int(chunk)), _choice(b, t, h, h * r, d, chunk)
        assert got in (0, c)
        if t <= c:
            assert got == 0
        elif t > 2048:
            assert got == c
        assert _choice(b, t, h, h * r, d, chunk, 0) == (0 if t <= c else c)
        retention.AUTO_CHUNK = True
        assert (retention.blocking(b, t, h, h * r, d, chunk or None) or 0) == got
        retention.AUTO_CHUNK = False
        assert retention.blocking(b, t, h, h * r, d, chunk or None) == (chunk or None)
    # sizes that the operator refuses: an answer, no crash
    for bad in ((0, 2000, 2, 2, 64, 128), (1, 2000, 0, 2, 64, 128), (1, 2000, 4, 2, 64, 128), (1, 2000, 2, 2, 80, 128),
                (1, 2000, 2, 2, 0, 128)):
        assert _choice(*bad) == 1024
    assert _choice(1, 0, 2, 2, 64, 128) == 0 and _choice(1, 2000, 2, 2, 64, 0) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("b,t,h,r,d,chunk,runs", [(4, 2048, 32, 1, 16, 1024, 1024), (1, 2048, 2, 12, 32, 128, 1024),
                                                  (1, 1999, 1, 16, 64, 1536, 768), (1, 2049, 2, 1, 64, 128, 768),
                                                  (1, 2049, 2, 2, 32, 1024, 1024), (1, 2000, 2, 1, 64, 128, None)])
def test_runs_as_chosen(cuda_device, b, t, h, r, d, chunk, runs):
    import retention_integration_b200 as prb
    from retention_integration_b200 import retention

    g = torch.Generator(cuda_device).manual_seed(t + d)
    R = lambda *s: torch.randn(*s, generator=g, device=cuda_device)
    leaves = [R(b, t, n, d).bfloat16().requires_grad_() for n in (h * r, h, h)] + [F.logsigmoid(R(b, t, h) + 2).requires_grad_()]
    dO = R(b, t, h * r, d).bfloat16()

    def run(auto, chunk, longest=2048):
        retention.AUTO_CHUNK, retention.QUADRATIC_TOKENS = auto, longest
        try:
            out = prb.power_retention(*leaves, chunk_size=chunk)
            return [out.detach(), *torch.autograd.grad(out, leaves, dO)]
        finally:
            retention.AUTO_CHUNK, retention.QUADRATIC_TOKENS = False, 2048

    same = lambda x, y: all(torch.equal(p, q) for p, q in zip(x, y))
    auto = run(True, chunk)
    assert same(auto, run(False, runs))
    assert same(run(True, chunk, 0), run(False, retention_chunk(t, chunk)))  # the limit is the one that Python names


def retention_chunk(t, chunk):
    from retention_integration_b200 import retention

    retention.AUTO_CHUNK = True
    try:
        return retention.effective_chunk(t, chunk)
    finally:
        retention.AUTO_CHUNK = False
