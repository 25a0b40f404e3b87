"""What the public calls accept and refuse of their plain arguments.  CPU tensors are refused last of all, so a call that
gets as far as that has had its other arguments accepted; nothing here needs a GPU."""
import math

import pytest
import torch

import retention_integration_b200 as prb
from retention_integration_b200 import retention

Q = torch.zeros(1, 256, 2, 64, dtype=torch.bfloat16)


@pytest.mark.parametrize("value", [math.inf, 512.0, 100.5, 0, -1, 2 ** 40, None])
def test_switch_over_may_be_any_number(value):
    with pytest.raises(prb.PRError, match="CUDA"):
        prb.power_retention(Q, Q, Q, chunk_size=128, switch_over_seq_len=value)
    with pytest.raises(prb.PRError, match="CUDA"):
        prb.power_retention_inference(Q, Q, Q, switch_over_seq_len=value)


def test_deg_may_be_a_whole_float():
    with pytest.raises(prb.PRError, match="CUDA"):
        prb.power_retention(Q, Q, Q, deg=2.0)
    with pytest.raises(prb.PRError, match="CUDA"):
        prb.power_retention_inference(Q, Q, Q, deg=2.0)
    with pytest.raises(prb.PRError, match="deg=4"):
        prb.power_retention_inference(Q, Q, Q, deg=4)
    with pytest.raises(AssertionError):
        prb.power_retention(Q, Q, Q, deg=2.5)


@pytest.mark.parametrize("auto", [False, True])
@pytest.mark.parametrize("chunk", [0, -1, -128])
def test_a_chunk_has_tokens(monkeypatch, auto, chunk):
    monkeypatch.setattr(retention, "AUTO_CHUNK", auto)
    with pytest.raises(prb.PRError, match="chunk_size"):
        prb.power_retention(Q, Q, Q, chunk_size=chunk)


def test_half_a_state_is_refused():
    sok = torch.zeros(1, 2, 2080)
    for pair in ((None, sok), (torch.zeros(1, 2, 2080, 64, dtype=torch.bfloat16), None)):
        with pytest.raises(prb.PRError, match="pair"):
            prb.power_retention(Q, Q, Q, initial_state=pair)


def _step(b=2, h=2, hq=4, d=64, dtype=torch.bfloat16):
    return [torch.zeros(b, 1, n, d, dtype=dtype) for n in (hq, h, h)] + [torch.zeros(b, 1, h)]


def _decode(q, k, v, g, dtype=torch.bfloat16):
    return prb.RetentionCache(2, 2, 64, dtype=dtype, device="cpu", recurrent=True).decode(q, k, v, g)


def test_a_recurrent_step_is_accepted_up_to_the_device():
    q, k, v, g = _step()
    for gates in (g, g[:, 0], None):
        with pytest.raises(prb.PRError, match="CUDA"):
            _decode(q, k, v, gates)


@pytest.mark.parametrize("change", [
    lambda q, k, v, g: (q, k[:1], v[:1], g),                       # fewer sequences than the queries have
    lambda q, k, v, g: (q, k[..., :32], v[..., :32], g),           # narrower keys
    lambda q, k, v, g: (q, k, v, g[:1]),                           # gates of fewer sequences
    lambda q, k, v, g: (q, k, v, g[..., :1]),                      # gates of fewer heads
    lambda q, k, v, g: (q, k, v, g.flatten()),
    lambda q, k, v, g: (q[:, :, :3], k, v, g),                     # heads that do not divide
])
def test_a_recurrent_step_of_other_shapes_is_refused(change):
    with pytest.raises(AssertionError):
        _decode(*change(*_step()))


def test_a_recurrent_step_of_another_dtype_than_the_state_is_refused():
    with pytest.raises(prb.PRError, match="state"):
        _decode(*_step(dtype=torch.float16))


def test_operator_wrappers_want_whole_chunks():
    """The tensors that the wrappers allocate hold whole chunks: a ragged sequence would be written past their ends."""
    from retention_integration_b200 import ops

    x, g, f = torch.zeros(1, 100, 2, 64, dtype=torch.bfloat16), torch.zeros(1, 100, 2), torch.zeros(1, 100, 2)
    xt = torch.zeros(1, 1, 2, 64, 64, dtype=torch.bfloat16)
    S, gr = torch.zeros(1, 1, 2, 2560, 64, dtype=torch.bfloat16), torch.zeros(1, 1, 2, 64, 64, dtype=torch.bfloat16)
    for call in (lambda: ops.gate_prep(x, g, 64, query_side=False),
                 lambda: ops.chunk_state(xt, None, x, 64, 2, True, True),
                 lambda: ops.expand_grad(x, x, S, gr, gr, None, None, f, 64, 2, True, 1.0, 2.0, 0, 0),
                 lambda: ops.chunk_dq(x, x, x, x, None, f, f, None, 64, 1.0),
                 lambda: ops.chunk_dkv(x, x, x, x, None, None, None, f, f, None, 64, -1, 1.0),
                 lambda: ops.gate_grad(f, None, f, None, None, None, 64)):
        with pytest.raises(prb.PRError, match="multiple of the chunk"):
            call()
