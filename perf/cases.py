"""The work that users of this package have it do, as cases for timing: training steps, prompts, decode steps and the
callers' glue, through the public entry points, from the smallest calls to the benchmark's own sizes.

A case is a dict of plain values; "kind" says which entry point it goes through:

    train      power_retention forward and backward
    prefill    power_retention_inference on a whole prompt, which is compressed into a state
    resume     power_retention that continues from a state and returns the next one (RetentionCache.prefill's call)
    extend     power_retention_inference of several new tokens against a state and the tokens cached since (these included)
    decode     power_retention_inference of one new token against a state and the tokens cached since (this one included)
    recurrent  RetentionCache.decode of one token without a token cache (the state advances)
    glue       prepare_qkvg forward and backward

Queries, keys, values and upstream gradients are N(0, 1); gates are logsigmoid(N(0, 1)) in training and
logsigmoid(6.906768 + N(0, 1)) in inference, as create_inputs has them.
"""
import torch
import torch.nn.functional as F

import retention_integration_b200 as prb

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}
GATE_BIAS = 6.906768
LARGEST = 65536 * 8  # tokens x heads of the largest training case


def listed():
    return [
        # a training step of one layer on a long sequence: the benchmark's headline workload
        dict(name="train_long", kind="train", b=1, t=65536, h=8, ratio=1, d=64, chunk=1024, dtype="bf16", gated=True),
        # grouped queries in fp16 without gates, a length that is no multiple of the chunk
        dict(name="train_gqa", kind="train", b=4, t=5000, h=2, ratio=4, d=64, chunk=1024, dtype="fp16", gated=False),
        # the odd length of the test grid with the reference's default chunk
        dict(name="train_ragged", kind="train", b=1, t=2000, h=2, ratio=1, d=64, chunk=128, dtype="bf16", gated=True),
        # create_inputs' defaults: a small model's layer, head dim 32, no chunking
        dict(name="train_d32", kind="train", b=2, t=1024, h=8, ratio=1, d=32, chunk=0, dtype="bf16", gated=True),
        # the shortest configuration of the benchmark: launches and host time
        dict(name="train_short", kind="train", b=1, t=1024, h=4, ratio=1, d=64, chunk=128, dtype="bf16", gated=True),
        # a batch of prompts compressed into states: the benchmark's prefill
        dict(name="prefill", kind="prefill", b=16, t=2048, h=32, ratio=1, d=64, dtype="bf16", gated=True),
        # the next piece of one long prompt, continuing from its state
        dict(name="resume", kind="resume", b=1, t=3001, h=8, ratio=4, d=64, chunk=1024, dtype="bf16", gated=True),
        # a few new tokens at once against a state (the inference test grid's sizes)
        dict(name="extend", kind="extend", b=1, tq=63, tk=64, h=2, ratio=12, d=64, dtype="bf16", gated=True),
        # a served batch generating: the benchmark's decode step in the middle of its cache
        dict(name="decode", kind="decode", b=16, tk=257, h=32, ratio=1, d=64, dtype="bf16", gated=True),
        # one user generating: latency
        dict(name="decode_one", kind="decode", b=1, tk=37, h=4, ratio=4, d=64, dtype="bf16", gated=True),
        # the same batch without a token cache: the state is read and written
        dict(name="recurrent", kind="recurrent", b=16, h=32, ratio=1, d=64, dtype="bf16"),
        # between projection and operator at the headline workload's size
        dict(name="glue", kind="glue", b=1, t=65536, h=8, ratio=1, d=64, dtype="bf16", gated=True, half_split=False),
    ]


def _log(rng, lo, hi):
    """A whole number of [lo, hi], spread over its logarithm."""
    return min(hi, max(lo, int(lo * (hi / lo) ** rng.random() + 0.5)))


def draw(rng):
    kind = rng.choice(["train", "train", "train", "train", "prefill", "resume", "extend", "decode", "decode",
                       "recurrent", "glue"])
    while True:
        c = dict(kind=kind, b=_log(rng, 1, 16), h=rng.choice([1, 2, 4, 8, 16, 32]), ratio=rng.choice([1, 1, 1, 2, 4, 8, 12]),
                 d=64, dtype=rng.choice(["bf16", "bf16", "bf16", "fp16"]), gated=rng.random() < 0.8)
        if kind in ("train", "resume", "glue"):
            c["t"] = _log(rng, 16, 65536)
            if rng.random() < 0.4:  # the powers of two and their multiples that most training runs use
                c["t"] = max(16, c["t"] // 256 * 256)
        if kind in ("train", "resume"):
            c["chunk"] = rng.choice([128, 256, 512, 1024, 1024])
        if kind == "train":
            c["d"] = rng.choice([64, 64, 64, 32])
            if c["t"] <= 2048 and rng.random() < 0.4:
                c["chunk"] = 0
        if kind == "prefill":
            c["t"] = _log(rng, 128, 4096)
        if kind == "extend":
            c["tq"] = _log(rng, 2, 256)
            c["tk"] = c["tq"] + _log(rng, 1, 512)
        if kind == "decode":
            c["tk"] = _log(rng, 1, 1000)
        if kind == "recurrent":
            c["dtype"] = "bf16"
            del c["gated"]
        if kind == "glue":
            c["half_split"] = rng.random() < 0.5
        heads = c["b"] * c["h"] * c["ratio"]
        if heads * c.get("t", c.get("tq", 1) * 16) <= LARGEST and c["b"] * c["h"] <= 512 and heads <= 2048:
            return c


def _randn(g, *shape, dtype=torch.float32):
    return torch.randn(*shape, generator=g, device="cuda", dtype=dtype)


def _state(g, b, h, d, dtype):
    """A state pair in the exact layout as some tokens leave it: sum_j phi(k_j) v_j^T and sum_j phi(k_j)."""
    n = 96
    a, c = torch.triu_indices(d, d, device="cuda")
    w = torch.where(a == c, 1.0, 2.0)
    state = torch.empty(b, h, a.numel(), d, device="cuda", dtype=dtype)
    sok = torch.empty(b, h, a.numel(), device="cuda")
    for i in range(b):
        k, v = _randn(g, h, n, d), _randn(g, h, n, d)
        phi = k[:, :, a] * k[:, :, c] * w
        state[i] = phi.transpose(1, 2) @ v
        sok[i] = phi.sum(1)
    return state, sok


def prepare(case, seed):
    g = torch.Generator("cuda").manual_seed(seed)
    kind, b, h, d = case["kind"], case["b"], case["h"], case["d"]
    hq, dt = h * case["ratio"], DTYPES[case["dtype"]]
    gated = case.get("gated", True)
    s = dict(case=case)
    if kind == "train":
        t = case["t"]
        leaves = [_randn(g, b, t, n, d, dtype=dt).requires_grad_() for n in (hq, h, h)]
        if gated:
            leaves.append(F.logsigmoid(_randn(g, b, t, h)).requires_grad_())
        s.update(leaves=leaves, dO=_randn(g, b, t, hq, d, dtype=dt))
    elif kind == "glue":
        t, used = case["t"], (hq + 2 * h) * d + (h if gated else 0)
        s["x"] = _randn(g, b, t, -(-used // 8) * 8, dtype=dt).requires_grad_()
        s["sin"], s["cos"] = prb.rotary_tables(t, d, "cuda")
        s["up"] = [_randn(g, b, t, n, d, dtype=dt) for n in (hq, h, h)] + ([_randn(g, b, t, h)] if gated else [])
    else:
        if kind in ("prefill", "resume"):
            tq = tk = room = case["t"]
        else:  # the cached tokens are the filled part of a longer preallocated cache
            tq, tk = case.get("tq", 1), case.get("tk", 1)
            room = tk if kind == "recurrent" else 1024
        s["q"] = _randn(g, b, tq, hq, d, dtype=dt)
        s["k"], s["v"] = (_randn(g, b, room, h, d, dtype=dt)[:, :tk] for _ in range(2))
        s["g"] = F.logsigmoid(GATE_BIAS + _randn(g, b, room, h))[:, :tk] if gated else None
        if kind != "prefill":
            s["state"], s["sok"] = _state(g, b, h, d, dt)
        if kind == "recurrent":
            cache = prb.RetentionCache(b, h, d, dtype=dt, recurrent=True)
            cache.update_state(s.pop("state"), s.pop("sok"))
            s["cache"] = cache
    return s


def run(s):
    c = s["case"]
    kind = c["kind"]
    if kind == "train":
        leaves = s["leaves"]
        out = prb.power_retention(*leaves, deg=2, chunk_size=c["chunk"] or None)
        return out.detach(), torch.autograd.grad(out, leaves, s["dO"])
    if kind == "glue":
        out = prb.prepare_qkvg(s["x"], s["sin"], s["cos"], c["h"], c["h"] * c["ratio"], c["d"], gated=c["gated"],
                               half_split=c["half_split"])
        out = out if c["gated"] else out[:3]
        return [x.detach() for x in out], torch.autograd.grad(out, s["x"], s["up"])
    if kind == "recurrent":
        y = s["cache"].decode(s["q"], s["k"], s["v"], s["g"])
        return y, s["cache"].state, s["cache"].sum_of_keys
    with torch.no_grad():
        if kind == "prefill":
            return prb.power_retention_inference(s["q"], s["k"], s["v"], s["g"], switch_over_seq_len=min(c["t"], 1024))
        if kind == "resume":
            return prb.power_retention(s["q"], s["k"], s["v"], s["g"], initial_state=(s["state"], s["sok"]),
                                       return_final_state=True, deg=2, chunk_size=c["chunk"])
        y, _, _ = prb.power_retention_inference(s["q"], s["k"], s["v"], s["g"], s["state"], s["sok"],
                                                switch_over_seq_len=1024)
        return y


def work(case):
    kind, b, h, d = case["kind"], case["b"], case["h"], case["d"]
    hq, D = h * case["ratio"], d * (d + 1) // 2
    gated = case.get("gated", True)
    tq, tk = case.get("t", case.get("tq", 1)), case.get("t", case.get("tk", 1))
    q, kv, gates, pair = 2 * b * tq * hq * d, 2 * b * tk * h * d, 4 * b * tk * h * gated, b * h * D * (2 * d + 4)
    if kind == "glue":  # projection <-> Q, K, V, gates each way, the sine and cosine tables, the gate column again
        return {"bytes": 2 * (2 * (q + 2 * kv) + 2 * b * tk * h * gated + gates) + 8 * tk * d, "flops": 0}
    if kind == "train":
        # within chunks of 1024 tokens by attention, between them through the expanded state; the whole sequence by
        # attention where it is no longer than two chunks
        chunk = tq if tq <= 2048 else 1024
        att = b * hq * tq * chunk * d
        exp = 2 * b * tq * D * d * (hq + h) * (tq > chunk)
        return {"bytes": 4 * q + 4 * kv + 2 * gates, "flops": 7 * att + 3 * exp}
    if kind in ("prefill", "resume"):
        chunk = min(tq, 1024)
        att = b * hq * tq * chunk * d
        read = kind == "resume" or tq > chunk
        exp = 2 * b * tq * D * d * (h + hq * read)
        return {"bytes": 2 * q + 2 * kv + gates + pair * (2 if kind == "resume" else 1), "flops": 2 * att + exp}
    if kind == "recurrent":
        return {"bytes": 2 * q + 2 * kv + gates + 2 * pair, "flops": 2 * b * D * d * (h + hq)}
    # every new token sees the cached tokens up to itself, and the state
    return {"bytes": 2 * q + 2 * kv + gates + pair, "flops": 2 * b * hq * tq * d * (D + 2 * tk - tq)}


def tolerance(case):
    # Results are 16-bit values, or sums of products of such.  In training a row's result is divided by the sum of its
    # weights (s q.k)^2, and fast gates leave a row few of them: where that sum happens to be tiny, the rounding of
    # a 16-bit operand shows as a large error of that one row (up to 0.8 of the root mean square between two
    # blockings of the same sequence), while the norm stays within the data type's.
    t = {"rel": 1e-2 if case["dtype"] == "bf16" else 5e-3}
    if case["kind"] == "train":
        t["max"] = 0.95
    return t
