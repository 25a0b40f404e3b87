"""The native host path (csrc/binding.cpp) under the tools that a caller may wrap around it."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


def _inputs(dev, b, t, h, hq, d=64, seed=0):
    g = torch.Generator(dev).manual_seed(seed)
    Q, K, V = (torch.randn(b, t, n, d, generator=g, device=dev).to(torch.bfloat16) for n in (hq, h, h))
    return [Q, K, V, F.logsigmoid(torch.randn(b, t, h, generator=g, device=dev))]


def _traced(fn, example, leaves):
    """(results, gradients) of the trace made from `example` and of `fn` itself, both on `leaves`."""
    out = []
    for f in (torch.jit.trace(fn, tuple(example), check_trace=False), fn):
        y = f(*leaves)
        y = list(y) if isinstance(y, (tuple, list)) else [y]
        out.append(y + list(torch.autograd.grad(sum((i + 1) * x.float().sum() for i, x in enumerate(y)), leaves)))
    return out


@pytest.mark.parametrize("t,d,chunk", [(256, 64, None), (256, 64, 64), (200, 64, 64), (96, 32, None)])
def test_a_trace_computes(cuda_device, t, d, chunk):
    """torch.jit.trace records the operator, not just the allocation of its result."""
    import retention_integration_b200 as prb

    leaves = [x.requires_grad_() for x in _inputs(cuda_device, 1, t, 2, 4, d, seed=1)]
    got, want = _traced(lambda *x: prb.power_retention(*x, chunk_size=chunk), _inputs(cuda_device, 1, t, 2, 4, d), leaves)
    for x, y in zip(got, want):
        # the traced path pads the sequence, which regroups no sum but those over whole zero tiles
        assert float((x.float() - y.float()).norm()) <= 1e-3 * float(y.float().norm())


@pytest.mark.parametrize("gated,half_split,extra", [(True, False, 0), (False, True, 0), (True, True, 6)])
def test_a_trace_of_the_glue_computes(cuda_device, gated, half_split, extra):
    import retention_integration_b200 as prb

    t, h, hq, d = 40, 2, 4, 64
    W = (hq + 2 * h) * d + (h if gated else 0) + extra
    g = torch.Generator(cuda_device).manual_seed(0)
    a, b = (torch.randn(2, t, W, generator=g, device=cuda_device).to(torch.bfloat16) for _ in range(2))
    sin, cos = prb.rotary_tables(t, d, cuda_device)
    fn = lambda x: tuple(y for y in prb.prepare_qkvg(x, sin, cos, h, hq, d, gated=gated, half_split=half_split)
                         if y is not None)
    got, want = _traced(fn, [a], [b.requires_grad_()])
    for x, y in zip(got, want):
        assert torch.equal(x, y)


@pytest.mark.parametrize("chunk", [None, 64])
def test_a_capture_leaves_other_streams_alone(cuda_device, chunk):
    """While one stream is being captured, forward and backward run on others, and the capture holds its own work alone.
    (More streams than the library keeps for overlapping, so that some share the captured caller's.)"""
    import retention_integration_b200 as prb

    def step(leaves, dO):
        return torch.autograd.grad(prb.power_retention(*leaves, chunk_size=chunk), leaves, dO)

    args = []
    for seed in (0, 1):
        leaves = [x.requires_grad_() for x in _inputs(cuda_device, 1, 256, 2, 4, seed=seed)]
        args.append((leaves, torch.randn_like(leaves[0])))
    want = [step(*a) for a in args]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(24)]
    for s in streams:  # memory for the calls below: the allocator need not ask the driver during the capture
        with torch.cuda.stream(s):
            step(*args[1])
    torch.cuda.synchronize()
    graph, others = torch.cuda.CUDAGraph(), []
    with torch.cuda.graph(graph, capture_error_mode="relaxed"):
        captured = [step(*args[0])]
        for s in streams:
            with torch.cuda.stream(s):
                others.append(step(*args[1]))
        captured.append(step(*args[0]))
    torch.cuda.synchronize()
    graph.replay()
    torch.cuda.synchronize()
    for got, ref in [(c, want[0]) for c in captured] + [(o, want[1]) for o in others]:
        for x, y in zip(got, ref):
            assert torch.equal(x, y)


def test_callers_on_many_streams_and_threads(cuda_device):
    """Backward passes enqueued from several threads on streams of their own, overlapping on the GPU."""
    import threading

    import retention_integration_b200 as prb

    cases = []
    for seed, (t, chunk) in enumerate([(256, None), (640, 128), (300, 128), (128, None)] * 3):
        leaves = [x.requires_grad_() for x in _inputs(cuda_device, 1, t, 2, 4, seed=seed)]
        cases.append((leaves, torch.randn_like(leaves[0]), chunk))

    def step(leaves, dO, chunk):
        return torch.autograd.grad(prb.power_retention(*leaves, chunk_size=chunk), leaves, dO)

    want = [step(*c) for c in cases]
    torch.cuda.synchronize()
    got = [None] * len(cases)

    def work(i):
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(20):
                got[i] = step(*cases[i])

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(cases))]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    torch.cuda.synchronize()
    for g, w in zip(got, want):
        for x, y in zip(g, w):
            assert torch.equal(x, y)


def _widened():
    """Saved 16-bit tensors come back in 32 bits, which the backward pass refuses before it launches anything."""
    return torch.autograd.graph.saved_tensors_hooks(lambda x: x, lambda x: x.float() if x.dtype == torch.bfloat16 else x)


@pytest.mark.parametrize("chunk", [None, 64])
def test_a_failed_backward_raises_the_packages_error(cuda_device, chunk):
    import retention_integration_b200 as prb

    leaves = [x.requires_grad_() for x in _inputs(cuda_device, 1, 256, 2, 4)]
    with _widened():
        out = prb.power_retention(*leaves, chunk_size=chunk)
    with pytest.raises(prb.PRError, match="float16"):
        out.sum().backward()
    with torch.autograd.detect_anomaly(check_nan=False):
        with _widened():
            out = prb.power_retention(*leaves, chunk_size=chunk)
        with pytest.raises(prb.PRError, match="float16"):
            out.sum().backward()


def test_a_failed_backward_of_the_glue_raises_the_packages_error(cuda_device):
    import retention_integration_b200 as prb

    x = torch.randn(1, 64, 4 * 64 + 8, device=cuda_device).to(torch.bfloat16).requires_grad_()
    sin, cos = prb.rotary_tables(64, 64, cuda_device)
    with _widened():
        Q, K, V, log_g = prb.prepare_qkvg(x, sin, cos, 1, 2, 64)
    with pytest.raises(prb.PRError, match="float16"):
        Q.sum().backward()


def _entry(name, dev):
    import retention_integration_b200 as prb

    Q, K, V, G = _inputs(dev, 1, 64, 1, 1)
    if name == "power_retention":
        return lambda: prb.power_retention(Q, K, V, G)
    if name == "prepare_qkvg":
        x = torch.zeros(1, 64, 200, device=dev, dtype=torch.bfloat16)
        sin, cos = prb.rotary_tables(64, 64, dev)
        return lambda: prb.prepare_qkvg(x, sin, cos, 1, 1, 64)
    one = [x[:, :1].contiguous() for x in (Q, K, V, G)]
    cache = prb.RetentionCache(1, 1, 64, recurrent=True)
    cache.decode(*one)
    if name == "recurrent":
        return lambda: cache.decode(*one)
    return lambda: prb.power_retention_inference(one[0], K, V, G, cache.state, cache.sum_of_keys)


@pytest.mark.parametrize("name", ["power_retention", "prepare_qkvg", "recurrent", "inference"])
def test_other_threads_run_while_a_launch_waits(cuda_device, name):
    """Behind half a second of GPU work the launch queue fills up, and one of the calls waits for room in it."""
    import threading
    import time

    call = _entry(name, cuda_device)
    with torch.no_grad():
        call()
        torch.cuda.synchronize()
        gaps, stop = [], threading.Event()

        def watch():
            last = time.perf_counter()
            while not stop.is_set():
                time.sleep(1e-3)
                last, before = time.perf_counter(), last
                gaps.append(last - before)

        watcher = threading.Thread(target=watch)
        watcher.start()
        torch.cuda._sleep(1_000_000_000)  # clocks
        longest = 0.0
        for _ in range(3000):
            t0 = time.perf_counter()
            call()
            longest = max(longest, time.perf_counter() - t0)
        stop.set()
        watcher.join()
        torch.cuda.synchronize()
    if longest < 0.1:
        pytest.skip("no launch had to wait")
    assert max(gaps) < longest / 2


def test_results_keep_the_queries_class(cuda_device):
    import retention_integration_b200 as prb

    class Marked(torch.Tensor):
        pass

    Q, K, V, G = _inputs(cuda_device, 1, 64, 2, 2)
    q = Q.as_subclass(Marked)
    assert type(prb.power_retention(q, K, V, G)) is Marked
    y, (state, sok) = prb.power_retention(q, K, V, G, return_final_state=True)
    assert type(y) is Marked and type(state) is torch.Tensor
    y, s, n = prb.power_retention_inference(q, K, V, G, state, sok, switch_over_seq_len=None)
    assert type(y) is Marked and s is state and n is sok
    leaf = torch.nn.Parameter(Q)
    out = prb.power_retention(leaf, K, V, G)
    assert type(out) is torch.Tensor
    want, = torch.autograd.grad(out.float().sum(), leaf)
    marked = Q.clone().as_subclass(Marked).requires_grad_()
    got, = torch.autograd.grad(prb.power_retention(marked, K, V, G).float().sum(), marked)
    assert torch.equal(got.as_subclass(torch.Tensor), want)
