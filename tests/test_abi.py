"""The C-ABI library builds, loads, and exports every symbol its header declares.
No compute call is made here (no GPU needed)."""
import ctypes
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _declared_symbols():
    text = open(os.path.join(ROOT, "include", "pr_b200.h")).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(pr_[a-z0-9_]+)\s*\(", text)))


def test_library_exports_every_declared_symbol():
    from retention_integration_b200 import build

    path = build.build()
    lib = ctypes.CDLL(path)
    names = _declared_symbols()
    assert len(names) >= 18
    for name in names:
        assert hasattr(lib, name), f"{name} is declared in include/pr_b200.h but not exported"
    assert lib.pr_abi_version() == 1


def test_bad_arguments_return_codes_not_crashes():
    from retention_integration_b200 import _lib

    lib = _lib.lib()
    # null pointers / unsupported head dim are refused before any CUDA call
    rc = lib.pr_chunk_state(0, 1, 128, 1, 1, 32, 128, None, None, None, None, None, 1, 0, None)
    assert rc == -1 and b"head dim" in lib.pr_last_error()
    rc = lib.pr_discumsum_fwd(0, 1, 4, 4, 1, ctypes.c_longlong(7), None, None, None, None, None, 0, None)
    assert rc == -1
    rc = lib.pr_selftest_umma(9, 0, 64, 64, None, None, None, 0, None)
    assert rc == -1 and b"variant" in lib.pr_last_error()


def test_pointers_that_a_kernel_would_fault_on_are_refused():
    """Addresses only: every one of these calls returns before it touches the device."""
    from retention_integration_b200 import _lib

    lib = _lib.lib()
    P = lambda a: ctypes.c_void_p(a)
    ok, off = P(1 << 20), P((1 << 20) + 16)  # 16 bytes short of the boundary that 32-byte stores want
    f = ctypes.c_float(1.0)
    rc = lib.pr_chunk_state(0, 1, 128, 1, 1, 64, 128, ok, ok, ok, off, None, 1, 0, None)
    assert rc == -1 and b"misaligned" in lib.pr_last_error()
    rc = lib.pr_expand_grad(0, 1, 128, 1, 1, 64, 128, ok, ok, ok, ok, ok, None, None, ok, 1, f, f, 0, 0, off, ok, 0, None)
    assert rc == -1 and b"misaligned" in lib.pr_last_error()

    class Problem(ctypes.Structure):
        _fields_ = [(n, ctypes.c_int) for n in ("dtype", "b", "t", "h", "hq", "d", "c")] + [("scale", ctypes.c_float)]

    prob = Problem(0, 1, 128, 1, 1, 64, 128, 1.0)
    for saved, scratch in ((off, ok), (ok, off)):
        rc = lib.pr_retention_fwd(ctypes.byref(prob), ok, ok, ok, None, None, None, ok, saved, scratch, None, None, 0, None)
        assert rc == -1 and b"32-byte" in lib.pr_last_error()
    # no keys, and a first chunk that does not read the state either
    rc = lib.pr_chunk_out(0, 1, 2, 128, 128, 1, 1, 64, ok, None, None, None, ok, ok, ok, 1, 0, 1, f, 2, ok, None, 0, None)
    assert rc == -1 and b"neither" in lib.pr_last_error()


def test_missing_library_fails_loudly(monkeypatch, tmp_path):
    from retention_integration_b200 import _lib

    monkeypatch.setattr(_lib, "_lib", None)
    monkeypatch.setattr(_lib, "LIB_PATH", str(tmp_path / "nope.so"))
    try:
        _lib.lib()
    except _lib.PRError as e:
        assert "no fallback" in str(e)
    else:
        raise AssertionError("a missing library must raise")


def test_cpu_tensors_are_rejected():
    import torch

    import retention_integration_b200 as prb

    q = torch.zeros(1, 128, 1, 64, dtype=torch.bfloat16)
    try:
        prb.power_retention(q, q, q, None, chunk_size=None)
    except prb.PRError as e:
        assert "CUDA" in str(e)
    else:
        raise AssertionError("CPU tensors must be rejected: there is no CPU path")
