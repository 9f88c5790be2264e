"""What the calls that bypass ctypes accept."""
import ctypes
import threading
import time

import pytest
import torch

from tnn_b200.ops import _lib


def test_call_takes_what_ctypes_takes():
    lib = ctypes.CDLL(_lib.lib_path())
    fn = lib.tnnb_gemm_bf16
    vp, i, ll = ctypes.c_void_p, ctypes.c_int, ctypes.c_longlong
    args = [vp, vp, vp, i, i, i, i, i, ll, ll, ll, vp, vp, vp, ll, vp, ll, i, i, i, vp, vp]
    t = torch.zeros(8, 8, dtype=torch.bfloat16)
    p = t.data_ptr()
    call = lambda f, a, **kw: f(a, a, a, kw.get("M", 0), 8, 8, 0, 0, 8, 8, 8, None, None, None, 0, None, 0, False, 0, 0, p, 0)
    fn.argtypes, fn.restype = args, i
    by_ctypes = call(fn, p)
    _lib.declare(lib, "tnnb_gemm_bf16", args)
    native = lib.tnnb_gemm_bf16
    assert native is not fn
    # a product without rows and one with a misaligned pitch are refused before anything is launched
    assert call(native, t) == call(native, p) == call(native, ctypes.c_void_p(p)) == by_ctypes == -2
    _lib.declare(lib, "tnnb_gemm_bf16", args)  # again: nothing changes
    assert lib.tnnb_gemm_bf16 is native
    with pytest.raises((TypeError, ctypes.ArgumentError)):
        call(native, 1.5)
    with pytest.raises((TypeError, ctypes.ArgumentError)):
        native(t)
    with pytest.raises(RuntimeError):  # a tensor without memory of its own
        call(native, torch.sparse_coo_tensor(torch.zeros(2, 1, dtype=torch.long), torch.ones(1), (8, 8)))


def test_other_signatures_go_through_ctypes():
    """A signature that is not compiled in: tensors, None and integers arrive as they would in ctypes."""
    class Lib:
        pass

    seen, lib, vp, i, f = {}, Lib(), ctypes.c_void_p, ctypes.c_int, ctypes.c_float
    lib.entry = ctypes.CFUNCTYPE(i, vp, i, vp, f)(lambda a, n, b, x: seen.update(a=a, n=n, b=b, x=x) or 7)
    _lib.declare(lib, "entry", [vp, i, vp, f])
    t = torch.zeros(3)
    assert lib.entry(t, 5, None, 0.5) == 7 and seen == {"a": t.data_ptr(), "n": 5, "b": None, "x": 0.5}
    assert lib.entry(ctypes.c_void_p(64), 5, t, 2) == 7 and seen == {"a": 64, "n": 5, "b": t.data_ptr(), "x": 2.0}
    with pytest.raises((TypeError, ctypes.ArgumentError)):
        lib.entry(object(), 5, None, 0.5)


def test_empty_is_torch_empty():
    like = torch.zeros(2, 3, dtype=torch.bfloat16, requires_grad=True)
    a, b = _lib.empty(like, 4, 5), _lib.empty(like, torch.float32, 7)
    assert (a.shape, a.dtype, a.device, a.requires_grad, a.is_contiguous()) == ((4, 5), torch.bfloat16, like.device, False, True)
    assert (b.shape, b.dtype) == ((7,), torch.float32)
    assert _lib.empty(like).shape == ()
    with pytest.raises(TypeError):
        _lib.empty([1, 2], 3)
    with pytest.raises(RuntimeError):
        _lib.empty(like, -1)


def test_an_allocation_leaves_the_interpreter_to_other_threads():
    """With memory filled on allocation, 2 GB take a while: time in which another thread runs."""
    like, longest, stop = torch.zeros(1, dtype=torch.uint8), [0.0], threading.Event()

    def watch():  # the longest time without a turn
        last = time.perf_counter()
        while not stop.is_set():
            now = time.perf_counter()
            longest[0] = max(longest[0], now - last)
            last = now

    before = torch.are_deterministic_algorithms_enabled()
    thread = threading.Thread(target=watch)
    torch.use_deterministic_algorithms(True)
    try:
        thread.start()
        shares = []
        for _ in range(3):
            time.sleep(0.02)
            longest[0] = 0.0
            start = time.perf_counter()
            _lib.empty(like, 2 << 30)
            shares.append(longest[0] / (time.perf_counter() - start))
    finally:
        stop.set()
        thread.join()
        torch.use_deterministic_algorithms(before)
    assert min(shares) < 0.5, shares
