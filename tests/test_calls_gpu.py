"""The native route of ``gemm`` against the general one, over everything it accepts and what it leaves to the general one."""
import pytest
import torch

from tnn_b200.ops import _lib
from tnn_b200.ops.gemm import LAUNCHES, gemm

pytestmark = pytest.mark.gpu


def _both(monkeypatch, *args, **kw):
    """Result of a call with and without the native route (or the exception's type), each on fresh copies of its outputs."""
    res = []
    for native in (True, False):
        k = {n: (t.clone(memory_format=torch.preserve_format) if n in ("out", "save_preact") and t is not None else t) for n, t in kw.items()}
        with monkeypatch.context() as m:
            if not native:
                m.setattr(_lib, "gemm", lambda *a: None)
            before = LAUNCHES["count"]
            try:
                r = gemm(*args, **k)
                assert LAUNCHES["count"] == before + 1 and (k.get("out") is None or r is k["out"])
                res.append((r, k.get("save_preact")))
            except (AssertionError, RuntimeError, ValueError) as e:
                res.append(type(e))
    _lib.check_status()
    return res


CASES = {
    "plain": {}, "f32": {"out_dtype": torch.float32}, "bias": {"bias": "n"}, "gelu": {"bias": "n", "gelu": True},
    "gelu_z": {"bias": "n", "gelu": True, "save_preact": "mn"}, "z_without_gelu": {"save_preact": "mn"}, "dgelu": {"dgelu_of": "mn"},
    "relu_resid": {"relu": True, "residual": "mn"}, "out": {"out": "mn"}, "out_f32": {"out": "mnf"}, "atomic": {"out": "mnf", "atomic": True},
    "accumulate": {"out": "mn", "accumulate": True}, "accumulate_f32": {"out": "mnf", "accumulate": True},
    # refused, or copied first: the general route's business
    "atomic_bf16": {"out": "mn", "atomic": True}, "split": {"split_k": 2}, "short_bias": {"bias": "short"}, "bias_f32": {"bias": "nf"},
    "wrong_out": {"out": "nm"}, "out_of_columns": {"out": "mn_t"},
}


@pytest.mark.parametrize("place", ["packed", "pitch", "odd", "columns"])
@pytest.mark.parametrize("a_t,b_t", [(False, False), (True, 1)])
@pytest.mark.parametrize("case", CASES)
def test_native_and_general_route(case, a_t, b_t, place, monkeypatch):
    M, N, K = 40, 24, 56
    g = torch.Generator(device="cuda").manual_seed(0)

    def rnd(*s, dtype=torch.bfloat16):
        return torch.randn(*s, generator=g, device="cuda").to(dtype)

    def operand(r, c):
        if place == "packed":
            return rnd(r, c)
        if place == "pitch":
            return rnd(r, c + 8)[:, :c]
        return rnd(r, c + 3)[:, :c] if place == "odd" else rnd(c, r).t()

    kinds = {"n": lambda: rnd(N), "nf": lambda: rnd(N, dtype=torch.float32), "short": lambda: rnd(N - 1), "mn": lambda: rnd(M, N),
             "mnf": lambda: rnd(M, N, dtype=torch.float32), "nm": lambda: rnd(N, M), "mn_t": lambda: rnd(N, M).t()}
    a, b = operand(*((K, M) if a_t else (M, K))), operand(*((K, N) if b_t else (N, K)))
    kw = {k: kinds[v]() if isinstance(v, str) else v for k, v in CASES[case].items()}
    x, y = _both(monkeypatch, a, b, a_t=a_t, b_t=b_t, **kw)
    if isinstance(x, type) or isinstance(y, type):
        assert x == y
        return
    assert x[0].dtype == y[0].dtype and x[0].stride() == y[0].stride() and torch.equal(x[0], y[0])
    if case == "gelu_z":
        assert torch.equal(x[1], y[1])


def test_wrong_shapes_are_refused(monkeypatch):
    a, b = torch.zeros(8, 16, device="cuda").bfloat16(), torch.zeros(8, 24, device="cuda").bfloat16()
    for args in ((a, b), (a, b.float()), (a.float(), a), (a[None], a[None]), (a[:0], a)):
        x, y = _both(monkeypatch, *args)
        assert isinstance(x, type) and x == y or isinstance(x, type) and isinstance(y, type)
