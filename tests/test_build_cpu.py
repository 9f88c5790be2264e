"""The native build: outputs appear whole, one process builds at a time, and what stays on the CPU needs no extension."""
import os
import subprocess
import sys
import threading

import pytest

from tnn_b200 import _build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(_build.__file__)))


def test_an_output_appears_whole_or_not_at_all(tmp_path, monkeypatch):
    out = str(tmp_path / "lib.so")

    def half_then_all(cmd, verbose):
        path = cmd[cmd.index("-o") + 1]
        assert path != out and os.path.dirname(path) == str(tmp_path)
        with open(path, "w") as f:
            f.write("half")
            f.flush()
            assert not os.path.exists(out)
            f.write(" and half")

    monkeypatch.setattr(_build, "_run", half_then_all)
    _build._link(["cc", "-o", out, "x.o"], out, False)
    assert open(out).read() == "half and half" and os.listdir(tmp_path) == ["lib.so"]

    def fails(cmd, verbose):
        open(cmd[cmd.index("-o") + 1], "w").close()
        raise RuntimeError("no")

    monkeypatch.setattr(_build, "_run", fails)
    with pytest.raises(RuntimeError):
        _build._link(["cc", "-o", out, "x.o"], out, False)
    assert open(out).read() == "half and half" and os.listdir(tmp_path) == ["lib.so"]


def test_one_build_at_a_time(tmp_path, monkeypatch):
    monkeypatch.setattr(_build, "LIB", str(tmp_path))
    inside, most, gate = [0], [0], threading.Barrier(3)

    @_build._serial
    def build():
        inside[0] += 1
        most[0] = max(most[0], inside[0])
        threading.Event().wait(0.05)
        inside[0] -= 1

    def start():
        gate.wait()
        build()

    threads = [threading.Thread(target=start) for _ in range(3)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert most[0] == 1


def test_the_extension_belongs_to_one_torch(monkeypatch):
    import torch
    here = _build.calls_path()
    monkeypatch.setattr(torch, "__version__", "99.0")
    assert _build.calls_path() != here


def test_the_cpu_needs_no_extension():
    code = """
from tnn_b200 import _build
def gone(*a, **k): raise RuntimeError("the extension was asked for")
_build.calls_path = _build.build_calls = gone
import torch
from tnn_b200.models import zoo
from tnn_b200.ops import functional as F
g = zoo.gpt2(16, 2, 1, "gpt", seq_len=4, vocab=8).compile(device="cpu", seed=0)
y = g.forward({"input": torch.zeros(1, 4, dtype=torch.long)})["output"]
g.backward({"output": torch.ones_like(y)})
F.linear(torch.ones(2, 4, requires_grad=True), torch.ones(3, 4, requires_grad=True)).sum().backward()
print("fine")
"""
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True)
    assert r.returncode == 0 and "fine" in r.stdout, r.stderr
