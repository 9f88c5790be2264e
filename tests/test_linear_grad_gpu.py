"""Weight gradients of ``functional.linear`` on both sides of the row count that decides how they are summed up."""
import pytest
import torch

from tnn_b200.ops import _lib, functional as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 127, 2048, 2049])
@pytest.mark.parametrize("K,N", [(320, 203), (64, 8), (72, 960)])
def test_weight_gradient(rows, K, N):
    g = torch.Generator(device="cuda").manual_seed(rows + K)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()
    x, w, dy = rnd(rows, K), rnd(N, K).requires_grad_(True), rnd(rows, N)
    F.linear(x, w).backward(dy)
    _lib.check_status()
    ref, mag = dy.double().t() @ x.double(), dy.double().abs().t() @ x.double().abs()
    assert w.grad.dtype == torch.bfloat16
    # fp32 sums (the tensor core truncates), one rounding to bf16
    assert bool(((w.grad.double() - ref).abs() <= 2.0 ** -19 * mag + 2.0 ** -8 * ref.abs() + 1e-6).all())


@pytest.mark.parametrize("rows,K,N,one", [(1024, 64, 64, True), (1025, 64, 64, False), (1500, 1024, 1024, True), (2049, 1024, 1024, False)])
def test_captured_weight_gradient(rows, K, N, one):
    """In a graph one walk over the rows is taken for few rows or many tiles only; both forms replay on new values."""
    rnd = lambda *s: torch.randn(*s, device="cuda").bfloat16()
    x, w, dy = rnd(rows, K), rnd(N, K).requires_grad_(True), rnd(rows, N)
    grad = lambda: torch.autograd.grad(F.linear(x, w), w, dy)[0]
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        grad()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            assert F._in_one_launch(rows, N, K) == one
            dw = grad()
    torch.cuda.current_stream().wait_stream(side)
    assert F._in_one_launch(rows, N, K) == (rows <= 2048)
    for _ in range(2):
        x.copy_(rnd(rows, K))
        graph.replay()
        ref, mag = dy.double().t() @ x.double(), dy.double().abs().t() @ x.double().abs()
        assert bool(((dw.double() - ref).abs() <= 2.0 ** -19 * mag + 2.0 ** -8 * ref.abs() + 1e-6).all())
    _lib.check_status()
