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
