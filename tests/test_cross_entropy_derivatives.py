"""What autograd can do with the gradient that enters the cross-entropy: differentiate it, batch it, carry a tangent."""
import pytest
import torch
from torch.autograd import forward_ad

from tnn_b200.ops import functional as F
from tnn_b200.ops import raw


def _loss(device, monkeypatch):
    torch.manual_seed(0)
    dtype = torch.bfloat16 if device == "cuda" else torch.float32
    logits = torch.randn(4, 24, device=device).to(dtype).requires_grad_(True)
    labels = torch.randint(0, 24, (4,), device=device)
    if device == "cpu":  # in the place of the launch: the numbers alone, as a kernel sees them
        monkeypatch.setattr(raw, "scale_by", lambda x, s: (x.float() * float(s)).to(x.dtype))
    loss = F.cross_entropy(logits, labels)
    one, = torch.autograd.grad(loss, logits, torch.ones((), device=device), retain_graph=True)
    return loss, logits, one.float()


DEVICES = ["cpu", pytest.param("cuda", marks=pytest.mark.gpu)]


@pytest.mark.parametrize("device", DEVICES)
def test_learned_loss_weight(device, monkeypatch):
    loss, logits, one = _loss(device, monkeypatch)
    w = torch.tensor(2.0, device=device, requires_grad=True)
    g, = torch.autograd.grad(loss, logits, w, create_graph=True)
    dw, = torch.autograd.grad((g.float() * one).sum(), w)
    assert torch.allclose(dw, one.square().sum(), rtol=2.0 ** -7)  # bf16 products


@pytest.mark.parametrize("device", DEVICES)
def test_batched_gradients(device, monkeypatch):
    loss, logits, one = _loss(device, monkeypatch)
    v = torch.tensor([1.0, 2.0, -4.0], device=device)  # powers of two: the products are exact
    g, = torch.autograd.grad(loss, logits, v, is_grads_batched=True)
    assert torch.equal(g.float(), v[:, None, None] * one)


@pytest.mark.parametrize("device", DEVICES)
def test_tangent_of_the_incoming_gradient(device, monkeypatch):
    loss, logits, one = _loss(device, monkeypatch)
    with forward_ad.dual_level():
        d = forward_ad.make_dual(torch.tensor(2.0, device=device), torch.tensor(4.0, device=device))
        g, = torch.autograd.grad(loss, logits, d)
        value, tangent = forward_ad.unpack_dual(g)
    assert torch.equal(value.float(), 2 * one)
    assert tangent is not None and torch.equal(tangent.float(), 4 * one)


@pytest.mark.gpu
def test_plain_gradient_takes_the_launch(monkeypatch):
    loss, logits, one = _loss("cuda", monkeypatch)
    calls = []
    launch = raw.scale_by
    monkeypatch.setattr(raw, "scale_by", lambda x, s: calls.append(1) or launch(x, s))
    g, = torch.autograd.grad(loss, logits, torch.tensor(0.5, device="cuda"))
    assert calls and torch.equal(g.float(), 0.5 * one)
