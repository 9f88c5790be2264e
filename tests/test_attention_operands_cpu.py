"""Attention calls whose tensors do not have the stated sizes are refused before anything is launched."""
import pytest
import torch

from tnn_b200.ops import functional as F
from tnn_b200.ops import raw

BF = torch.bfloat16


def _operands(B, S, H, D):
    return {"qkv": torch.zeros(B * S, 3 * H * D, dtype=BF), "out": torch.zeros(B * S, H * D, dtype=BF),
            "dout": torch.zeros(B * S, H * D, dtype=BF), "lse": torch.zeros(B, H, S)}


@pytest.mark.parametrize("width", [290, 287, 2, 0])
def test_packed_width(width):
    with pytest.raises(ValueError):
        F.causal_self_attention(torch.zeros(2, 5, width, dtype=BF), 12)


@pytest.mark.parametrize("shape", [(10, 290), (9, 288), (10, 286), (11, 288)])
def test_packed_projection_of_another_size(shape):
    with pytest.raises(ValueError, match="qkv"):
        raw._attn_fwd_generic(torch.zeros(*shape, dtype=BF), 2, 5, 12, 8, True, 1.0)


@pytest.mark.parametrize("name,change", [("qkv", lambda t: t[1:]), ("out", lambda t: t[:, 1:]), ("dout", lambda t: t[1:]), ("lse", lambda t: t[1:]),
                                         ("dout", lambda t: t.float()), ("lse", lambda t: t.to(BF)), ("out", lambda t: t.to("meta"))])
@pytest.mark.parametrize("D", [8, 64])
def test_backward_operands(name, change, D):
    ops = _operands(2, 5, 3, D)
    raw._attn_operands(2, 5, 3, D, **ops)
    ops[name] = change(ops[name])
    with pytest.raises(ValueError, match=name):
        raw._attn_operands(2, 5, 3, D, **ops)
    if D != 64:
        with pytest.raises(ValueError, match=name):
            raw._attn_bwd_generic(ops["qkv"], ops["out"], ops["dout"], ops["lse"], 2, 5, 3, D, True, 1.0)


def test_flash_kernels_take_the_first_rows_of_a_longer_buffer():
    ops = _operands(2, 6, 3, 64)
    raw._attn_operands(2, 5, 3, 64, **ops)


def test_backward_of_an_empty_batch():
    ops = _operands(0, 5, 3, 8)
    d = raw._attn_bwd_generic(ops["qkv"], ops["out"], ops["dout"], ops["lse"], 0, 5, 3, 8, True, 1.0)
    assert d.shape == (0, 72) and d.dtype == BF
