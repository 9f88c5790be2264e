"""Epilogues of the tcgen05 GEMM: in whole lines, with the tensor beside the output fetched by the copy unit, and row by row.
Every fused operation, tile width and placement of the tensors against fp64, with the surroundings of the output left alone."""
import pytest
import torch

from tnn_b200.ops import _lib
from tnn_b200.ops.gemm import gemm

pytestmark = pytest.mark.gpu

# (M, N, K, force_bn): one partial tile; ragged edges; more tiles than CTAs, so that tiles follow one another in a CTA
SHAPES = [(1, 8, 8, 0), (33, 72, 40, 0), (129, 130, 72, 0), (300, 200, 136, 1024 + 256), (4200, 1100, 72, 64),
          (20000, 56, 600, 0), (4200, 1100, 72, 128), (4200, 1100, 72, 256),
          (4200, 1100, 72, 1024 + 256), (10000, 776, 40, 1024 + 384), (4200, 1100, 200, 1024 + 384)]
KINDS = ["plain", "bias", "gelu", "gelu_z", "dgelu", "resid", "relu_resid", "inplace", "f32", "atomic", "add", "add_f32",
         "relu_add_resid"]


def _placed(M, N, dtype, place, fill):
    """A [M, N] view inside a larger buffer: aligned with a padded pitch, an odd pitch, or off a 16-byte boundary."""
    pad = {"aligned": (N + 7) // 8 * 8 + 16, "odd": (N + 7) // 8 * 8 + 3, "shifted": (N + 7) // 8 * 8 + 16}[place]
    buf = torch.full((M + 2, pad), 7.0, dtype=dtype, device="cuda")
    shift = 1 if place == "shifted" else 8
    view = buf[1:M + 1, shift:shift + N] if place != "odd" else buf[1:M + 1, :N]
    view.copy_(fill)
    return buf, view


def _gelu(x):
    return torch.nn.functional.gelu(x, approximate="tanh")


CASES = [(*s, p) for s in SHAPES for p in ("aligned", "odd", "shifted")] + [(40, 24, 16, 0, "shifted")]
# K ranges in clusters of 2 and 4: a short last range, ragged edges, several tiles; and the sizes where the rule takes them
CASES += [(33, 72, 136, 2048 + 2, "aligned"), (129, 130, 584, 2048 + 4, "aligned"), (300, 264, 1000, 2048 + 4, "aligned"),
          (69, 768, 1800, 0, "aligned"), (7, 200, 1288, 0, "aligned")]


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("M,N,K,bn,place", CASES)
def test_epilogue(M, N, K, bn, place, kind):
    if bn > 2048 and kind in ("atomic", "relu_add_resid"):
        pytest.skip("added products are split another way; with a tensor beside an output that is read, too, none are split")
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda").to(torch.bfloat16)
    a, b = rnd(M, K), rnd(N, K) * 0.25
    bias, aux = rnd(N), rnd(M, N)
    out_dtype = torch.float32 if kind in ("f32", "atomic", "add_f32") else torch.bfloat16
    start = torch.randn(M, N, generator=g, device="cuda").to(out_dtype)
    buf, out = _placed(M, N, out_dtype, place, start)
    abuf, aview = _placed(M, N, torch.bfloat16, place, aux)
    acc = a.double() @ b.double().t()
    mag = a.double().abs() @ b.double().abs().t()
    x = acc + bias.double()
    grow = torch.ones_like(x)  # what the fused operation does to an error of its argument, at most
    kw, ref = {}, None
    if kind == "plain":
        ref = acc
    elif kind == "bias":
        kw, ref = {"bias": bias}, x
    elif kind in ("gelu", "gelu_z"):
        kw, ref = {"bias": bias, "gelu": True}, _gelu(x)
        grow = 1.2 * grow
        if kind == "gelu_z":
            kw["save_preact"] = aview
    elif kind == "dgelu":
        z = aux.double().requires_grad_(True)
        slope, = torch.autograd.grad(_gelu(z).sum(), z)
        kw, ref = {"dgelu_of": aview}, acc * slope
        grow = 1.2 * grow
    elif kind in ("resid", "relu_resid", "inplace"):
        res = aux if kind != "inplace" else start
        kw = {"bias": bias, "residual": aview if kind != "inplace" else out, "relu": kind == "relu_resid"}
        ref = (x.clamp_min(0) if kind == "relu_resid" else x) + res.double()
    elif kind == "f32":
        kw, ref = {"bias": bias}, x
    elif kind in ("add", "add_f32"):
        kw, ref = {"accumulate": True}, start.double() + acc
    elif kind == "relu_add_resid":  # the output is added to behind a residual of its own
        kw, ref = {"relu": True, "residual": aview, "accumulate": True}, acc.clamp_min(0) + aux.double() + start.double()
    else:
        kw, ref = {"atomic": True}, start.double() + acc
    gemm(a, b, out=out, force_bn=bn, **kw)
    _lib.check_status()
    # fp32 accumulation (truncating): 2^-20 of the absolute products; tanh.approx: 2^-10.9 of |x| / 2 (GELU) or of
    # |acc| (1 + z^2) (its derivative); one rounding of the result
    bound = grow * mag * 2.0 ** -20 + ref.abs() * (2.0 ** -8 if out_dtype == torch.bfloat16 else 2.0 ** -22) + 1e-6
    if kind in ("gelu", "gelu_z"):
        bound = bound + x.abs() * 2.0 ** -11
    if kind == "dgelu":
        bound = bound + acc.abs() * (1 + aux.double() ** 2) * 2.0 ** -10
    err = (out.double() - ref).abs()
    assert bool((err <= bound).all()), float((err / bound).max())
    if kind == "gelu_z":
        zerr = (aview.double() - x).abs()
        assert bool((zerr <= x.abs() * 2.0 ** -8 + mag * 2.0 ** -20 + 1e-6).all())
    for whole, view in ((buf, out), (abuf, aview)):  # nothing around the views was written
        view.fill_(7.0)
        assert bool((whole == 7.0).all())


@pytest.mark.parametrize("kind", ["gelu", "gelu_f32", "dgelu", "resid"])
def test_rounding_does_not_depend_on_the_placement(kind):
    """The same product into a tensor that takes whole lines and into one that does not: two epilogues, one result, to the
    last bit. (8 M values: a difference in the last place of fp32 reaches the bf16 result once in 65536.)"""
    g = torch.Generator(device="cuda").manual_seed(11)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda").to(torch.bfloat16)
    M, N = 4096, 2048
    a, b, aux = rnd(M, 64), rnd(N, 64) * 0.25, rnd(M, N)
    dtype = torch.float32 if kind == "gelu_f32" else torch.bfloat16
    kw = {"gelu": {"gelu": True}, "gelu_f32": {"gelu": True}, "dgelu": {"dgelu_of": aux}, "resid": {"residual": aux}}[kind]
    lines, rows = (_placed(M, N, dtype, place, 0.0 * aux.to(dtype))[1] for place in ("aligned", "odd"))
    gemm(a, b, out=lines, **kw)
    gemm(a, b, out=rows, **kw)
    _lib.check_status()
    assert torch.equal(lines, rows)
