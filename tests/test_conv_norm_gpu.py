"""A convolution and the batch norm behind it in one kernel (inference): every route against fp64, and the graph executor's
use of it against the layers one by one."""
import pytest
import torch

from tnn_b200.models import zoo
from tnn_b200.nn.graph import infer_shapes
from tnn_b200.ops import _lib, conv, raw

pytestmark = pytest.mark.gpu

# (n, h, c, o, k, stride, pad): 1 x 1; implicit with one tile and with many (K ranges of clusters or not); input window with
# halo; patch matrix; strided; channel counts past one column block
GEOMETRIES = [(2, 7, 64, 256, 1, 1, 0), (7, 14, 256, 1024, 1, 1, 0), (1, 8, 512, 512, 3, 1, 1), (1, 4, 256, 192, 3, 1, 1),
              (3, 9, 128, 320, 3, 2, 1), (40, 28, 128, 256, 3, 1, 1), (2, 20, 64, 64, 3, 1, 1), (3, 17, 3, 16, 7, 2, 3),
              (2, 6, 24, 40, 3, 1, 1)]


@pytest.mark.parametrize("n,h,c,o,k,s,p", GEOMETRIES)
@pytest.mark.parametrize("relu,resid,post", [(False, False, False), (True, False, False), (True, True, False), (True, True, True)])
@pytest.mark.parametrize("affine", [True, False])
def test_conv_norm(n, h, c, o, k, s, p, relu, resid, post, affine):
    g = torch.Generator(device="cuda").manual_seed(n * h + c + o)
    rnd = lambda *shape: torch.randn(*shape, generator=g, device="cuda")
    x, w = rnd(n, h, h, c).bfloat16(), (rnd(o, k, k, c) * (k * k * c) ** -0.5).bfloat16()
    bias = rnd(o).bfloat16() if affine else None
    gamma, beta = ((1 + 0.1 * rnd(o)).bfloat16(), rnd(o).bfloat16()) if affine else (None, None)
    mean, var = 0.1 * rnd(o), 0.5 + rnd(o).abs()
    oh = (h + 2 * p - k) // s + 1
    res = rnd(n, oh, oh, o).bfloat16() if resid else None
    y = conv.conv2d_norm_infer(x, w, bias, (s, s), (p, p), gamma, beta, mean, var, 1e-5, relu, resid=res, post_add=post)
    _lib.check_status()
    xd, wd = x.double().permute(0, 3, 1, 2), w.double().permute(0, 3, 1, 2)
    acc = torch.nn.functional.conv2d(xd, wd, stride=s, padding=p).permute(0, 2, 3, 1)
    mag = torch.nn.functional.conv2d(xd.abs(), wd.abs(), stride=s, padding=p).permute(0, 2, 3, 1)
    b = bias.double() if affine else 0.0
    scale = (var.double() + 1e-5).rsqrt() * (gamma.double() if affine else 1.0)
    pre = (acc + b - mean.double()) * scale + (beta.double() if affine else 0.0)
    ref = pre
    if resid:
        ref = pre.clamp_min(0) + res.double() if post else (pre + res.double()).clamp_min(0)
    elif relu:
        ref = pre.clamp_min(0)
    # fp32 sums (truncating) scaled by the norm, one rounding of the normalised value and one of the sum
    bound = 2.0 ** -20 * (mag + 2) * (1 + scale.abs()) + 2.0 ** -8 * (pre.abs() + ref.abs()) + 1e-6
    assert bool(((y.double() - ref).abs() <= bound).all())


@pytest.mark.parametrize("c,o,k,p", [(64, 128, 1, 0), (128, 64, 3, 1), (64, 64, 3, 1), (3, 32, 3, 1)])
def test_residual_off_a_16_byte_boundary_is_refused(c, o, k, p):
    """As the norm kernels refuse it, in training and for layers run one by one."""
    x, w = torch.ones(2, 8, 8, c, device="cuda").bfloat16(), torch.ones(o, k, k, c, device="cuda").bfloat16()
    res = torch.zeros(2 * 64 * o + 8, device="cuda", dtype=torch.bfloat16)[1:1 + 2 * 64 * o].view(2, 8, 8, o)
    mean, var = torch.zeros(o, device="cuda"), torch.ones(o, device="cuda")
    with pytest.raises(RuntimeError):
        conv.conv2d_norm_infer(x, w, None, (1, 1), (p, p), None, None, mean, var, 1e-5, False, resid=res)
    with pytest.raises(RuntimeError):
        raw.batchnorm_infer(torch.ones_like(res), None, None, mean, var, 1e-5, False, resid=res)


@pytest.mark.parametrize("model,batch", [("cifar10_resnet9", 1), ("cifar10_resnet9", 33), ("cifar100_wrn16_8", 2),
                                         ("imagenet100_resnet50", 3)])
def test_evaluation_is_that_of_the_layers(model, batch):
    g = zoo.create(model).compile(device="cuda", seed=1)
    x = torch.randn((batch,) + zoo.INPUT_SHAPES[model], device="cuda").bfloat16()
    g.set_training(False)
    pairs, fused = g._norm_after, g.forward({"input": x})["output"].float()
    g._norm_after = {}
    plain = g.forward({"input": x})["output"].float()
    _lib.check_status()
    assert model == "cifar100_wrn16_8" or pairs
    # one rounding to bf16 less in each of up to fifty layers
    assert float((fused - plain).norm() / plain.norm()) < 0.02
