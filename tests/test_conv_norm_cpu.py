"""Which convolutions the executor runs together with the batch norm behind them in evaluation mode."""
import ctypes

import pytest
import torch

from tnn_b200.nn.graph import Graph
from tnn_b200.nn.layers import BatchNorm, Conv2D
from tnn_b200.ops import _lib
from tnn_b200.ops.gemm import EPI_RESID


def _graph(features=16, tap=False, branch=False):
    g = Graph()
    y = Conv2D(8, features, 3, 3, 1, 1, 1, 1, name="conv")(g.input("input"))
    z = BatchNorm(features, use_relu=True, name="bn")(y)
    if branch:  # the convolution's output is used twice
        z = z + y
    z.set_uid("output")
    if tap:  # ... or asked for
        g.set_output(y)
    g.set_output(z)
    return g.compile(device="cpu", seed=0)


def test_pairs_of_convolution_and_norm():
    assert list(_graph()._norm_after) == [0]
    assert not _graph(tap=True)._norm_after and not _graph(branch=True)._norm_after
    assert not _graph(features=12)._norm_after  # the norm kernels take multiples of eight channels
    g, x = _graph(), torch.randn(2, 5, 5, 8)
    g.set_training(False)
    both = g.forward({"input": x})["output"]
    g._norm_after = {}
    assert torch.equal(both, g.forward({"input": x})["output"])  # off the GPU the layers run one by one


@pytest.mark.parametrize("n,ldd,ld_res,d,res,code", [(64, 64, 64, 0, 2, -4), (64, 64, 64, 8, 0, -4), (64, 72, 68, 0, 0, -3),
                                                     (64, 68, 64, 0, 0, -3), (60, 64, 64, 0, 0, -3)])
def test_product_with_norm_refuses_what_the_norm_refuses(n, ldd, ld_res, d, res, code):
    """Outputs and residuals that cannot be read and written in 16-byte vectors: before anything is launched."""
    lib = ctypes.CDLL(_lib.lib_path())
    vp, ll, i, f = ctypes.c_void_p, ctypes.c_longlong, ctypes.c_int, ctypes.c_float
    fn = lib.tnnb_gemm_bf16_norm
    fn.argtypes, fn.restype = [vp, vp, vp, i, i, i, ll, ll, ll, vp, vp, vp, vp, vp, f, vp, ll, i, i, vp, vp], i
    at = 1 << 20  # never read
    assert fn(at, at, at + d, 32, n, 64, 64, 64, ldd, None, None, None, at, at, 1e-5, at + res, ld_res, EPI_RESID, 0, at, None) == code
