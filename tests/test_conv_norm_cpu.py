"""Which convolutions the executor runs together with the batch norm behind them in evaluation mode."""
import torch

from tnn_b200.nn.graph import Graph
from tnn_b200.nn.layers import BatchNorm, Conv2D


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
