"""An evaluation gives an input the same output, to the last bit, whatever its batch holds beside it - unless the graph was told
that it need not."""
import pytest
import torch

from tnn_b200.models import zoo
from tnn_b200.ops import _lib, functional as F

pytestmark = pytest.mark.gpu


def _inputs(model, batch):
    """A compiled graph in evaluation mode and ``batch`` inputs."""
    g = torch.Generator(device="cuda").manual_seed(5)
    if model == "gpt":  # rows enough for one tile, sums of 1536 and 384 values
        graph = zoo.gpt2(384, 6, 2, "gpt", seq_len=48, vocab=500).compile(device="cuda", seed=1)
        x = torch.randint(0, 500, (batch, 48), generator=g, device="cuda")
    else:
        graph = zoo.create(model).compile(device="cuda", seed=1)
        x = torch.randn((batch,) + zoo.INPUT_SHAPES[model], generator=g, device="cuda").bfloat16()
    graph.set_training(False)
    return graph, x


@pytest.mark.parametrize("model,batch", [("gpt", 40), ("cifar10_resnet9", 40), ("cifar100_wrn16_8", 24), ("cifar10_vgg", 33),
                                         ("tiny_imagenet_resnet50", 17), ("tiny_imagenet_flash_vit", 9)])
def test_outputs_alone_and_among_others(model, batch):
    graph, x = _inputs(model, batch)
    run = lambda t: graph.forward({"input": t.contiguous()})["output"].clone()
    among, alone, few = run(x), run(x[:1]), run(x[:3])
    _lib.check_status()
    assert torch.equal(among[:1], alone) and torch.equal(among[:3], few)
    graph.set_batch_independent(False)
    other = run(x[:1]).float()
    graph.set_batch_independent(True)
    assert torch.equal(run(x[:1]), alone)
    assert float((other - alone.float()).norm() / alone.float().norm()) < 0.02  # single roundings to bf16, in up to fifty layers


@pytest.mark.parametrize("gelu", [False, True])
def test_linear_rows_alone_and_among_others(gelu):
    g = torch.Generator(device="cuda").manual_seed(6)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()
    x, w, b = rnd(3000, 2048), rnd(520, 2048), rnd(520)
    whole = F.linear(x, w, b, gelu=gelu)
    for rows in (1, 33, 700):
        assert torch.equal(F.linear(x[:rows], w, b, gelu=gelu), whole[:rows])
    _lib.check_status()
