"""Greedy decoding over the tokens so far on the GPU: the kernels at the lengths it uses against a full-length pass."""
import pytest
import torch

from tnn_b200.inference import _prefix_suffices, greedy_generate
from tnn_b200.models import zoo

pytestmark = pytest.mark.gpu
SEQ, VOCAB = 200, 203


@pytest.mark.parametrize("fuse", [True, False])
@pytest.mark.parametrize("embed,heads", [(128, 2), (192, 2)])  # heads of 64 and of 96
def test_logits_at_the_last_token(fuse, embed, heads):
    """The positions behind the last token change nothing but the order of sums: one bf16 rounding (2**-8) per residual sum
    and product, of which the two blocks and the head have nine in a row."""
    g = zoo.gpt2(embed, heads, 2, "p", seq_len=SEQ, vocab=VOCAB).compile(device="cuda", seed=3, fuse=fuse)
    g.set_training(False)
    assert _prefix_suffices(g, SEQ)
    torch.manual_seed(0)
    text = torch.randint(0, VOCAB, (1, SEQ), device="cuda")
    for n in (1, 63, 64, 65, 127, 128, 129, 192, 193, SEQ - 1, SEQ):
        x = text.clone()
        x[0, n:] = 0
        full = g.forward({"input": x})["output"][0, n - 1].float()
        short = g._forward({"input": x[:, :min(SEQ, (n + 63) // 64 * 64)].contiguous()}, 0, True)["output"][0, n - 1].float()
        assert float((short - full).norm()) <= 9 * 2.0 ** -8 * float(full.norm()), n


def test_tokens():
    """Each token is the likeliest of a full-length pass, or ties with it to a bf16 rounding of the largest logit."""
    g = zoo.gpt2(128, 2, 2, "p", seq_len=SEQ, vocab=VOCAB).compile(device="cuda", seed=4)
    tokens = greedy_generate(g, [5, 9, 2], num_new=70, eos=None)
    assert len(tokens) == 73
    g.set_training(False)
    x = torch.zeros(1, SEQ, dtype=torch.long)
    x[0, :73] = torch.tensor(tokens)
    logits = g.forward({"input": x.cuda()})["output"][0].float()
    for k in range(3, 73):
        row = logits[k - 1]
        assert float(row[tokens[k]]) >= float(row.max()) - 2.0 ** -7 * float(row.abs().max()), k
