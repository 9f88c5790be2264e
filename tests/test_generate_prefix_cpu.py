"""Greedy decoding over the tokens so far against a full-length forward pass per token."""
import pytest
import torch

from tnn_b200.inference import _prefix_suffices, greedy_generate
from tnn_b200.models import zoo
from tnn_b200.nn.graph import Graph
from tnn_b200.nn.layers import Dense, Embedding, PositionalEmbedding, Transpose


def _full(g, prompt, n, S):
    tokens = list(prompt)
    g.set_training(False)
    for _ in range(n):
        use = tokens[-S:]
        x = torch.zeros(1, S, dtype=torch.long)
        x[0, :len(use)] = torch.tensor(use)
        tokens.append(int(g.forward({"input": x})["output"][0, len(use) - 1].argmax()))
    return tokens


@pytest.mark.parametrize("seq,prompt,new", [(80, 3, 6), (80, 62, 5), (80, 78, 6), (20, 1, 25)])
@pytest.mark.parametrize("fuse", [True, False])
def test_same_tokens(seq, prompt, new, fuse):
    g = zoo.gpt2(128, 2, 2, "p", seq_len=seq, vocab=97).compile(device="cpu", seed=3, fuse=fuse)
    torch.manual_seed(seq + prompt)
    start = torch.randint(0, 97, (prompt,)).tolist()
    assert _prefix_suffices(g, seq)
    assert greedy_generate(g, start, num_new=new, eos=None) == _full(g, start, new, seq)


def test_other_models_run_at_full_length():
    g = zoo.gpt2(128, 2, 1, "p", seq_len=16, vocab=50).compile(device="cpu", seed=0)
    assert not _prefix_suffices(g, 12)                       # a length the positional table does not have
    with pytest.raises(ValueError):
        greedy_generate(g, [1, 2], num_new=1, eos=None, seq_len=12)
    with pytest.raises(ValueError):                          # a plain forward pass still takes the full length only
        g.forward({"input": torch.zeros(1, 8, dtype=torch.long)})
    h = Graph()
    x = Embedding(50, 16)(h.input("input"))
    x = PositionalEmbedding(16, 16)(x)
    y = Dense(16, 50)(Transpose(1, 2)(Dense(16, 16)(Transpose(1, 2)(x))))  # mixes positions
    y.set_uid("output")
    h.set_output(y)
    h.compile(device="cpu", seed=1)
    assert not _prefix_suffices(h, 16)
    assert greedy_generate(h, [1, 2, 3], num_new=3, eos=None) == _full(h, [1, 2, 3], 3, 16)
