"""Inference helpers: validation of a saved or fresh model and greedy text generation.

Reference: examples/inferencer.cpp:12-70 (validation loss / accuracy from ``model_path`` or a fresh zoo
model) and examples/gpt2_inference.cpp:16-114 (greedy decoding: the prompt is right-padded with zeros to
the model's sequence length, the logits at the last real position pick the next token, decoding stops
at token 50256).
"""
from __future__ import annotations

from typing import Callable, Dict, Iterable, List, Optional

import torch

from .nn.blocks import FlashAttentionBlock
from .nn.graph import Graph
from .nn.layers import (Add, Dense, Div, Dropout, ELU, Embedding, GELU, LayerNorm, LeakyReLU, Mul, PositionalEmbedding, ReLU,
                        Sigmoid, Sub, Tanh)

_PER_POSITION = (Add, Dense, Div, Dropout, ELU, Embedding, GELU, LayerNorm, LeakyReLU, Mul, ReLU, Sigmoid, Sub, Tanh)


def model_seq_len(graph: Graph) -> Optional[int]:
    """Sequence length fixed by the positional embedding of a language model (None if there is none)."""
    for layer in graph.layers():
        if isinstance(layer, PositionalEmbedding):
            return int(layer.seq_len)
    return None


def _prefix_suffices(graph: Graph, S: int) -> bool:
    """True when the output at a position depends on the positions up to it alone: every layer works on one position at
    a time or is causal attention, and positional tables hold the ``S`` positions of a full forward pass. The logits
    behind the last token then follow from the tokens themselves and the padding after them need not be computed."""
    if len(graph.input_nodes) != 1 or len(graph.output_nodes) != 1:
        return False
    for layer in graph.layers():
        if getattr(layer, "tp", 1) != 1:  # tensor-parallel ranks exchange rows of the full sequence
            return False
        if type(layer) is PositionalEmbedding:
            if layer.seq_len != S:
                return False
        elif type(layer) is FlashAttentionBlock:
            if not layer.is_causal:
                return False
        elif type(layer) not in _PER_POSITION:
            return False
    return True


@torch.no_grad()
def greedy_generate(graph: Graph, prompt: Iterable[int], num_new: int = 50, eos: Optional[int] = 50256,
                    seq_len: Optional[int] = None, on_token: Optional[Callable[[int], None]] = None) -> List[int]:
    """Greedy decoding with a forward pass per token (the reference has no KV cache either), over the tokens so far,
    rounded up to 64, where the model allows it (:func:`_prefix_suffices`) and over the full length otherwise.

    ``seq_len`` defaults to the model's positional-embedding length; the window slides once the text is
    longer than that. Returns prompt + generated tokens.
    """
    tokens = [int(t) for t in prompt]
    if not tokens:
        raise ValueError("empty prompt")
    S = seq_len or model_seq_len(graph) or len(tokens) + num_new
    was_training = graph.training
    graph.set_training(False)
    prefix = _prefix_suffices(graph, S)
    try:
        for _ in range(num_new):
            use = tokens[-S:]
            x = torch.zeros(1, min(S, (len(use) + 63) // 64 * 64) if prefix else S, dtype=torch.long)
            x[0, :len(use)] = torch.tensor(use)
            inputs = {graph.input_nodes[0].uid(): x.to(graph.device)}
            out = (graph._forward(inputs, 0, True) if prefix else graph.forward(inputs))[graph.output_nodes[0].uid()]
            logits = out[0, len(use) - 1].float()
            best = torch.argmax(logits)
            nxt, bad = torch.stack((best, torch.isnan(logits[0]).to(best.dtype))).tolist()  # one wait for the device
            if bad:
                raise FloatingPointError("model output contains NaNs (the model probably diverged in training)")
            tokens.append(nxt)
            if on_token is not None:
                on_token(nxt)
            if eos is not None and nxt == eos:
                break
    finally:
        graph.set_training(was_training)
    return tokens


@torch.no_grad()
def evaluate(trainer, max_batches: Optional[int] = None) -> Dict[str, float]:
    """Validation loss / accuracy (and perplexity for token models) through the trainer's own loop."""
    return dict(trainer.validate(max_batches=max_batches))
