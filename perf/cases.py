"""The work this framework is used for, as measurable cases over its public entry points.

Six kinds of work, each with a range of sizes:

``lm_train``     one optimizer step of a GPT-2 style language model through ``Trainer.train_step``; ``graph`` says whether
                 the step was captured in a CUDA graph beforehand (``cuda_graph`` of the training configuration)
``lm_score``     logits of a batch of token sequences through ``Graph.forward`` in evaluation mode (prefill, validation)
``lm_generate``  greedy decoding with ``greedy_generate``, then one scoring pass over the text it produced
``image_train``  one optimizer step of an image model of the zoo through ``Trainer.train_step``
``image_infer``  logits of a batch of images through ``Graph.forward`` in evaluation mode
``block``        a transformer block with a classification head, written with the ``ops.functional`` bridges: loss and
                 ``backward()``

The model shapes are those of the zoo (``tnn_b200/models/zoo.py``) and of its ``gpt2`` builder with other widths, depths,
sequence lengths and vocabularies; batch sizes and optimizers are those of ``configs/`` and ``bench.py`` and what lies
around them.
"""
import math

import torch

from tnn_b200.inference import greedy_generate
from tnn_b200.models import zoo
from tnn_b200.nn.graph import infer_shapes
from tnn_b200.nn.blocks import FlashAttentionBlock
from tnn_b200.nn.layers import Add, BatchNorm, Conv2D, Dense, Dropout
from tnn_b200.ops import functional as F
from tnn_b200.trainer import Trainer
from tnn_b200.utils.config import TrainingConfig

DEV = "cuda"

ADAMW = {"type": "adamw", "learning_rate": 3e-4, "beta1": 0.9, "beta2": 0.95, "epsilon": 1e-8, "weight_decay": 0.1}
SGD = {"type": "sgd", "learning_rate": 0.01, "momentum": 0.9}

#: Image models of the zoo, the number of classes each ends in and the largest batch that a case of it uses.
IMAGE_MODELS = {
    "mnist_cnn": (10, 2048), "cifar10_vgg": (10, 1024), "cifar10_resnet9": (10, 512), "cifar100_resnet18": (100, 512),
    "cifar100_wrn16_8": (100, 192), "tiny_imagenet_resnet18": (200, 256), "tiny_imagenet_resnet50": (200, 192),
    "tiny_imagenet_flash_vit": (200, 256), "imagenet100_resnet50": (100, 256),
}
IMAGE_NAMES = sorted(IMAGE_MODELS)


# ------------------------------------------------------------------------------------------------------------- cases
def listed():
    return [
        # configs/gpt2_small.json and bench.py: the headline training step, captured in a CUDA graph
        {"name": "gpt2_small_train", "kind": "lm_train", "embed": 768, "heads": 12, "layers": 12, "seq": 1024, "vocab": 50257,
         "batch": 8, "graph": True},
        # a small model on short sequences of odd length and a vocabulary of its own: a first experiment, run eagerly
        {"name": "gpt_tiny_train", "kind": "lm_train", "embed": 256, "heads": 4, "layers": 4, "seq": 203, "vocab": 5003,
         "batch": 6, "graph": False},
        # validation loss / scoring with the medium model: prefill of full-length sequences
        {"name": "gpt2_medium_score", "kind": "lm_score", "embed": 1024, "heads": 16, "layers": 24, "seq": 1024, "vocab": 50257,
         "batch": 4},
        # `generate` on the command line: a short prompt, a few dozen new tokens, batch 1
        {"name": "gpt2_small_generate", "kind": "lm_generate", "embed": 768, "heads": 12, "layers": 12, "seq": 1024,
         "vocab": 50257, "prompt": 45, "new": 24},
        # configs/resnet50_imagenet100.json: epoch mode, so every step is launched from the host
        {"name": "resnet50_train", "kind": "image_train", "model": "imagenet100_resnet50", "batch": 256, "graph": False},
        # configs/wrn16_8_cifar100.json: the same for the wide residual network (channel counts from 16 to 512)
        {"name": "wrn16_8_train", "kind": "image_train", "model": "cifar100_wrn16_8", "batch": 128, "graph": False},
        # configs/cnn_mnist.json on a GPU: a network so small that launches and host work decide
        {"name": "mnist_train", "kind": "image_train", "model": "mnist_cnn", "batch": 256, "graph": False},
        # the vision transformer: sequences of 257 tokens, no causal mask, an odd batch, captured step
        {"name": "vit_train", "kind": "image_train", "model": "tiny_imagenet_flash_vit", "batch": 125, "graph": True},
        # serving images in small odd batches
        {"name": "resnet50_infer", "kind": "image_infer", "model": "imagenet100_resnet50", "batch": 7},
        # one small image: the shortest call there is, latency only
        {"name": "resnet9_infer_1", "kind": "image_infer", "model": "cifar10_resnet9", "batch": 1},
        # a module written with the autograd bridges, heads of 96 (the attention micro-benchmark's shape)
        {"name": "block_d96", "kind": "block", "batch": 16, "seq": 512, "heads": 8, "dim": 96, "causal": True,
         "vocab": 1024},
        # the same for a small ragged shape without mask, the common head size
        {"name": "block_d64_ragged", "kind": "block", "batch": 3, "seq": 333, "heads": 5, "dim": 64, "causal": False,
         "vocab": 203},
    ]


def _log_int(rng, lo, hi):
    """A whole number from lo to hi, spread evenly over its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _draw_once(rng):
    kind = rng.choice(["lm_train", "lm_score", "lm_generate", "image_train", "image_train", "image_infer", "block"])
    if kind in ("image_train", "image_infer"):
        model = rng.choice(IMAGE_NAMES)
        top = IMAGE_MODELS[model][1]
        if kind == "image_infer":
            return {"kind": kind, "model": model, "batch": _log_int(rng, 1, top)}
        return {"kind": kind, "model": model, "batch": _log_int(rng, 8, top), "graph": rng.random() < 0.5}
    if kind == "block":
        return {"kind": kind, "batch": _log_int(rng, 1, 32), "seq": _log_int(rng, 16, 1500), "heads": _log_int(rng, 1, 16),
                "dim": rng.choice([32, 48, 64, 64, 64, 80, 96, 128]), "causal": rng.random() < 0.7,
                "vocab": _log_int(rng, 64, 8192)}
    heads = _log_int(rng, 2, 20)
    case = {"kind": kind, "embed": 64 * heads, "heads": heads, "layers": _log_int(rng, 2, 24), "seq": _log_int(rng, 48, 1536),
            "vocab": _log_int(rng, 200, 50257)}
    if kind == "lm_generate":
        case["prompt"] = _log_int(rng, 4, case["seq"] // 2)
        case["new"] = _log_int(rng, 4, 32)
        return case
    case["batch"] = _log_int(rng, 1, 24)
    if kind == "lm_train":
        case["graph"] = rng.random() < 0.6
    return case


def draw(rng):
    """One more case of the same ranges, no more work than the headline training step."""
    most = work(listed()[0])["flops"]
    while True:
        case = _draw_once(rng)
        if case["kind"] == "block" and case["batch"] * case["seq"] > 16384:
            continue
        if work(case)["flops"] <= most:
            return case


# ------------------------------------------------------------------------------------------------------------ models
def _graph_of(case):
    """The uncompiled graph of a case and the shape of its input."""
    if case["kind"].startswith("lm"):
        g = zoo.gpt2(case["embed"], case["heads"], case["layers"], "gpt", seq_len=case["seq"], vocab=case["vocab"])
        return g, (case.get("batch", 1), case["seq"])
    return zoo.create(case["model"]), (case["batch"],) + zoo.INPUT_SHAPES[case["model"]]


def _compiled(case, seed):
    """A model as it is after loading: the zoo's own initialisation, drawn on the GPU from the seed, in the flat fp32
    buffer and its bf16 copy. Dropout masks follow from the seed too (a layer's own base would follow from Python's
    string hash, which is another one in every process)."""
    g, _ = _graph_of(case)
    g.compile(device=DEV, init=False)
    gen = torch.Generator(device=DEV).manual_seed(seed)
    for k, layer in enumerate(g.layers()):
        for spec, m in zip(layer.param_specs(), layer.masters):
            kind, val = spec.init
            if kind == "normal":
                m.normal_(0.0, val, generator=gen)
            else:
                m.fill_(1.0 if kind == "ones" else 0.0)
        if isinstance(layer, Dropout):
            layer.seed_base = (seed * 7907 + k) * 65537 - (hash(layer.name) & 0xFFFFFFFF) * 1000003
    return g, gen


def _tokens(shape, vocab, gen):
    """Token ids with the frequencies of text: the id's logarithm is uniform, so a few ids are everywhere."""
    u = torch.rand(shape, generator=gen, device=DEV, dtype=torch.float64)
    return (vocab ** u).long().sub_(1).clamp_(0, vocab - 1)


def _trained_transformer(case, g, gen):
    """Weights with what training gives a transformer and a fresh one has not: projections whose scores are of order one
    (the blocks scale them by 1, so training learns the 1 / sqrt(head size)), scaled output projections that keep the
    tokens visible in the residual stream, and, for a language model, one next token that is clearly the likeliest - so
    that the results do not hang on the last bit of a score or of a logit."""
    layers = {layer.name: layer for layer in g.layers()}
    blocks = [layer for layer in g.layers() if isinstance(layer, FlashAttentionBlock)]
    shrink = 1.0 / math.sqrt(2 * max(1, len(blocks)))
    for layer in blocks:
        layer.masters[0][:2 * layer.embed_dim].mul_(layer.head_dim ** -0.25)
        layer.masters[2].mul_(shrink)
    for layer in g.layers():
        if layer.name.endswith("_mlp_fc2"):
            layer.masters[0].mul_(shrink)
    if "token_embed" in layers:
        wte, head = layers["token_embed"].masters[0], layers["head"].masters[0]
        wte.normal_(0.0, 0.5, generator=gen)
        follows = torch.randperm(case["vocab"], generator=gen, device=DEV)
        head.mul_(0.5)
        head[follows] += wte / math.sqrt(case["embed"])


def _settled(g, gen):
    """Batch-norm statistics and scales as training leaves them: near the data's, not exactly 0 and 1."""
    for layer in g.layers():
        if isinstance(layer, BatchNorm):
            gamma, beta, mean, var = layer.masters
            gamma.normal_(1.0, 0.1, generator=gen)
            beta.normal_(0.0, 0.1, generator=gen)
            mean.normal_(0.0, 0.1, generator=gen)
            var.uniform_(0.5, 1.5, generator=gen)


def _well_conditioned(g):
    """What training soon gives an image model and a fresh one has not: residual branches that correct their shortcut
    instead of drowning it (the scale of a block's closing batch norm is a fraction of 1) and logits of order one. With
    the plain initialisation a deep model's gradient hangs on single bits of its activations: weights that differ by
    one part in a million give velocities that differ by half their size (0.53 for the 50-layer model)."""
    for e in g.edges:
        if isinstance(e.layer, BatchNorm) and not e.layer.name.endswith(("shortcut_bn", "bn3")):
            out = e.consumers[0]
            if any(type(f.layer) is Add and out in f.producers for f in g.edges):
                e.layer.masters[0].mul_(0.25)
    if isinstance(g.edges[-1].layer, Dense):
        g.edges[-1].layer.masters[0].mul_(0.1)


def _resumed(trainer, weights, gen):
    """The trainer as it is when training goes on from a snapshot: these weights, and an optimizer that has seen some
    steps (Adam's second moments near the squares of such gradients, so that a step is not the sign of the gradient)."""
    g, opt = trainer.graph, trainer.optimizer
    g.master_flat.copy_(weights)
    g.sync_params_from_master()
    g.zero_grads()
    state = opt.state_dict()
    for k, t in _optimizer_state(opt).items():
        t.zero_()
        if k == "v":
            t.uniform_(0.5e-6, 1.5e-6, generator=gen)
    opt.load_state_dict(dict(state, step=torch.tensor(1000)))
    trainer.global_step = 0
    trainer.step_counter.zero_()


# ------------------------------------------------------------------------------------------------ prepare, run
def prepare(case, seed):
    kind = case["kind"]
    if kind == "block":
        return _prepare_block(case, seed)
    g, gen = _compiled(case, seed)
    _trained_transformer(case, g, gen)
    if kind == "image_infer":
        _settled(g, gen)
    if kind == "image_train":
        _well_conditioned(g)
    g.sync_params_from_master()
    weights = g.master_flat.clone() if kind.endswith("train") else None
    state = {"kind": kind, "graph": g}
    _, shape = _graph_of(case)
    if kind.startswith("lm"):
        ids = _tokens((shape[0], shape[1] + 1), case["vocab"], gen)
        data, labels = ids[:, :-1].contiguous(), ids[:, 1:].contiguous()
    else:
        data = torch.randn(shape, generator=gen, device=DEV).to(torch.bfloat16)
        labels = torch.randint(0, IMAGE_MODELS[case["model"]][0], (shape[0],), generator=gen, device=DEV)
    if kind in ("lm_train", "image_train"):
        cfg = TrainingConfig.from_dict({"model_name": "case", "batch_size": shape[0], "device_type": "CUDA",
                                        "optimizer": ADAMW if kind == "lm_train" else SGD, "scheduler": {"type": "no_op"},
                                        "loss": {"type": "logsoftmax_crossentropy"}})
        trainer = Trainer(cfg, graph=g, device=torch.device(DEV), log=False)
        if case["graph"]:
            trainer.enable_cuda_graph(data, labels)
        _resumed(trainer, weights, gen)
        state.update(trainer=trainer, data=data, labels=labels)
    elif kind == "lm_generate":
        g.set_training(False)
        state.update(prompt=[int(t) for t in data[0, :case["prompt"]].cpu()], new=case["new"], seq=case["seq"])
    else:
        g.set_training(False)
        state["data"] = data
    return state


def _prepare_block(case, seed):
    """A torch.nn style block: bf16 parameters that autograd collects gradients for, activations and their gradient."""
    gen = torch.Generator(device=DEV).manual_seed(seed)
    e = case["heads"] * case["dim"]

    def make(*shape, scale):
        return (torch.randn(*shape, generator=gen, device=DEV) * scale).to(torch.bfloat16)

    w = {"g1": 1 + make(e, scale=0.1), "b1": make(e, scale=0.1), "g2": 1 + make(e, scale=0.1), "b2": make(e, scale=0.1),
         "wqkv": make(3 * e, e, scale=e ** -0.5), "bqkv": make(3 * e, scale=0.1), "wo": make(e, e, scale=e ** -0.5),
         "bo": make(e, scale=0.1), "w1": make(4 * e, e, scale=e ** -0.5), "bb1": make(4 * e, scale=0.1),
         "w2": make(e, 4 * e, scale=(4 * e) ** -0.5), "bb2": make(e, scale=0.1), "gf": 1 + make(e, scale=0.1),
         "bf": make(e, scale=0.1), "head": make(case["vocab"], e, scale=e ** -0.5)}
    for t in w.values():
        t.requires_grad_(True)
    x = make(case["batch"], case["seq"], e, scale=1.0).requires_grad_(True)
    labels = torch.randint(0, case["vocab"], (case["batch"], case["seq"]), generator=gen, device=DEV)
    return {"kind": "block", "w": w, "x": x, "labels": labels, "heads": case["heads"], "causal": case["causal"]}


def _run_block(state):
    w, x = state["w"], state["x"]
    for t in w.values():
        t.grad = None
    x.grad = None
    h, s = F.add_layer_norm(x, None, w["g1"], w["b1"])
    a = F.causal_self_attention(F.linear(h, w["wqkv"], w["bqkv"]), state["heads"], causal=state["causal"])
    h, s = F.add_layer_norm(s, F.linear(a, w["wo"], w["bo"]), w["g2"], w["b2"])
    y = F.linear(F.linear(h, w["w1"], w["bb1"], gelu=True), w["w2"], w["bb2"])
    h, _ = F.add_layer_norm(s, y, w["gf"], w["bf"])
    logits = F.linear(h, w["head"])
    loss = F.cross_entropy(logits, state["labels"])
    loss.backward()
    return {"loss": loss, "logits": logits, "dx": x.grad, "dw": {k: t.grad for k, t in w.items()}}


def run(state):
    kind = state["kind"]
    if kind == "block":
        return _run_block(state)
    g = state["graph"]
    if kind in ("lm_train", "image_train"):
        loss = state["trainer"].train_step(state["data"], state["labels"])
        return {"loss": loss, "weights": g.master_flat, "optimizer": _optimizer_state(state["trainer"].optimizer)}
    if kind == "lm_generate":
        tokens = greedy_generate(g, state["prompt"], num_new=state["new"], eos=None)
        text = torch.zeros(1, state["seq"], dtype=torch.long)
        text[0, :len(tokens)] = torch.tensor(tokens)
        return {"tokens": torch.tensor(tokens), "logits": g.forward({"input": text})["output"]}
    return g.forward({"input": state["data"]})["output"]


def _optimizer_state(opt):
    """What the update keeps for the next step: the moments, or the velocity."""
    state = opt.state_dict()
    return {k: state[k] for k in ("m", "v", "velocity") if k in state}


# ------------------------------------------------------------------------------------------------ work, tolerance
def _layer_work(case):
    """(forward flops, elements that layers hand to each other, parameters) of one forward pass of a zoo graph."""
    g, shape = _graph_of(case)
    shapes = infer_shapes(g, {"input": shape})
    flops, between, params = 0.0, 0.0, 0.0
    for e in g.edges:
        layer = e.layer
        out = shapes[e.consumers[0].uid()]
        n = math.prod(out)
        for spec in layer.param_specs():
            params += math.prod(spec.shape)
        if isinstance(layer, Conv2D):
            flops += 2.0 * n * layer.kernel_h * layer.kernel_w * layer.in_channels
            between += n
        elif isinstance(layer, Dense):
            flops += 2.0 * n * layer.input_features
            between += n
        elif isinstance(layer, FlashAttentionBlock):
            b, s, width = out
            flops += 8.0 * b * s * width * width + 4.0 * b * s * s * width * (0.5 if layer.is_causal else 1.0)
            between += 5.0 * n
    return flops, between, params, math.prod(shape), math.prod(shapes["output"])


def work(case):
    """Bytes and operations that one pass cannot do without.

    Training: three times the forward products; weights in bf16 read, gradients and optimizer state in fp32 read and
    written once; every product's result kept in bf16 from the forward to the backward pass (written once, read once).
    Evaluation: weights, inputs and outputs. Decoding: the prompt once, then the weights once per new token."""
    kind = case["kind"]
    if kind == "block":
        e, rows = case["heads"] * case["dim"], case["batch"] * case["seq"]
        att = 4.0 * rows * case["seq"] * e * (0.5 if case["causal"] else 1.0)
        params = 12.0 * e * e + case["vocab"] * e
        flops = 3 * 2.0 * rows * params + 3.5 * att
        return {"bytes": 2.0 * (2 * rows * e + 2 * params + 2 * 11 * rows * e + 2 * rows * case["vocab"]), "flops": flops}
    flops, between, params, n_in, n_out = _layer_work(case)
    elem = 8 if kind.startswith("lm") else 2
    if kind in ("lm_train", "image_train"):
        opt = 30 if kind == "lm_train" else 22
        return {"bytes": float(elem * n_in + 4 * between + params * (4 + opt)), "flops": 3 * flops}
    if kind == "lm_generate":
        tables = (case["vocab"] + case["seq"]) * case["embed"]  # looked up, not read through
        cells = params - tables
        # a token's own products, decoding step by step, and one whole scoring pass
        per_token = 2.0 * cells
        return {"bytes": float(2 * cells * (case["new"] + 1) + 2 * n_out), "flops": flops + per_token * (case["prompt"] + case["new"])}
    return {"bytes": float(elem * n_in + 2 * params + 2 * n_out), "flops": flops}


def tolerance(case):
    """bf16 weights and activations with fp32 sums. Each number is about four times the largest difference measured over
    several sizes:

    * ``block``: against the same block in fp64 on the same bf16 values (worst: the gradient of a layer-norm scale, 0.0065);
    * ``lm_train``: Adam's first moment against the layer-by-layer executor, which rounds at other places, and against
      fp32 on the CPU (0.0022 to 0.0046); ``lm_score``, ``lm_generate``: logits likewise (0.0076 to 0.0114);
    * ``image_infer``: logits against fp32 on the CPU (0.0025 to 0.0032);
    * ``image_train``: the velocity after one and after two steps, with the weights moved by one part in a million, so
      that a few of them round the other way (0.006 to 0.027; VGG, a plain stack without shortcuts, 0.20). Each ReLU
      mask or pooling index that flips is a whole gradient entry, so single values are not bounded.

    Tokens are whole numbers: one in a hundred may differ where two logits tie."""
    kind = case["kind"]
    if kind == "block":
        return {"rel": 0.026, "max": 0.15}
    if kind == "lm_train":
        return {"rel": 0.018, "max": 0.4}
    if kind == "lm_score":
        return {"rel": 0.03, "max": 0.3}
    if kind == "lm_generate":
        return {"rel": 0.03, "max": 0.3, "differ": 0.01}
    if kind == "image_infer":
        return {"rel": 0.013, "max": 0.04}
    return {"rel": 0.8 if case["model"] == "cifar10_vgg" else 0.11}
