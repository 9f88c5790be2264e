"""Kernels that may become resident while the kernel before them still writes their inputs (csrc/kernels/launch.cuh)."""
import glob
import os
import re

import tnn_b200

KERNELS = os.path.join(os.path.dirname(tnn_b200.__file__), "csrc", "kernels")


def _kernels():
    """(name, parameters, body) of every kernel definition."""
    for path in sorted(glob.glob(os.path.join(KERNELS, "*.cu"))):
        text = open(path).read()
        for m in re.finditer(r"__global__ void\s", text):
            brace = text.index("{", m.end())
            head = text[m.end():brace]
            end = text.index("\n}", brace)
            name = re.findall(r"(\w+)\(", head.split("__launch_bounds__")[-1].split("\n", 1)[-1] if "__launch_bounds__" in head else head)[0]
            yield name, head, text[brace:end]


def test_no_input_is_promised_to_be_constant():
    waiting = [(name, head) for name, head, body in _kernels() if "grid_dep_wait()" in body]
    assert {"ln_fwd_kernel", "ln_bwd_kernel", "bn_bwd_apply_kernel", "colsum_kernel", "attn_bwd_kernel"} <= {name for name, _ in waiting}
    assert [name for name, head in waiting if "__restrict__" in head] == []


def _launched_early():
    """Names of the kernels behind every ``launch_dependent`` and ``launch_dependent_cluster``, also those that go through a
    variable: the last ``auto kern = ...;`` before the launch."""
    for path in sorted(glob.glob(os.path.join(KERNELS, "*.cu"))):
        text = open(path).read()
        for m in re.finditer(r"\blaunch_dependent(?:_cluster)?\(\s*(\w+)", text):
            name = m.group(1)
            if name.endswith("_kernel"):
                yield path, {name}
                continue
            held = re.findall(rf"\bauto {name} =([^;]+);", text[:m.start()])
            yield path, set(re.findall(r"\w+_kernel\b", held[-1])) if held else set()


def test_every_kernel_launched_early_waits():
    launches = list(_launched_early())
    assert all(names for _, names in launches), launches  # a launch whose kernel is not found tests nothing
    launched = set().union(*(names for _, names in launches))
    assert {"conv_fwd_halo_kernel", "conv_fwd_ranges_kernel", "conv_fwd_implicit_kernel", "gemm_bf16_tcgen05_kernel",
            "gemm_bf16_tcgen05_ranges_kernel", "gemm_bf16_tcgen05_pair_kernel", "attn_fwd_kernel", "ln_fwd_kernel"} <= launched
    waiting = {name for name, _, body in _kernels() if "grid_dep_wait()" in body}
    assert launched <= waiting, launched - waiting
