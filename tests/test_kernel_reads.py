"""Kernels are resident while the launch in front still writes (programmatic launches), and what is read through the non-coherent path must
not be written during a kernel's lifetime: only weights are."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "naivert_b200", "csrc")
# file -> what its non-coherent loads, and the helpers made of them, may read
HELPERS = {"stack_rows.cu": "bf4", "stack_state.cu": "bf4", "stack_step.cu": "ldw4"}
WEIGHTS = {
    "stack_rows.cu": {"a.join_w", "a.join_w2", "emb", "a.post_w", "a.add", "a.pre_w"},
    "stack_state.cu": {"a.rate", "a.mu", "w"},
    "stack_step.cu": {"a.in_w", "a.post_w", "a.join_w", "a.join_w2", "emb", "a.add", "mu"},
    "draft.cu": {"wr", "r", "a.w1", "embed", "mask"},           # rows of the factors
    "gemm.cuh": {"p.ngamma", "ws0", "ws1"},
    "moe_fused.cu": {"ws0", "ws1", "p.down_s"},
    "router.cuh": {"a.gamma", "a.w", "a.bias"},
    "target_kernels.cu": {"table", "gamma"},
    "wide_gemm.cu": {"ws0", "ws1"},
}


def source(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def read_by(text, function):
    """Names of the pointers that calls of ``function`` are given."""
    out = set()
    for m in re.finditer(rf"\b{function}\(", text):
        if re.search(r"(float4|uint2)\s+$", text[:m.start()]):                       # its definition
            continue
        arg = re.sub(r"^(reinterpret_cast<[^>]*>)?\(*", "", text[m.end():m.end() + 200])
        out.add(re.match(r"[\w.]+", arg)[0])
    return out


@pytest.mark.parametrize("name", sorted(n for n in os.listdir(CSRC) if n.endswith((".cu", ".cuh"))))
def test_only_weights_are_read_past_the_coherent_path(name):
    text = source(name)
    helper = HELPERS.get(name)
    got = read_by(text, "__ldg")
    if helper:
        got = (got - {"p"}) | {n for n in read_by(text, helper) if n not in ("p.post", "p.in", "ldw4")}
    got |= set(re.findall(r"const\s[\w\s]+\*\s*__restrict__\s+(\w+)", text))         # what a kernel reads only, and says so
    assert got == WEIGHTS.get(name, set())
    assert not re.search(r"\.nc\b", text)
