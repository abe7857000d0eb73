"""Rules that the CUDA sources keep so that no launch can wait for ever; read from their text, without a GPU."""

import os
import re

import pytest

import ferrisinfer_b200

CSRC = os.path.join(os.path.dirname(ferrisinfer_b200.__file__), "csrc")


def kernels_with(word):
    """(file, kernel's name, body without comments) of every kernel whose body holds ``word``."""
    found = []
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith((".cu", ".cuh")):
            continue
        with open(os.path.join(CSRC, name)) as f:
            text = re.sub(r"//[^\n]*|/\*.*?\*/", "", f.read(), flags=re.S)
        for m in re.finditer(r"__global__", text):
            at = text.index("{", m.end())
            if ";" in text[m.end():at]:
                continue  # a declaration
            depth, end = 1, at + 1
            while depth:
                depth += {"{": 1, "}": -1}.get(text[end], 0)
                end += 1
            if word in text[at:end]:
                kernel = re.findall(r"(\w+)\s*\(", re.sub(r"__launch_bounds__\s*\((?:[^()]|\([^()]*\))*\)", "", text[m.end():at]))[0]
                found.append((name, kernel, text[at:end]))
    return found


def block_after(body, at):
    """What follows position ``at`` up to the end of the block that holds it."""
    depth, end = 0, at
    while depth >= 0:
        depth += {"{": 1, "}": -1}.get(body[end], 0)
        end += 1
    return body[at:end]


ALLOCATING = kernels_with("tmem_alloc")


def test_the_kernels_that_allocate_tensor_memory_are_found():
    assert {k for _, k, _ in ALLOCATING} == {"gemm_tcgen05_kernel", "gemm_tokens_m_kernel", "gemm_tokens_pair_kernel",
                                             "prefill_attention_tc5_kernel"}


@pytest.mark.parametrize("file, kernel, body", ALLOCATING, ids=[k for _, k, _ in ALLOCATING])
def test_tensor_memory_is_allocated_before_dependents_are_let_in(file, kernel, body):
    """A dependent launch that is let in first may take an SM's tensor memory and then wait for this one, which waits for
    the tensor memory: neither wait has a limit.  (A CTA that returns without allocating may let them in.)"""
    allocated = body.index("tmem_alloc")
    triggers = [m.start() for m in re.finditer(r"pdl_launch_dependents\(\)", body)]
    assert any(at > allocated for at in triggers)
    for at in triggers:
        if at < allocated:
            assert "return;" in block_after(body, at), f"{file}: {kernel} lets dependents in before it has its tensor memory"


def test_only_the_attention_of_listed_tokens_lets_the_next_launch_in_after_its_wait():
    """The attention of portions may run beside it without a wait of its own, which is safe only when the launches before have
    ended; every other launch behind this kernel waits by itself and is let in at once."""
    (_, _, body), = [k for k in kernels_with("LISTED") if k[1] == "decode_attention_kernel"]
    wait = body.index("pdl_wait();")
    assert "if (!LISTED) pdl_launch_dependents();" in body[:wait]
    assert body[wait:].split("pdl_wait();")[1].strip().startswith("if (LISTED) pdl_launch_dependents();")
