"""Shared memory of another CTA of a cluster may be touched only once that CTA is known to run, and nothing but a barrier of the
cluster says so.  Read from the sources, since a kernel without the barrier works nearly always."""

import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "lite_lang_b200", "csrc")


def _body(text, at):
    """The braces' contents from the first one at or behind ``at``."""
    start = text.index("{", at)
    depth = 0
    for i in range(start, len(text)):
        depth += (text[i] == "{") - (text[i] == "}")
        if depth == 0:
            return text[start:i + 1]
    raise AssertionError("no end")


def _text(name):
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name), encoding="utf-8").read())
    for inc in re.findall(r'#include "([^"]+\.cuh)"', text):
        text = _text(inc) + text
    return text


def _helpers(text, instruction):
    """Names of the device functions whose bodies hold ``instruction``."""
    out = set()
    for m in re.finditer(r"__device__ __forceinline__ \w+ (\w+)\(", text):
        if instruction in _body(text, m.end()):
            out.add(m.group(1))
    return out


FILES = sorted(f for f in os.listdir(CSRC) if f.endswith(".cu") and "mapa." in _text(f))


@pytest.mark.parametrize("name", FILES)
def test_a_barrier_of_the_cluster_comes_before_its_shared_memory(name):
    text = _text(name)
    peer = _helpers(text, "mapa.shared::cluster")
    waits = sorted(_helpers(text, "barrier.cluster.wait"))
    assert peer and waits
    wait = re.compile("|".join([r"barrier\.cluster\.wait"] + [rf"\b{w}\(" for w in waits]))
    seen = 0
    for m in re.finditer(r"__global__", text):
        body = _body(text, m.end())
        uses = [u.start() for u in re.finditer("|".join(rf"\b{p}\(" for p in sorted(peer)), body)]
        if not uses:
            continue
        seen += 1
        first = wait.search(body)
        assert first is not None and first.start() < uses[0], f"{name}: {body[max(0, uses[0] - 200):uses[0] + 60]}"
        if "barrier.cluster.wait" == first.group(0):      # a wait of its own: the arrival stands above it
            assert 0 <= body.find("barrier.cluster.arrive") < first.start()
    assert seen


def test_the_sources_with_such_kernels_are_found():
    assert {"attention_decode.cu", "attention_mma.cu", "gemm_f32.cu", "gemm_group.cu", "gemm_pair.cu", "latent_attention_mma.cu"} <= set(FILES)
