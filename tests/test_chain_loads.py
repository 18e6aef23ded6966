"""Kernels that start while their predecessors run (csrc/chain.cuh) read what
those write with chain_load only: the read-only path (__ldg, or const
__restrict__ parameters) is for the chain's inputs. Checked on the sources, as a
load that comes too early shows on the GPU only by chance."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "minimumlbvh_b200", "csrc")
INPUTS = {"tris", "off", "offsets"}  # triangles; mesh offsets
LOCAL = {"t": "a triangle", "t4": "the triangles", "q": "a triangle", "src": "the triangles"}


def functions(name):
    """(head, body) of every function of a source file, comments out."""
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
    return re.findall(r"\n((?:template|static|__global__|__device__)[^;{}]*?\([^;{}]*\)[^;{}]*)\{\n(.*?)\n\}", text, re.S)


@pytest.mark.parametrize("name", ["build.cu", "batch.cu", "ploc.cu", "onesweep.cuh", "tree.cuh", "climb.cuh"])
def test_read_only_loads_are_of_inputs(name):
    found = 0
    for head, body in functions(name):
        if "__global__" in head and "chain_begin()" not in body:  # no part of a chain
            continue
        found += 1
        wrong = set(re.findall(r"__ldg\(\s*(?:reinterpret_cast<[^>]*>\()?&?(\w+)", body)) - INPUTS - set(LOCAL)
        assert not wrong, (head, wrong)
        if "chain_begin()" in body:
            const = re.findall(r"const\s+[\w:]+\*\s*__restrict__\s+(\w+)", head)
            assert set(const) <= INPUTS, (head, const)
    assert found


def test_every_chained_kernel_waits_first():
    """A kernel that is launched chained calls chain_begin before any global access."""
    launched = set()
    for name in ("build.cu", "batch.cu", "ploc.cu", "tree.cuh"):
        launched |= set(re.findall(r"launch_chained\((k_\w+)", open(os.path.join(CSRC, name)).read()))
    launched |= {"k_onesweep"}
    assert launched >= {"k_keys", "k_tree_tiles", "k_tree_groups", "k_tree_cross", "k_ploc_init", "k_batch_keys"}
    seen = set()
    for name in ("build.cu", "batch.cu", "ploc.cu", "onesweep.cuh", "tree.cuh"):
        for head, body in functions(name):
            k = set(re.findall(r"\b(k_\w+)\s*\(", head)) & launched
            if k:
                seen |= k
                before = body[:body.index("chain_begin()")]
                assert not re.search(r"__ldc?g|chain_load|atomic|\*\s*reinterpret|\[blockIdx", before), head
    assert seen == launched
