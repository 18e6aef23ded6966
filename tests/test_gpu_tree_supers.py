"""A tree of more than 32 supers (csrc/tree.cuh: 8,388,608 leaves), whose top
nodes' ranges cross blocks of the top level, against the oracle."""
import pytest

import _gpu as G
import _oracle as O
from minimumlbvh_b200 import scenes

pytestmark = pytest.mark.gpu


def test_more_than_32_supers(cuda):
    tris = scenes.gaussian_soup(8_650_000, clusters=64, seed=9)
    _, _, out = G.build(tris)
    G.assert_build_equal(out, O.build(tris))
