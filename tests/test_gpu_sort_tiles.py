"""The sort passes of the build at the edges of their small tiles (1024 keys)
and of the size where the large ones (4096) take over, against the oracle's
stable order, bit for bit."""
import numpy as np
import pytest

import _gpu as G
import _oracle as O
from minimumlbvh_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [33, 1023, 1024, 1025, 4 * 1024 + 1, 9 * 1024 - 1, 454_655, 454_656, 454_657])
def test_sorted_keys_and_order(cuda, n):
    tris = scenes.gaussian_soup(n, clusters=5, seed=n)
    tris[n // 3: n // 2] = tris[n // 3]  # equal keys: the order of the indices shows
    for option in (0, 1):
        _, _, out = G.build(tris, option)
        keys, idx = out["keys"].copy(), out["indices"].copy()
        ref = O.build(tris, option)
        np.testing.assert_array_equal(keys, ref["keys"])
        np.testing.assert_array_equal(idx, ref["indices"])
