"""Scratch sizes never fall as n grows, so scratch sized for the largest scene
serves every smaller one: at the edges of the sort's small tiles (454,656
keys) and of the PLOC build's (151,552 clusters)."""
import minimumlbvh_b200 as mb


def test_scratch_sizes_grow_with_n():
    L = mb.lib()
    sizes = sorted({m + d for m in (1024, 4096, 8192, 65536, 151552, 262144, 398977, 454656, 500000, 517888, 524288,
                                    1 << 20, 1 << 25) for d in (-1, 0, 1)})
    for f in (L.mlbvh_build_scratch_bytes, L.mlbvh_build_ploc_scratch_bytes):
        got = [f(n) for n in sizes]
        assert got == sorted(got), [(n, s) for n, s, t in zip(sizes, got, got[1:]) if t < s]
