"""The device mesh rebuild against the host build at the sizes where its kernel changes course: a warp's 32 items, the
256 triangles above which a node takes a CTA, a CTA's 512 threads, and bounds that are zeros of either sign."""
import numpy as np
import pytest

import neraulgraphics_b200 as ng

pytestmark = pytest.mark.gpu


def soup(rng, triangles, kind):
    """Separate triangles: spread, on a lattice (many equal centres and bounds that are -0 or +0), in clusters (places
    falling by powers of two, sizes not), or in a chain whose tree is deep and lopsided (places and sizes falling by
    powers of two, 120 of them)."""
    if kind == "lattice":
        c = rng.integers(-2, 3, size=(triangles, 1, 3)).astype(np.float32)
        v = c + rng.integers(-1, 2, size=(triangles, 3, 3))
        return np.where(rng.random(v.shape) < 0.5, -v, v).astype(np.float32) * np.float32(0.5) * rng.choice([-1.0, 1.0])
    c = rng.uniform(-1.0, 1.0, size=(triangles, 1, 3))
    if kind == "clusters":
        c = c * (0.5 ** (np.arange(triangles) % 40))[:, None, None]
    size = np.full(triangles, 0.02)
    if kind == "chain":
        fall = 0.5 ** np.linspace(0.0, 120.0, triangles)
        c, size = (c + 1.5) * fall[:, None, None], size * fall
    return (c + rng.normal(0.0, 1.0, size=(triangles, 3, 3)) * size[:, None, None]).astype(np.float32)


def depth(nodes):
    """The tree's depth, the root's children at 1 (a node's words: lo.xyz, first child or triangle, hi.xyz, count)."""
    deepest, level, below = 0, [0], []
    while level:
        below = [c for n in level if nodes[n, 7] == 0 for c in (nodes[n, 3], nodes[n, 3] + 1)]
        deepest, level = deepest + bool(below), below
    return deepest


@pytest.mark.parametrize("kind", ["spread", "lattice", "clusters", "chain"])
@pytest.mark.parametrize("triangles", [1, 2, 5, 31, 32, 33, 64, 255, 256, 257, 513, 1500, 5000, 12000])
def test_rebuilt_tree_is_the_hosts(triangles, kind):
    rng = np.random.default_rng(triangles)
    first, second = soup(rng, triangles, "spread"), soup(rng, triangles, kind)
    index = np.arange(3 * triangles, dtype=np.uint32)
    r = ng.BatchRenderer(8, 8, 1, 1, meshes=[ng.Mesh(first.reshape(-1, 3), index)], instances=[ng.Instance(0)])
    r.update_mesh(0, second.reshape(-1, 3))
    got = r.inspect_mesh(0)
    want = ng.build_meshes([ng.Mesh(second.reshape(-1, 3), index)])
    if kind == "chain" and triangles >= 1500:  # to the deepest levels (the builds stop at 60)
        assert depth(want["nodes"].reshape(-1, 8)) >= (60 if triangles == 12000 else 45)
    for name in ("nodes", "triangle_index"):
        assert np.array_equal(got[name], want[name]), name
    for name in ("triangles", "bounds"):
        assert np.array_equal(got[name].view(np.uint32), want[name].view(np.uint32)), name
