"""The device mesh rebuild against the host build at the sizes where its kernel changes course: a warp's 32 items, the
256 triangles above which a node takes a CTA, a CTA's 512 threads, and bounds that are zeros of either sign."""
import numpy as np
import pytest

import neraulgraphics_b200 as ng

pytestmark = pytest.mark.gpu


def soup(rng, triangles, kind):
    """Separate triangles: spread, on a lattice (many equal centres and bounds that are -0 or +0), or in a chain whose
    tree is deep and lopsided (sizes falling by powers of two)."""
    if kind == "lattice":
        c = rng.integers(-2, 3, size=(triangles, 1, 3)).astype(np.float32)
        v = c + rng.integers(-1, 2, size=(triangles, 3, 3))
        return np.where(rng.random(v.shape) < 0.5, -v, v).astype(np.float32) * np.float32(0.5) * rng.choice([-1.0, 1.0])
    c = rng.uniform(-1.0, 1.0, size=(triangles, 1, 3))
    if kind == "chain":
        c = c * (0.5 ** (np.arange(triangles) % 40))[:, None, None]
    return (c + rng.normal(0.0, 0.02, size=(triangles, 3, 3))).astype(np.float32)


@pytest.mark.parametrize("kind", ["spread", "lattice", "chain"])
@pytest.mark.parametrize("triangles", [1, 2, 5, 31, 32, 33, 64, 255, 256, 257, 513, 1500, 5000])
def test_rebuilt_tree_is_the_hosts(triangles, kind):
    rng = np.random.default_rng(triangles)
    first, second = soup(rng, triangles, "spread"), soup(rng, triangles, kind)
    index = np.arange(3 * triangles, dtype=np.uint32)
    r = ng.BatchRenderer(8, 8, 1, 1, meshes=[ng.Mesh(first.reshape(-1, 3), index)], instances=[ng.Instance(0)])
    r.update_mesh(0, second.reshape(-1, 3))
    got = r.inspect_mesh(0)
    want = ng.build_meshes([ng.Mesh(second.reshape(-1, 3), index)])
    for name in ("nodes", "triangle_index"):
        assert np.array_equal(got[name], want[name]), name
    for name in ("triangles", "bounds"):
        assert np.array_equal(got[name].view(np.uint32), want[name].view(np.uint32)), name
