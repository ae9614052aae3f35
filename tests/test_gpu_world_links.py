"""The tree over all worlds' keys at the sizes where the per-world build changes course: a world's first and last nodes,
which reach other worlds by their numbers alone, worlds of one instance, world counts around powers of two, and the
counts (a CTA's threads) up to which the build's last CTA fits the inter-world nodes itself; against the oracle and, for uneven worlds
(empty ones among them), against the global tree of the same keys built here."""
import numpy as np
import pytest

import neraulgraphics_b200 as ng
import oracle as O

pytestmark = pytest.mark.gpu


def placed(rng, shape):
    q = rng.normal(size=shape + (4,))
    q /= np.linalg.norm(q, axis=-1, keepdims=True)
    flat = [ng.make_transform(p, k, 0.5).matrix for p, k in zip(rng.uniform(-3, 3, size=shape + (3,)).reshape(-1, 3),
                                                                q.reshape(-1, 4))]
    return np.array(flat, np.float32).reshape(shape + (3, 4))


@pytest.mark.parametrize("worlds,instances", [(1, 2), (2, 1), (3, 1), (7, 1), (64, 1), (127, 1), (128, 1), (129, 1), (1024, 1), (2047, 2), (2049, 1), (5, 2), (6, 3),
                                              (33, 5), (128, 3), (129, 3), (9, 31), (4, 32), (5, 33), (3, 64), (17, 100), (1500, 2),
                                              (3, 200), (2, 513), (128, 300), (129, 300), (129, 200)])
def test_batched_trees_are_the_oracles(worlds, instances):
    rng = np.random.default_rng(worlds * 1000 + instances)
    m = placed(rng, (worlds, instances))
    if instances > 2:
        m[0, 1] = m[0, 0]  # equal keys
    args = (8, 8, worlds, 1)
    kw = dict(meshes=[ng.make_box((0.4, 0.3, 0.2))], instances=[ng.Instance(0)] * instances)
    r = ng.BatchRenderer(*args, **kw)
    want = None
    for build in (1, 2, 1):  # twice: the counters are left as they were
        r.set_build(build)
        r.set_instance_transforms(m)
        r.synchronize()
        got = r.inspect_tlas()
        if want is None:
            o = O.Oracle(ng.SceneDesc(*args, **kw))
            o.set_instance_transforms(m)
            want = o.tlas()
        for name in ("keys", "sorted_ids", "nodes", "roots"):
            assert np.array_equal(got[name], np.asarray(want[name]).reshape(got[name].shape)), (name, build)


def radix_links(keys):
    """Children of the radix tree over sorted 64-bit keys, equal keys told apart by position, by plain recursion."""
    n = len(keys)
    links = np.zeros((n - 1, 2), np.int64)

    def prefix(i, j):
        return 64 + 32 - int(i ^ j).bit_length() if keys[i] == keys[j] else 64 - int(keys[i] ^ keys[j]).bit_length()

    for p in range(n - 1):
        at = lambda x: prefix(p, x) if 0 <= x < n else -1
        d = 1 if at(p + 1) > at(p - 1) else -1
        j = p
        while at(j + d) > at(p - d):
            j += d
        g = p
        while g + d != j and at(g + d) > at(j):
            g += d
        g += min(d, 0)
        lo, hi = min(p, j), max(p, j)
        links[p] = (n - 1 + g if lo == g else g), (n + g if hi == g + 1 else g + 1)
    return links


@pytest.mark.parametrize("counts", [[3, 0, 0, 5, 1, 1, 0, 40], [0, 7, 0], [1, 1], [2, 0, 0, 0, 0, 0, 0, 0, 1], [33] * 6,
                                    [0, 1, 2, 3, 4, 5, 6, 7, 8, 9, 0, 0, 12, 64, 200, 0]])
def test_uneven_trees_follow_their_keys(counts):
    rng = np.random.default_rng(len(counts))
    r = ng.UnevenBatchRenderer([(8, 8, [ng.Instance(0)] * c) for c in counts], meshes=[ng.make_box((0.4, 0.3, 0.2))],
                               lights=[ng.Light((0.0, 5.0, 0.0))])
    n = sum(counts)
    r.set_instance_transforms(placed(rng, (n,)))
    keys, ids = np.zeros(n, np.uint64), np.zeros(n, np.int32)
    nodes, roots, mats = np.zeros((2 * n - 1, 8), np.int32), np.zeros(len(counts), np.int32), np.zeros((n, 12), np.float32)
    import ctypes as C
    vp = lambda a: a.ctypes.data_as(C.c_void_p)
    assert r._lib.ngb_inspect_tlas(r._h, vp(keys), vp(ids), vp(nodes), vp(roots), vp(mats)) == 0
    k = [int(x) for x in keys[ids]]
    assert k == sorted(k)
    want = radix_links(k)
    assert np.array_equal(nodes[:n - 1, [3, 7]], want)
    # Every node's box is its children's.
    box = nodes.view(np.float32)[:, [0, 1, 2, 4, 5, 6]]
    l, h = box[want[:, 0]], box[want[:, 1]]
    assert np.array_equal(box[:n - 1], np.concatenate([np.minimum(l[:, :3], h[:, :3]), np.maximum(l[:, 3:], h[:, 3:])], 1))
