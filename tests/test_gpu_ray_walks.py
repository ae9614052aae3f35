"""Ray queries by warp packets and by lanes walking alone (the default picks per warp by how its rays look) against the
per-thread kernel, which walks each ray in the reference's way: the same hits, but for rays with two surfaces within
rounding of each other (packets visit a world's instances in another order; under one ray in 10,000)."""
import numpy as np
import pytest

import neraulgraphics_b200 as ng

pytestmark = pytest.mark.gpu


def renderer(worlds, instances, rng):
    meshes = [ng.make_icosphere(0.5, 2), ng.make_box((0.4, 0.4, 0.4)), ng.cylinder(0.4, 0.5, 24)]
    r = ng.BatchRenderer(16, 16, worlds, 1, spheres=[ng.Sphere((0.3, 0.4, 0.0), 0.3)],
                         floor=ng.Plane(y=-2.0, half_extent_x=5.0, z_min=-5.0, z_max=5.0), meshes=meshes,
                         instances=[ng.Instance(i % 3) for i in range(instances)])
    if instances:
        q = rng.normal(size=(worlds, instances, 4))
        pos = rng.uniform(-2.0, 2.0, size=(worlds, instances, 3)) * max(1.0, (instances / 20.0) ** (1.0 / 3.0))
        r.set_instance_transforms(np.stack([[ng.make_transform(p, k / np.linalg.norm(k), 0.6).matrix for p, k in zip(ps, qs)]
                                            for ps, qs in zip(pos, q)]).astype(np.float32))
    return r


def directions(kind, worlds, rays, rng):
    scan = 2.0 * np.pi * np.arange(rays) / max(rays, 700)
    d = np.broadcast_to(np.stack([np.cos(scan), 0.1 * np.ones(rays), np.sin(scan)], -1), (worlds, rays, 3)).copy()
    if kind == "all ways":
        d = rng.normal(size=(worlds, rays, 3))
    elif kind == "mixed":  # some warps of either kind, and rays that are misses for their length
        d[:, rays // 2:] = rng.normal(size=(worlds, rays - rays // 2, 3))
        d[:, ::7] = 0.0
        d[:, 3::11] *= 1e20
    return d.astype(np.float32)


@pytest.mark.parametrize("kind", ["scan", "all ways", "mixed"])
@pytest.mark.parametrize("worlds,instances,rays", [(3, 0, 40), (3, 1, 33), (5, 20, 1), (4, 20, 31), (2, 20, 700),
                                                   (2, 60, 129), (1, 300, 500)])
def test_default_walks_give_the_per_thread_kernels_hits(worlds, instances, rays, kind):
    rng = np.random.default_rng(rays)
    r = renderer(worlds, instances, rng)
    origins = rng.uniform(-1.0, 1.0, size=(worlds, rays, 3)).astype(np.float32)
    if kind == "scan":
        origins[:] = origins[:, :1]
    d = directions(kind, worlds, rays, rng)
    got = r.cast_rays(origins, d, 6.0)
    r.set_ray_kernel(1)
    want = r.cast_rays(origins, d, 6.0)
    for name in want:
        differ = (got[name] != want[name]).reshape(worlds * rays, -1).any(-1).sum()
        assert differ <= worlds * rays * 1e-4, (name, differ)


@pytest.mark.parametrize("rays,dead", [(7, ()), (16, ()), (48, ()), (32, (16,)), (31, (16, 20)), (2, ())])
def test_the_walk_does_not_depend_on_where_a_sensor_faces(rays, dead):
    """Two meshes share a square; rays from the left enter the first's box before the second's, rays from the right the
    other way round. Which of the two coincident surfaces a ray reports shows which walk its warp took, so a scene
    turned round, sensor and all, has to report the same ones."""
    square = np.array([(-1, -1, -1), (1, -1, -1), (1, 1, -1), (-1, 1, -1)], np.float32)
    fins = [np.array([(s * 3, 0.9, 0), (s * 3, 0.8, 0), (s * 3, 0.9, -0.1)], np.float32) for s in (-1, 1)]
    index = np.array([0, 1, 2, 0, 2, 3, 4, 5, 6], np.uint32)
    side = np.where(np.arange(rays) % 3 == 2, 1.0, -1.0)  # two rays in three from the left
    o = np.stack([2.2 * side, np.linspace(-0.4, 0.4, rays), np.ones(rays)], -1)[None].astype(np.float32)
    d = np.stack([-0.6 * side, np.zeros(rays), np.full(rays, -0.8)], -1)[None].astype(np.float32)
    d[:, list(dead)] = 0.0
    found = []
    for turn in (1.0, -1.0):  # half a turn about y
        t = np.array([turn, 1.0, turn], np.float32)
        r = ng.BatchRenderer(8, 8, 1, 1, meshes=[ng.Mesh(np.concatenate([square, f]) * t, index) for f in fins],
                             instances=[ng.Instance(0), ng.Instance(1)])
        found.append(r.cast_rays(o * t, d * t, 10.0))
    live = ~np.isin(np.arange(rays), dead)
    assert np.isfinite(found[0]["distance"][0]).tolist() == live.tolist()
    assert np.array_equal(found[0]["distance"], found[1]["distance"])
    assert np.array_equal(found[0]["object_id"], found[1]["object_id"])


def crowd(worlds, rays):
    import torch
    rng = np.random.default_rng(worlds + rays)
    r = ng.BatchRenderer(8, 8, worlds, 1, meshes=[ng.make_icosphere(0.5, 1)], instances=[ng.Instance(0)] * 2)
    m = np.zeros((worlds, 2, 3, 4), np.float32)
    m[..., [0, 1, 2], [0, 1, 2]] = 1.0
    m[..., 3] = rng.uniform(-1.5, 1.5, size=(worlds, 2, 3))
    r.set_instance_transforms(m)
    d = rng.normal(size=(worlds, rays, 3)).astype(np.float32)
    return r, torch.from_numpy(np.zeros_like(d)).cuda(), torch.from_numpy(d).cuda()


@pytest.mark.parametrize("worlds,rays", [(32768, 4), (32769, 4), (32769, 5), (40961, 5), (65536, 9)])
def test_many_worlds_of_few_rays_give_the_per_thread_kernels_hits(worlds, rays):
    import torch
    r, o, d = crowd(worlds, rays)
    got = r.cast_rays(o, d, 5.0)
    r.set_ray_kernel(1)
    want = r.cast_rays(o, d, 5.0)
    torch.cuda.synchronize()
    assert int(torch.isfinite(want["distance"]).sum()) > worlds * rays // 20
    for name in want:
        differ = (got[name] != want[name]).reshape(worlds * rays, -1).any(-1).sum().item()
        assert differ <= worlds * rays * 1e-4, (name, differ)


def test_many_worlds_of_one_ray_take_no_longer_than_on_the_persistent_kernel():
    r, o, d = crowd(262144, 1)
    ms = {}
    for kernel in (0, 2, 0, 2):
        r.set_ray_kernel(kernel)
        for _ in range(5):
            r.cast_rays(o, d, 5.0)
            r.synchronize()
            ms[kernel] = min(r.last_kernel_ms, ms.get(kernel, 1e9))
    assert ms[0] <= 1.5 * ms[2], ms  # packets of one ray each: 3.8 times
