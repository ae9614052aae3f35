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
