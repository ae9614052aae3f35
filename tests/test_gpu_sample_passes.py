"""Pictures of several samples, lights or mirrors on the tile kernels (sample passes) against the per-pixel kernel, which
runs the reference's loop for each pixel: the arithmetic and its order are the same, so the images are, but for pixels
with two surfaces within rounding of each other along a ray (the walks visit a world's instances in other orders; under
one pixel in 10,000)."""
import numpy as np
import pytest

import neraulgraphics_b200 as ng

pytestmark = pytest.mark.gpu

LIGHTS = [ng.Light((-3.0 + i, 6.0, 4.0 - 2.0 * i), 0.5 + 0.1 * i, 0.1 * i, spot_angle=0.9 if i == 3 else 0.0,
                   direction=(0.0, -1.0, -0.5), falloff=6.0 if i == 2 else 0.0, color=(1.0, 0.8, 0.5 + 0.1 * i))
          for i in range(8)]


def scene(worlds, instances, lights, mirror, width, height, cameras=1, seed=0):
    rng = np.random.default_rng(seed)
    meshes = [ng.make_icosphere(0.5, 2), ng.make_box((0.4, 0.4, 0.4)), ng.cylinder(0.4, 0.5, 24)]
    mat = [ng.Material(diffuse_color=(0.8, 0.3, 0.2)), ng.Material(reflectivity=0.6 if mirror else 0.0),
           ng.Material(diffuse_color=(0.2, 0.4, 0.9), specular_exponent=5.0)]
    inst = [ng.Instance(i % 3, material=mat[i % 3]) for i in range(instances)]
    r = ng.BatchRenderer(width, height, worlds, cameras,
                         spheres=[ng.Sphere((0.5, 0.5, 0.0), 0.4, ng.Material(reflectivity=0.3 if mirror else 0.0))],
                         lights=LIGHTS[:lights], floor=ng.Plane(y=-1.5, half_extent_x=5.0, z_min=-5.0, z_max=5.0),
                         meshes=meshes, instances=inst)
    if instances:
        q = rng.normal(size=(worlds, instances, 4))
        q /= np.linalg.norm(q, axis=-1, keepdims=True)
        spread = 1.2 * max(1.0, (instances / 8.0) ** (1.0 / 3.0))
        mats = np.stack([[ng.make_transform(p, k, 0.6).matrix for p, k in zip(ps, ks)]
                         for ps, ks in zip(rng.uniform(-spread, spread, size=(worlds, instances, 3)), q)])
        r.set_instance_transforms(mats.astype(np.float32))
    r.ambient = 0.1
    eye = rng.uniform(-0.5, 0.5, size=(worlds * cameras, 3)) + np.array([0.0, 1.0, 4.0])
    return r, ng.look_at(eye, np.zeros(3), up=(0.0, 1.0, 0.0))


def images(r, cams, kernel, spp, **outputs):
    r.set_tuning(kernel=kernel, threads_per_block=128, registers=64)
    return r.render(cams, 1.0, spp, frame=3, **outputs)


@pytest.mark.parametrize("spp,lights,mirror,instances,worlds,width,height,cameras", [
    (2, 1, False, 5, 3, 33, 17, 1),       # ragged tiles
    (1, 2, False, 8, 2, 40, 40, 2),       # lights alone, two cameras
    (1, 1, True, 8, 2, 40, 40, 1),        # mirrors alone
    (3, 0, True, 6, 2, 21, 30, 1),        # no light
    (5, 8, True, 8, 1, 37, 23, 1),        # every light
    (2, 2, True, 0, 2, 24, 24, 1),        # spheres and the floor alone
    (2, 2, True, 1, 2, 24, 24, 1),
    (2, 2, True, 40, 2, 48, 32, 1),       # lists above 32
    (2, 2, True, 300, 1, 64, 48, 1),      # a world walked as packets
])
def test_passes_give_the_per_pixel_kernels_images(spp, lights, mirror, instances, worlds, width, height, cameras):
    r, cams = scene(worlds, instances, lights, mirror, width, height, cameras)
    outputs = dict(rgb=True, depth=True, normals=True, object_ids=True)
    want = images(r, cams, 1, spp, **outputs)
    got = images(r, cams, 0, spp, **outputs)
    pixels = want["depth"].size
    for name in outputs:
        differ = (got[name] != want[name]).reshape(pixels, -1).any(-1).sum()
        assert differ <= pixels * 1e-4, (name, differ, pixels)
    assert np.array_equal(images(r, cams, 0, spp, rgb=True)["rgb"], got["rgb"])  # unpaired tiles
    alone = images(r, cams, 0, spp, rgb=False, depth=True)["depth"]
    assert np.array_equal(alone.view(np.uint32), got["depth"].view(np.uint32))
    r.set_rows(5, 8)
    band = images(r, cams, 0, spp, rgb=True)["rgb"]
    assert np.array_equal(band, got["rgb"][:, 5:13])


def test_a_capture_without_a_render_before_it_takes_the_kernel_that_needs_no_scratch():
    import torch
    r, cams = scene(2, 6, 2, True, 32, 32)
    dev = torch.from_numpy(cams).cuda()
    into = {"rgb": torch.zeros((2, 32, 32, 3), dtype=torch.uint8, device="cuda")}
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        r.render(dev, 1.0, 2, frame=3, rgb=True, into=into)
    g.replay()
    torch.cuda.synchronize()
    want = images(r, cams, 0, 2, rgb=True)["rgb"]
    differ = (into["rgb"].cpu().numpy() != want).any(-1).sum()
    assert differ <= 2 * 32 * 32 * 1e-3


def test_a_captured_render_outlives_renders_of_more_samples():
    import torch
    r, cams = scene(2, 6, 2, True, 32, 32)
    dev = torch.from_numpy(cams).cuda()
    into = {"rgb": torch.zeros((2, 32, 32, 3), dtype=torch.uint8, device="cuda")}
    r.render(dev, 1.0, 2, frame=3, rgb=True, into=into)
    torch.cuda.synchronize()
    want = into["rgb"].clone()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        r.render(dev, 1.0, 2, frame=3, rgb=True, into=into)
    r.render(dev, 1.0, 9, frame=1, rgb=True, into=into)
    into["rgb"].zero_()
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(into["rgb"], want)


@pytest.mark.parametrize("lights,rgb", [(1, True), (0, True), (1, False)])
def test_stage_times_of_one_pass(lights, rgb):
    r, cams = scene(4, 8, lights, False, 64, 64)
    for _ in range(2):
        r.render(cams, 1.0, 1, rgb=rgb, depth=True)
        stages = r.last_stage_ms
        assert len(stages) == 3 and stages[0] > 0.0 and (stages[1] > 0.0) == rgb and (stages[2] > 0.0) == (rgb and lights == 1)
        assert abs(sum(stages) - r.last_kernel_ms) <= 1e-5 and r.last_kernel_ms < 50.0


def test_times_read_while_the_render_runs_are_whole():
    import torch
    r, cams = scene(64, 8, 1, False, 64, 64)
    dev = torch.from_numpy(cams).cuda()
    into = {"rgb": torch.zeros((64, 64, 64, 3), dtype=torch.uint8, device="cuda")}
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    for _ in range(200):
        with torch.cuda.stream(stream):
            r.render(dev, 1.0, 1, rgb=True, into=into)
        stages, ms = r.last_stage_ms, r.last_kernel_ms  # a poll that may meet the last warp's writes
        assert len(stages) == 3 and min(stages) > 0.0 and abs(sum(stages) - ms) <= 1e-5 and ms < 50.0


@pytest.mark.parametrize("spp", [1, 2])
def test_a_capture_keeps_the_times_of_the_render_before_it(spp):
    import torch
    r, cams = scene(4, 8, 1, False, 64, 64)
    dev = torch.from_numpy(cams).cuda()
    into = {"rgb": torch.zeros((4, 64, 64, 3), dtype=torch.uint8, device="cuda")}
    r.render(dev, 1.0, spp, rgb=True, into=into)
    torch.cuda.synchronize()
    r.render(dev, 1.0, 1, rgb=True, into=into)
    want = r.last_stage_ms, r.last_kernel_ms
    assert len(want[0]) == 3
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        r.render(dev, 1.0, spp, rgb=True, into=into)
    g.replay()
    torch.cuda.synchronize()
    assert (r.last_stage_ms, r.last_kernel_ms) == want
    del g


@pytest.mark.parametrize("instances,worlds,size,coarse", [(8, 1, 8, True), (8, 1, 9, False), (256, 4, 15, True),
                                                          (256, 4, 16, False), (257, 2, 25, True), (257, 2, 26, False),
                                                          (300, 56, 24, True), (300, 57, 24, False)])
def test_coarse_pictures_take_the_per_pixel_kernel(instances, worlds, size, coarse):
    r, cams = scene(worlds, instances, 2, True, size, size)
    want = images(r, cams, 1, 2, rgb=True, depth=True)
    before = ng.device_bytes()
    got = images(r, cams, 0, 2, rgb=True, depth=True)
    pixels = worlds * size * size
    if coarse:  # it needs no scratch
        assert ng.device_bytes() == before
        assert all(np.array_equal(got[k], want[k]) for k in want)
    else:
        assert ng.device_bytes() - before >= 70 * pixels
        for k in want:
            differ = (got[k] != want[k]).reshape(pixels, -1).any(-1).sum()
            assert differ <= max(pixels * 1e-4, 1), (k, differ)
    tuned = images(r, cams, 3, 2, rgb=True, depth=True)  # the tile kernels' shape chosen, as autotune does
    assert all(np.array_equal(tuned[k], got[k]) for k in want)
    assert (ng.device_bytes() == before) == coarse
    # A band of rows takes the whole image's kernel.
    r, cams = scene(worlds, instances, 2, True, size, size)
    r.set_rows(4, 4)
    images(r, cams, 1, 2, rgb=True, depth=True)
    before = ng.device_bytes()
    band = images(r, cams, 0, 2, rgb=True, depth=True)
    assert (ng.device_bytes() == before) == coarse
    assert all(np.array_equal(band[k], got[k][:, 4:8]) for k in band)
