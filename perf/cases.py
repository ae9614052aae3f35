"""The work that programs have this framework do, as measurable cases.

Each case is one call sequence through the public entry points, at a size from the repository's own workloads,
tests and benchmark or a generic one:

- frame: a batch of worlds placed (matrices, body poses or geom poses, as simulators hand them over) and
  rendered, from 16 small worlds to the 4096-world headline, with one or several cameras per world, odd image
  sizes, colour or depth and normals alone, and multi-sample renders with two lights and mirrors;
- uneven: worlds of different instance counts and image sizes in one renderer;
- large: one world of up to 100,000 instances rendered and swept by a LiDAR;
- rays: range sensors in every world of a batch (cast_rays);
- gradient: differentiable depth and normals, forward and backward, from poses to pose gradients;
- mesh: a deformable mesh whose vertices move every step, its tree rebuilt on the GPU, then a render;
- view: a single-view renderer averaging frames of a scene.

Inputs follow the seeded distributions of neraulgraphics_b200.workloads (body_worlds, icosphere_worlds,
uneven_worlds, large_world, differentiable_worlds), drawn here with numpy so that many can be made quickly.
`exact` restates what the calls return (depth, normals, distances, gradients) by brute force in 64 bits with
plain torch: every ray against every triangle of every instance it can meet.
"""

import functools
import math

import numpy as np
import torch

import neraulgraphics_b200 as ng
from neraulgraphics_b200 import autodiff

INF = float("inf")


def listed():
    frame = {"kind": "frame", "cameras": 1, "spp": 1, "lights": 1, "mirror": False}
    return [
        # A handful of environments while developing: the smallest call, where launches and host work count
        # (icosphere_worlds, the first configuration of the benchmark).
        dict(frame, name="frame_small", place="matrices", worlds=16, bodies=8, width=64, height=64,
             outputs="rgb depth object_ids"),
        # The headline: vision for reinforcement learning over 4096 environments (body_worlds).
        dict(frame, name="frame_bodies", place="bodies", worlds=4096, bodies=20, width=64, height=64,
             outputs="rgb depth object_ids"),
        # Depth-and-normal observations from two cameras per environment, odd image sizes and counts.
        dict(frame, name="frame_depth", place="bodies", worlds=1023, bodies=13, width=75, height=53, cameras=2,
             outputs="depth normals"),
        # Cluttered environments whose poses come from a MuJoCo-style simulator's geoms.
        dict(frame, name="frame_geoms", place="geoms", worlds=512, bodies=120, width=80, height=60,
             outputs="rgb depth"),
        # Better pictures: four samples per pixel, two lights, some mirrors (as the tests' template scene).
        dict(frame, name="frame_samples", place="bodies", worlds=96, bodies=20, width=96, height=96, spp=4, lights=2,
             mirror=True, outputs="rgb depth object_ids"),
        # Curricula and domain randomisation: every world its own size (uneven_worlds).
        {"name": "uneven", "kind": "uneven", "worlds": 640, "most": 200},
        # One big outdoor-like world, a camera frame and a LiDAR sweep per step (large_world).
        {"name": "large", "kind": "large", "instances": 100_000, "width": 1280, "height": 720, "beams": 64,
         "azimuths": 2048},
        # A planar-and-tilted range sensor in each of 1024 environments.
        {"name": "rays", "kind": "rays", "worlds": 1024, "bodies": 20, "beams": 720},
        # Pose estimation by gradient descent on depth and normals (differentiable_worlds).
        {"name": "gradient", "kind": "gradient", "worlds": 1024, "bodies": 12, "width": 128, "height": 128,
         "normals": True},
        # A soft body of 5120 triangles in every world, rebuilt each step.
        {"name": "mesh", "kind": "mesh", "subdivisions": 4, "worlds": 64, "bodies": 6, "width": 64, "height": 64},
        # An interactive viewer: two averaged frames of a 2000-instance scene with its depth and IDs.
        {"name": "view", "kind": "view", "instances": 2000, "width": 1280, "height": 720, "frames": 2},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame"] * 5 + ["uneven", "large", "rays", "gradient", "mesh", "view"])
    if kind == "frame":
        spp = rng.choice([1, 1, 1, 1, 2, 3])
        lights = rng.choice([1, 1, 1, 1, 0, 2])
        mirror = rng.random() < 0.15
        plain = spp == 1 and lights <= 1 and not mirror
        most = 8_000_000 if plain else 600_000 // spp
        width, height, cameras = _log(rng, 17, 200), _log(rng, 17, 200), rng.choice([1, 1, 1, 2, 3])
        bodies = _log(rng, 1, 40) if rng.random() < 0.8 else _log(rng, 40, 250)
        if bodies > 40:
            most //= 3
        worlds = _log(rng, 1, max(1, min(4096, most // (width * height * cameras))))
        return {"kind": kind, "place": rng.choice(["matrices", "bodies", "bodies", "geoms"]), "worlds": worlds,
                "bodies": bodies, "width": width, "height": height, "cameras": cameras, "spp": spp, "lights": lights,
                "mirror": mirror, "outputs": rng.choice(["rgb depth object_ids", "rgb depth object_ids", "rgb",
                                                         "rgb depth", "depth", "depth normals",
                                                         "rgb depth normals object_ids"])}
    if kind == "uneven":
        return {"kind": kind, "worlds": _log(rng, 3, 400), "most": _log(rng, 4, 200)}
    if kind == "large":
        return {"kind": kind, "instances": _log(rng, 300, 60_000), "width": _log(rng, 160, 1280),
                "height": _log(rng, 120, 720), "beams": _log(rng, 1, 64), "azimuths": _log(rng, 90, 2048)}
    if kind == "rays":
        return {"kind": kind, "worlds": _log(rng, 1, 1024), "bodies": _log(rng, 1, 60), "beams": _log(rng, 7, 720)}
    if kind == "gradient":
        return {"kind": kind, "worlds": _log(rng, 1, 512), "bodies": _log(rng, 1, 24), "width": _log(rng, 24, 128),
                "height": _log(rng, 24, 128), "normals": rng.random() < 0.5}
    if kind == "mesh":
        return {"kind": kind, "subdivisions": rng.choice([1, 2, 3, 4]), "worlds": _log(rng, 1, 64),
                "bodies": _log(rng, 1, 12), "width": _log(rng, 17, 100), "height": _log(rng, 17, 100)}
    return {"kind": kind, "instances": _log(rng, 2, 2000), "width": _log(rng, 160, 1280), "height": _log(rng, 120, 720),
            "frames": rng.choice([1, 2])}


# ------------------------------------------------------------------------------------------------- inputs --

PALETTE = [(0.80, 0.25, 0.20), (0.20, 0.55, 0.80), (0.25, 0.70, 0.30), (0.85, 0.75, 0.20), (0.60, 0.30, 0.75),
           (0.90, 0.50, 0.15), (0.30, 0.75, 0.70), (0.75, 0.75, 0.75)]
LIGHTS = [ng.Light((-10.0, 20.0, 10.0), 1.6, 1.0), ng.Light((6.0, 9.0, -5.0), 0.8, 0.5, color=(1.0, 0.9, 0.7))]


@functools.lru_cache(maxsize=None)
def _mesh(name):
    """The workloads' meshes (geometry only, the same for every seed)."""
    if name == "box":
        return ng.make_box((0.4, 0.4, 0.4))
    if name == "cylinder":
        return ng.cylinder(1.0, 1.0, 128)
    m = ng.make_icosphere(0.5, int(name[3]))
    if name.endswith("smooth"):
        return ng.Mesh(m.vertices, m.triangles, normals=m.vertices / 0.5)
    return m


@functools.lru_cache(maxsize=None)
def _instance(mesh, colour, mirror=False):
    return ng.Instance(mesh, material=ng.Material(diffuse_color=PALETTE[colour], reflectivity=0.35 if mirror else 0.0))


def _quaternions(rng, *shape):
    q = rng.normal(size=shape + (4,))
    return q / np.linalg.norm(q, axis=-1, keepdims=True)


def _rotation(q):
    x, y, z, w = np.moveaxis(q, -1, 0)
    r = np.stack([1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w),
                  2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w),
                  2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)], -1)
    return r.reshape(q.shape[:-1] + (3, 3))


def _matrices(pos, q, scale):
    return np.concatenate([_rotation(q) * scale[..., None, :], pos[..., None]], -1).astype(np.float32)


def _ring(rng, n, radius, height):
    a = 2.0 * np.pi * (np.arange(n) / n + rng.uniform())
    r, h = np.broadcast_to(radius, n), np.broadcast_to(height, n)
    return ng.look_at(np.stack([r * np.cos(a), h, r * np.sin(a)], -1), np.zeros(3), up=(0.0, 1.0, 0.0))


def _scales(rng, names, shape=()):
    """Per instance: uniform 0.6 to 1.2, the cylinders squeezed to the other meshes' size."""
    s = np.repeat(rng.uniform(0.6, 1.2, size=shape + (len(names), 1)), 3, axis=-1)
    s[..., [n == "cylinder" for n in names], :] *= np.array([0.3, 0.3, 0.5])
    return s


def _inputs(case, seed):
    """Everything a case's calls read, as numpy arrays and scene objects, from the seed alone."""
    rng = np.random.default_rng(seed)
    k = {"floor": ng.Plane(y=-2.5, half_extent_x=8.0, z_min=-8.0, z_max=8.0, checker_scale=1.0), "lights": LIGHTS[:1]}
    kind = case["kind"]
    W = case.get("worlds", 1)
    if kind in ("frame", "rays"):
        P = case["bodies"]
        icospheres = case.get("place") == "matrices"
        k["meshes"] = ["ico2"] if icospheres else ["ico3", "box", "cylinder"]
        M = len(k["meshes"])
        k["slot"] = [i % M for i in range(P)]
        k["instances"] = [_instance(i % M, i % 8, case.get("mirror", False) and i % 5 == 2) for i in range(P)]
        k["lights"] = LIGHTS[:case.get("lights", 1)]
        names = [k["meshes"][m] for m in k["slot"]]
        spread = 2.0 * max(1.0, (P / 20.0) ** (1.0 / 3.0))  # the density of body_worlds
        pos, q = rng.uniform(-spread, spread, size=(W, P, 3)), _quaternions(rng, W, P)
        scale = _scales(rng, names)
        k["cameras"] = _ring(rng, W * case.get("cameras", 1), 2.0 * spread, spread / 2.0)
        place = case.get("place", "bodies")
        if place == "bodies":
            k["local"] = np.concatenate([rng.uniform(-0.1, 0.1, size=(P, 3)), _quaternions(rng, P)], -1).astype(np.float32)
            k["scale"] = scale.astype(np.float32)
            k["poses"] = np.concatenate([pos, q], -1).astype(np.float32)
            lp, bp = k["local"].astype(np.float64), k["poses"].astype(np.float64)
            unit = lambda v: v / np.linalg.norm(v, axis=-1, keepdims=True)  # noqa: E731
            rb, rl = _rotation(unit(bp[..., 3:])), _rotation(unit(lp[..., 3:]))
            r = rb @ rl * k["scale"].astype(np.float64)[:, None, :]
            k["exact_matrices"] = np.concatenate([r, (bp[..., :3] + (rb @ lp[..., :3, None])[..., 0])[..., None]], -1)
        elif place == "geoms":
            k["scale"] = scale.astype(np.float32)
            k["xpos"], k["xmat"] = pos.astype(np.float32), _rotation(q).astype(np.float32)
            k["exact_matrices"] = np.concatenate([k["xmat"].astype(np.float64) * k["scale"].astype(np.float64)[:, None, :],
                                                  k["xpos"].astype(np.float64)[..., None]], -1)
        else:
            k["matrices"] = _matrices(pos, q, np.broadcast_to(scale, (W, P, 3)))
        if kind == "rays":
            R = case["beams"]
            az = 2.0 * np.pi * np.arange(R) / R
            el = np.radians(np.where(np.arange(R) % 2, -12.0, 3.0))
            d = np.stack([np.cos(el) * np.cos(az), np.sin(el), np.cos(el) * np.sin(az)], -1)
            k["origins"] = np.broadcast_to(rng.uniform(-1.0, 1.0, size=(W, 1, 3)), (W, R, 3)).astype(np.float32)
            k["directions"] = np.broadcast_to(d, (W, R, 3)).astype(np.float32)
    elif kind == "uneven":
        k["meshes"] = ["box", "ico2", "cylinder", "ico3", "ico4", "ico5"]
        spread = np.random.default_rng(7 * W + case["most"])  # the worlds' sizes are the case's, the same for every seed
        counts = spread.integers(1, case["most"] + 1, size=W)
        sizes = np.array([32, 64, 128])[spread.integers(0, 3, size=W)]
        k["worlds"] = [(int(s), int(s), [_instance(i % 6, i % 8) for i in range(c)]) for s, c in zip(sizes, counts)]
        r = 2.0 * (counts / 20.0) ** (1.0 / 3.0)
        n = int(counts.sum())
        each = np.repeat(r, counts)[:, None]
        within = np.concatenate([np.arange(c) for c in counts])
        scale = np.repeat(rng.uniform(0.6, 1.2, size=(n, 1)), 3, axis=1)
        scale[within % 6 == 2] *= np.array([0.3, 0.3, 0.5])
        k["matrices"] = _matrices(rng.uniform(-each, each, size=(n, 3)), _quaternions(rng, n), scale)
        k["cameras"] = _ring(rng, W, 2.0 * r, r / 2.0)
        k["floor"] = ng.Plane(y=-float(r.max()) - 0.5, half_extent_x=4 * float(r.max()), z_min=-4 * float(r.max()),
                              z_max=4 * float(r.max()), checker_scale=1.0)
    elif kind in ("large", "view"):
        n = case["instances"]
        k["meshes"] = ["box", "ico2", "cylinder", "ico3", "ico5"]
        k["slot"] = [i % 5 for i in range(n)]
        k["instances"] = [_instance(i % 5, i % 8) for i in range(n)]
        half = 100.0 * math.sqrt(n / 100_000.0)  # the density of large_world
        pos = rng.uniform((-half, -10.0, -half), (half, 10.0, half), size=(n, 3))
        scale = np.ones((n, 3))
        scale[2::5] = (0.3, 0.3, 0.5)
        k["matrices"] = _matrices(pos, _quaternions(rng, n), scale)[None]
        k["floor"] = ng.Plane(y=-11.0, half_extent_x=120.0, z_min=-120.0, z_max=120.0, checker_scale=1.0)
        eye = (float(rng.uniform(-5.0, 5.0)), 2.0, -half)
        k["camera"] = ng.make_camera(eye, (0.0, 0.0, 0.0), width=case["width"], height=case["height"], fov=1.0)
        k["cameras"] = k["camera"].matrix[None]
        if kind == "large":
            e, a = np.meshgrid(np.radians(np.linspace(-15.0, 15.0, case["beams"])),
                               np.radians(np.linspace(0.0, 360.0, case["azimuths"], endpoint=False)), indexing="ij")
            d = np.stack([np.cos(e) * np.sin(a), np.sin(e), np.cos(e) * np.cos(a)], -1).reshape(1, -1, 3)
            k["directions"] = d.astype(np.float32)
            k["origins"] = np.broadcast_to(rng.uniform(-1.0, 1.0, size=3), d.shape).astype(np.float32)
    elif kind == "gradient":
        P = case["bodies"]
        k["meshes"] = ["ico3smooth", "box"]
        k["slot"] = [i % 2 for i in range(P)]
        k["instances"] = [_instance(i % 2, i % 8) for i in range(P)]
        k["positions"] = (rng.uniform(-2.0, 2.0, size=(W, P, 3)) + np.array([0.0, 0.0, -6.0])).astype(np.float32)
        k["quaternions"] = _quaternions(rng, W, P).astype(np.float32)
        k["scales"] = np.repeat(rng.uniform(0.6, 1.2, size=(W, P, 1)), 3, axis=-1).astype(np.float32)
        k["floor"] = ng.Plane(y=-2.5, half_extent_x=12.0, z_min=-30.0, z_max=-2.0, checker_scale=0.0)
        eye = np.array([0.0, 1.0, 0.0]) + rng.uniform(-0.2, 0.2, size=(W, 3))
        k["cameras"] = ng.look_at(eye, np.array([0.0, 0.0, -6.0]), up=(0.0, 1.0, 0.0))
        # The measured depth: a coarse random relief around the scene's distance, with sensor noise.
        h, w = case["height"], case["width"]
        relief = rng.uniform(-1.0, 1.0, size=(W, 8, 8)).astype(np.float32)
        rows, cols = (np.arange(h) * 8) // h, (np.arange(w) * 8) // w
        k["target"] = 6.0 + relief[:, rows][:, :, cols] + 0.1 * (rng.random((W, h, w), np.float32) - 0.5)
        k["target_normal"] = np.array([0.0, 0.5, math.sqrt(0.75)], np.float32)
    elif kind == "mesh":
        P = case["bodies"]
        k["meshes"] = ["ico%dsmooth" % case["subdivisions"], "box"]
        k["slot"] = [i % 2 for i in range(P)]
        k["instances"] = [_instance(i % 2, i % 8) for i in range(P)]
        k["matrices"] = _matrices(rng.uniform(-1.5, 1.5, size=(W, P, 3)), _quaternions(rng, W, P),
                                  np.broadcast_to(_scales(rng, ["a"] * P), (W, P, 3)))
        k["cameras"] = _ring(rng, W, 4.0, 1.0)
        v = _mesh(k["meshes"][0]).vertices
        a, b = rng.uniform(1.0, 6.0, size=(3, 3)), rng.uniform(0.0, 6.28, size=3)
        k["vertices"] = (v * (1.0 + 0.25 * np.sin(v @ a + b))).astype(np.float32)
    return k


def _gpu(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _outputs(case):
    names = case["outputs"].split()
    return {n: n in names for n in ("rgb", "depth", "normals", "object_ids")}


def prepare(case, seed):
    k = _inputs(case, seed)
    meshes = [_mesh(n) for n in k["meshes"]]
    s = {"kind": case["kind"], "case": case}
    common = dict(lights=k["lights"], floor=k["floor"], meshes=meshes)
    kind = case["kind"]
    if kind == "uneven":
        s["renderer"] = ng.UnevenBatchRenderer(k["worlds"], **common)
    elif kind == "view":
        s["renderer"] = ng.Renderer(case["width"], case["height"], instances=k["instances"], **common)
        s["camera"] = k["camera"]
    else:
        s["renderer"] = ng.BatchRenderer(case.get("width", 64), case.get("height", 64), case.get("worlds", 1),
                                         case.get("cameras", 1), instances=k["instances"], **common)
    P = len(k.get("slot", []))
    if "poses" in k:
        s["renderer"].bind_bodies(np.arange(P, dtype=np.int32), k["local"], k["scale"], P)
        s["poses"] = _gpu(k["poses"])
    elif "xpos" in k:
        s["renderer"].bind_geoms(np.arange(P, dtype=np.int32), k["scale"], P)
        s["xpos"], s["xmat"] = _gpu(k["xpos"]), _gpu(k["xmat"])
    elif "matrices" in k:
        s["matrices"] = _gpu(k["matrices"])
    for name in ("cameras", "origins", "directions", "vertices", "scales", "target", "target_normal"):
        if name in k:
            s[name] = _gpu(k[name])
    if kind == "gradient":
        s["positions"] = _gpu(k["positions"]).requires_grad_()
        s["quaternions"] = _gpu(k["quaternions"]).requires_grad_()
    if kind == "mesh":
        s["renderer"].set_instance_transforms(s["matrices"])
        s["normals"] = torch.nn.functional.normalize(s["vertices"], dim=1)
    return s


def _place(s):
    if "poses" in s:
        s["renderer"].set_body_poses(s["poses"])
    elif "xpos" in s:
        s["renderer"].set_geom_poses(s["xpos"], s["xmat"])
    else:
        s["renderer"].set_instance_transforms(s["matrices"])


def _loss(depth, normals, target, target_normal, with_normals):
    """Squared depth error of the pixels that see something, and how far their normals turn from the target's."""
    seen = torch.isfinite(depth)
    loss = (torch.where(seen, depth - target, 0.0) ** 2).sum()
    if with_normals:
        loss = loss + torch.where(seen, 1.0 - (normals * target_normal).sum(-1), 0.0).sum()
    return loss


def run(state):
    s, case, r = state, state["case"], state["renderer"]
    kind = s["kind"]
    if kind == "frame":
        _place(s)
        return r.render(s["cameras"], 1.0, case["spp"], zero_copy=True, **_outputs(case))
    if kind == "uneven":
        _place(s)
        return r.render(s["cameras"], 1.0, 1, rgb=True, depth=True, object_ids=True, zero_copy=True)
    if kind == "large":
        _place(s)
        return {"frame": r.render(s["cameras"], 1.0, 1, rgb=True, depth=True, object_ids=True, zero_copy=True),
                "lidar": r.cast_rays(s["origins"], s["directions"], 150.0)}
    if kind == "rays":
        _place(s)
        return r.cast_rays(s["origins"], s["directions"], 20.0)
    if kind == "gradient":
        s["positions"].grad = s["quaternions"].grad = None
        m = autodiff.pose_matrices(s["positions"], s["quaternions"], s["scales"])
        depth, normals = autodiff.render_depth_normals(r, m, s["cameras"], 1.0)
        _loss(depth, normals, s["target"], s["target_normal"], case["normals"]).backward()
        return {"depth": depth.detach(), "normals": normals.detach(), "positions": s["positions"].grad,
                "quaternions": s["quaternions"].grad}
    if kind == "mesh":
        r.update_mesh(0, s["vertices"], s["normals"])
        return r.render(s["cameras"], 1.0, 1, rgb=False, depth=True, normals=True, zero_copy=True)
    r.set_instance_transforms(s["matrices"])
    for f in range(case["frames"] - 1):
        r.render_frame(s["camera"], f, 1, rgb=True, zero_copy=True)
    frame = r.render_frame(s["camera"], case["frames"] - 1, 1, rgb=True, depth=True, object_ids=True, zero_copy=True)
    return {n: image.clone() for n, image in frame.items()}  # the images are the renderer's: a viewer that keeps them copies them


def work(case):
    """Inputs read once and outputs written once; of the arithmetic, one instance transform, one box and one
    triangle test for each ray that is asked for (about 100 operations), which no ray that hits can do without."""
    kind = case["kind"]
    tris = {"box": 12, "ico1": 80, "ico2": 320, "cylinder": 512, "ico3": 1280, "ico4": 5120, "ico5": 20480}
    per_pixel = {"rgb": 3, "depth": 4, "normals": 12, "object_ids": 4}
    scene = lambda *names: sum(tris[n] * 18 for n in names)  # noqa: E731  (36-byte triangles shared in pairs)
    if kind == "frame":
        o = [n for n, on in _outputs(case).items() if on]
        px = case["worlds"] * case["cameras"] * case["width"] * case["height"]
        each = {"matrices": 48, "bodies": 28, "geoms": 48}[case["place"]]
        rays = px * ((case["spp"] * (1 + case["lights"]) if "rgb" in o else 0) + (0 if o == ["rgb"] else 1))
        return {"bytes": px * sum(per_pixel[n] for n in o) + case["worlds"] * (case["bodies"] * each + 48 * case["cameras"])
                + scene("ico3", "box", "cylinder"), "flops": 100.0 * rays}
    if kind == "uneven":
        px = case["worlds"] * 7168  # the mean of 32, 64 and 128 squared
        return {"bytes": px * 11 + case["worlds"] * (24 * case["most"] + 48) + scene("box", "ico2", "cylinder", "ico3", "ico4", "ico5"),
                "flops": 100.0 * 3 * px}
    if kind == "large":
        px, beams = case["width"] * case["height"], case["beams"] * case["azimuths"]
        return {"bytes": px * 11 + beams * 44 + case["instances"] * 48 + scene("box", "ico2", "cylinder", "ico3", "ico5"),
                "flops": 100.0 * (3 * px + beams)}
    if kind == "rays":
        n = case["worlds"] * case["beams"]
        return {"bytes": n * 44 + case["worlds"] * case["bodies"] * 28 + scene("ico3", "box", "cylinder"), "flops": 100.0 * n}
    if kind == "gradient":
        px, n = case["worlds"] * case["width"] * case["height"], case["worlds"] * case["bodies"]
        return {"bytes": px * 20 + n * (40 + 28) + case["worlds"] * 48 + scene("ico3", "box"), "flops": 400.0 * px}
    if kind == "mesh":
        px, t = case["worlds"] * case["width"] * case["height"], 20 * 4 ** case["subdivisions"]
        return {"bytes": px * 16 + t * (12 + 12 + 12 + 18) + case["worlds"] * case["bodies"] * 48,
                "flops": 100.0 * px + 100.0 * t * math.log2(t)}
    px = case["width"] * case["height"]
    return {"bytes": px * (case["frames"] * 3 + 8) + case["instances"] * 48, "flops": 100.0 * px * (2 * case["frames"] + 1)}


def tolerance(case):
    """The images of two correct walks of one scene differ where two surfaces lie within rounding of each other
    along a ray (3 pixels in a million of the 4096-world batch between the framework's own kernels) and, in
    colour, by a level where a transcendental function rounds the other way (5 in a million against other
    builds of the same shading). Depth and distance follow from 32-bit arithmetic: 1e-7 relative where 64 bits
    see the same surface, and a pixel on a silhouette that sees another one moves by its whole value. Gradients
    are 32-bit sums over thousands of pixels in no fixed order: 6e-7, the largest 1e-5, between two passes."""
    return {"rel": 1e-5, "max": 1e-3, "differ": 5e-5}


# -------------------------------------------------------------------------------------------- 64-bit truth --

def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _f64(a):
    return torch.as_tensor(np.asarray(a, np.float64), device=_device())


class _Geometry:
    """A mesh's triangles and the tables that turn a ray-triangle test into products with (o x d, d) and o."""

    def __init__(self, vertices, triangles, normals):
        v, t = _f64(vertices), torch.as_tensor(np.asarray(triangles, np.int64), device=_device())
        v0, v1, v2 = v[t[:, 0]], v[t[:, 1]], v[t[:, 2]]
        # Edges as the packed triangles hold them, rounded to 32 bits.
        e1, e2 = (v1 - v0).float().double(), (v2 - v0).float().double()
        self.v0, self.e1, self.e2, self.n = v0, e1, e2, torch.linalg.cross(e1, e2)
        self.u = torch.cat([e2, -torch.linalg.cross(e2, v0)], 1).T.contiguous()
        self.v = torch.cat([-e1, -torch.linalg.cross(v0, e1)], 1).T.contiguous()
        self.t0 = (v0 * self.n).sum(1)
        self.centre = v.mean(0)
        self.radius = float((v - self.centre).norm(dim=1).max()) * 1.0001 + 1e-9
        self.normals = None if normals is None else torch.stack([_f64(normals)[t[:, i]] for i in range(3)], 1)


def _closest(o, d, A, slot, geometry, floor):
    """Per ray (W, R): the closest surface's distance (inf: none), its instance (-1: the floor or none), triangle
    and barycentrics; o, d (W, R, 3), A (W, P, 3, 4) world from mesh."""
    t = (floor.y - o[..., 1]) / d[..., 1]
    at = o + d * t[..., None]
    on = (d[..., 1].abs() > 1e-3) & (t > 0) & (at[..., 0].abs() < floor.half_extent_x) & (at[..., 2] > floor.z_min) & (at[..., 2] < floor.z_max)
    best = torch.where(on, t, INF).flatten()
    inst = torch.full(best.shape, -1, dtype=torch.int64, device=best.device)
    tri, bu, bv = torch.zeros_like(inst), torch.zeros_like(best), torch.zeros_like(best)
    Ai = torch.linalg.inv(A[..., :3])
    for i, m in enumerate(slot):
        g = geometry[m]
        lo = (o - A[:, None, i, :, 3]) @ Ai[:, i].transpose(1, 2)
        ld = d @ Ai[:, i].transpose(1, 2)
        q = lo - g.centre
        dd = (ld * ld).sum(-1)
        near = (q * q).sum(-1) * dd - (q * ld).sum(-1) ** 2 <= g.radius ** 2 * dd
        at = near.flatten().nonzero()[:, 0]
        step = max(1, 16_000_000 // g.n.shape[0])
        for first in range(0, at.numel(), step):
            j = at[first:first + step]
            oj, dj = lo.reshape(-1, 3)[j], ld.reshape(-1, 3)[j]
            x = torch.cat([torch.linalg.cross(oj, dj), dj], 1)
            det = -(dj @ g.n.T)
            u, v = (x @ g.u) / det, (x @ g.v) / det
            t = (oj @ g.n.T - g.t0) / det
            t[~((u >= 0) & (v >= 0) & (u + v <= 1) & (t > 0))] = INF
            t, k = t.min(1)
            closer = t < best[j]
            j, k = j[closer], k[closer]
            best[j], inst[j], tri[j] = t[closer], i, k
            bu[j], bv[j] = u[closer].gather(1, k[:, None])[:, 0], v[closer].gather(1, k[:, None])[:, 0]
    return tuple(x.reshape(o.shape[:2]) for x in (best, inst, tri, bu, bv))


def _at_hit(hit, slot, geometry, i):
    """The hit triangle's record of every ray on instance i's mesh (the boolean mask, triangles, barycentrics)."""
    on = hit[1] == i
    return on, geometry[slot[i]], hit[2][on], hit[3][on], hit[4][on]


def _normals(hit, o, d, A, slot, geometry):
    """The shading normal of every hit, facing the ray; zero where nothing is hit."""
    up = torch.zeros(3, dtype=o.dtype, device=o.device)
    up[1] = 1.0
    n = torch.where(torch.isfinite(hit[0])[..., None], up, torch.zeros_like(up)).expand(o.shape).clone()
    world = torch.arange(o.shape[0], device=o.device)[:, None].expand(o.shape[:2])
    for i in range(len(slot)):
        on, g, tri, u, v = _at_hit(hit, slot, geometry, i)
        if tri.numel():
            n[on] = _surface(g, tri, u, v, torch.linalg.inv(A[world[on], i][:, :, :3]), d[on])
    return n


def _surface(g, tri, u, v, Ai, d):
    unit = lambda x: x / x.norm(dim=-1, keepdim=True)  # noqa: E731
    turn = lambda x: (Ai.transpose(1, 2) @ x[..., None])[..., 0]  # noqa: E731
    face = unit(turn(g.n[tri]))
    face = torch.where((face * d).sum(-1, keepdim=True) > 0, -face, face)
    if g.normals is None:
        return face
    n0, n1, n2 = g.normals[tri].unbind(1)
    smooth = unit(turn(n0 * (1 - u - v)[:, None] + n1 * u[:, None] + n2 * v[:, None]))
    return torch.where((smooth * face).sum(-1, keepdim=True) < 0, -smooth, smooth)


def _centre_rays(cameras, width, height, worlds):
    """Origins, directions (W, R, 3) and forwards of every view's pixel centres, fov 1."""
    c = _f64(cameras)
    unit = lambda x: x / x.norm(dim=-1, keepdim=True)  # noqa: E731
    right, up, fwd = unit(c[:, :, 0]), unit(c[:, :, 1]), unit(-c[:, :, 2])
    scale = math.tan(0.5)
    x = (2 * (torch.arange(width, device=c.device, dtype=torch.float64) + 0.5) / width - 1) * scale * (width / height)
    y = -(2 * (torch.arange(height, device=c.device, dtype=torch.float64) + 0.5) / height - 1) * scale
    d = unit(right[:, None, None] * x[None, None, :, None] + up[:, None, None] * y[None, :, None, None] + fwd[:, None, None])
    o = c[:, None, None, :, 3].expand(d.shape)
    f = fwd[:, None, None].expand(d.shape)
    return tuple(v.reshape(worlds, -1, 3) for v in (o, d, f))


def exact(case, seed):
    kind = case["kind"]
    if kind in ("uneven", "large"):
        return None  # a brute-force pass over these scenes takes minutes
    k = _inputs(case, seed)
    geometry = []
    for i, name in enumerate(k["meshes"]):
        m = _mesh(name)
        v = k["vertices"] if kind == "mesh" and i == 0 else m.vertices
        normals = m.normals
        if kind == "mesh" and i == 0:
            normals = (k["vertices"] / np.linalg.norm(k["vertices"], axis=1, keepdims=True)).astype(np.float32)
        geometry.append(_Geometry(v, m.triangles, normals))
    slot, floor = k["slot"], k["floor"]
    if kind == "gradient":
        return _exact_gradient(case, k, geometry)
    A = _f64(k["exact_matrices"] if "exact_matrices" in k else k["matrices"])
    if kind == "rays":
        o, d = _f64(k["origins"]), _f64(k["directions"])
        d = d / d.norm(dim=-1, keepdim=True)
        hit = _closest(o, d, A, slot, geometry, floor)
        hit = (torch.where(hit[0] <= 20.0, hit[0], INF), torch.where(hit[0] <= 20.0, hit[1], -1)) + hit[2:]
        return {"distance": hit[0], "normal": _normals(hit, o, d, A, slot, geometry), "object_id": None}
    W, h, w = case.get("worlds", 1), case["height"], case["width"]
    views = W * case.get("cameras", 1)
    o, d, f = _centre_rays(k["cameras"], w, h, W)
    hit = _closest(o, d, A, slot, geometry, floor)
    out = {"depth": (hit[0] * (d * f).sum(-1)).reshape(views, h, w)}
    if kind == "mesh" or "normals" in case.get("outputs", ""):
        out["normals"] = _normals(hit, o, d, A, slot, geometry).reshape(views, h, w, 3)
    if kind == "view":
        return {"rgb": None, "depth": out["depth"][0], "object_ids": None}
    if kind == "mesh":
        return out
    out = {n: out.get(n) for n, on in _outputs(case).items() if on}
    return out if "depth" in out else None  # colour alone: bytes


def _exact_gradient(case, k, geometry):
    """The same loss through the surfaces that each pixel sees, by autograd in 64 bits."""
    W, h, w, slot = case["worlds"], case["height"], case["width"], k["slot"]
    p, q = _f64(k["positions"]).requires_grad_(), _f64(k["quaternions"]).requires_grad_()
    x, y, z, v = (q / q.norm(dim=-1, keepdim=True)).unbind(-1)
    R = torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - z * v), 2 * (x * z + y * v), 2 * (x * y + z * v),
                     1 - 2 * (x * x + z * z), 2 * (y * z - x * v), 2 * (x * z - y * v), 2 * (y * z + x * v),
                     1 - 2 * (x * x + y * y)], -1).unflatten(-1, (3, 3)) * _f64(k["scales"])[..., None, :]
    A = torch.cat([R, p[..., None]], -1)
    o, d, f = _centre_rays(k["cameras"], w, h, W)
    with torch.no_grad():
        hit = _closest(o, d, A, slot, geometry, k["floor"])
    t, normal = hit[0], _normals(hit, o, d, A.detach(), slot, geometry)
    world = torch.arange(W, device=o.device)[:, None].expand(t.shape)
    for i in range(len(slot)):
        on, g, tri, _, _ = _at_hit(hit, slot, geometry, i)
        if not tri.numel():
            continue
        wi, oi, di = world[on], o[on], d[on]
        Ai = torch.linalg.inv(A[:, i, :, :3])[wi]
        b = A[wi, i, :, 3]
        n = (Ai.transpose(1, 2) @ g.n[tri][..., None])[..., 0]
        vertex = (A[wi, i, :, :3] @ g.v0[tri][..., None])[..., 0] + b
        ti = (n * (vertex - oi)).sum(-1) / (n * di).sum(-1)
        local = (Ai @ (oi + di * ti[:, None] - b)[..., None])[..., 0] - g.v0[tri]
        nn = (g.n[tri] ** 2).sum(-1)
        u = (torch.linalg.cross(local, g.e2[tri]) * g.n[tri]).sum(-1) / nn
        v = (torch.linalg.cross(g.e1[tri], local) * g.n[tri]).sum(-1) / nn
        t = t.masked_scatter(on, ti)
        normal = normal.masked_scatter(on[..., None].expand_as(normal), _surface(g, tri, u, v, Ai, di))
    depth, normal = (t * (d * f).sum(-1)).reshape(W, h, w), normal.reshape(W, h, w, 3)
    _loss(depth, normal, _f64(k["target"]), _f64(k["target_normal"]), case["normals"]).backward()
    return {"depth": depth.detach(), "normals": normal.detach(), "positions": p.grad, "quaternions": q.grad}
