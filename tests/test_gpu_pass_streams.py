"""Renders of several samples, lights or mirrors from several streams at once, and in captures that are replayed beside
them or outlive a growth of the renderer's scratch: each picture is the one its render gives alone."""
import numpy as np
import pytest

from test_gpu_sample_passes import scene

pytestmark = pytest.mark.gpu

SIZE = (32, 64, 48, 3)  # worlds, height, width


def buffers(torch, count):
    return [{"rgb": torch.zeros(SIZE, dtype=torch.uint8, device="cuda")} for _ in range(count)]


def moved(torch, cams, k):
    c = torch.from_numpy(cams).cuda()
    c[:, :, 3] += 0.3 * k
    return c


def test_renders_on_several_streams_do_not_meet(torch_cuda):
    torch = torch_cuda
    r, cams = scene(32, 8, 2, True, 48, 64)
    samples = (3, 2, 1, 4)  # 1: the mirrors and the second light take passes for one sample too
    views = [moved(torch, cams, k) for k in range(4)]
    alone, got = buffers(torch, 4), buffers(torch, 4)
    for k in range(4):
        r.render(views[k], 1.0, samples[k], frame=k, rgb=True, into=alone[k])
        torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(4)]
    for _ in range(5):
        for g in got:
            g["rgb"].zero_()
        torch.cuda.synchronize()
        for k in range(4):
            with torch.cuda.stream(streams[k]):
                r.render(views[k], 1.0, samples[k], frame=k, rgb=True, into=got[k])
        torch.cuda.synchronize()
        for k in range(4):
            assert torch.equal(got[k]["rgb"], alone[k]["rgb"]), k


def test_a_replayed_capture_does_not_meet_other_renders(torch_cuda):
    torch = torch_cuda
    r, cams = scene(32, 8, 2, True, 48, 64)
    views = [moved(torch, cams, k) for k in range(2)]
    alone, got = buffers(torch, 2), buffers(torch, 2)
    for k in range(2):
        r.render(views[k], 1.0, 3, frame=k, rgb=True, into=alone[k])
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        r.render(views[0], 1.0, 3, frame=0, rgb=True, into=got[0])
    streams = [torch.cuda.Stream() for _ in range(2)]
    for _ in range(5):
        for b in got:
            b["rgb"].zero_()
        torch.cuda.synchronize()
        with torch.cuda.stream(streams[0]):
            g.replay()
        with torch.cuda.stream(streams[1]):
            r.render(views[1], 1.0, 3, frame=1, rgb=True, into=got[1])
        with torch.cuda.stream(streams[0]):
            g.replay()
        torch.cuda.synchronize()
        for k in range(2):
            assert torch.equal(got[k]["rgb"], alone[k]["rgb"]), k
    del g


def test_a_captured_band_outlives_renders_of_more_rows(torch_cuda):
    torch = torch_cuda
    r, cams = scene(32, 8, 2, True, 48, 64)
    dev = torch.from_numpy(cams).cuda()
    band = {"rgb": torch.zeros((32, 8, 48, 3), dtype=torch.uint8, device="cuda")}
    r.set_rows(16, 8)
    r.render(dev, 1.0, 2, frame=3, rgb=True, into=band)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        r.render(dev, 1.0, 2, frame=3, rgb=True, into=band)
    r.set_rows(0, 64)
    whole = buffers(torch, 1)[0]
    r.render(dev, 1.0, 2, frame=3, rgb=True, into=whole)
    band["rgb"].zero_()
    g.replay()
    torch.cuda.synchronize()
    # The capture may have taken the per-pixel kernel: pixels with two surfaces within rounding may differ.
    differ = (band["rgb"] != whole["rgb"][:, 16:24]).any(-1).sum().item()
    assert differ <= 32 * 8 * 48 * 1e-4, differ
    del g
