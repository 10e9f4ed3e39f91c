"""Which Gaussians a dense scene of stochastic transparency queues: by how many the queue holds, never by what wins.

The clear pass estimates how many AABBs lie above 256, 512 and 1024 pixels (WorkQueue::larger), and the scatter pass
queues those above the first of these sizes that fit, else those above 2048. The framebuffers must be the same
bit for bit, also at image sizes below a tile, a quad and a claim's worth of items. (Scenes of fewer than 8192
Gaussians, or of fewer than 137 million covered pixels, are never dense.)
"""
import numpy as np
import pytest
import torch

import sgs_scenes
from oracle import cpu
from sgs_testing import assert_bitwise
from test_gpu_schedule import KEYS, cam_dict
from test_gpu_st_queue import dense_scene

pytestmark = pytest.mark.gpu


def call(scene, cam, samples=1, **flags):
    from StochasticGSCudaBackend import _C

    dev = scene.means.device
    cam = cam.to(dev)
    n_fb = cam.width * cam.height
    e = torch.empty(0)
    kb = (torch.empty((0, n_fb, 2), dtype=torch.int32, device=dev), torch.empty((0, n_fb, 4), device=dev))
    _C.set_frame_index(40)
    _, ws, at = _C.render_samples_with_workspace(
        samples, *scene.tensors(), cam.w2c, cam.position, cam.width, cam.height, cam.focal_x, cam.focal_y,
        cam.center_x, cam.center_y, cam.near_plane, cam.far_plane, False, 1, False, flags.get("hybrid", False), False,
        torch.empty(0, dtype=torch.uint8, device=dev), *kb, e, e, e, e, torch.eye(4, device=dev), 0)
    fb = ws[at.framebuffer:at.framebuffer + 8 * n_fb * samples].view(torch.int64).cpu().numpy()
    header = ws[at.queue:at.queue + 128]
    counts = header[24:36].view(torch.int32).tolist()  # entries, items, items listed
    return fb, *counts, header[80:128].view(torch.float32).view(3, 4).sum(dim=1).tolist()


@pytest.mark.parametrize("samples", [1, 3])
def test_every_size_gives_the_same(samples, cuda_device):
    from StochasticGSCudaBackend import _C

    scene = dense_scene(150_000, -2.6).to(cuda_device)
    cam = sgs_scenes.front_camera(450, 253)
    fb, entries, items, listed, larger = call(scene, cam, samples)
    assert larger[0] > larger[1] > larger[2] > 1000 and listed > 0
    queued = [entries]
    try:
        for room in (int(larger[1]), int(larger[2]), int(larger[2] * 0.5)):  # sizes above 512, 1024 and 2048 pixels
            _C.set_queue_limit(room)
            got, n, _, listed, _ = call(scene, cam, samples)
            queued.append(n)
            assert listed > 0
            assert_bitwise(f"room for {room}", got, fb)
    finally:
        _C.set_queue_limit(0)
    assert queued == sorted(queued, reverse=True) and len(set(queued)) == 4


@pytest.mark.parametrize("width,height,hybrid,n", [(7, 5, False, 9000), (8, 8, False, 9000), (127, 57, True, 100_000),
                                                   (33, 257, False, 100_000), (257, 131, True, 60_000)])
def test_dense_scenes_at_the_edges_of_tiles(width, height, hybrid, n, cuda_device):
    """The depth-ordered queue: most Gaussians are large, and its items listed."""
    scene = sgs_scenes.make_scene(sgs_scenes.SceneSpec(n=n, log_scale_mean=1.0, log_scale_std=0.8), seed=11)
    if width > 200:
        scene = dense_scene(n, -1.5)
    scene.scales[::5] = -9.0  # (the queue has room for 15 of 16)
    cam = sgs_scenes.front_camera(width, height)
    fb, entries, items, listed, _ = call(scene.to(cuda_device), cam, hybrid=hybrid)
    if width * height > 256:
        assert entries > 1000 and listed > 1000
    want = cpu.accumulate({k: t.numpy() for k, t in zip(KEYS, scene.tensors())}, cam_dict(cam),
                          dict(aa=False, ss=1, gps=False, hybrid=hybrid), 40)
    # a knife-edge pixel may differ in an image of fewer than 10,000
    assert float((fb == want).mean()) >= 0.9999 or int((fb != want).sum()) <= 1
    assert np.unique(fb).size > 1
