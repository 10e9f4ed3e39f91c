"""What the coverage estimate of the clear pass leaves to the passes in depth order (WorkQueue::covered, covered_all).

Faint Gaussians hide little, however much they cover: their scenes are drawn as they lie, whatever the footprints. So are
scenes of few covered pixels, for which the order takes longer than it saves: in small images however dense.
"""
import numpy as np
import pytest
import torch

import sgs_scenes
from oracle import cpu
from test_gpu_front_dispatch import HEIGHT, WIDTH, binned, covered_all, render
from test_gpu_front_to_back import deep_scene
from test_gpu_schedule import KEYS, cam_dict
from test_gpu_st_queue import dense_scene
from test_gpu_st_queue_sizes import call

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,shift,width,height,ordered", [
    (60_000, 0.0, 321, 181, True), (60_000, -5.0, 321, 181, False), (9_000, 0.0, 321, 181, False), (120_000, 0.0, 81, 46, False),
    (100_000, 0.0, 500, 280, True)])
def test_queues_of_faint_and_small_scenes_are_not_ordered(n, shift, width, height, ordered, cuda_device):
    scene = dense_scene(n, -2.0)
    scene.opacities += shift
    cam = sgs_scenes.front_camera(width, height)
    fb, entries, items, listed, _ = call(scene.to(cuda_device), cam)
    assert items > 1000 and (listed > 0) == ordered
    want = cpu.accumulate({k: t.numpy() for k, t in zip(KEYS, scene.tensors())}, cam_dict(cam),
                          dict(aa=False, ss=1, gps=False, hybrid=False), 40)
    assert float((fb == want).mean()) >= 0.9999
    assert np.unique(fb).size > 1


@pytest.mark.parametrize("gps", [False, True])
def test_deep_faint_scenes_are_drawn_as_they_lie(gps, cuda_device):
    estimates = []
    for shift in (0.0, -5.0):
        scene = deep_scene((1 << 21) + 45, -5.0)
        scene.opacities += shift
        estimates.append(covered_all(render(scene.to(cuda_device).tensors(), cuda_device, samples=2, mode=1, gps=gps)[2]))
    assert estimates[0] > 58 * WIDTH * HEIGHT > estimates[1] > 0


def test_footprints_too_large_for_the_tests_do_not_count(cuda_device):
    """Passes in depth order test Gaussians of few tiles only."""
    n_fb = WIDTH * HEIGHT
    header = render(deep_scene((1 << 21) + 45, -1.0).to(cuda_device).tensors(), cuda_device, samples=2, mode=1, gps=False)[2]
    larger = float(header[48:64].view(torch.float32).sum())
    assert larger > 10_000 * n_fb and covered_all(header) < 0.1 * larger


def test_queues_that_may_fill_hinder_the_order(cuda_device):
    """What finds a dense scene's queue full comes last in depth order, and together: such scenes are drawn as they lie."""
    from StochasticGSCudaBackend import _C

    scene = deep_scene((1 << 21) + 45, -3.8).to(cuda_device).tensors()
    _, ordered, header = render(scene, cuda_device, samples=2, mode=1, gps=False, hybrid=True)
    larger = header[80:128].view(torch.float32).view(3, 4).sum(dim=1).tolist()
    listed = int(header[32:36].view(torch.int32))
    assert covered_all(header) > 58 * WIDTH * HEIGHT and listed > 0
    try:
        _C.set_queue_limit(max(int(larger[2] * 0.8), 1))
        _, as_they_lie, full = render(scene, cuda_device, samples=2, mode=1, gps=False, hybrid=True)
    finally:
        _C.set_queue_limit(0)
    assert binned(header) < binned(full)  # groups that are left out are not counted
    np.testing.assert_array_equal(as_they_lie, ordered)
