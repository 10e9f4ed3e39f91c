"""The depth-ordered queue's list has room for the parts of all queued Gaussians, however large these are.

16,000 Gaussians over the whole image have more parts of 32 quads than the list has places: the parts grow instead.
"""
import pytest
import torch

import sgs_scenes
from oracle import cpu
from test_gpu_schedule import KEYS, cam_dict
from test_gpu_st_queue import dense_scene

pytestmark = pytest.mark.gpu


def test_parts_of_huge_gaussians_fit_the_list(cuda_device):
    from StochasticGSCudaBackend import _C

    scene = dense_scene(20_000, 0.5)
    scene.scales[::5] = -9.0  # (the queue has room for 15 of 16)
    cam = sgs_scenes.front_camera(257, 257)
    n_fb = cam.width * cam.height
    on = cam.to(cuda_device)
    e = torch.empty(0)
    kb = (torch.empty((0, n_fb, 2), dtype=torch.int32, device=cuda_device), torch.empty((0, n_fb, 4), device=cuda_device))
    _C.set_frame_index(40)
    _, ws, at = _C.render_with_workspace(
        *scene.to(cuda_device).tensors(), on.w2c, on.position, on.width, on.height, on.focal_x, on.focal_y, on.center_x,
        on.center_y, on.near_plane, on.far_plane, False, 1, False, False, False,
        torch.empty(0, dtype=torch.uint8, device=cuda_device), *kb, e, e, e, e, torch.eye(4, device=cuda_device), 0)
    header = ws[at.queue:at.queue + 36].view(torch.int32).tolist()
    overflow, entries, items, listed = header[3], *header[6:9]
    assert entries > 15_000 and overflow == 0 and listed == items > 3 * entries
    fb = _C.workspace_views(ws, at, n_fb, False)["framebuffer"].cpu().numpy()
    want = cpu.accumulate({k: t.numpy() for k, t in zip(KEYS, scene.tensors())}, cam_dict(cam),
                          dict(aa=False, ss=1, gps=False, hybrid=False), 40)
    assert float((fb == want).mean()) >= 0.9999
