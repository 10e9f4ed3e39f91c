"""The binned GPS Gaussians taken front to back, against the same Gaussians taken as they came.

From 8192 queue places on, hybrid GPS lists its binned Gaussians in depth order and skips those that lie
behind every pixel they can reach (csrc/accumulate_gps.cu); a smaller queue is taken in arrival order.
Point seeds are counter-based, so both must give the same framebuffer bit for bit. Image sizes lie around
the 8 x 8 tiles and the 64 x 64 blocks of depth bounds; needles have ellipses too thin for their extents.
"""
import pytest
import torch

import sgs_scenes
from sgs_testing import assert_bitwise

pytestmark = pytest.mark.gpu


def needles(n, seed=9):
    """Long thin Gaussians at random rotations: 1 / (1 - rho^2) of their footprints passes 1000."""
    scene = sgs_scenes.make_scene(sgs_scenes.SceneSpec(n=n, log_scale_mean=-6.0, log_scale_std=0.3), seed=seed)
    scales = scene.scales.clone()
    scales[:, 0] = 0.2
    return sgs_scenes.Scene(scene.means, scales, scene.rotations, scene.opacities, scene.sh_coefficients)


def heavy(n, log_scale, seed=3):
    return sgs_scenes.make_scene(sgs_scenes.SceneSpec(n=n, log_scale_mean=log_scale, log_scale_std=1.0), seed=seed)


@pytest.mark.parametrize("kind,width,height,ss,max_fragments", [
    ("heavy", 64, 64, 3, 0), ("heavy", 65, 129, 2, 700), ("heavy", 321, 181, 1, 0), ("heavy", 257, 120, 2, 5000),
    ("needles", 200, 150, 2, 0), ("needles", 121, 87, 3, 1024)])
@pytest.mark.parametrize("samples", [1, 3])
def test_depth_order_keeps_the_framebuffer(kind, width, height, ss, max_fragments, samples, cuda_device):
    from StochasticGSCudaBackend import _C

    n = 12_000
    scene = (needles(n) if kind == "needles" else heavy(n, -3.2)).to(cuda_device)
    cam = sgs_scenes.front_camera(width, height).to(cuda_device)
    n_fb = width * height * ss * ss
    e = torch.empty(0)
    kb = (torch.empty((0, n_fb, 2), dtype=torch.int32, device=cuda_device),
          torch.empty((0, n_fb, 4), device=cuda_device))
    args = (*scene.tensors(), cam.w2c, cam.position, width, height, cam.focal_x, cam.focal_y, cam.center_x, cam.center_y,
            cam.near_plane, cam.far_plane, False, ss, True, True, False,
            torch.empty(0, dtype=torch.uint8, device=cuda_device), *kb, e, e, e, e, torch.eye(4, device=cuda_device), 0)
    got = {}
    for max_binned in (0, 8191):
        _C.set_frame_index(17)
        _, ws, layout = _C.render_samples_with_workspace(samples, *args, max_fragments=max_fragments,
                                                         max_binned=max_binned)
        entries = int(ws[layout.queue:layout.queue + 8].view(torch.int64)) >> 40
        assert 50 < entries < 8191, f"{entries} Gaussians binned"
        got[max_binned] = ws[layout.framebuffer:layout.framebuffer + 8 * n_fb * samples].view(torch.int64).cpu().numpy()
    assert (got[0] != -1).sum() > 1000
    assert_bitwise("framebuffer", got[0], got[8191])
