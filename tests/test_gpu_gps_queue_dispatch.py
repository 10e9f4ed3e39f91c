"""Which queues of binned point-splatting Gaussians are listed in depth order, and that either way gives the same.

Of fewer than 4096 Gaussians in the queue, those of 32,768 chunks (256 points each) and more are taken as they came,
all others in depth order (csrc/accumulate_st.cu, order_kernel). A queue with fewer than 8192 places is always
taken as it came: the framebuffers must be the same bit for bit, at image sizes around the tiles and blocks.
"""
import pytest
import torch

import sgs_scenes
from sgs_testing import assert_bitwise
from test_gpu_gps_queue import heavy

pytestmark = pytest.mark.gpu

NOT_LISTED = 0xFFFFFFFF


def over_a_filled_image(n_large, n_small=30_000):
    """Large Gaussians among small ones that fill the image: most items' tests go over many closed tiles."""
    small = sgs_scenes.make_scene(sgs_scenes.SceneSpec(n=n_small, log_scale_mean=-3.6, log_scale_std=0.3,
                                                       opacity_logit_std=3.0), seed=4, morton=False)
    large = sgs_scenes.make_scene(sgs_scenes.SceneSpec(n=n_large, log_scale_mean=-0.7, log_scale_std=0.3), seed=6,
                                  morton=False)
    return sgs_scenes.Scene(*(torch.cat(pair) for pair in zip(small.tensors(), large.tensors())))


def call(scene, width, height, ss, samples, max_binned, device):
    from StochasticGSCudaBackend import _C

    cam = sgs_scenes.front_camera(width, height).to(device)
    n_fb = width * height * ss * ss
    e = torch.empty(0)
    kb = (torch.empty((0, n_fb, 2), dtype=torch.int32, device=device), torch.empty((0, n_fb, 4), device=device))
    _C.set_frame_index(17)
    _, ws, at = _C.render_samples_with_workspace(
        samples, *scene.tensors(), cam.w2c, cam.position, width, height, cam.focal_x, cam.focal_y, cam.center_x,
        cam.center_y, cam.near_plane, cam.far_plane, False, ss, True, True, False,
        torch.empty(0, dtype=torch.uint8, device=device), *kb, e, e, e, e, torch.eye(4, device=device), 0,
        max_binned=max_binned)
    fb = ws[at.framebuffer:at.framebuffer + 8 * n_fb * samples].view(torch.int64).cpu().numpy()
    packed = int(ws[at.queue:at.queue + 8].view(torch.int64))
    # the last sample's WorkQueue: entries and chunks, items listed
    return fb, packed >> 40, packed & ((1 << 40) - 1), int(ws[at.queue + 32:at.queue + 36].view(torch.int32)) & NOT_LISTED


@pytest.mark.parametrize("scene,width,height,ss,listed", [
    ("heavy", 321, 181, 2, True), ("heavy", 449, 257, 1, True),       # 4096 Gaussians and more
    ("filled", 321, 181, 1, True), ("filled", 65, 129, 3, True),      # few Gaussians, few chunks
    ("filled", 1283, 721, 1, False),                                  # few Gaussians, many chunks
])
@pytest.mark.parametrize("samples", [1, 2])
def test_listed_or_as_they_came(scene, width, height, ss, listed, samples, cuda_device):
    made = (heavy(12_000, -2.0) if scene == "heavy" else over_a_filled_image(400)).to(cuda_device)
    fb, entries, chunks, items = call(made, width, height, ss, samples, 0, cuda_device)
    assert (4096 <= entries < 8191) if scene == "heavy" else (300 <= entries < 4096)
    if scene == "filled":
        assert (chunks < 1 << 15) == listed
    assert (0 < items < NOT_LISTED) if listed else items == NOT_LISTED
    as_they_came, entries_2, _, _ = call(made, width, height, ss, samples, 8191, cuda_device)
    assert entries_2 == entries and (fb != -1).sum() > 1000
    assert_bitwise("framebuffer", fb, as_they_came)
