"""Scatter passes front to back (csrc/sgs_front.cuh): what they drop must not have been able to win.

Deep scenes of some millions of Gaussians run in depth order and drop what lies behind their tiles' bounds. The
winners must be those of the CPU restatement (>= 99.99 % identical, its float tolerance), and several samples per
call, whose passes run front to back from fewer Gaussians on, those of single calls bit for bit. Image sizes are
ragged against the 8 x 8 tiles and the quads of four, counts against the groups of 32.
"""
import numpy as np
import pytest
import torch

import sgs_scenes
from oracle import cpu
from sgs_testing import assert_bitwise, render_once
from test_gpu_schedule import KEYS, cam_dict

pytestmark = pytest.mark.gpu


def deep_scene(n, log_scale):
    """A box filled with Gaussians that cover the image of `front_camera` a hundred times and more."""
    spec = sgs_scenes.SceneSpec(n=n, means="uniform", means_scale=2.0, log_scale_mean=log_scale, log_scale_std=0.6,
                                opacity_logit_std=2.0, sh_bases=1)
    return sgs_scenes.make_scene(spec, seed=5)


@pytest.mark.parametrize("n,log_scale,width,height,gps,hybrid", [
    ((5 << 19) + 13, -5.0, 643, 481, False, False),
    (5 << 19, -4.5, 801, 447, False, True),
    ((1 << 22) + 1, -5.0, 643, 481, True, False),
])
def test_the_winners_are_those_of_the_restatement(n, log_scale, width, height, gps, hybrid, cuda_device):
    scene = deep_scene(n, log_scale)
    cd = cam_dict(sgs_scenes.front_camera(width, height))
    flags = dict(aa=False, ss=1, gps=gps, hybrid=hybrid)
    dev_scene = {k: t.to(cuda_device) for k, t in zip(KEYS, scene.tensors())}
    got = render_once(dev_scene, cd, flags, 9)["fb"]
    want = cpu.accumulate({k: t.numpy() for k, t in zip(KEYS, scene.tensors())}, cd, flags, 9)
    agree = float((got == want).mean())
    assert agree >= 0.9999, f"{agree:.6f} of the winners agree"
    assert np.unique(got).size > 1000


@pytest.mark.parametrize("gps,layout,aa,ss,samples", [(False, "float", False, 1, 3), (False, "quant", True, 1, 2),
                                                      (True, "pre", False, 1, 3), (True, "quant", True, 2, 2)])
def test_samples_of_a_deep_scene_equal_single_calls(gps, layout, aa, ss, samples, cuda_device):
    from StochasticGSCudaBackend import _C

    n, width, height = (1 << 21) + 45, 645 // ss, 483 // ss
    scene = deep_scene(n, -5.0).to(cuda_device)
    cam = sgs_scenes.front_camera(width, height).to(cuda_device)
    extra = {}
    if layout == "pre":
        extra["preactivated"] = _C.preactivate(*scene.tensors()[1:4])
    elif layout == "quant":
        extra["quantized"] = _C.quantize(*scene.tensors())
    e = torch.empty(0)
    n_fb = width * height * ss * ss
    kb = (torch.empty((0, n_fb, 2), dtype=torch.int32, device=cuda_device),
          torch.empty((0, n_fb, 4), device=cuda_device))
    args = (*scene.tensors(), cam.w2c, cam.position, width, height, cam.focal_x, cam.focal_y, cam.center_x, cam.center_y,
            cam.near_plane, cam.far_plane, aa, ss, gps, False, False,
            torch.empty(0, dtype=torch.uint8, device=cuda_device), *kb, e, e, e, e, torch.eye(4, device=cuda_device), 0)
    _C.set_frame_index(40)
    _, ws, layout = _C.render_samples_with_workspace(samples, *args, **extra)
    together = ws[layout.framebuffer:layout.framebuffer + 8 * n_fb * samples].view(torch.int64).view(samples, n_fb)
    for s in range(samples):
        _C.set_frame_index(40 + s)
        _, ws1, layout1 = _C.render_with_workspace(*args, **extra)
        one = _C.workspace_views(ws1, layout1, n_fb, False)["framebuffer"]
        assert_bitwise(f"sample {s}", together[s].cpu().numpy(), one.cpu().numpy())
    assert np.unique(together.cpu().numpy()).size > 1000
