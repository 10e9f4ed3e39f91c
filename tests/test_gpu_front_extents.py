"""What a front-to-back pass drops before the projection must lie inside the extents that it tests.

A curtain closes the left of the image; Gaussians behind it are dropped in groups when the tiles within their
extents are closed (csrc/sgs_front.cuh). Here their projections reach past the curtain's edge although rough
extents would not, by cancellation or by parameters that are not finite. With 2^21 to 5 * 2^19 Gaussians several samples per call run front to back and single
calls draw the Gaussians as they lie: both must give the same framebuffers bit for bit.
"""
import math

import numpy as np
import pytest
import torch

import sgs_scenes
from sgs_testing import assert_bitwise

pytestmark = pytest.mark.gpu

WIDTH, HEIGHT, FOCAL = 640, 480, 1500.0
CENTER_X, CENTER_Y = -1200.0, HEIGHT / 2.0  # the image lies beside the optical axis, up to 50 degrees off it
EDGE = 369.0  # the curtain's right edge, within a tile
N_CURTAIN = 1 << 21


def camera():
    return sgs_scenes.Camera(sgs_scenes.look_at((0.0, 0.0, 0.0), (0.0, 0.0, 1.0)), torch.zeros(3), WIDTH, HEIGHT, FOCAL,
                             FOCAL, CENTER_X, CENTER_Y)


def at_pixel(x, y, z):
    return torch.stack([(x - CENTER_X) / FOCAL * z, (y - CENTER_Y) / FOCAL * z, z], dim=1)


def uniform(g, n, lo, hi):
    return lo + (hi - lo) * torch.rand(n, generator=g)


def with_curtain(g, means, scales, rotations, opacities):
    """The curtain at depths of 0.6 to 0.9 in Morton order, then the given Gaussians in groups of 32."""
    z = uniform(g, N_CURTAIN, 0.6, 0.9)
    c_means = at_pixel(uniform(g, N_CURTAIN, -10.0, EDGE), uniform(g, N_CURTAIN, -10.0, HEIGHT + 10.0), z)
    c_means = c_means[torch.argsort(sgs_scenes.morton_codes(c_means), stable=True)]
    unit = torch.tensor([1.0, 0.0, 0.0, 0.0])
    n = N_CURTAIN + means.shape[0]
    assert means.shape[0] % 32 == 0 and n < 5 << 19
    return (torch.cat([c_means, means]), torch.cat([torch.full((N_CURTAIN, 3), -7.4), scales]),
            torch.cat([unit.expand(N_CURTAIN, 4), rotations]), torch.cat([torch.full((N_CURTAIN,), 3.0), opacities]),
            torch.randn((n, 1, 3), generator=g) * 0.5)


def framebuffers(scene, layout, gps, device, samples=2):
    """Framebuffers of `samples` frames: from one call, and from single calls."""
    from StochasticGSCudaBackend import _C

    scene = [t.float().contiguous().to(device) for t in scene]
    cam = camera().to(device)
    extra = {}
    if layout == "pre":
        extra["preactivated"] = _C.preactivate(*scene[1:4])
    elif layout == "quant":
        extra["quantized"] = _C.quantize(*scene)
    e = torch.empty(0)
    n_fb = WIDTH * HEIGHT
    kb = (torch.empty((0, n_fb, 2), dtype=torch.int32, device=device), torch.empty((0, n_fb, 4), device=device))
    args = (*scene, cam.w2c, cam.position, WIDTH, HEIGHT, cam.focal_x, cam.focal_y, cam.center_x, cam.center_y,
            cam.near_plane, cam.far_plane, False, 1, gps, False, False,
            torch.empty(0, dtype=torch.uint8, device=device), *kb, e, e, e, e, torch.eye(4, device=device), 0)
    _C.set_frame_index(40)
    _, ws, at = _C.render_samples_with_workspace(samples, *args, **extra)
    together = ws[at.framebuffer:at.framebuffer + 8 * n_fb * samples].view(torch.int64).view(samples, n_fb)
    # the clear pass's estimate of the pixels that all Gaussians cover (WorkQueue::covered_all)
    covered = float(ws[at.queue + 64:at.queue + 80].view(torch.float32).sum())
    assert covered > 110 * n_fb, "the several samples did not run front to back"
    single = []
    for s in range(samples):
        _C.set_frame_index(40 + s)
        _, ws1, at1 = _C.render_with_workspace(*args, **extra)
        single.append(_C.workspace_views(ws1, at1, n_fb, False)["framebuffer"].cpu().numpy())
    return together.cpu().numpy(), np.stack(single)


@pytest.mark.parametrize("gps", [False, True])
def test_needles_along_their_rays_in_the_preactivated_layout(gps, cuda_device):
    """A needle along its ray has a projected variance that cancels down to rounding residue of its squared length
    in pixels, tens of pixels squared and more here; the quadratic form that the extents come from must allow for it."""
    g = torch.Generator().manual_seed(1)
    n = 4096
    z = uniform(g, n, 1.2, 2.0)
    means = at_pixel(uniform(g, n, EDGE - 20.0, EDGE - 4.0), uniform(g, n, 0.0, HEIGHT), z)
    d = means / means.norm(dim=1, keepdim=True)
    # half-way quaternion from the x axis, the needle's own, to the ray
    q = torch.stack([1.0 + d[:, 0], torch.zeros(n), -d[:, 2], d[:, 1]], dim=1)
    q = q / q.norm(dim=1, keepdim=True)
    scales = torch.tensor([math.log(30.0), math.log(1.0e-4), math.log(1.0e-4)]).expand(n, 3)
    copies = [t.repeat_interleave(32, dim=0) for t in (means, scales, q, torch.full((n,), 3.0))]
    together, single = framebuffers(with_curtain(g, *copies), "pre", gps, cuda_device)
    won = (single != -1) & ((single & 0xFFFFFFFF) >= N_CURTAIN)
    assert won.sum() > 100, "the needles reach past the curtain"
    assert_bitwise("framebuffers", together, single)


POISON = {  # (log-scale of one axis, factor on the quaternion)
    "nan_scale": (float("nan"), 1.0),
    "inf_scale": (float("inf"), 1.0),
    "nan_quaternion": (-6.4, float("nan")),
    "huge_quaternion": (-6.4, 1.0e25),
}


@pytest.mark.parametrize("layout,poison", [("float", "nan_scale"), ("float", "inf_scale"), ("float", "nan_quaternion"),
                                           ("float", "huge_quaternion"), ("pre", "nan_scale"),
                                           ("pre", "huge_quaternion"), ("quant", "nan_scale")])
def test_parameters_that_are_not_finite(layout, poison, cuda_device):
    """One such Gaussian among the 32 of a group: its projection is bounded by the whole image."""
    g = torch.Generator().manual_seed(2)
    n = 32 * 32
    x, y = uniform(g, 32, 100.0, 300.0), uniform(g, 32, 100.0, 400.0)  # groups some ten pixels wide
    means = at_pixel(x.repeat_interleave(32) + uniform(g, n, -8.0, 8.0),
                     y.repeat_interleave(32) + uniform(g, n, -8.0, 8.0), torch.full((n,), 1.5))
    scales, q = torch.full((n, 3), -6.4), torch.tensor([1.0, 0.5, -0.25, 0.125]).repeat(n, 1)
    scales[5::32, 1], factor = POISON[poison]
    q[5::32] *= factor
    together, single = framebuffers(with_curtain(g, means, scales, q, torch.zeros(n)), layout, False, cuda_device)
    if poison == "nan_scale":
        won = (single != -1) & ((single & 0xFFFFFFFF) >= N_CURTAIN)
        assert won.sum() > 1000, "the Gaussian is drawn beside the curtain"
    assert_bitwise("framebuffers", together, single)
