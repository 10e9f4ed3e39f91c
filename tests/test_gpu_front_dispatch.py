"""Which passes are prepared to run front to back, by what the clear pass leaves in the queue's header.

Its estimate of the pixels that all Gaussians cover (WorkQueue::covered_all) is written by the passes of point
splatting that are prepared for depth order, and by all of stochastic transparency.
"""
import pytest
import torch

import sgs_scenes
from test_gpu_front_to_back import deep_scene

pytestmark = pytest.mark.gpu

WIDTH, HEIGHT = 645, 483


def render(scene, device, *, samples=1, mode=0, reuse=False, gps=True, hybrid=False, layout="float", blue=None,
           camera=None, **caps):
    """The outputs, the framebuffer of the first sample and the queue's header (as bytes) of one call."""
    from StochasticGSCudaBackend import _C

    cam = (camera or sgs_scenes.front_camera(WIDTH, HEIGHT)).to(device)
    n_fb = WIDTH * HEIGHT
    entries = _C.k_buffer_size if reuse else 0
    kb = (torch.full((entries, n_fb, 2), -1, dtype=torch.int32, device=device),
          torch.zeros((entries, n_fb, 4), device=device))
    history = [torch.zeros((HEIGHT, WIDTH, c), device=device) for c in (3, 1, 1, 1)]
    args = (*scene, cam.w2c, cam.position, WIDTH, HEIGHT, cam.focal_x, cam.focal_y, cam.center_x, cam.center_y,
            cam.near_plane, cam.far_plane, False, 1, gps, hybrid, reuse,
            torch.empty(0, dtype=torch.uint8, device=device) if blue is None else blue, *kb, *history,
            torch.eye(4, device=device), mode)
    extra = dict(caps)
    if layout == "pre":
        extra["preactivated"] = _C.preactivate(*scene[1:4])
    elif layout == "quant":
        extra["quantized"] = _C.quantize(*scene)
    outputs = [torch.empty_like(h) for h in history]
    size = _C.samples_workspace_size(samples, *args, **caps)
    raw = torch.zeros(size + 256, dtype=torch.uint8, device=device)
    workspace = raw[-raw.data_ptr() % 256:][:size]
    _C.set_frame_index(21)
    _C.render_samples_into(outputs, workspace, samples, *args, **extra)
    fb = workspace[256:256 + 8 * n_fb].view(torch.int64).cpu().numpy()
    return outputs, fb, workspace[:256].cpu()


def covered_all(header):
    return float(header[64:80].view(torch.float32).sum())


@pytest.mark.parametrize("more", [dict(mode=2), dict(mode=1, reuse=True), dict(mode=1, hybrid=True, max_binned=1 << 22)])
def test_passes_of_one_sample_keep_the_rule_of_one_sample(more, cuda_device):
    """2^21 Gaussians of point splatting: front to back pays for passes of several samples, not of one."""
    scene = deep_scene((1 << 21) + 45, -5.0).to(cuda_device).tensors()
    _, _, together = render(scene, cuda_device, samples=2, mode=1)
    assert covered_all(together) > 58 * WIDTH * HEIGHT
    _, _, apart = render(scene, cuda_device, samples=2, **more)
    assert covered_all(apart) == 0


def binned(header):
    return int(header[20:24].view(torch.int32))  # WorkQueue::binned


def test_a_small_bin_of_stochastic_transparency_fills_as_the_gaussians_lie(cuda_device):
    """Hybrid scheduling evaluates the first max_binned Gaussians above 512 pixels in another form; depth order, and
    groups left out of the count, would change which these are."""
    scene = deep_scene((1 << 21) + 45, -4.2).to(cuda_device).tensors()
    _, _, alone = render(scene, cuda_device, gps=False, hybrid=True, max_binned=64)
    assert binned(alone) > 1000
    _, _, small = render(scene, cuda_device, gps=False, hybrid=True, max_binned=64, samples=2)
    assert binned(small) == binned(alone)
    # a bin that cannot fill does not hinder the order, which leaves most of them out
    _, _, full = render(scene, cuda_device, gps=False, hybrid=True, samples=2)
    assert binned(full) < binned(alone)


@pytest.mark.parametrize("layout", ["float", "pre", "quant"])
def test_points_of_models_in_no_order_are_drawn_as_they_lie(layout, cuda_device):
    """Groups of Gaussians from all over the scene are not compact: their coverage does not count."""
    scene = deep_scene((1 << 21) + 45, -5.0)
    ordered = render(scene.to(cuda_device).tensors(), cuda_device, samples=2, mode=1, layout=layout)[2]
    perm = torch.randperm(scene.means.shape[0], generator=torch.Generator().manual_seed(3))
    shuffled = [t[perm].contiguous().to(cuda_device) for t in scene.tensors()]
    at_random = render(shuffled, cuda_device, samples=2, mode=1, layout=layout)[2]
    n_fb = WIDTH * HEIGHT
    assert covered_all(ordered) > 110 * n_fb and 0 < covered_all(at_random) < 58 * n_fb
