"""Front-to-back passes in the layouts, modes and cameras that other tests of them leave out, bit for bit.

With 2^21 to 5 * 2^19 Gaussians of stochastic transparency, calls of several samples run front to back and single
calls draw the Gaussians as they lie. Hybrid point splatting runs front to back where its queue has a place for every
Gaussian, and as they lie with the default 2^20 places; either way the same Gaussians are queued.
"""
import pytest
import torch

import sgs_scenes
from sgs_testing import assert_bitwise
from test_gpu_front_dispatch import HEIGHT, WIDTH, covered_all
from test_gpu_front_to_back import deep_scene

pytestmark = pytest.mark.gpu

N_FB = WIDTH * HEIGHT


def arguments(scene, device, camera, gps, hybrid, reuse, blue):
    cam = camera.to(device)
    noise = sgs_scenes.synthetic_blue_noise(2) if blue else torch.empty(0, dtype=torch.uint8)
    head = (*scene, cam.w2c, cam.position, WIDTH, HEIGHT, cam.focal_x, cam.focal_y, cam.center_x, cam.center_y,
            cam.near_plane, cam.far_plane, False, 1, gps, hybrid, reuse, noise.to(device))
    return head


def k_buffers(device, reuse):
    from StochasticGSCudaBackend import _C

    k = _C.k_buffer_size if reuse else 0
    return (torch.full((k, N_FB, 2), -1, dtype=torch.int32, device=device), torch.full((k, N_FB, 4), 0.5, device=device))


def inside_camera():
    """In the middle of the scene, with what lies up to half a unit behind it still drawn."""
    return sgs_scenes.pinhole((0.0, 0.0, -0.3), WIDTH, HEIGHT, near_plane=-0.5)


@pytest.mark.parametrize("layout,blue,hybrid,camera", [
    ("pre", False, False, "front"), ("float", True, False, "front"), ("pre", True, True, "front"),
    ("quant", False, True, "front"), ("float", False, False, "inside"), ("pre", False, False, "inside"),
    ("quant", True, False, "inside")])
def test_samples_of_stochastic_transparency(layout, blue, hybrid, camera, cuda_device):
    from StochasticGSCudaBackend import _C

    scene = deep_scene((1 << 21) + 45, -5.0).to(cuda_device).tensors()
    extra = {}
    if layout == "pre":
        extra["preactivated"] = _C.preactivate(*scene[1:4])
    elif layout == "quant":
        extra["quantized"] = _C.quantize(*scene)
    e = torch.empty(0)
    head = arguments(scene, cuda_device, sgs_scenes.front_camera(WIDTH, HEIGHT) if camera == "front" else inside_camera(),
                     False, hybrid, False, blue)
    args = (*head, *k_buffers(cuda_device, False), e, e, e, e, torch.eye(4, device=cuda_device), 0)
    _C.set_frame_index(130)
    _, ws, at = _C.render_samples_with_workspace(2, *args, **extra)
    together = ws[at.framebuffer:at.framebuffer + 16 * N_FB].view(torch.int64).view(2, N_FB)
    assert covered_all(ws[at.queue:at.queue + 128]) > 58 * N_FB
    for s in range(2):
        _C.set_frame_index(130 + s)
        _, ws1, at1 = _C.render_with_workspace(*args, **extra)
        one = _C.workspace_views(ws1, at1, N_FB, False)["framebuffer"]
        assert (one != -1).sum() > 1000
        assert_bitwise(f"sample {s}", together[s].cpu().numpy(), one.cpu().numpy())


@pytest.mark.parametrize("reuse,mode", [(False, 2), (True, 2), (True, 1)])
def test_samples_with_a_history(reuse, mode, cuda_device):
    """Each sample's pass runs by itself: outputs and k-buffers as of one call after the other."""
    from StochasticGSCudaBackend import _C

    scene = deep_scene((1 << 21) + 45, -5.0).to(cuda_device).tensors()
    e = torch.empty(0)
    head = arguments(scene, cuda_device, sgs_scenes.front_camera(WIDTH, HEIGHT), False, False, reuse, False)
    eye = torch.eye(4, device=cuda_device)
    _C.set_frame_index(9)
    history = _C.render(*head, *k_buffers(cuda_device, reuse), e, e, e, e, eye, 0)
    got_k, want_k = k_buffers(cuda_device, reuse), k_buffers(cuda_device, reuse)
    _C.set_frame_index(10)
    got, ws, at = _C.render_samples_with_workspace(2, *head, *got_k, *history, eye, mode)
    assert covered_all(ws[at.queue:at.queue + 128]) > 58 * N_FB
    _C.set_frame_index(10)
    want = _C.render(*head, *want_k, *history, eye, mode)
    want = _C.render(*head, *want_k, *want, eye, 1)
    for name, a, b in zip(("image", "depth", "alpha", "weight mass", "primitives", "occlusion"), (*got, *got_k),
                          (*want, *want_k)):
        assert_bitwise(name, a.cpu().numpy(), b.cpu().numpy())


@pytest.mark.parametrize("samples", [1, 2])
def test_hybrid_point_splatting(samples, cuda_device):
    from StochasticGSCudaBackend import _C

    n = (1 << 22) + 7
    scene = deep_scene(n, -4.6).to(cuda_device).tensors()
    e = torch.empty(0)
    head = arguments(scene, cuda_device, sgs_scenes.front_camera(WIDTH, HEIGHT), True, True, False, False)
    fbs, entries = [], []
    for places in (n, 1 << 20):
        _C.set_frame_index(55)
        _, ws, at = _C.render_samples_with_workspace(
            samples, *head, *k_buffers(cuda_device, False), e, e, e, e, torch.eye(4, device=cuda_device), 0,
            max_binned=places)
        if places == n:
            assert covered_all(ws[at.queue:at.queue + 128]) > 110 * N_FB
        entries.append(int(ws[at.queue:at.queue + 8].view(torch.int64)) >> 40)
        fbs.append(ws[at.framebuffer:at.framebuffer + 8 * samples * N_FB].view(torch.int64).cpu().numpy())
    assert 10 < entries[0] <= entries[1] < 1 << 20
    assert_bitwise("framebuffers", fbs[0], fbs[1])
