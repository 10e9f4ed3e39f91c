"""The fused backward walk's two queues where they fill: footprints above 2048 pixels, and those above 256.

Each holds min(N, 2^18) entries, both together min(N, 2^19) places that they take from the two ends. What does not fit
is walked by its warp. The gradients are those of one walk per sample, which has no queue. The Gaussians are so faint
that tiles keep empty pixels and none is left out.
"""
import ctypes

import numpy as np
import pytest
import torch

import sgs_scenes
from StochasticGSCudaBackend import Settings

pytestmark = pytest.mark.gpu

WIDTH, HEIGHT, SAMPLES = 3840, 2160, 2
FULL = 1 << 18


def faint_scene(n, huge, device):
    """n Gaussians of some 300 pixels, every `huge`-th of some 3000."""
    gen = torch.Generator().manual_seed(n + huge)
    means = torch.randn((n, 3), generator=gen)
    scales = torch.randn((n, 3), generator=gen) * 0.05 - 4.44
    opacities = torch.randn(n, generator=gen) * 0.1 - 3.9
    scales[::huge] += 1.55
    opacities[::huge] -= 0.7
    rotations = torch.randn((n, 4), generator=gen)
    rotations /= rotations.norm(dim=1, keepdim=True)
    sh = torch.randn((n, 4, 3), generator=gen) * 0.3
    return [t.contiguous().to(device) for t in (means, scales, rotations, opacities, sh)]


@pytest.mark.parametrize("n,huge,full", [(600_000, 300, (False, True)), (1_100_000, 2, (True, True)),
                                         (520_000, 20, (False, True)), (300_001, 2, (False, False))])
def test_full_queues(n, huge, full, cuda_device):
    from StochasticGSCudaBackend import _abi
    from StochasticGSCudaBackend.autograd import _render_all, _render_one, _structs

    lib = _abi.load()
    tensors = faint_scene(n, huge, cuda_device)
    cam = sgs_scenes.front_camera(WIDTH, HEIGHT).to(cuda_device)
    settings = Settings(cam.w2c, cam.position, WIDTH, HEIGHT, cam.focal_x, cam.focal_y, cam.center_x, cam.center_y,
                        cam.near_plane, cam.far_plane, False, 1, False, False, False)
    g, c, s = _structs(*tensors, settings)
    gen = torch.Generator().manual_seed(5)
    grads = [torch.randn((HEIGHT, WIDTH, k), generator=gen).to(cuda_device) / (WIDTH * HEIGHT) for k in (3, 1, 1)]
    gp = [ctypes.c_void_p(t.data_ptr()) for t in grads]
    weight = ctypes.c_float(1.0 / SAMPLES)
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    nbytes = lib.sgs_backward_workspace_size(n)

    def finish(bw):
        outs = [torch.empty_like(t) for t in tensors]
        assert lib.sgs_backward_finish(ctypes.byref(g), ctypes.byref(c), ctypes.byref(s), ctypes.c_void_p(bw.data_ptr()),
                                       *(ctypes.c_void_p(t.data_ptr()) for t in outs), stream) == _abi.SGS_OK
        return [t.cpu().numpy() for t in outs]

    e = torch.empty(0)
    hist, bw = (e, e, e, e), torch.empty(nbytes, dtype=torch.uint8, device=cuda_device)
    for k in range(SAMPLES):
        hist, ws, _ = _render_one(tensors, settings, hist, min(k, 1), 700 + k)
        assert lib.sgs_backward_accumulate(ctypes.byref(g), ctypes.byref(c), ctypes.byref(s),
                                           ctypes.c_void_p(ws.data_ptr()), *gp, weight, int(k == 0),
                                           ctypes.c_void_p(bw.data_ptr()), stream) == _abi.SGS_OK
    want = finish(bw)

    _, ws, layout = _render_all(tensors, settings, SAMPLES, 700)
    scratch = torch.empty(lib.sgs_backward_samples_scratch_size(ctypes.byref(c), ctypes.byref(s), SAMPLES),
                          dtype=torch.uint8, device=cuda_device)
    assert lib.sgs_backward_accumulate_framebuffers(
        ctypes.byref(g), ctypes.byref(c), ctypes.byref(s), ctypes.c_void_p(ws.data_ptr() + layout.framebuffer), SAMPLES,
        *gp, weight, 1, ctypes.c_void_p(scratch.data_ptr()), ctypes.c_void_p(bw.data_ptr()), stream) == _abi.SGS_OK
    got = finish(bw)

    # the queues' headers lie behind the colours and the accumulators, each section 256-byte aligned
    def up(v):
        return (v + 255) & ~255

    at = up(4 * ((3 * n + 3) & ~3)) + up(8 * 10 * n)
    headers = bw[at:at + 512].view(torch.int64).cpu().numpy()  # 160 bytes each: entries << 40 | chunks, ...
    entries = [int(headers[0]) >> 40, int(headers[20]) >> 40]
    assert [v > FULL for v in entries] == list(full) and min(entries) > 1000, entries
    for name, a, b in zip(("means", "scales", "rotations", "opacities", "sh"), want, got):
        scale = np.abs(a).max()
        assert scale > 0, name
        # as in the walk's other tests: single precision per fragment, double in the sums
        np.testing.assert_allclose(b, a, rtol=2e-3, atol=2e-5 * scale, err_msg=name)
