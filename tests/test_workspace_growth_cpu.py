"""A workspace that is large enough for a scene and an image serves every smaller one, without a GPU.

Callers keep one workspace for the largest scene and framebuffer that they expect ("reused"): its size must not
shrink when the number of Gaussians, the image or the number of samples per call grows.
"""
import ctypes

import pytest

from StochasticGSCudaBackend import _abi

COUNTS = sorted({int(2 ** (i / 3)) for i in range(0, 84)}
                | {1 << 18, (1 << 18) + 1, 1 << 20, 1 << 21, (5 << 19) - 1, 5 << 19, 1 << 22, 6_000_000})
# aspect 4:3 from one tile up to 3900 pixels, odd sizes among them; then single steps over the edges of tiles and quads
SIZES = [(int(8 * 1.12 ** i), int(6 * 1.12 ** i)) for i in range(52)]
STEPS = [(w, 480) for w in range(600, 680)] + [(680, h) for h in range(480, 520)]


def size(n, width, height, gps, hybrid, reuse, samples):
    g = _abi.Gaussians(0, 0, 0, 0, 0, n, 16)
    c = _abi.Camera(0, 0, width, height, 500.0, 500.0, width / 2, height / 2, 0.2, 100.0)
    s = _abi.SettingsC(0, 1, gps, hybrid, reuse, 0, None, None, 0, 0, None)
    args = [ctypes.byref(x) for x in (g, c, s)]
    lib = _abi.load()
    return lib.sgs_workspace_size(*args) if samples == 1 else lib.sgs_samples_workspace_size(*args, samples)


MODES = [(0, 0, 0), (0, 1, 0), (0, 0, 1), (1, 0, 0), (1, 1, 0), (1, 1, 1)]


@pytest.mark.parametrize("gps,hybrid,reuse", MODES)
@pytest.mark.parametrize("samples", [1, 3, 8])
def test_more_gaussians_need_no_less(gps, hybrid, reuse, samples):
    for width, height in SIZES:
        sizes = [size(n, width, height, gps, hybrid, reuse, samples) for n in COUNTS]
        assert sizes[0] > 0 and sizes == sorted(sizes), (width, height)


@pytest.mark.parametrize("gps,hybrid,reuse", MODES)
@pytest.mark.parametrize("samples", [1, 3, 8])
def test_larger_images_need_no_less(gps, hybrid, reuse, samples):
    for n in COUNTS:
        for images in (SIZES, STEPS):
            sizes = [size(n, width, height, gps, hybrid, reuse, samples) for width, height in images]
            assert sizes[0] > 0 and sizes == sorted(sizes), n


@pytest.mark.parametrize("gps,hybrid,reuse", MODES)
def test_more_samples_need_no_less(gps, hybrid, reuse):
    for n in COUNTS[::3]:
        for width, height in SIZES[::3]:
            sizes = [size(n, width, height, gps, hybrid, reuse, samples) for samples in (1, 2, 3, 8, 16)]
            assert sizes == sorted(sizes), (n, width, height)
