"""Workspace of the stochastic-transparency queue: its sizes through the C ABI, without a GPU.

The queue's own entries, the tile bounds, the depth histogram and the item list must not make a one-sample
workspace larger than the 64 MiB scratch of sgs_render_no_alloc where the 60 bytes per entry of a
2^18-entry queue, which that entry point's documentation promises, fit.
"""
import ctypes

import pytest

from StochasticGSCudaBackend import _abi

SCRATCH = 64 << 20


def up(v):
    return (v + 255) // 256 * 256


def promised(n, n_fb):
    q = min(n, 1 << 18)
    return 256 + up(8 * n_fb) + up(16 * n_fb) + up(8 * q) + 3 * up(16 * q) + up(4 * q)


def size(n, width, height, ss=1):
    g = _abi.Gaussians(0, 0, 0, 0, 0, n, 16)
    c = _abi.Camera(0, 0, width, height, 500.0, 500.0, width / 2, height / 2, 0.2, 100.0)
    s = _abi.SettingsC(0, ss, 0, 0, 0, 0, None, None, 0, 0, None)
    return _abi.load().sgs_workspace_size(ctypes.byref(g), ctypes.byref(c), ctypes.byref(s))


@pytest.mark.parametrize("n", [1, 31, 1000, 65_536, 262_144, 262_145, 500_000, 1_048_575, 1_048_576, 6_000_000,
                               4_000_000_000])
@pytest.mark.parametrize("width,height,ss", [(1, 1, 1), (7, 5, 1), (160, 120, 1), (640, 480, 1), (333, 127, 3),
                                             (1279, 719, 1), (1920, 1080, 1), (2048, 1040, 1), (1336, 400, 2)])
def test_what_fitted_the_fixed_scratch_still_does(n, width, height, ss):
    if promised(n, width * height * ss * ss) <= SCRATCH:
        assert 0 < size(n, width, height, ss) <= SCRATCH


def test_the_queue_grows_with_the_scene_and_stays_bounded():
    sizes = [size(n, 800, 800) for n in (1, 1000, 100_000, 1_000_000, 100_000_000)]
    assert sizes == sorted(sizes) and sizes[0] < sizes[-1] <= SCRATCH
