"""Colours of the quantised layout: degree-3 SH as 16-byte loads, everything else coefficient by coefficient.

Both read the same coefficients in the same order of operations, so an SH array that does not start on 16 bytes
must give the image of one that does, and a model of fewer bases that of the same model filled up with
zeros, bit for bit.
"""
import dataclasses

import pytest
import torch

import sgs_scenes
from StochasticGSCudaBackend import _C
from sgs_testing import assert_bitwise
from test_gpu_quantized import _args

pytestmark = pytest.mark.gpu


def image(scene, quantized, ss, samples):
    cam = sgs_scenes.front_camera(97 if ss == 1 else 41, 61)
    e = torch.empty(0)
    args = _args(scene, cam, dict(aa=False, ss=ss, gps=False, hybrid=False), (e, e, e, e), 0)
    _C.set_frame_index(5)
    outs = _C.render_samples(samples, *args, quantized=quantized) if samples > 1 else _C.render(*args, quantized=quantized)
    return outs[0].cpu().numpy()


@pytest.mark.parametrize("bases", [1, 4, 9, 16])
@pytest.mark.parametrize("ss,samples", [(1, 1), (2, 1), (1, 3)])
def test_colours_do_not_depend_on_the_loads(bases, ss, samples, cuda_device):
    spec = sgs_scenes.SceneSpec(n=5000, log_scale_mean=-2.5, log_scale_std=0.6, sh_bases=bases, sh_rest_std=0.2)
    scene = sgs_scenes.make_scene(spec, seed=3).to("cuda")
    q = _C.quantize(*scene.tensors())
    got = image(scene, q, ss, samples)
    if bases == 16:
        flat = torch.empty(q.sh_half.numel() + 1, dtype=torch.float16, device="cuda")
        flat[1:] = q.sh_half.reshape(-1)
        other, other_scene = _C.Quantized(q.records, q.chunks, flat[1:].view(q.sh_half.shape)), scene
    else:
        filled = torch.zeros((5000, 16, 3), device="cuda")
        filled[:, :bases] = scene.sh_coefficients
        other_scene = dataclasses.replace(scene, sh_coefficients=filled)
        other = _C.quantize(*other_scene.tensors())
    assert_bitwise("image", got, image(other_scene, other, ss, samples))
    assert float(got.std()) > 0.05
