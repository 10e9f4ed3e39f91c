"""The work that a user of this library has it do, as timed cases: renders, training steps, the learned resolve.

Every case goes through the public entry points: `render` and `_C.render_samples` for sample-frames,
`autograd.render_samples` with a backward for training, `denoise.Denoiser` and `denoise.denoise_train`
for the learned resolve. Scenes follow the specifications of `sgs_scenes.SCENES` (and the smoke test's
small scene), drawn on the GPU and put in Morton order like a loaded model.
"""
import math
import sys
from pathlib import Path

import torch
import torch.nn.functional as F

# the tree this file is asked to measure is the working folder, not the one the file lies in
sys.path.insert(0, str(Path("stochastic-gaussian-splatting_b200").resolve()))

import sgs_scenes  # noqa: E402
from StochasticGSCudaBackend import History, Settings, TemporalMode, _C, autograd, denoise, render  # noqa: E402

# scene name: (specification, orbit radius of its cameras)
SCENES = {
    "smoke": (sgs_scenes.SceneSpec(n=3000, log_scale_mean=-2.5, log_scale_std=0.6), 4.0),
    "st_100k": (sgs_scenes.SCENES["st_100k"], 4.0),
    "gps_1m": (sgs_scenes.SCENES["gps_1m"], 4.0),
    "batch_6m": (sgs_scenes.SCENES["batch_6m"], 25.0),
    "train_500k": (sgs_scenes.SCENES["train_500k"], 4.0),
}


def _render(name, scene, n, width, height, **more):
    case = dict(name=name, kind="render", scene=scene, n=n, width=width, height=height, ss=1, gps=False, hybrid=False,
                reuse=False, mode="static", samples=1, blue=False, layout="float", aa=False, bases=16,
                max_fragments=0)
    case.update(more)
    return case


def _train(name, scene, n, width, height, **more):
    case = dict(name=name, kind="train", scene=scene, n=n, width=width, height=height, ss=1, gps=False, hybrid=False,
                samples=8, aa=False, bases=16)
    case.update(more)
    return case


def listed():
    return [
        # a preview of a few thousand Gaussians: nothing but launches and the call itself
        _render("st_3k_160x120", "smoke", 3000, 160, 120, mode="reset"),
        # the plain progressive viewer on a small scene
        _render("st_100k_640x480", "st_100k", 100_000, 640, 480),
        # the benchmark's headline: one more progressive sample of a large scene
        _render("st_6m_1080p", "batch_6m", 6_000_000, 1920, 1080),
        # the same with Gaussian point splatting
        _render("gps_6m_1080p", "batch_6m", 6_000_000, 1920, 1080, gps=True),
        # a viewer frame of 8 samples per pixel in one call, on the preactivated model
        _render("st_6m_1080p_x8_pre", "batch_6m", 6_000_000, 1920, 1080, samples=8, layout="pre"),
        # the largest image, from the quantised model
        _render("st_6m_4k_quant", "batch_6m", 6_000_000, 3840, 2160, layout="quant"),
        # a moving camera with temporal reuse on heavy-tailed footprints, ragged size, blue noise
        _render("st_hybrid_400k_1279x719", "gps_1m", 400_000, 1279, 719, hybrid=True, mode="reproject", blue=True),
        # spatio-temporal reuse with binned point splatting, supersampled: the progressive benchmark, 4 samples (the
        # queue holds every Gaussian that qualifies: past a smaller one's end the binned ones are those that come first)
        _render("gps_hybrid_1m_720p_ss2_x4", "gps_1m", 1_000_000, 1280, 720, ss=2, gps=True, hybrid=True, reuse=True,
                mode="reproject", samples=4, max_fragments=1024),
        # forward and backward of one training view
        _train("train_500k_800x800_x8", "train_500k", 500_000, 800, 800),
        # the same through Gaussian point splatting
        _train("train_gps_100k_640x480_x4", "st_100k", 100_000, 640, 480, gps=True, samples=4),
        # the learned resolve of one frame
        dict(name="denoise_1080p", kind="denoise", batch=1, width=1920, height=1080),
        # one training step of the learned resolve on a batch of crops
        dict(name="denoise_train_16x128", kind="denoise_train", batch=16, width=128, height=128),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("small", "st", "gps", "samples", "layout", "heavy", "reuse", "train", "train_gps", "denoise",
                       "denoise_train"))
    if kind == "small":
        case = _render(None, "smoke", _log_int(rng, 1000, 30_000), _log_int(rng, 97, 640), _log_int(rng, 61, 480),
                       mode=rng.choice(("reset", "static")), ss=rng.choice((1, 2)), gps=rng.random() < 0.3,
                       bases=rng.choice((1, 4, 9, 16)))
    elif kind in ("st", "gps"):
        case = _render(None, "batch_6m", _log_int(rng, 300_000, 6_000_000), _log_int(rng, 640, 1920),
                       _log_int(rng, 360, 1080), gps=kind == "gps", hybrid=rng.random() < 0.3,
                       mode=rng.choice(("reset", "static", "reproject")), aa=rng.random() < 0.3)
    elif kind == "samples":
        case = _render(None, "batch_6m", _log_int(rng, 300_000, 6_000_000), _log_int(rng, 640, 1920),
                       _log_int(rng, 360, 1080), gps=rng.random() < 0.3, samples=rng.choice((2, 4, 8)),
                       layout=rng.choice(("float", "pre")))
    elif kind == "layout":
        case = _render(None, "batch_6m", _log_int(rng, 600_000, 6_000_000), _log_int(rng, 1280, 3840),
                       _log_int(rng, 720, 2160), layout=rng.choice(("quant", "pre")), blue=rng.random() < 0.3)
    elif kind == "heavy":
        case = _render(None, "gps_1m", _log_int(rng, 40_000, 400_000), _log_int(rng, 320, 1279),
                       _log_int(rng, 180, 719), hybrid=rng.random() < 0.5, blue=rng.random() < 0.5,
                       mode=rng.choice(("static", "reproject")))
    elif kind == "reuse":
        gps = rng.random() < 0.7
        case = _render(None, "gps_1m", _log_int(rng, 60_000, 1_000_000 if gps else 200_000), _log_int(rng, 320, 640),
                       _log_int(rng, 180, 360), ss=rng.choice((1, 2)), gps=gps, hybrid=True, reuse=True,
                       mode=rng.choice(("static", "reproject")), samples=rng.choice((1, 2, 4)),
                       max_fragments=1024)
    elif kind == "train":
        case = _train(None, "train_500k", _log_int(rng, 30_000, 500_000), _log_int(rng, 200, 800),
                      _log_int(rng, 200, 800), samples=rng.choice((2, 4, 8)), hybrid=rng.random() < 0.3,
                      bases=rng.choice((4, 16)))
    elif kind == "train_gps":
        case = _train(None, "st_100k", _log_int(rng, 10_000, 100_000), _log_int(rng, 200, 640),
                      _log_int(rng, 160, 480), gps=True, samples=rng.choice((2, 4)), hybrid=rng.random() < 0.3)
    elif kind == "denoise":
        case = dict(kind="denoise", batch=rng.choice((1, 2)), width=_log_int(rng, 320, 1280),
                    height=_log_int(rng, 180, 800))
    else:
        case = dict(kind="denoise_train", batch=rng.randint(2, 16), width=_log_int(rng, 64, 128),
                    height=_log_int(rng, 64, 128))
    case.pop("name", None)
    return case


def _scene(case, gen):
    spec, _ = SCENES[case["scene"]]
    n, dev = case["n"], "cuda"

    def normal(*shape):
        return torch.randn(shape, generator=gen, device=dev)

    if spec.means == "uniform":
        means = (torch.rand((n, 3), generator=gen, device=dev) * 2.0 - 1.0) * spec.means_scale
    else:
        means = normal(n, 3) * spec.means_scale
    scales = normal(n, 3) * spec.log_scale_std + spec.log_scale_mean
    rotations = normal(n, 4)
    rotations = rotations / rotations.norm(dim=1, keepdim=True).clamp_min(1e-12)
    opacities = normal(n) * spec.opacity_logit_std
    sh = normal(n, case["bases"], 3) * spec.sh_rest_std
    sh[:, 0, :] *= spec.sh_dc_std / spec.sh_rest_std
    order = torch.argsort(sgs_scenes.morton_codes(means), stable=True)
    return tuple(t[order].contiguous() for t in (means, scales, rotations, opacities, sh))


def _camera(case, angle):
    radius = SCENES[case["scene"]][1]
    return sgs_scenes.pinhole((radius * math.sin(angle), 0.0, -radius * math.cos(angle)), case["width"],
                              case["height"])


def _settings(case, cam):
    return Settings(cam.w2c.cuda(), cam.position.cuda(), cam.width, cam.height, cam.focal_x, cam.focal_y, cam.center_x,
                    cam.center_y, cam.near_plane, cam.far_plane, case["aa"], case["ss"], case["gps"], case["hybrid"],
                    case.get("reuse", False))


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    if case["kind"] == "denoise":
        b, h, w = case["batch"], case["height"], case["width"]
        return dict(case, features=_features(gen, b, h, w), model=denoise.Denoiser(_denoise_params(seed)))
    if case["kind"] == "denoise_train":
        b, h, w = case["batch"], case["height"], case["width"]
        return dict(case, features=_features(gen, b, h, w),
                    target=torch.rand((b, h, w, 3), generator=gen, device="cuda"),
                    params=[p.requires_grad_(True) for p in _denoise_params(seed)])
    scene = _scene(case, gen)
    angle = 2.0 * math.pi * ((seed * 0.6180339887) % 1.0)
    cam = _camera(case, angle)
    settings = _settings(case, cam)
    frame = 1000 + seed % 1000
    if case["kind"] == "train":
        shape = (case["height"], case["width"])
        pixels = shape[0] * shape[1]
        # the upstream gradient of a mean absolute error, and of a light mask and depth term
        return dict(case, params=[t.requires_grad_(True) for t in scene], settings=settings, frame=frame,
                    grads=(torch.sign(torch.randn((*shape, 3), generator=gen, device="cuda")) / (3 * pixels),
                           torch.randn((*shape, 1), generator=gen, device="cuda") * (0.01 / pixels),
                           torch.randn((*shape, 1), generator=gen, device="cuda") * (0.1 / pixels)))
    blue = (sgs_scenes.synthetic_blue_noise(0) if case["blue"] else torch.empty(0, dtype=torch.uint8)).cuda()
    n_fb = case["width"] * case["height"] * case["ss"] ** 2
    entries = _C.k_buffer_size if case["reuse"] else 0
    k_buffer = (torch.full((entries, n_fb, 2), -1, dtype=torch.int32, device="cuda"),
                torch.zeros((entries, n_fb, 4), device="cuda"))
    extra = dict(max_fragments=case["max_fragments"])
    if case["layout"] == "pre":
        extra["preactivated"] = _C.preactivate(*scene[1:4])
    elif case["layout"] == "quant":
        extra["quantized"] = _C.quantize(*scene)
    empty = torch.empty(0)
    history, view_to_previous = History(empty, empty, empty, empty), torch.eye(4, device="cuda")
    if case["mode"] != "reset":
        # the frame before: the same view, or the view of a camera that has since moved a little
        before = _camera(case, angle - 0.01) if case["mode"] == "reproject" else cam
        _C.set_frame_index(frame - 1)
        history = History(*_C.render(*scene, *_settings(dict(case, reuse=False), before).as_tuple(), blue,
                                     torch.empty((0, n_fb, 2), dtype=torch.int32, device="cuda"),
                                     torch.empty((0, n_fb, 4), device="cuda"), *history, view_to_previous, 0, **extra))
        view_to_previous = (before.w2c @ cam.c2w).contiguous().cuda()
    return dict(case, scene=scene, settings=settings, frame=frame, blue=blue, k_buffer=k_buffer, extra=extra,
                history=history, view_to_previous=view_to_previous)


def _features(gen, b, h, w):
    """Denoiser inputs with the ranges of rendered features: colour, alpha, depth / 32, noise, change rate, 0."""
    x = torch.rand((b, h, w, 8), generator=gen, device="cuda")
    x[..., 5] *= 0.2
    x[..., 7] = 0.0
    return x.half()


def _denoise_params(seed):
    params = denoise.init_params(seed)
    g = torch.Generator().manual_seed(seed + 1)
    params[10] = (torch.randn(params[10].shape, generator=g) * 0.02).cuda()  # trained: the last layer is not zero
    for l in range(6):
        params[2 * l + 1] = (torch.randn(params[2 * l + 1].shape, generator=g) * 0.05).cuda()
    return params


MODES = {"reset": TemporalMode.RESET, "static": TemporalMode.STATIC, "reproject": TemporalMode.REPROJECT}


def run(s):
    if s["kind"] == "denoise":
        return s["model"](s["features"])
    if s["kind"] == "denoise_train":
        out = denoise.denoise_train(s["features"], s["params"])
        loss = F.mse_loss(out, s["target"])
        return out.detach(), torch.autograd.grad(loss, s["params"])
    if s["kind"] == "train":
        outs = autograd.render_samples(*s["params"], s["settings"], n_samples=s["samples"], first_frame=s["frame"])
        return tuple(t.detach() for t in outs), torch.autograd.grad(outs, s["params"], grad_outputs=s["grads"])
    _C.set_frame_index(s["frame"])  # the same sample on every pass
    k_prims, k_occlusion = s["k_buffer"]
    if s["reuse"]:
        k_prims.fill_(-1)  # a frame after a change of the scene: an empty k-buffer
        k_occlusion.zero_()
    if s["samples"] > 1 or s["blue"].numel():
        args = (*s["scene"], *s["settings"].as_tuple(), s["blue"], k_prims, k_occlusion, *s["history"],
                s["view_to_previous"], int(MODES[s["mode"]]))
        outs = _C.render_samples(s["samples"], *args, **s["extra"]) if s["samples"] > 1 else _C.render(*args, **s["extra"])
    else:
        outs = render(*s["scene"], s["settings"], s["k_buffer"], s["history"], s["view_to_previous"], MODES[s["mode"]],
                      **s["extra"])
    return tuple(outs) + ((k_prims, k_occlusion) if s["reuse"] else ())


def work(case):
    px = case["width"] * case["height"]
    if case["kind"].startswith("denoise"):
        px *= case["batch"]
        macs = 9 * (7 * 32 + 4 * 32 * 32 + 32 * 3)
        if case["kind"] == "denoise":
            return {"bytes": px * (16 + 12), "flops": 2 * macs * px}
        # forward, weight gradients, data gradients of every layer but the first
        return {"bytes": px * (16 + 12 + 12), "flops": 2 * px * (2 * macs + macs - 9 * 7 * 32)}
    n, fb = case["n"], px * case["ss"] ** 2
    # about a fifth of the subpixels have a winner of their own, whose mean and SH are read
    winners = (12 + 12 * case["bases"]) * min(n, fb) // 5
    if case["kind"] == "train":
        # parameters, their gradients, outputs, upstream gradients
        return {"bytes": n * 2 * (44 + 12 * case["bases"]) + px * 40, "flops": 0}
    per = {"float": 44, "pre": 44, "quant": 16}[case["layout"]]
    total = n * per + (winners // 2 if case["layout"] == "quant" else winners) + 24 * px
    if case["mode"] != "reset":
        total += 24 * px
    if case["reuse"]:
        total += fb * 4 * 24 * 2
    return {"bytes": total, "flops": 0}


def exact(case, seed):
    # A render's outputs hang on which of two float32 numbers is the larger at every fragment (the threshold and the
    # alpha), and the gradients on the same winners: 64-bit arithmetic has other winners, not a more exact value.
    if case["kind"] not in ("denoise", "denoise_train"):
        return None
    s = prepare(case, seed)
    params = [p.detach().double() for p in (s["model"].params if case["kind"] == "denoise" else s["params"])]
    if case["kind"] == "denoise_train":
        params = [p.requires_grad_(True) for p in params]
    features = s["features"].double().permute(0, 3, 1, 2)
    x = features[:, :7]
    for l in range(6):
        x = F.conv2d(x, params[2 * l], params[2 * l + 1], padding=1)
        if l < 5:
            x = F.relu(x)
    out = (x + features[:, :3]).permute(0, 2, 3, 1).contiguous()
    if case["kind"] == "denoise":
        return out
    loss = F.mse_loss(out, s["target"].double())
    return out.detach(), torch.autograd.grad(loss, params)
