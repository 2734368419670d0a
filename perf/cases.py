"""The work a user of the rasterizer has it do, as measurable cases.

Each case is one pass through the public Python surface (`htgs_b200.torch_bindings`, `htgs_b200.glue`): a rendered frame, a short
sequence of frames, a training step, the importance update, or the 3D-filter update of all training views.  Scenes are the seeded
synthetic ones of `htgs_b200.scenes` (same distributions, drawn on the GPU); sizes are those of the benchmark configurations and
of the tests.  All tensors are float32, the only type the rasterizer takes.
"""
import math

import numpy as np
import torch
import torch.nn.functional as F

import htgs_b200.torch_bindings as tb
from htgs_b200 import glue, scenes

HYBRID, FIRST_K, GLOBAL, OIT = 0, 1, 2, 3
DEVICE = "cuda"


def _case(kind, n, width, height, focal, mode=HYBRID, K=16, sh=3, active=None, layout="mixture", components=64, ball=10.0, log_scale=-4.5,
          views=1, hwc=False, median=False, rows=0, distance_scaling=False):
    return {"kind": kind, "n": n, "width": width, "height": height, "focal": focal, "mode": mode, "K": K, "sh": sh, "active": sh if active is None else active,
            "layout": layout, "components": components, "ball": ball, "log_scale": log_scale, "views": views, "hwc": hwc, "median": median, "rows": rows,
            "distance_scaling": distance_scaling}


def listed():
    return [
        # An object viewer's frame: few Gaussians, small window, one blocking call per mouse move; latency is all there is.
        dict(_case("render", 16384, 256, 256, 256.0, sh=0, layout="cloud", log_scale=-3.0), name="render_tiny"),
        # A mid-sized object in a ragged window, first-K blending, SH degree 2.
        dict(_case("render", 300_001, 501, 333, 437.0, mode=FIRST_K, K=8, sh=2, log_scale=-3.9), name="render_ragged_first_k"),
        # The headline frame: outdoor scene at full evaluation resolution (image + mean depth).
        dict(_case("render", 3_000_000, 1297, 840, 1150.0), name="render_outdoor"),
        # Evaluation of a test set: views of the outdoor scene one after the other, frames queued without a host wait on two streams.
        dict(_case("frames", 3_000_000, 1297, 840, 1150.0, views=8), name="frames_outdoor"),
        # Globally sorted blending with median depth, image handed on as HWC (what a viewer or an encoder wants).
        dict(_case("render", 1_500_000, 980, 545, 580.0, mode=GLOBAL, K=1, components=32, ball=6.0, hwc=True, median=True), name="render_compact_global"),
        # The largest frame: 8 M Gaussians with dense clusters in front of the cameras, 4K, deep buffer.
        dict(_case("render", 8_000_000, 3840, 2160, 3000.0, K=32, layout="stress", log_scale=-5.5), name="render_4k"),
        # The relaxed-precision path on the headline frame (frame rate benchmarks, interactive viewing).
        dict(_case("fast", 3_000_000, 1297, 840, 1150.0), name="fast_outdoor"),
        # A training step early on: about as many Gaussians as a structure-from-motion cloud has points, SH not yet active, densification
        # statistics gathered, training images at reduced resolution.
        dict(_case("train", 100_003, 649, 420, 575.0, active=0, log_scale=-3.5, rows=2), name="train_start"),
        # A training step at full size, after densification.
        dict(_case("train", 3_000_000, 1297, 840, 1150.0), name="train_outdoor"),
        # A training step under global ordering while the densification statistics (with absolute gradients) are gathered.
        dict(_case("train", 1_500_000, 980, 545, 580.0, mode=GLOBAL, K=1, components=32, ball=6.0, rows=3, distance_scaling=True), name="train_compact_global"),
        # One view of importance pruning: the largest blending weight of every Gaussian.
        dict(_case("weights", 3_000_000, 1297, 840, 1150.0), name="weights_outdoor"),
        # The 3D filter after densification: every training view against every Gaussian.
        dict(_case("filter", 3_000_000, 1297, 840, 1150.0, views=200), name="filter_views"),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["render", "frames", "fast", "train", "weights", "filter"], [30, 8, 20, 28, 7, 7])[0]
    if kind == "filter":
        n, width = _log_uniform(rng, 16384, 8_000_000), _log_uniform(rng, 256, 3840)
        return _case(kind, n, width, max(144, int(width * rng.uniform(0.55, 0.75))), width * rng.uniform(0.59, 1.0), views=rng.randint(1, 300))
    # whole frames go up to the largest scene at 4K; training and its companions run at up to 1600 pixels, as the method's datasets do
    n_hi, w_hi = (8_000_000, 3840) if kind in ("render", "fast") else (3_000_000, 1600) if kind in ("train", "weights") else (3_000_000, 1297)
    n, width = _log_uniform(rng, 16384, n_hi), _log_uniform(rng, 256, w_hi)
    height = max(144, int(width * rng.uniform(0.55, 1.0 if width < 1000 else 0.66)))
    mode = rng.choices([HYBRID, FIRST_K, GLOBAL, OIT], [55, 15, 15, 15])[0]
    K = rng.choice([4, 8, 16, 16, 16, 32] if kind != "frames" else [8, 16]) if mode in (HYBRID, FIRST_K) else 1
    sh = rng.choice([0, 1, 2, 3, 3, 3])
    layout = "cloud" if n < 100_000 and rng.random() < 0.5 else "mixture"
    # denser scenes have smaller Gaussians, as densification makes them
    log_scale = -3.0 - 0.4 * math.log(n / 16384.0) + rng.uniform(-0.3, 0.2)
    return _case(kind, n, width, height, width * rng.uniform(0.59, 1.0), mode, K, sh, rng.randint(0, sh) if kind == "train" else sh, layout,
                 rng.choice([32, 64]), rng.choice([6.0, 10.0]), log_scale, views=rng.randint(2, 8) if kind == "frames" else 1, hwc=rng.random() < 0.3,
                 median=rng.random() < 0.3, rows=rng.choice([0, 2, 3]) if kind == "train" else 0, distance_scaling=rng.random() < 0.3)


def _camera(case, rng):
    """World -> view matrix and position of one camera: the identity for a cloud in front of it, else a point of the orbit."""
    if case["layout"] == "cloud":
        return np.eye(4), np.zeros(3)
    phi = 2.0 * math.pi * rng.integers(0, 200) / 200
    position = np.array([4.0 * math.cos(phi), 1.5, 4.0 * math.sin(phi)])
    return scenes.look_at(position), position


def _settings(case, w2c, position):
    return glue.extract_settings(w2c, case["focal"], case["focal"], case["width"] / 2.0, case["height"] / 2.0, case["width"], case["height"], 0.2,
                                 100.0 if case["layout"] == "cloud" else 1000.0, position, case["mode"], case["K"], (case["active"] + 1) ** 2)


def _positions(case, g):
    n = case["n"]
    rand, randn = (lambda *s: torch.rand(*s, device=DEVICE, generator=g)), (lambda *s: torch.randn(*s, device=DEVICE, generator=g))
    if case["layout"] == "cloud":
        return torch.cat([2.0 * rand(n, 2) - 1.0, 2.0 + 4.0 * rand(n, 1)], dim=1)

    def mixture(count):
        centres = F.normalize(randn(case["components"], 3)) * (case["ball"] * rand(case["components"], 1) ** (1.0 / 3.0))
        sigma = 0.3 + 1.7 * rand(case["components"], 1)
        which = torch.randint(0, case["components"], (count,), device=DEVICE, generator=g)
        return centres[which] + sigma[which] * randn(count, 3)

    if case["layout"] == "mixture":
        return mixture(n)
    # half of the Gaussians in a ring of 64 dense clusters, 1.5 units in front of 64 cameras of the orbit
    cameras = np.stack([(4.0 * math.cos(a), 1.5, 4.0 * math.sin(a)) for a in 2.0 * np.pi * np.arange(64) / 64])
    centres = torch.as_tensor(np.stack([p + 1.5 * scenes.look_at(p)[2, :3] for p in cameras]), dtype=torch.float32, device=DEVICE)
    which = torch.randint(0, 64, (n // 2,), device=DEVICE, generator=g)
    return torch.cat([centres[which] + 0.5 * randn(n // 2, 3), mixture(n - n // 2)])[torch.randperm(n, device=DEVICE, generator=g)]


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    g = torch.Generator(device=DEVICE).manual_seed(int(seed))
    n, rest = case["n"], (case["sh"] + 1) ** 2 - 1
    state = {"case": case, "cameras": [_camera(case, rng) for _ in range(case["views"])], "positions": _positions(case, g)}
    if case["kind"] == "filter":
        state["w2cs"] = torch.as_tensor(np.stack([w2c for w2c, _ in state["cameras"]]), dtype=torch.float32)
        return state

    def randn(*shape):
        return torch.randn(*shape, device=DEVICE, generator=g)

    raw_scales = case["log_scale"] + (0.5 if case["layout"] == "cloud" else 1.0) * randn(n, 3)
    raw_rotations, raw_opacities = randn(n, 4), (1.0 if case["layout"] == "cloud" else 1.5) * randn(n, 1)
    sh_0, sh_rest = 0.3 * randn(n, 1, 3), 0.05 * randn(n, rest, 3)
    if case["kind"] == "train":     # raw parameters with gradients, the view's target image, and the running densification statistics
        state["raw"] = [t.requires_grad_() for t in (state.pop("positions"), raw_scales, raw_rotations, raw_opacities, sh_0, sh_rest)]
        state["target"] = torch.rand(3, case["height"], case["width"], device=DEVICE, generator=g)
        state["densification"] = torch.zeros(case["rows"], n, 1, device=DEVICE) if case["rows"] else torch.empty(0, device=DEVICE)
        return state
    # a loaded model: activated once, then rendered from many cameras
    scales, rotations, opacities = glue.activate(raw_scales, raw_rotations, raw_opacities)
    state["model"] = [state["positions"], scales, rotations, opacities, sh_0, sh_rest]
    return state


_streams = []


def _frames(state):
    """Frames in flight on two streams from one host thread; their status is checked once, at the end."""
    case = state["case"]
    if not _streams:
        _streams.extend(torch.cuda.Stream() for _ in range(2))
    caller = torch.cuda.current_stream()
    outputs = []
    tb.rasterization.set_deferred_checks(True)
    try:
        for s in _streams:
            s.wait_stream(caller)
        for k, camera in enumerate(state["cameras"]):
            with torch.cuda.stream(_streams[k % 2]):
                outputs.append(tb.rasterize(*state["model"], _settings(case, *camera), not case["hwc"], case["median"]))
        for s in _streams:
            caller.wait_stream(s)
        tb.rasterization.frame_results()
    finally:
        tb.rasterization.set_deferred_checks(False)
    return outputs


def _train(state):
    case, raw = state["case"], state["raw"]
    for p in raw:
        p.grad = None
    positions, raw_scales, raw_rotations, raw_opacities, sh_0, sh_rest = raw
    scales, rotations, opacities = glue.activate(raw_scales, raw_rotations, raw_opacities)
    image = tb.diff_rasterize(positions, scales, rotations, opacities, sh_0, sh_rest, state["densification"], _settings(case, *state["cameras"][0]),
                              case["distance_scaling"])
    F.l1_loss(image, state["target"]).backward()
    return {"image": image.detach(), "gradients": [p.grad for p in raw], "densification": state["densification"]}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "frames":
        return _frames(state)
    if kind == "train":
        return _train(state)
    if kind == "filter":
        n, views = case["n"], case["views"]
        filter_3d = torch.full((n, 1), torch.finfo(torch.float32).max, device=DEVICE)
        visible = torch.zeros(n, dtype=torch.bool, device=DEVICE)
        tb.update_3d_filter_views(state["positions"], state["w2cs"], filter_3d, visible, [case["width"]] * views, [case["height"]] * views,
                                  [case["focal"]] * views, [case["focal"]] * views, [case["width"] / 2.0] * views, [case["height"] / 2.0] * views,
                                  [0.2] * views, 0.15, 0.2 ** 0.5 / case["focal"])
        return {"filter": filter_3d, "visible": visible}
    settings = _settings(case, *state["cameras"][0])
    if kind == "weights":
        weights = torch.zeros(case["n"], 1, device=DEVICE)
        tb.update_max_weights(weights, *state["model"][:4], settings, 0.01)
        return weights
    if kind == "fast":
        return tb.fast_rasterize(*state["model"], settings, not case["hwc"])
    return tb.rasterize(*state["model"], settings, not case["hwc"], case["median"])


def work(case):
    """Inputs once in, outputs once out; arithmetic from the expected number of accepted fragments: a sixth of the Gaussians is visible,
    and each covers pi * 9 * sigma_1 * sigma_2 pixels at a typical depth."""
    n, pixels, kind = case["n"], case["width"] * case["height"], case["kind"]
    if kind == "filter":
        return {"bytes": n * (12 + 4 + 1), "flops": n * case["views"] * 8.0}
    coefficients = 3 * (case["active"] + 1) ** 2
    spread, depth = (0.5, 4.0) if case["layout"] == "cloud" else (1.0, 6.0)
    area = min(float(pixels), math.pi * 9.0 * math.exp(2.0 * case["log_scale"] + spread * spread) * (case["focal"] / depth) ** 2)
    fragments = n * (1.0 if case["layout"] == "cloud" else 1.0 / 6.0) * area
    per_fragment = 114.0 + (7.0 * case["K"] if case["mode"] in (HYBRID, FIRST_K) else 0.0)
    forward = 250.0 * n + per_fragment * fragments
    if kind == "train":     # parameters in, gradients out (every coefficient's gradient is written, active or not), image, target, statistics
        return {"bytes": 4.0 * (n * (11 + coefficients + 11 + 3 * (case["sh"] + 1) ** 2 + 2 * case["rows"]) + 6 * pixels), "flops": 3.0 * forward}
    if kind == "weights":
        return {"bytes": 4.0 * n * 12, "flops": forward}
    frames = case["views"] if kind == "frames" else 1
    return {"bytes": 4.0 * (n * (11 + coefficients) + frames * pixels * (3 if kind == "fast" else 4)), "flops": frames * forward}


def tolerance(case):
    kind = case["kind"]
    if kind == "fast":      # colours are buffered in half precision; now and then a fragment changes sides between buffer and tail
        return {"rel": 5e-4, "max": 0.05}
    if kind == "train":     # float32 sums over thousands of pixels in no fixed order; single rows cancel
        return {"rel": 5e-5, "max": 0.05}
    if kind == "filter":
        return {"rel": 1e-6, "max": 1e-5, "differ": 1e-6}
    return {"rel": 1e-5, "max": 1e-3}
