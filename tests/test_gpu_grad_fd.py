"""GPU: gradients of `diff_rasterize` against central finite differences of the float64 CPU oracle's forward.

An independent check of the backward pass (the other gradient tests compare with the reference's gradients): for a tiny
scene the loss L = mean |image - target| is evaluated with the oracle at theta +- h for a sample of parameter entries, and
(L+ - L-) / 2h must agree with the CUDA gradient.  The forward has thresholds (alpha cutoffs, K-buffer membership and
order), so an entry whose two one-sided differences disagree (a discontinuity inside the step) is skipped; at least
two thirds of the sampled entries must remain and agree to 2 % (plus a small absolute floor)."""
import copy

import numpy as np
import pytest

import harness
from htgs_b200 import scenes
from golden.make_golden import target_image

pytestmark = pytest.mark.gpu

PARAMS = ("positions", "scales", "rotations", "opacities", "sh_0", "sh_rest")


def oracle_loss(oracle_lib, scene, view, mode, K, target):
    img, _, _, _ = oracle_lib.render(scene, view, mode=mode, K=K, dtype=np.float64)
    return float(np.abs(img - target).mean())


@pytest.mark.parametrize("mode,K", [(0, 4), (1, 4), (2, 1), (3, 1)])
def test_gradients_against_finite_differences(oracle_lib, mode, K):
    import torch
    scene = scenes.tiny_scene(n=48, size=32, seed=77 + mode, sh_degree=1)
    scene.scales *= 2.5                       # larger footprints: every Gaussian covers many pixels
    scene.opacities[:] = np.clip(scene.opacities, 0.15, 0.85)
    view = scene.views[0]
    target = target_image(view.height, view.width, 1000 + mode).astype(np.float64) * 0.2   # keep |image - target| away from its kink
    ours = harness.ours()
    leaves = [t.clone().requires_grad_(True) for t in harness.scene_tensors(scene)]
    st = harness.settings_for(ours, scene, view, mode, K)
    image = ours.diff_rasterize(*leaves, torch.empty(0, device="cuda"), st, False)
    assert image.max().item() < 1.0           # the oracle's inference image is clamped to [0, 1]; stay below the clamp
    loss = (image - torch.from_numpy(target).float().cuda()).abs().mean()
    loss.backward()
    grads = {name: leaf.grad.cpu().numpy().astype(np.float64) for name, leaf in zip(PARAMS, leaves)}
    base = oracle_loss(oracle_lib, scene, view, mode, K, target)
    assert abs(base - loss.item()) <= 1e-5 * max(1.0, abs(base))

    rng = np.random.default_rng(5 + mode)
    checked = agreed = skipped = 0
    for name in PARAMS:
        arr = getattr(scene, name)
        if arr.size == 0:
            continue
        g = grads[name].reshape(arr.shape)
        # sample among the entries with a noticeable gradient
        flat = np.argsort(-np.abs(g).reshape(-1))[: max(8, arr.size // 8)]
        for idx in rng.choice(flat, size=min(6, flat.size), replace=False):
            ix = np.unravel_index(int(idx), arr.shape)
            h = 1e-4 * max(1.0, abs(float(arr[ix])))
            losses = []
            for sign in (+1.0, -1.0):
                s2 = copy.deepcopy(scene)
                a2 = getattr(s2, name).astype(np.float64)
                a2[ix] += sign * h
                setattr(s2, name, a2.astype(np.float32))
                step = float(getattr(s2, name)[ix]) - float(arr[ix])   # the step actually taken in float32
                losses.append((oracle_loss(oracle_lib, s2, view, mode, K, target), step))
            (lp, hp), (lm, hm) = losses
            if hp == 0.0 or hm == 0.0:
                continue
            d_plus, d_minus = (lp - base) / hp, (lm - base) / hm
            checked += 1
            if abs(d_plus - d_minus) > 0.05 * max(abs(d_plus), abs(d_minus)) + 1e-9:
                skipped += 1                  # a threshold or a change of order inside the step
                continue
            fd = (lp - lm) / (hp - hm)
            if name == "rotations":
                # the rasterizer treats the quaternion as given (no normalisation inside), so does the oracle: comparable as is
                pass
            assert abs(fd - g[ix]) <= 0.02 * abs(fd) + 2e-7, f"{name}{ix}: finite difference {fd:.6e} vs gradient {g[ix]:.6e}"
            agreed += 1
    assert checked >= 20 and agreed >= (2 * checked) // 3, (checked, agreed, skipped)


@pytest.mark.parametrize("mode", [0, 1, 2, 3])
@pytest.mark.parametrize("rows", [0, 3])
@pytest.mark.parametrize("value", [float("nan"), float("inf")])
def test_bad_pixel_gradient_stays_with_the_gaussians_of_the_pixel(mode, rows, value):
    # a NaN or an infinity in one pixel's gradient reaches the Gaussians that the pixel accepted and no other; those are the ones that
    # have a gradient when only this pixel has one
    import torch
    tb = harness.ours()
    scene = scenes.tiny_scene(n=2000, size=64, seed=5, mode=mode, K=8, sh_degree=1)

    def gradients(grad_image):
        leaves = [t.requires_grad_() for t in harness.scene_tensors(scene)]
        densification = torch.zeros(rows, scene.n, 1, device="cuda") if rows else torch.empty(0, device="cuda")
        tb.diff_rasterize(*leaves, densification, harness.settings_for(tb, scene, scene.views[0], mode, 8), False).backward(grad_image)
        return torch.cat([t.grad.reshape(scene.n, -1) for t in leaves] + ([densification[1:].reshape(rows - 1, scene.n).T] if rows else []), dim=1)

    generator = torch.Generator(device="cuda").manual_seed(1)
    everywhere = torch.rand(3, 64, 64, device="cuda", generator=generator) + 0.5
    for y, x in ((20, 37), (32, 32), (47, 24)):
        only_here, without, bad = torch.zeros_like(everywhere), everywhere.clone(), everywhere.clone()
        only_here[:, y, x], without[:, y, x], bad[:, y, x] = 1.0, 0.0, value
        touched = (gradients(only_here) != 0).any(dim=1)
        assert touched.any() and not touched.all()
        got, want = gradients(bad), gradients(without)
        assert torch.isfinite(got[~touched]).all() and not torch.isfinite(got[touched]).all()
        # sums of one Gaussian over its pixels in another order: a few float32 roundings of the largest gradient
        assert torch.allclose(got[~touched], want[~touched], rtol=1e-4, atol=1e-5 * float(want.abs().max()))
