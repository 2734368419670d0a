"""CPU: the oracle's float64 gradients against the reference extension's golden gradients and against finite differences of the
oracle's own forward pass."""
import copy
import os

import numpy as np
import pytest

from golden.make_golden import CASES, target_image
from htgs_b200 import scenes
from test_oracle_golden import GOLDEN, all_cases

NAMES = ("positions", "scales", "rotations", "opacities", "sh_0", "sh_rest")


def gradients(oracle, scene, view, mode, K, grad_image):
    pre = oracle.preprocess(scene, view, mode, dtype=np.float64, with_clamp=True)
    grid_w, grid_h = oracle.grid_of(view, mode)
    bins = oracle.bin_instances(pre["n_touched"], pre["bounds"], grid_w, grid_w * grid_h, pre["mt3"][:, 3] if mode == 2 else None)
    return oracle.backward(scene, view, mode, K, bins["ranges"], bins["sorted_prims"], grad_image, pre)


@pytest.mark.parametrize("name,mode,K", list(all_cases()))
def test_gradients_match_the_reference(oracle_lib, name, mode, K):
    scene = scenes.tiny_scene(**CASES[name]["kwargs"])
    view = scene.views[0]
    gold = np.load(os.path.join(GOLDEN, f"{name}.npz"))
    tag = f"m{mode}_k{K}"
    difference = gold[f"{tag}_train_image"].astype(np.float64) - target_image(view.height, view.width, 1000 + mode)
    got = gradients(oracle_lib, scene, view, mode, K, np.sign(difference) / difference.size)
    for grad, field in zip(got, NAMES):
        want = gold[f"{tag}_grad_{field}"]
        if want.size:       # the reference sums in float32, and a fragment on a threshold may fall on either side
            assert np.linalg.norm(grad - want) <= 1e-3 * np.linalg.norm(want), field


@pytest.mark.parametrize("mode,K", [(0, 4), (1, 4), (2, 1), (3, 1)])
def test_gradients_match_finite_differences(oracle_lib, mode, K):
    scene = scenes.tiny_scene(n=24, size=24, seed=5 + mode, sh_degree=3)
    scene.scales *= 2.5
    scene.opacities[:] = np.clip(scene.opacities, 0.15, 0.85)
    view = scene.views[0]
    weights = np.random.default_rng(mode).standard_normal((3, view.height, view.width))
    grads = gradients(oracle_lib, scene, view, mode, K, weights)
    agreed = 0
    for grad, field in zip(grads, NAMES):
        for index in np.argsort(-np.abs(grad).ravel())[:4]:
            at = np.unravel_index(index, grad.shape)
            values = []
            for sign in (1.0, 0.0, -1.0):
                moved = copy.deepcopy(scene)
                array = getattr(moved, field)
                array[at] += np.float32(sign * 2e-4)
                image = oracle_lib.render(moved, view, mode=mode, K=K, dtype=np.float64)[0]
                assert image.max() < 1.0            # the rendered image is clamped, the training image is not
                values.append((float((image * weights).sum()), float(array[at])))
            (up, x_up), (mid, x_mid), (down, x_down) = values
            one_sided = (up - mid) / (x_up - x_mid), (mid - down) / (x_mid - x_down)
            if abs(one_sided[0] - one_sided[1]) > 0.02 * max(map(abs, one_sided)):
                continue                            # a threshold or a change of order inside the step
            assert abs((up - down) / (x_up - x_down) - grad[at]) <= 0.01 * abs(grad[at]), (field, at)
            agreed += 1
    assert agreed >= 14
