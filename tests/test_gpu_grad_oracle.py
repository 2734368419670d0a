"""GPU: gradients of `diff_rasterize` against the oracle's float64 gradients."""
import numpy as np
import pytest

import harness
from htgs_b200 import scenes
from test_oracle_backward import gradients

pytestmark = pytest.mark.gpu


def tilted_scene(seed):
    """Long, thin Gaussians close to the camera whose long axis points 75 degrees out of the image plane: perspective moves their outlines
    far from their projected centres, and each reaches over hundreds of tiles."""
    scene = scenes.tiny_scene(n=16, size=768, seed=seed, sh_degree=0)
    rng = np.random.default_rng(seed)
    scene.positions[:, 2] = rng.uniform(0.42, 0.5, scene.n)
    scene.positions[:, :2] = rng.uniform(-0.4, 0.4, (scene.n, 2)) * scene.positions[:, 2:]
    scene.scales[:] = (0.006, 0.06, 0.006)
    tilt, turn = np.radians(rng.uniform(67, 83, scene.n)) / 2, rng.uniform(0, 2 * np.pi, scene.n) / 2
    scene.rotations[:] = np.stack([np.cos(turn) * np.cos(tilt), np.cos(turn) * np.sin(tilt), np.sin(turn) * np.sin(tilt), np.sin(turn) * np.cos(tilt)], 1)
    scene.opacities[:] = rng.uniform(0.3, 0.9, (scene.n, 1))
    return scene, scene.views[0]


def needle_scene(seed):
    """Gaussians a hundred times as long as thick, at all angles."""
    scene = scenes.tiny_scene(n=16, size=768, seed=seed, sh_degree=0)
    rng = np.random.default_rng(seed)
    scene.positions[:, 2] = rng.uniform(3.0, 6.0, scene.n)
    scene.positions[:, :2] = rng.uniform(-0.3, 0.3, (scene.n, 2)) * scene.positions[:, 2:]
    scene.scales[:] = (0.005, 0.5, 0.005)
    scene.opacities[:] = rng.uniform(0.5, 0.9, (scene.n, 1))
    return scene, scene.views[0]


@pytest.mark.parametrize("mode,K", [(0, 16), (0, 32), (1, 8), (2, 1), (3, 1)])
@pytest.mark.parametrize("seed", [0, 1, 2, 3])
@pytest.mark.parametrize("make_scene", [tilted_scene, needle_scene])
def test_sums_over_many_tiles(oracle_lib, mode, K, seed, make_scene):
    """Against float64 sums over the same rounded rows and core entries: what is left is the rounding of the pairs and of the sums.  A Gaussian has
    up to 3000 partial sums, added in no fixed order: roundings of 2^-25 on average give sqrt(3000) * 2^-25 = 1.6e-6 of a sum."""
    import torch
    tb = harness.ours()
    scene, view = make_scene(seed)
    leaves = [t.requires_grad_() for t in harness.scene_tensors(scene)]
    image = tb.diff_rasterize(*leaves, torch.empty(0, device="cuda"), harness.settings_for(tb, scene, view, mode, K), False)
    weights = np.random.default_rng(7 + seed).choice([-1.0, 1.0], image.shape)       # signs, as an L1 loss gives them
    blobs = [t.cpu().numpy() for t in image.grad_fn.saved_tensors[-4:]]
    n_instances = image.grad_fn.n_instances
    image.backward(torch.from_numpy(weights).float().cuda())
    rows, ranges, prims, core = harness.training_blobs(scene, view, mode, K, blobs, n_instances)
    want = oracle_lib.backward(scene, view, mode, K, ranges, prims, weights, rows, core)
    for leaf, grad, name in zip(leaves[:4], want, ("positions", "scales", "rotations", "opacities")):
        assert np.linalg.norm(leaf.grad.cpu().numpy() - grad) <= 3e-6 * np.linalg.norm(grad), name


def mirrored_pair_scene():
    """One Gaussian on the optical axis of an 8 x 8 image: pixels 3 and 4 of a row lie symmetrically about it."""
    scene = scenes.tiny_scene(n=1, size=8, seed=1, sh_degree=0)
    scene.positions[:] = (0.0, 0.0, 4.0)
    scene.scales[:] = 0.8
    scene.rotations[:] = (1.0, 0.0, 0.0, 0.0)
    scene.opacities[:] = 0.5
    scene.sh_0[:] = 0.5
    return scene, scene.views[0]


@pytest.mark.parametrize("mode,K", [(0, 4), (1, 4), (2, 1), (3, 1)])
def test_opposite_gradients_of_a_mirrored_pair(oracle_lib, mode, K):
    """The gradients of colour and opacity cancel, that of the position does not."""
    import torch
    tb = harness.ours()
    scene, view = mirrored_pair_scene()
    weights = np.zeros((3, 8, 8))
    weights[:, 2, 3], weights[:, 2, 4] = 1.0, -1.0
    leaves = [t.requires_grad_() for t in harness.scene_tensors(scene)]
    image = tb.diff_rasterize(*leaves, torch.empty(0, device="cuda"), harness.settings_for(tb, scene, view, mode, K), False)
    image.backward(torch.from_numpy(weights).float().cuda())
    want = gradients(oracle_lib, scene, view, mode, K, weights)
    assert abs(want[0][0, 0]) > 0.1
    for leaf, grad in zip(leaves[:5], want):         # a few dozen float32 operations on numbers of this size
        assert np.abs(leaf.grad.cpu().numpy() - grad).max() <= 1e-5 * abs(want[0][0, 0])
