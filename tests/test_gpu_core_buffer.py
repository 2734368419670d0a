"""GPU: the K-buffer's two forms (unsorted keys, insertion chain) and the pixel blocks at ragged edges.

The unsorted form serves depth ranges its keys cover, the chain everything else; a far plane of 3e38 selects the chain for a
scene that both see in full, so the two renders have to agree bit for bit, ties in depth included.
"""
import numpy as np
import pytest

import harness
from htgs_b200 import scenes

pytestmark = pytest.mark.gpu


def scene_with_ties(n, width, height, K, mode, seed=5):
    scene = scenes.tiny_scene(n=n, size=max(width, height), seed=seed, mode=mode, K=K, sh_degree=1)
    # every third Gaussian sits where its predecessor sits, with the same shape: equal depth at every pixel, other colour and opacity
    for a in (scene.positions, scene.scales, scene.rotations):
        a[2::3] = a[1::3][: len(a[2::3])]
    view = scene.views[0]
    view.width, view.height = width, height
    return scene, view


def render(scene, view, mode, K, near, far, median):
    import torch
    tb = harness.ours()
    wide = scenes.make_view(view.M, view.width, view.height, 256.0, 256.0, view.width / 2.0, view.height / 2.0, near, far)
    st = harness.settings_for(tb, scene, wide, mode, K)
    image, depth = tb.rasterize(*harness.scene_tensors(scene), st, True, median)
    torch.cuda.synchronize()
    return image.cpu().numpy(), depth.cpu().numpy()


@pytest.mark.parametrize("mode,K", [(0, 4), (0, 8), (0, 16), (0, 32), (1, 4), (1, 8), (1, 16), (1, 32)])
@pytest.mark.parametrize("n,width,height", [(6000, 256, 256), (40, 7, 3), (900, 129, 61), (3000, 33, 250)])
def test_unsorted_buffer_equals_the_chain(mode, K, n, width, height):
    scene, view = scene_with_ties(n, width, height, K, mode)
    for median in (False, True):
        got = render(scene, view, mode, K, 0.2, 100.0, median)
        want = render(scene, view, mode, K, 0.2, 3e38, median)
        assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
        assert got[0].max() > 0.0


@pytest.mark.parametrize("mode,K", [(0, 8), (1, 16)])
def test_training_forward_and_gradients_agree_between_the_two_forms(mode, K):
    import torch
    tb = harness.ours()
    scene, view = scene_with_ties(3000, 131, 77, K, mode)
    outs = []
    for near, far in ((0.2, 100.0), (0.2, 3e38)):
        wide = scenes.make_view(view.M, view.width, view.height, 256.0, 256.0, view.width / 2.0, view.height / 2.0, near, far)
        tensors = [t.requires_grad_() for t in harness.scene_tensors(scene)]
        image = tb.diff_rasterize(*tensors, torch.empty(0, device="cuda"), harness.settings_for(tb, scene, wide, mode, K), False)
        image.square().sum().backward()
        outs.append((image.detach(), [t.grad for t in tensors]))
    assert torch.equal(outs[0][0], outs[1][0])
    for a, b in zip(outs[0][1], outs[1][1]):
        assert torch.allclose(a, b, rtol=1e-4, atol=1e-5 * float(b.abs().max()))


def scene_with_copies(n, size, K, mode, copies, seed):
    """Every Gaussian `copies` times, at random places of the list: between two copies of one Gaussian others arrive in front of and
    behind them.  Colours and opacities differ."""
    scene = scenes.tiny_scene(n=n, size=size, seed=seed, mode=mode, K=K, sh_degree=1)
    of = np.random.default_rng(seed).permutation(n) // copies
    for a in (scene.positions, scene.scales, scene.rotations):
        a[:] = a[of]
    scene.scales *= 1.5
    scene.opacities[:] = np.clip(scene.opacities, 0.1, 0.6)
    return scene, scene.views[0]


@pytest.mark.parametrize("mode,K", [(0, 4), (0, 8), (0, 16), (0, 32), (1, 4), (1, 8), (1, 16), (1, 32)])
@pytest.mark.parametrize("copies", [3, 4, 7])
def test_three_and_more_entries_of_one_depth(mode, K, copies):
    # 64 x 64 pixels run the form that keeps colours, 512 x 512 the other one
    for size, n in ((64, 3000), (512, 6000)):
        scene, view = scene_with_copies(n, size, K, mode, copies, seed=31 + copies)
        for median in (False, True):
            got = render(scene, view, mode, K, 0.2, 100.0, median)
            want = render(scene, view, mode, K, 0.2, 3e38, median)
            assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])


@pytest.mark.parametrize("mode,K", [(0, 8), (1, 16)])
def test_training_forward_with_three_entries_of_one_depth(mode, K):
    import torch
    tb = harness.ours()
    scene, view = scene_with_copies(4000, 160, K, mode, 3, seed=6)
    images = []
    for near, far in ((0.2, 100.0), (0.2, 3e38)):
        wide = scenes.make_view(view.M, view.width, view.height, 256.0, 256.0, view.width / 2.0, view.height / 2.0, near, far)
        with torch.no_grad():
            images.append(tb.diff_rasterize(*harness.scene_tensors(scene), torch.empty(0, device="cuda"), harness.settings_for(tb, scene, wide, mode, K), False))
    assert torch.equal(*images)


@pytest.mark.parametrize("mode,K", [(0, 4), (0, 8), (0, 16), (0, 32), (1, 4), (1, 16), (1, 32)])
@pytest.mark.parametrize("order", ["front first", "back first", "mixed", "one depth"])
def test_buffer_filled_to_the_last_entry(mode, K, order):
    # every pixel sees the same Gaussians, one short of a full buffer to one more, and all of them enter: the step from an empty place
    # to an entry that falls out; 64 x 64 pixels run the form that keeps colours, 512 x 512 the other one
    for size in (64, 512):
        for n in (K - 1, K, K + 1, 2 * K + 1):
            scene = scenes.tiny_scene(n=n, size=size, seed=n, mode=mode, K=K, sh_degree=1)
            depth = np.linspace(2.0, 4.0, n)
            if order == "back first":
                depth = depth[::-1]
            elif order == "mixed":
                depth = np.random.default_rng(n).permutation(depth)
            elif order == "one depth":
                depth[:] = 3.0
            scene.positions[:] = 0.0
            scene.positions[:, 2] = depth
            scene.scales[:] = 1.0 if order == "one depth" else 0.2 * depth[:, None]
            scene.scales[:, 2] = 1e-3
            scene.rotations[:] = np.array([1.0, 0.0, 0.0, 0.0], dtype=np.float32)
            scene.opacities[:] = np.random.default_rng(K).uniform(0.2, 0.5, scene.opacities.shape)
            for median in (False, True):
                got = render(scene, scene.views[0], mode, K, 0.2, 100.0, median)
                want = render(scene, scene.views[0], mode, K, 0.2, 3e38, median)
                assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
                assert got[0].max() > 0.0


@pytest.mark.parametrize("far", [100.0, 3e38])
@pytest.mark.parametrize("K", [4, 8, 16, 32])
def test_statistics_of_a_buffer_that_every_candidate_enters(K, far):
    # K Gaussians that every pixel accepts: every time a warp comes to the insertion all of its lanes insert, whatever form the buffer has
    import torch
    from htgs_b200 import _native
    from htgs_b200.torch_bindings import _C
    scene = scenes.tiny_scene(n=K, size=64, seed=K, mode=0, K=K, sh_degree=1)
    depth = np.linspace(4.0, 2.0, K)
    scene.positions[:] = 0.0
    scene.positions[:, 2] = depth
    scene.scales[:] = depth[:, None]
    scene.scales[:, 2] = 1e-3
    scene.rotations[:] = np.array([1.0, 0.0, 0.0, 0.0], dtype=np.float32)
    scene.opacities[:] = 0.5
    lib, ctx = _native.lib(), _native.context(0)
    lib.htgs_set_collect_stats(ctx, 1)
    try:
        image, _ = render(scene, scene.views[0], 0, K, 0.2, far, False)
        info = _C.last_frame_info
    finally:
        lib.htgs_set_collect_stats(ctx, 0)
    assert image.min() > 0.0 and info.accepted_fragments == info.lane_insertions == K * 64 * 64
    assert info.warp_trips == info.warp_trips_inserting == K * 64 * 64 // 32


@pytest.mark.parametrize("width,height", [(752, 776), (752, 784), (1000, 1000)])
@pytest.mark.parametrize("n", [3, 4, 5, 9, 6000])
def test_four_entries_with_and_without_colours(n, width, height):
    # on either side of the number of tiles from which a buffer of four entries does without colours and inserts per candidate (148 multiprocessors of 31 blocks)
    scene, view = scene_with_ties(n, width, height, 4, 0)
    if n < 10:      # Gaussians that every pixel near the centre sees, one short of a full buffer to more than fit
        scene.positions[:, :2] = 0.0
        scene.scales[:] = 0.5
        scene.opacities[:] = 0.4
    for median in (False, True):
        got = render(scene, view, 0, 4, 0.2, 100.0, median)
        want = render(scene, view, 0, 4, 0.2, 3e38, median)
        assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
        assert got[0].max() > 0.0
