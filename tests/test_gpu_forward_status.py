"""GPU: the device status of a training forward is reported before anything uses its gradients.

The forward returns while its kernels run.  A kernel that gives up a bounded wait sets the error word of the status at the head of the
per-Gaussian blob; here the tests set it themselves, behind the forward.
"""
import pytest

import harness
from htgs_b200 import scenes
from htgs_b200.torch_bindings import rasterization

pytestmark = pytest.mark.gpu

ERROR_BYTE = 12          # FrameStatus::error


def forward(tb, scene, mode, requires_grad=True):
    import torch
    leaves = [t.requires_grad_(requires_grad) for t in harness.scene_tensors(scene)]
    image = tb.diff_rasterize(*leaves, torch.empty(0, device="cuda"), harness.settings_for(tb, scene, scene.views[0], mode, 8), False)
    return leaves, image


def fail(image):
    per_primitive = image.grad_fn.saved_tensors[-4]
    per_primitive.data[ERROR_BYTE] = 1          # .data: not an in-place change to autograd


@pytest.mark.parametrize("mode", [0, 1, 2, 3])
def test_backward_raises_for_a_failed_forward(mode):
    import torch
    tb = harness.ours()
    scene = scenes.tiny_scene(n=2000, size=128, seed=3, mode=mode, K=8, sh_degree=1)
    for _ in range(2):      # the second forward is queued ahead of its instance count
        leaves, image = forward(tb, scene, mode)
        fail(image)
        with pytest.raises(RuntimeError, match="internal error"):
            image.square().sum().backward()
        leaves, image = forward(tb, scene, mode)
        image.square().sum().backward()
        assert torch.isfinite(leaves[0].grad).all() and leaves[0].grad.any()


@pytest.mark.parametrize("split_pass", [True, False])
def test_backward_by_ranges_raises_before_the_first_hand_over(split_pass):
    tb = harness.ours()
    scene = scenes.tiny_scene(n=2000, size=128, seed=3, mode=0, K=8, sh_degree=1)
    handed_over = []

    class Hook:
        def __init__(self):
            self.split_pass = split_pass

        def ranges(self, n, mode):
            return [(0, 1000), (1000, n - 1000)]

        def after_range(self, k, first, count, grads):
            handed_over.append(k)

        def finish(self, grads):
            handed_over.append("finish")

    rasterization.set_backward_hook(Hook())
    try:
        leaves, image = forward(tb, scene, 0)
        image.square().sum().backward()
        assert handed_over == [0, 1, "finish"]
        del handed_over[:]
        leaves, image = forward(tb, scene, 0)
        fail(image)
        with pytest.raises(RuntimeError, match="internal error"):
            image.square().sum().backward()
        assert handed_over == []
    finally:
        rasterization.set_backward_hook(None)


def test_forward_without_a_backward_pass_is_checked_at_once(monkeypatch):
    import torch
    tb = harness.ours()
    scene = scenes.tiny_scene(n=500, size=64, seed=4, mode=0, K=8, sh_degree=0)
    calls = []
    check = rasterization._impl.check_training_forwards

    class Recorder:
        def __getattr__(self, name):
            return getattr(impl, name)

        def check_training_forwards(self, *args):
            calls.append(args)
            return check(*args)

    impl = rasterization._impl
    monkeypatch.setattr(rasterization, "_impl", Recorder())
    forward(tb, scene, 0, requires_grad=False)
    with torch.no_grad():
        forward(tb, scene, 0)
    assert len(calls) == 2
    forward(tb, scene, 0)
    assert len(calls) == 2
    tb.rasterization.frame_results()
