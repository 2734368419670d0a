"""GPU: a training forward that is queued before its instance count is known (htgs_forward_ahead).

The guess is the previous forward's capacity; a view that exceeds it, one that needs a fraction of it and one without instances have to
give what the forward in two halves gives, which tracking the visible rows selects.
"""
import pytest

import harness
from htgs_b200 import scenes
from htgs_b200.torch_bindings import rasterization

pytestmark = pytest.mark.gpu


def step(tb, scene, mode, factor, behind):
    import torch
    tensors = harness.scene_tensors(scene)
    tensors[1] = tensors[1] * factor
    if behind:
        tensors[0] = tensors[0] - torch.tensor([0.0, 0.0, 100.0], device="cuda")
    tensors = [t.detach().clone().requires_grad_() for t in tensors]
    image = tb.diff_rasterize(*tensors, torch.empty(0, device="cuda"), harness.settings_for(tb, scene, scene.views[0], mode, 8), False)
    image.square().sum().backward()
    return image.detach(), [t.grad for t in tensors]


@pytest.mark.parametrize("mode", [0, 1, 2, 3])
def test_views_above_and_below_the_guess(mode):
    import torch
    tb = harness.ours()
    scene = scenes.tiny_scene(n=3000, size=256, seed=11, mode=mode, K=8, sh_degree=1)
    cases = [(0.05, False), (3.0, False), (0.05, False), (1.0, True), (1.0, False), (1.0, False)]
    got = [step(tb, scene, mode, *c) for c in cases]
    rasterization.track_training_visibility(True)
    try:
        want = [step(tb, scene, mode, *c) for c in cases]
    finally:
        rasterization.track_training_visibility(False)
    for (image, grads), (image_w, grads_w) in zip(got, want):
        assert torch.equal(image, image_w)
        for a, b in zip(grads, grads_w):
            assert torch.allclose(a, b, rtol=1e-4, atol=1e-5 * float(b.abs().max()))
    assert float(want[1][0].max()) > 0.0 and not float(want[3][0].abs().max()) > 0.0


@pytest.mark.parametrize("mode", [0, 1, 2, 3])
def test_second_half_again(mode):
    # htgs_forward_finish reads the per-Gaussian blob that htgs_forward_begin filled: it may be called on it any number of times
    import ctypes
    import torch
    from htgs_b200 import _native
    from htgs_b200.torch_bindings import _C
    scene = scenes.tiny_scene(n=3000, size=256, seed=11, mode=mode, K=8, sh_degree=1)
    tensors = harness.scene_tensors(scene)
    st = harness.settings_for(harness.ours(), scene, scene.views[0], mode, 8)
    lib, ctx, stream = _native.lib(), _native.context(0), torch.cuda.current_stream().cuda_stream
    s, v = _C._scene_view(tensors, st.M, st.VPM, st.cam_position, mode, 8, st.active_sh_bases, st.width, st.height, st.near_plane, st.far_plane, 1.0)
    sizes = [ctypes.c_size_t() for _ in range(3)]
    _native.check(lib.htgs_forward_blob_sizes(ctypes.byref(s), ctypes.byref(v), *(ctypes.byref(x) for x in sizes)))
    primitive, tile, pixel = (torch.empty(x.value, dtype=torch.uint8, device="cuda") for x in sizes)
    count = ctypes.c_uint32()
    _native.check(lib.htgs_forward_begin(ctx, ctypes.byref(s), ctypes.byref(v), primitive.data_ptr(), primitive.numel(), stream, ctypes.byref(count)))
    instance = torch.empty(lib.htgs_forward_instance_bytes(ctypes.byref(v), count.value), dtype=torch.uint8, device="cuda")
    blobs = _native.HtgsTrainBlobs(*(x for t in (primitive, tile, instance, pixel) for x in (t.data_ptr(), t.numel())))
    first = primitive.clone()
    images = []
    for _ in range(3):
        image = torch.zeros(3, st.height, st.width, device="cuda")
        _native.check(lib.htgs_forward_finish(ctx, ctypes.byref(s), ctypes.byref(v), ctypes.byref(blobs), count.value, image.data_ptr(), stream,
                                              ctypes.byref(_native.HtgsFrameInfo())))
        assert torch.equal(primitive[64:], first[64:])        # behind the status at its head, the first half's results are only read
        images.append(image)
    assert float(images[0].max()) > 0.0 and torch.equal(images[0], images[1]) and torch.equal(images[0], images[2])


def first_half(mode):
    """A scene's training forward up to the instance count: (library, context, scene, view, blob sizes, per-Gaussian blob, count, what has to stay alive)."""
    import ctypes
    import torch
    from htgs_b200 import _native
    from htgs_b200.torch_bindings import _C
    scene = scenes.tiny_scene(n=3000, size=256, seed=11, mode=mode, K=8, sh_degree=1)
    tensors = harness.scene_tensors(scene)
    st = harness.settings_for(harness.ours(), scene, scene.views[0], mode, 8)
    lib, ctx = _native.lib(), _native.context(0)
    s, v = _C._scene_view(tensors, st.M, st.VPM, st.cam_position, mode, 8, st.active_sh_bases, st.width, st.height, st.near_plane, st.far_plane, 1.0)
    sizes = [ctypes.c_size_t() for _ in range(3)]
    _native.check(lib.htgs_forward_blob_sizes(ctypes.byref(s), ctypes.byref(v), *(ctypes.byref(x) for x in sizes)))
    primitive = torch.empty(sizes[0].value, dtype=torch.uint8, device="cuda")
    count = ctypes.c_uint32()
    _native.check(lib.htgs_forward_begin(ctx, ctypes.byref(s), ctypes.byref(v), primitive.data_ptr(), primitive.numel(),
                                         torch.cuda.current_stream().cuda_stream, ctypes.byref(count)))
    return lib, ctx, s, v, [x.value for x in sizes], primitive, count.value, (tensors, st)


def second_half(lib, ctx, s, v, sizes, primitive, count, instance=None):
    """Status, image and the tiles' ranges and order of a second half with blobs of its own, filled with zeros, which are valid tile numbers."""
    import ctypes
    import torch
    from htgs_b200 import _native
    if instance is None:
        instance = torch.zeros(lib.htgs_forward_instance_bytes(ctypes.byref(v), count), dtype=torch.uint8, device="cuda")
    tile, pixel = (torch.zeros(x, dtype=torch.uint8, device="cuda") for x in sizes[1:])
    blobs = _native.HtgsTrainBlobs(*(x for t in (primitive, tile, instance, pixel) for x in (t.data_ptr(), t.numel())))
    image = torch.zeros(3, v.height, v.width, device="cuda")
    status = lib.htgs_forward_finish(ctx, ctypes.byref(s), ctypes.byref(v), ctypes.byref(blobs), count, image.data_ptr(), torch.cuda.current_stream().cuda_stream,
                                     ctypes.byref(_native.HtgsFrameInfo()))
    torch.cuda.synchronize()
    n_tiles = (256 // 8) ** 2 if v.mode != 2 else (256 // 16) ** 2
    words = tile[:12 * n_tiles].view(torch.int32)
    return status, image, words[:2 * n_tiles].reshape(n_tiles, 2), words[2 * n_tiles:]


@pytest.mark.parametrize("mode", [0, 1, 2, 3])
def test_second_half_with_other_blobs(mode):
    # htgs_forward_finish leaves the per-Gaussian blob that htgs_forward_begin filled as it was: it may be called on it any number of times, with
    # other blobs for what it writes (an order of the tiles that is missing leaves only tile 0)
    import torch
    *first, primitive, count, _alive = first_half(mode)
    before = primitive.clone()
    results = [second_half(*first, primitive, count) for _ in range(3)]
    assert torch.equal(primitive, before)
    for status, image, ranges, order in results:
        assert status == 0 and torch.equal(order.sort().values, torch.arange(len(order), dtype=torch.int32, device="cuda"))
        assert torch.equal(ranges, results[0][2]) and torch.equal(image, results[0][1])
    assert float(results[0][1].max()) > 0.0


@pytest.mark.parametrize("mode", [0, 1, 2, 3])
@pytest.mark.parametrize("share", [0.0, 0.3, 1.0])
def test_second_half_with_a_smaller_count(mode, share):
    # a count below that of the first half cuts the lists; nothing is written beyond the blob that belongs to that count, which may have room
    # for fewer instances than there are visible Gaussians
    import ctypes
    import torch
    *first, primitive, count, _alive = first_half(mode)
    lib, _, _, v = first[:4]
    fewer = max(int(count * share), 3)
    size = lib.htgs_forward_instance_bytes(ctypes.byref(v), fewer)
    room = torch.full((lib.htgs_forward_instance_bytes(ctypes.byref(v), 2 * count) + (1 << 20),), 0x5a, dtype=torch.uint8, device="cuda")
    status, image, ranges, _order = second_half(*first, primitive, fewer, room[:size])
    assert status == 0 and bool((room[size:] == 0x5a).all()) and bool(torch.isfinite(image).all())
    assert int((ranges[:, 1] - ranges[:, 0]).sum()) == fewer and int(ranges.max()) == fewer


@pytest.mark.parametrize("mode", [0, 1, 2, 3])
def test_second_half_after_an_error(mode):
    # with the error flag set, as a wait that gave up leaves it, no list is read: every tile is empty, and the call says so
    import torch
    from htgs_b200 import _native
    *first, primitive, count, _alive = first_half(mode)
    primitive[12:16].view(torch.int32).fill_(2)
    status, image, ranges, order = second_half(*first, primitive, count)
    assert status == _native.HTGS_ERR_DEVICE_FLAG and not bool(ranges.any()) and not bool(image.any())
    assert torch.equal(order.sort().values, torch.arange(len(order), dtype=torch.int32, device="cuda"))
    primitive[12:16].view(torch.int32).fill_(0)
    status, image, ranges, _order = second_half(*first, primitive, count)
    assert status == 0 and bool(image.any()) and int(ranges.max()) == count
