"""GPU: emission and radix sort at the edges of their tiles, against the CPU oracle: one instance, a part of a sort block, several
groups of sort blocks, one Gaussian over the whole image among small ones, one tile row and one tile column."""
import numpy as np
import pytest

import harness
from htgs_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [0, 2])
@pytest.mark.parametrize("n,width,height,large", [(1, 256, 256, 0), (257, 8, 8, 0), (300, 17, 9, 1), (5000, 1000, 8, 0), (5000, 8, 900, 3), (60_000, 640, 480, 5),
                                                  (40_000, 2100, 1500, 40)])
def test_sorted_instances_and_ranges(oracle_lib, mode, n, width, height, large):
    import torch
    from htgs_b200.torch_bindings import _C
    tb = harness.ours()
    scene = scenes.tiny_scene(n=n, size=max(width, height), seed=n + mode)
    scene.scales[:large] *= 40.0
    focal = float(max(width, height))
    view = scenes.make_view(np.eye(4), width, height, focal, focal, width / 2.0, height / 2.0, 0.2, 100.0)
    tb.rasterize(*harness.scene_tensors(scene), harness.settings_for(tb, scene, view, mode, 4), True, False)
    torch.cuda.synchronize()
    info = _C.last_frame_info
    got = harness.our_intermediates(0, scene.n, info.n_instances)
    depth = got["eval"][:, 3, 3] if mode == scenes.ALPHA_BLEND_GLOBAL_ORDERING else None
    want = oracle_lib.bin_instances(got["n_touched"], got["bounds"].astype(np.uint32), got["grid_w"], got["n_tiles"], depth)
    assert info.n_instances == int(got["n_touched"].sum())
    assert np.array_equal(want["sorted_prims"], got["prims_sorted"]) and np.array_equal(want["ranges"], got["ranges"])


@pytest.mark.parametrize("near,far", [(0.2, 100.0), (0.2, 3e38), (3.0, 3.0625), (0.0, 100.0), (-1.0, 100.0)])
@pytest.mark.parametrize("n,width,height", [(1, 16, 16), (257, 16, 16), (5000, 250, 131), (9000, 4128, 4112)])
def test_global_ordering_lists(oracle_lib, near, far, n, width, height):
    # sorted by depth first and by tile then: windows of depth bits of one to four passes and none, ties in depth (every Gaussian twice,
    # the copies far apart), one tile (no pass over it), and more than 65536 tiles
    import torch
    from htgs_b200.torch_bindings import _C
    tb = harness.ours()
    scene = scenes.tiny_scene(n=n, size=max(width, height), seed=n, mode=2, K=1, sh_degree=1)
    half = n // 2
    for a in (scene.positions, scene.scales, scene.rotations):
        a[half:2 * half] = a[:half]
    if far < 4.0:
        scene.positions[:, 2] = near + (far - near) * np.random.default_rng(n).uniform(0.3, 0.7, n)
        scene.scales[:] *= 1e-2
    focal = float(max(width, height))
    view = scenes.make_view(np.eye(4), width, height, focal, focal, width / 2.0, height / 2.0, near, far)
    tb.rasterize(*harness.scene_tensors(scene), harness.settings_for(tb, scene, view, 2, 1), True, False)
    torch.cuda.synchronize()
    info = _C.last_frame_info
    inter = harness.our_intermediates(0, n, info.n_instances)
    ob = oracle_lib.bin_instances(inter["n_touched"], inter["bounds"].astype(np.uint32), inter["grid_w"], inter["n_tiles"], inter["eval"][:, 3, 3])
    assert np.array_equal(ob["sorted_prims"], inter["prims_sorted"])
    assert np.array_equal(ob["ranges"], inter["ranges"])
    assert np.array_equal(ob["sorted_keys"], inter["keys_sorted"])
    assert info.n_instances > 0 or near <= 0.0 or n == 1


ULP = 2.0 ** -22        # of float32 between 2 and 4


@pytest.mark.parametrize("far", [3.0625, 3.0 + 16000 * ULP, 3.0 + 200 * ULP, 3.0 + 100 * ULP, 3.0 + ULP, 3.0])
@pytest.mark.parametrize("n,width,height", [(1, 16, 16), (257, 16, 16), (5000, 250, 131), (9000, 4128, 4112)])
def test_global_ordering_narrow_windows(oracle_lib, far, n, width, height):
    # windows of 19, 14, 8, 7 and one bits of depth (of none: the same depth for all), so that the sort takes three passes to one, with the ties in depth of
    # every Gaussian twice, the copies far apart
    import torch
    from htgs_b200.torch_bindings import _C
    tb = harness.ours()
    scene = scenes.tiny_scene(n=n, size=max(width, height), seed=n, mode=2, K=1, sh_degree=1)
    near = 3.0
    scene.positions[:, 2] = near + ULP * np.random.default_rng(n).integers(0, round((far - near) / ULP) + 1, n)
    half = n // 2
    for a in (scene.positions, scene.scales, scene.rotations):
        a[half:2 * half] = a[:half]
    focal = float(max(width, height))
    view = scenes.make_view(np.eye(4), width, height, focal, focal, width / 2.0, height / 2.0, 0.2, 100.0)
    view.near_plane, view.far_plane = near, far           # of the centres; the matrix's planes, for the extents, are wide apart
    tb.rasterize(*harness.scene_tensors(scene), harness.settings_for(tb, scene, view, 2, 1), True, False)
    torch.cuda.synchronize()
    info = _C.last_frame_info
    inter = harness.our_intermediates(0, n, info.n_instances)
    ob = oracle_lib.bin_instances(inter["n_touched"], inter["bounds"].astype(np.uint32), inter["grid_w"], inter["n_tiles"], inter["eval"][:, 3, 3])
    assert np.array_equal(ob["sorted_prims"], inter["prims_sorted"])
    assert np.array_equal(ob["ranges"], inter["ranges"])
    assert np.array_equal(ob["sorted_keys"], inter["keys_sorted"])
    if n > 1:
        depths = inter["eval"][inter["n_touched"] != 0, 3, 3]
        assert len(np.unique(depths)) < len(depths) and depths.min() >= near and depths.max() <= far


@pytest.mark.parametrize("own", [True, False])
def test_global_ordering_keys_are_written_while_the_memory_is_the_frames(oracle_lib, own):
    # the 64-bit keys of a frame, asked for twice; of a caller's workspace also after it went back to the allocator and another tensor has its
    # memory: the call must not touch that
    import ctypes
    import torch
    from htgs_b200 import _native
    from htgs_b200.torch_bindings import _C
    tb = harness.ours()
    scene = scenes.tiny_scene(n=4000, size=200, seed=3, mode=2, K=1, sh_degree=1)
    st = harness.settings_for(tb, scene, scene.views[0], 2, 1)
    tensors = harness.scene_tensors(scene)
    lib, ctx = _native.lib(), _native.context(0)
    s, v = _C._scene_view(tensors, st.M, st.VPM, st.cam_position, 2, 1, st.active_sh_bases, st.width, st.height, st.near_plane, st.far_plane, 1.0)
    image, depth = torch.empty(3, st.height, st.width, device="cuda"), torch.empty(st.height, st.width, device="cuda")
    info = _native.HtgsFrameInfo()
    workspace = None if own else torch.empty(lib.htgs_render_workspace_bytes(ctypes.byref(s), ctypes.byref(v), 1 << 18), dtype=torch.uint8, device="cuda")
    _native.check(lib.htgs_render(ctx, ctypes.byref(s), ctypes.byref(v), image.data_ptr(), depth.data_ptr(), None, 1, 0, None if own else workspace.data_ptr(),
                                  0 if own else workspace.numel(), torch.cuda.current_stream().cuda_stream, ctypes.byref(info)))
    for _ in range(2):
        got = harness.our_intermediates(0, scene.n, info.n_instances)
        want = oracle_lib.bin_instances(got["n_touched"], got["bounds"].astype(np.uint32), got["grid_w"], got["n_tiles"], got["eval"][:, 3, 3])
        assert info.n_instances > 1000 and np.array_equal(want["sorted_keys"], got["keys_sorted"]) and np.array_equal(want["sorted_prims"], got["prims_sorted"])
    if not own:
        size, address = workspace.numel(), workspace.data_ptr()
        del workspace
        other = torch.full((size,), 0x7f, dtype=torch.uint8, device="cuda")
        assert other.data_ptr() == address
        torch.cuda.synchronize()
        inter = _native.HtgsIntermediates()
        _native.check(lib.htgs_get_intermediates(ctx, ctypes.byref(inter)))
        torch.cuda.synchronize()
        assert address <= inter.keys_sorted < address + size and bool((other == 0x7f).all())


@pytest.mark.parametrize("far", [100.0, 3e38])
@pytest.mark.parametrize("n", [1 << 19, (1 << 19) + 1])
def test_global_ordering_digits(oracle_lib, n, far):
    # on either side of the number of Gaussians from which the sort by depth takes more and shorter digits, with windows of 27 and 31 bits
    import torch
    from htgs_b200.torch_bindings import _C
    tb = harness.ours()
    scene = scenes.tiny_scene(n=n, size=512, seed=n, mode=2, K=1, sh_degree=0)
    scene.scales[:] *= 0.1
    half = n // 2
    for a in (scene.positions, scene.scales, scene.rotations):
        a[half:2 * half] = a[:half]
    view = scenes.make_view(np.eye(4), 512, 512, 512.0, 512.0, 256.0, 256.0, 0.2, far)
    tb.rasterize(*harness.scene_tensors(scene), harness.settings_for(tb, scene, view, 2, 1), True, False)
    torch.cuda.synchronize()
    info = _C.last_frame_info
    inter = harness.our_intermediates(0, n, info.n_instances)
    ob = oracle_lib.bin_instances(inter["n_touched"], inter["bounds"].astype(np.uint32), inter["grid_w"], inter["n_tiles"], inter["eval"][:, 3, 3])
    assert info.n_instances > n          # so that the buffers do not bound the number of visible Gaussians
    assert np.array_equal(ob["sorted_prims"], inter["prims_sorted"]) and np.array_equal(ob["ranges"], inter["ranges"])
    assert np.array_equal(ob["sorted_keys"], inter["keys_sorted"])
