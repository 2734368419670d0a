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
