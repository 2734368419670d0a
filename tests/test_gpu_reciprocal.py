"""GPU: the blend kernels' reciprocal against CUDA's division, for every float of its range, and frames that need the division."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

import harness
from htgs_b200 import build, scenes

pytestmark = pytest.mark.gpu

SOURCE = r'''
#include "common.cuh"
// counts[0]: floats from 2^-126 to 2^126; [1]: of these, those whose reciprocal differs from the quotient
__global__ void compare(unsigned long long* counts) {
    unsigned long long in_range = 0, different = 0;
    const uint64_t step = uint64_t(gridDim.x) * blockDim.x;
    for (uint64_t bits = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; bits < (uint64_t(1) << 32); bits += step) {
        const float x = __uint_as_float(uint32_t(bits));
        if (!(x >= 0x1p-126f && x <= 0x1p126f)) continue;
        ++in_range;
        if (__float_as_uint(htgs::reciprocal_rn(x)) != __float_as_uint(1.0f / x)) ++different;
    }
    atomicAdd(counts, in_range);
    atomicAdd(counts + 1, different);
}
extern "C" int run(unsigned long long* host) {
    unsigned long long* device = nullptr;
    cudaError_t err = cudaMalloc(&device, 2 * sizeof(*device));
    if (err == cudaSuccess) err = cudaMemset(device, 0, 2 * sizeof(*device));
    if (err == cudaSuccess) { compare<<<148 * 8, 256>>>(device); err = cudaGetLastError(); }
    if (err == cudaSuccess) err = cudaMemcpy(host, device, 2 * sizeof(*device), cudaMemcpyDeviceToHost);
    cudaFree(device);
    return int(err);
}
'''


def test_reciprocals_of_all_floats(tmp_path):
    (tmp_path / "compare.cu").write_text(SOURCE)
    library = tmp_path / "compare.so"
    subprocess.run([build._nvcc(), *build.NVCC_FLAGS, "-shared", "-I", os.path.join(harness.REPO, "htgs_b200", "csrc"), str(tmp_path / "compare.cu"), "-o", str(library)], check=True)
    counts = (ctypes.c_ulonglong * 2)()
    assert ctypes.CDLL(str(library)).run(counts) == 0
    assert counts[0] == (252 << 23) + 1 and counts[1] == 0


def one_gaussian(scale, depth):
    """A round Gaussian on the optical axis, which meets the centre of pixel (3, 3) exactly: m = 0 there.  |d|^2 is about (8 scale)^4."""
    scene = scenes.tiny_scene(n=1, size=8, seed=1, sh_degree=0)
    scene.positions[:] = (0.0, 0.0, depth)
    scene.scales[:] = scale
    scene.rotations[:] = (1.0, 0.0, 0.0, 0.0)
    scene.opacities[:] = 0.5
    scene.sh_0[:] = 0.5
    view = scenes.make_view(np.eye(4), 8, 8, 8.0, 8.0, 3.5, 3.5, 0.2, 100.0 if depth < 50.0 else 3e38)
    return scene, view


# |d|^2 of 2^-127 (subnormal, its reciprocal is not), of 1, and of 2^126.5 (normal, its reciprocal is subnormal)
@pytest.mark.parametrize("scale,depth", [(2.0 ** -34.75, 4.0), (0.125, 4.0), (2.0 ** 28.625, 2.0 ** 31)])
@pytest.mark.parametrize("mode,K", [(0, 1), (0, 8), (0, 16), (0, 32), (1, 8), (2, 1), (3, 1)])
def test_frames_beyond_the_reciprocals_range(oracle_lib, mode, K, scale, depth):
    import torch
    tb = harness.ours()
    scene, view = one_gaussian(scale, depth)
    want = oracle_lib.render(scene, view, mode=mode, K=K, dtype=np.float64)[0]
    assert want[0, 3, 3] == pytest.approx(0.5 * (0.5 + 0.28209479177387814 * 0.5), rel=1e-6)
    settings = harness.settings_for(tb, scene, view, mode, K)
    image = tb.rasterize(*harness.scene_tensors(scene), settings, True, False)[0]
    near = np.ix_(range(3), (2, 3, 4), (2, 3, 4))       # |m|^2 overflows farther out for the largest one
    # a subnormal |d|^2 has 22 bits
    assert np.abs(image.cpu().numpy() - want)[near].max() <= 1e-6
    with torch.no_grad():
        image = tb.diff_rasterize(*harness.scene_tensors(scene), torch.empty(0, device="cuda"), settings, False)
    assert np.abs(image.cpu().numpy() - want)[near].max() <= 1e-6


@pytest.mark.parametrize("mode,K", [(0, 2), (0, 8), (0, 16), (0, 32), (1, 16), (2, 1), (3, 1)])
def test_dividing_form_equals_the_others(mode, K):
    """A Gaussian of no extent that meets no pixel centre makes the whole frame divide (5120 blocks of pixels, more than the grid of that form)."""
    import torch
    tb = harness.ours()
    images = []
    for extent in (0.02, 1e-12):
        scene = scenes.tiny_scene(n=6000, size=640, seed=9, mode=mode, K=K, sh_degree=1)
        scene.positions[17] = (0.30001, 0.20001, 3.0)
        scene.scales[17], scene.opacities[17] = extent, 1e-3 if extent > 1e-3 else 0.9      # neither shows
        view = scene.views[0]
        view.height = 512
        settings = harness.settings_for(tb, scene, view, mode, K)
        outputs = list(tb.rasterize(*harness.scene_tensors(scene), settings, True, False))
        with torch.no_grad():
            outputs.append(tb.diff_rasterize(*harness.scene_tensors(scene), torch.empty(0, device="cuda"), settings, False))
        weights = torch.zeros((scene.n, 1), device="cuda")
        tb.update_max_weights(weights, *harness.scene_tensors(scene)[:4], settings, 0.01)
        images.append(outputs + [weights])
    for a, b in zip(*images):
        assert torch.equal(a, b)
