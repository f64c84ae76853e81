"""Candidate grids of the spherical projections against the exhaustive search
where their stored vectors and the cosine test before acosf could go wrong:
lengths from 1e-12 to 1e12, clusters of nearly equal directions, and an eye
that changes between two frames.  Equal pixel for pixel: both searches
compare the same computed angles."""
import numpy as np
import pytest

import eyeRendererHelperFunctions as eh
from test_gpu_projections import KINDS, _both, _eye, _set_ommatidia

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 33, 4099])
@pytest.mark.parametrize("kind", KINDS)
def test_lengths_clusters_and_changed_eyes(lib, small, kind, n):
    eh.lastError(lib)
    lib.loadGlTFscene(small["gltf"].encode())
    eh.gotoFirstCompoundEye(lib)
    lib.setCurrentEyeSamplesPerOmmatidium(2)
    rng = np.random.default_rng(n)
    for scale in (0.0, 1e-7):
        e = _eye(rng, n)
        e[:, 0:3] *= 10.0 ** rng.uniform(-12, 12, size=(n, 1))
        e[:, 3:6] *= 10.0 ** rng.uniform(-12, 12, size=(n, 1))
        if scale:
            centre = rng.normal(size=(max(1, n // 16), 3))
            d = centre[rng.integers(0, len(centre), size=n)]
            d = d / np.linalg.norm(d, axis=1, keepdims=True) + rng.normal(scale=scale, size=(n, 3))
            e[:, 0:3], e[:, 3:6] = d, -d
        _set_ommatidia(lib, e)
        a, b = _both(lib, kind, 97, 45)
        assert np.array_equal(a, b)


def test_projection_memory_is_optional(lib, small):
    """Under a memory cap of what the candidate grids need without their kept
    vectors, a spherical frame is still drawn, the same; and what is kept gives
    way to a later render."""
    import ctypes

    import torch

    n, w, h = 5000, 201, 101
    rng = np.random.default_rng(2)
    d = rng.normal(0, 1, (n, 3))
    d /= np.linalg.norm(d, axis=1)[:, None]
    omm = np.zeros((n, 8), np.float32)
    omm[:, 0:3], omm[:, 3:6], omm[:, 6] = d * 0.001, d, 0.05
    lib.setOmmatidia.argtypes = [ctypes.c_void_p, ctypes.c_size_t]
    sets = [n - 1, n - 1, int((omm[1:, 0] < 0).sum()), int((omm[1:, 0] > 0).sum())]
    side = [max(1, min(128, round(0.33 * k ** 0.5))) for k in sets]
    grids = sum(4 * (g ** 3 + 1) + 4 * k for g, k in zip(side, sets))
    poses = torch.zeros((4, 16), device="cuda")
    poses[:, 4] = poses[:, 9] = poses[:, 14] = 1.0
    poses[:, 1] = 0.5
    out = torch.zeros((4, n, 3), device="cuda")
    torch.cuda.synchronize()
    got = []
    for cap in (False, True):
        lib.loadGlTFscene(small["gltf"].encode())
        eh.gotoFirstCompoundEye(lib)
        lib.setOmmatidia(omm.ctypes.data, n)
        lib.setCurrentEyeSamplesPerOmmatidium(8)
        eh.setRenderSize(lib, w, h)
        lib.setCurrentEyeShaderName(b"single_dimension")
        assert lib.renderFrame() >= 0
        held = lib.crGetDeviceMemoryHeld()
        lib.setCurrentEyeShaderName(b"spherical_orientationwise")
        try:
            if cap:
                lib.crSetDeviceMemoryCap(held + 8 * n + grids)
            assert lib.renderFrame() >= 0, eh.lastError(lib)
            got.append(eh.getFrame(lib, w, h))
            lib.crSetDeviceMemoryCap(0)
            if not cap:  # grids, vectors and lengths are kept; a render takes what it needs from them
                kept = lib.crGetDeviceMemoryHeld()
                assert kept >= held + grids + 8 * n + 16 * sum(sets)
                draws = 4 * n * 8 * 8
                assert kept - held < draws <= kept - held + 900000
                lib.crSetDeviceMemoryCap(kept + 900000)
                assert lib.crRenderPosesDevice(poses.data_ptr(), 4, out.data_ptr()) == 0, eh.lastError(lib)
                assert lib.crSynchronize() == 0
                lib.crSetDeviceMemoryCap(0)
                assert lib.crGetDeviceMemoryHeld() == held + draws
        finally:
            lib.crSetDeviceMemoryCap(0)
    assert np.array_equal(got[0], got[1])
