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
