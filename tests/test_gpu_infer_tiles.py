"""The tcgen05 inference's four tiles in flight: one tile and less, a tile and
one row, as many tiles as groups, and enough tiles that every block takes each
of its buffers more than once.  Against the mma.sync kernel, with the bound of
the other inference test (8 bf16 steps of the output's terms)."""
import numpy as np
import pytest

import eyeRendererHelperFunctions as eh
import mlp_ref
import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,P", [(7, 1), (129, 1), (256, 2), (701, 300)])
def test_tcgen05_inference_tiles(lib, tmp_path, n, P):
    info = scenes.terrain_scene(str(tmp_path), cells=48, extent=40.0, cones=30, n_omm=n, poses=4)
    rng = np.random.default_rng(n)
    poses = scenes.random_poses(info["height_fn"], P, rng, 10.0)

    def load():
        lib.loadGlTFscene(info["gltf"].encode())
        assert eh.lastError(lib) == ""
        eh.gotoFirstCompoundEye(lib)

    load()
    assert lib.getCurrentEyeOmmatidialCount() == n
    assert lib.crDenoiserInit(4) == 0
    rows = n * P
    X = np.zeros((rows, mlp_ref.FEAT), np.uint16)
    base = np.zeros((rows, 3), np.float32)
    assert lib.crDenoiserFeatureRows(poses, P, 8, X, base) == 0, eh.lastError(lib)
    out = []
    try:
        for kernel in (0, 1):
            load()  # restarts the feature streams
            assert lib.crSetDenoiserKernel(kernel) == 0
            got = np.zeros((P, n, 3), np.float32)
            assert lib.crDenoiserRenderPoses(poses, P, 8, got) == 0, eh.lastError(lib)
            out.append(got.reshape(-1, 3))
    finally:
        lib.crSetDenoiserKernel(1)
    params = np.zeros(mlp_ref.N_PARAMS, np.float32)
    grads = np.zeros(mlp_ref.N_PARAMS, np.float32)
    assert lib.crDenoiserGradient(X[:1].copy(), base[:1].copy(), base[:1].copy(), 1, grads, params) >= 0
    _, (_, _, H3), (_, _, _, W4b) = mlp_ref.forward_parts(params, mlp_ref.from_bits(X))
    tol = 2.0 ** -5 * (np.abs(H3) @ np.abs(W4b))[:, :3] + 1e-7
    err = np.abs(out[1] - out[0])
    assert (err <= tol).all(), ((err > tol).sum(), (err / tol).max())
