"""The fused tcgen05 training step at the edges of its tiles of 128 rows (one
row, a tile less one, a tile, a tile and one) and past the 512 tiles of one
launch, where the gradient sums are carried over: gradients against the numpy
reference with the bounds of the other gradient tests."""
import pytest

from test_gpu_denoiser import _gradients_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 127, 128, 129, 65537])
def test_fused_step_gradients(lib, rows):
    assert lib.crSetDenoiserKernel(1) == 0
    _gradients_case(lib, rows)


@pytest.mark.parametrize("rows_poses,batch", [(2, 700), (5, 900)])
def test_training_queued_behind_other_work(lib, small, tmp_path, rows_poses, batch):
    """The epochs' orders are drawn and uploaded while the stream is still busy
    with earlier work: every step sees its own, so the parameters are those of
    a run on an idle stream, bit for bit (epochs of one and several steps)."""
    import numpy as np
    import torch

    import eyeRendererHelperFunctions as eh
    import scenes

    p12 = scenes.open_poses(small["boxes"], rows_poses, np.random.default_rng(1))
    st = torch.cuda.Stream()
    torch.cuda.synchronize()
    got = []
    assert lib.crSetStream(st.cuda_stream) == 0 and lib.crSetDenoiserKernel(1) == 0
    try:
        for busy in (False, True, True):
            lib.loadGlTFscene(small["gltf"].encode())  # restarts the feature and target draws
            eh.gotoFirstCompoundEye(lib)
            assert lib.crDenoiserInit(5) == 0
            assert lib.crDenoiserAddTrainingPoses(p12, rows_poses, 8, 32) == 0, eh.lastError(lib)
            assert batch <= lib.crDenoiserTrainingRows()
            if busy:
                with torch.cuda.stream(st):
                    torch.cuda._sleep(100_000_000)  # about 50 ms
            assert lib.crDenoiserTrain(60, batch, 1e-3, 7, None) == 0, eh.lastError(lib)
            path = tmp_path / "net.bin"
            assert lib.crDenoiserSave(str(path).encode()) == 0
            got.append(path.read_bytes())
    finally:
        lib.crSetStream(None)
        lib.crDenoiserRelease()
    assert got[0] == got[1] == got[2]
