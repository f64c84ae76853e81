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
