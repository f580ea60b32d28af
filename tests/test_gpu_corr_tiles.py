"""The correlation's fused x pass at the sizes where its tiles change or end:
axes of one cell, (y, z) column counts that leave a remainder in the last tile,
long axes up to the limit of 256 cells.  Results are whole numbers and equal the oracle's exactly."""
import numpy as np
import pytest

from oracle import psb_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 1, 1), (1, 9, 2), (2, 1, 1), (256, 1, 1), (255, 3, 5), (2, 2, 256), (64, 17, 33),
                                   (33, 64, 1), (7, 1, 130)])
def test_correlation_tiles(gpu_core, shape):
    rng = np.random.default_rng(sum(shape))
    a = rng.integers(0, 4, shape).astype(np.int32)
    b = (rng.random(shape) < 0.3).astype(np.int32)
    assert np.array_equal(gpu_core.dft_corr3(a, b), O.dft_corr3(a, b))
    assert np.array_equal(gpu_core.dft_conv3(a, b), O.dft_conv3(a, b))
