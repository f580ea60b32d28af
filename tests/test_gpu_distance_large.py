"""The distance field of a grid with more z lines than a 32-bit count of the
kernel's threads holds (32 threads per line, 2^27 lines), against the L1
distances to its sources."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(16384, 8193, 1), (8193, 129, 2)])
def test_distance_of_many_lines(gpu_core, shape):
    nx, ny, nz = shape
    sources = [(5, 7, 0), (nx - 2, ny // 2, nz - 1), (nx // 2, ny - 1, 0)]
    grid = np.zeros(shape, np.int32)
    for s in sources:
        grid[s] = 1
    got = gpu_core.calculate_distance(grid)
    far = nx + ny + nz + 10
    y, z = np.arange(ny, dtype=np.int32)[:, None], np.arange(nz, dtype=np.int32)[None, :]
    flat = [np.abs(y - s[1]) + np.abs(z - s[2]) for s in sources]
    for x in range(nx):
        want = np.minimum.reduce([f + abs(x - s[0]) for f, s in zip(flat, sources)])
        assert np.array_equal(got[x], np.minimum(want, far)), x
