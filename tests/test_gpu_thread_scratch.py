"""Device scratch that a stateless call keeps for its thread goes with the thread."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_short_lived_threads_leave_no_scratch_behind(gpu_core):
    import torch
    from psacking_b200.voxelize import voxelize_mesh
    a, b, c, d = np.float32([[0, 0, 0], [1, 0.2, 0.1], [0.1, 0.9, 0.2], [0.3, 0.1, 0.8]])
    mesh = np.ascontiguousarray([[a, c, b], [a, b, d], [a, d, c], [b, c, d]])
    grid = np.zeros((120, 110, 100), np.int32)
    grid[3, 4, 5] = 1
    want = voxelize_mesh(mesh, 301), gpu_core.calculate_distance(grid)
    bad = []

    def work():
        got = voxelize_mesh(mesh, 301), gpu_core.calculate_distance(grid)   # about 0.2 GB of scratch
        if not all(np.array_equal(g, w) for g, w in zip(got, want)):
            bad.append(1)

    free = torch.cuda.mem_get_info()[0]
    for _ in range(16):
        t = threading.Thread(target=work)
        t.start()
        t.join()
    assert not bad and free - torch.cuda.mem_get_info()[0] < 1 << 30
