"""The score-bound kernels' shared state (best score, list length, blocked
directions) under many writers: crowded trays whose items find many survivors
and lower the best score all the time, interlocking-free, several trays at once
and over again, against the transforms."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _key(r):
    return [(p.success, p.position, p.orientation_index, p.score) for p in r.placements]


@pytest.mark.parametrize("nz", [40, 150])   # both widths of the free bits
def test_crowded_trays_over_again(gpu_core, nz):
    from psacking_b200 import BinPacker, workloads
    rng = np.random.default_rng(nz)
    trays = []
    for k in range(4):
        items = workloads.config1_items(40 + k, 60)
        items += [np.ones(tuple(int(v) for v in rng.integers(1, 4, 3)), np.int32) for _ in range(20)]
        trays.append(((48 + 3 * k, 44, nz), items))
    packer = BinPacker((8, 8, 8), num_orientations=24, interlocking_free=True)
    gpu_core.set_cand_filter(False)
    try:
        want = packer.pack_many(trays, concurrency=4)
    finally:
        gpu_core.set_cand_filter(True)
    for _ in range(4):
        for got, w in zip(packer.pack_many(trays, concurrency=4), want):
            assert _key(got) == _key(w)
            np.testing.assert_array_equal(got.tray, w.tray)
