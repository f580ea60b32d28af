"""The packing loop's search by score bounds against the transform flow.

With the candidate filter off every item goes through the transforms, the
flood fill and the exact re-scoring; with the defaults the loop decides items
by score bounds and falls back to the transforms where it cannot.  Both are
exact, so placements, scores and trays must be equal, on trays whose sides end
inside, on and after the kernels' tiles (32 rows, 32 and 128 cells of z), on
trays that fill up, start partly filled, or hold a concave source.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _key(r):
    return [(p.success, p.position, p.orientation_index, p.score) for p in r.placements]


def _both(core, items, dims, n_orient, interlock, initial=None):
    from psacking_b200 import BinPacker
    packer = BinPacker(dims, num_orientations=n_orient, interlocking_free=interlock)
    got = packer.pack_voxels(items, initial_tray=initial)
    core.set_cand_filter(False)
    try:
        want = packer.pack_voxels(items, initial_tray=initial)
    finally:
        core.set_cand_filter(True)
    assert _key(got) == _key(want)
    np.testing.assert_array_equal(got.tray, want.tray)
    assert got.density == want.density
    return got


SIZES = [(33, 31, 32), (32, 32, 33), (40, 65, 31), (9, 7, 8), (64, 33, 128), (36, 40, 129), (50, 34, 140)]


@pytest.mark.parametrize("interlock", [False, True])
@pytest.mark.parametrize("dims", SIZES)
def test_bound_search_edges(gpu_core, dims, interlock):
    """Box unions until they stop fitting: first item, open space, full tray."""
    from psacking_b200 import workloads
    items = workloads.config1_items(sum(dims), 40)
    got = _both(gpu_core, items, dims, 6, interlock)
    assert got.num_placed > 0


@pytest.mark.parametrize("interlock", [False, True])
@pytest.mark.parametrize("n_orient", [1, 4, 24])
def test_bound_search_shapes(gpu_core, n_orient, interlock):
    """Curved, ring and hook shapes in a crowded tray, both scoring modes."""
    from psacking_b200 import workloads
    items = workloads.config3_items(17)[:24] + workloads.config2_items(18)[:16]
    _both(gpu_core, items, (100, 64, 64), n_orient, interlock)


@pytest.mark.parametrize("interlock", [False, True])
def test_bound_search_initial_tray(gpu_core, interlock):
    """A partly filled start: the sources form a concave ring in the middle of
    the tray (the bounds hold but are loose), other cells are no sources."""
    from psacking_b200 import workloads
    tray = np.zeros((60, 50, 40), np.int32)
    tray[20:40, 15:35, 10:20] = 1
    tray[24:36, 19:31, :] = 0
    tray[0:30, 0:10, 0:8] = 5
    tray[50:60, 40:50, 0:30] = 3
    _both(gpu_core, workloads.config1_items(5, 30), (60, 50, 40), 4, interlock, tray)
    # no source at all: the distance field is constant
    _both(gpu_core, workloads.config1_items(6, 6), (60, 50, 40), 4, interlock, np.where(tray == 1, 2, tray))


def test_bound_search_weighted_items(gpu_core):
    """Item values above 1 weigh the proximity; an item without voxels and one
    that fits nowhere sit between the others."""
    from psacking_b200 import workloads
    rng = np.random.default_rng(3)
    items = [i * int(rng.integers(1, 4)) for i in workloads.config1_items(9, 12)]
    items[3] = items[3] * rng.integers(0, 3, items[3].shape).astype(np.int32)
    items.insert(2, np.zeros((3, 4, 5), np.int32))
    items.insert(5, np.ones((80, 3, 3), np.int32))
    for interlock in (False, True):
        _both(gpu_core, items, (48, 40, 36), 6, interlock)


def test_bound_search_trays_at_once(gpu_core):
    """Several trays on their own streams and threads equal single runs."""
    from psacking_b200 import BinPacker, workloads
    trays = [((40 + 7 * k, 50 - 3 * k, 33 + 31 * k), workloads.config1_items(20 + k, 24)) for k in range(5)]
    many = BinPacker((8, 8, 8), num_orientations=6, interlocking_free=True).pack_many(trays, concurrency=5)
    for (dims, items), r in zip(trays, many):
        one = BinPacker(dims, num_orientations=6, interlocking_free=True).pack_voxels(items)
        assert _key(r) == _key(one)
        np.testing.assert_array_equal(r.tray, one.tray)


def _search(core, tray, phi, items, flags):
    core.gpu_tray_init(tray, phi)
    try:
        return core.search_detail(items, flags, per_orientation=False)["best"]
    finally:
        core.gpu_tray_cleanup()


@pytest.mark.parametrize("flags", [0, 1, 1 | 0x10])   # scan, block, block with interlocking
@pytest.mark.parametrize("shape", [(9, 7, 8), (33, 31, 32), (40, 65, 33), (36, 40, 129), (64, 64, 64)])
def test_bound_search_calls(gpu_core, shape, flags):
    """One synchronous search of explicit arrays, analysed on the device,
    against the transforms: random trays, sparse and weighted items, an array
    larger than the tray, distance fields of the tray, of another tray and
    partly negative ones."""
    rng = np.random.default_rng(sum(shape) + flags)
    for trial in range(4):
        tray = np.zeros(shape, np.int32)
        for b in range([3, 12, 40, 6][trial]):
            e = [int(rng.integers(1, max(2, s // 4))) for s in shape]
            o = [int(rng.integers(0, s - ee + 1)) for s, ee in zip(shape, e)]
            tray[o[0]:o[0] + e[0], o[1]:o[1] + e[1], o[2]:o[2] + e[2]] = 1 + b % 5
        items = []
        for k in range(5):
            e = [int(rng.integers(1, max(2, s // 3))) for s in shape]
            it = (rng.random(e) < [1.0, 0.6, 0.1, 0.9, 0.5][k]).astype(np.int32) * int(rng.integers(1, 4))
            it.flat[0] = 1
            items.append(it)
        items.insert(2, np.ones((shape[0] + 1, 2, 2), np.int32))
        phi = gpu_core.calculate_distance(tray)
        for p in (phi, gpu_core.calculate_distance(np.roll(tray, 3, 1)), phi // 2 - 4):
            got = _search(gpu_core, tray, p, items, flags)
            gpu_core.set_cand_filter(False)
            try:
                want = _search(gpu_core, tray, p, items, flags)
            finally:
                gpu_core.set_cand_filter(True)
            assert got == want


def test_bound_search_calls_errors_and_empties(gpu_core):
    tray = np.zeros((20, 18, 16), np.int32)
    tray[:6, :6, :6] = 1
    phi = gpu_core.calculate_distance(tray)
    bad = np.ones((3, 3, 3), np.int32)
    bad[1, 1, 1] = -2
    ok = np.ones((2, 3, 4), np.int32)
    gpu_core.gpu_tray_init(tray, phi)
    with pytest.raises(RuntimeError, match="orientation 1 holds negative"):
        gpu_core.search_detail([ok, bad], 1, per_orientation=False)
    a = gpu_core.search_detail([ok], 1, per_orientation=False)["best"]   # the context stays usable
    assert a[1]
    gpu_core.gpu_tray_cleanup()
    # an empty tray: the first array that fits, at the origin
    empty = np.zeros((20, 18, 16), np.int32)
    for items in ([np.ones((30, 2, 2), np.int32), ok], [np.ones((30, 2, 2), np.int32)], [np.zeros((2, 2, 2), np.int32)]):
        pos, found, score = gpu_core.fft_search_placement(items[-1], empty)
        gpu_core.set_cand_filter(False)
        try:
            gpu_core.gpu_tray_init(empty, gpu_core.calculate_distance(empty))
            want = gpu_core.search_detail([items[-1]], 0, per_orientation=False)["best"]
        finally:
            gpu_core.set_cand_filter(True)
            gpu_core.gpu_tray_cleanup()
        assert (tuple(pos), found) == (tuple(want[0]), want[1]) and (not found or score == want[2])
