"""Tray calls of the C ABI (psb_tray_set, psb_tray_search, psb_tray_place) on
the inputs where their shortcuts and limits lie, against the transform flow
(candidate filter off), which every search can fall back to, or against plain
numpy."""
import ctypes
from pathlib import Path

import numpy as np
import pytest

from oracle import psb_oracle as O

pytestmark = pytest.mark.gpu

LIB = Path(__file__).resolve().parent.parent / "psacking_b200" / "libpsb200.so"
SCAN, BLOCK, INTERLOCK = 0, 1, 0x10
PSB_ERR_ARG, PSB_ERR_OVERLAP = 1, 4


class Res(ctypes.Structure):
    _fields_ = [("x", ctypes.c_int32), ("y", ctypes.c_int32), ("z", ctypes.c_int32),
                ("found", ctypes.c_int32), ("score", ctypes.c_double), ("orientation", ctypes.c_int32),
                ("diag", ctypes.c_uint32), ("n_candidates", ctypes.c_int32), ("err_ratio", ctypes.c_float)]


class Tray:
    """A tray handle; phi None: the tray's own distance field."""

    def __init__(self, tray, phi=None):
        self.lib = lib = ctypes.CDLL(str(LIB))
        P, I = ctypes.c_void_p, ctypes.c_int
        lib.psb_last_error.argtypes = [ctypes.c_char_p, ctypes.c_size_t]
        lib.psb_tray_create.argtypes = [I, I, I, P]
        lib.psb_tray_destroy.argtypes = [P]
        lib.psb_tray_set.argtypes = [P, P, P]
        lib.psb_tray_get.argtypes = [P, P, P]
        lib.psb_tray_search.argtypes = [P, P, P, I, I, P, P]
        lib.psb_tray_place.argtypes = [P, P, I, I, I, I, I, I, ctypes.c_int32]
        self.shape, self.h = tray.shape, P()
        self.check(lib.psb_tray_create(*tray.shape, ctypes.byref(self.h)))
        self.set(tray, phi)

    def __enter__(self):
        return self

    def __exit__(self, *a):
        assert self.lib.psb_tray_destroy(self.h) == 0

    def err(self):
        buf = ctypes.create_string_buffer(1024)
        self.lib.psb_last_error(buf, 1024)
        return buf.value.decode()

    def check(self, st):
        assert st == 0, self.err()

    def set(self, tray, phi=None):
        tray = np.ascontiguousarray(tray, np.int32)
        phi = None if phi is None else np.ascontiguousarray(phi, np.int32)
        self.check(self.lib.psb_tray_set(self.h, tray.ctypes.data, None if phi is None else phi.ctypes.data))

    def get(self):
        tray, phi = np.empty(self.shape, np.int32), np.empty(self.shape, np.int32)
        self.check(self.lib.psb_tray_get(self.h, tray.ctypes.data, phi.ctypes.data))
        return tray, phi

    def search_status(self, items, flags):
        items = [np.ascontiguousarray(i, np.int32) for i in items]
        ptrs = (ctypes.c_void_p * len(items))(*[i.ctypes.data for i in items])
        dims = np.array([i.shape for i in items], np.int32).ravel()
        r = Res()
        return self.lib.psb_tray_search(self.h, ptrs, dims.ctypes.data, len(items), flags, ctypes.byref(r), None), r

    def search(self, items, flags):
        st, r = self.search_status(items, flags)
        self.check(st)
        return (r.found, r.x, r.y, r.z, r.orientation, r.score)


def by_transforms(core, tray, phi, items, flags):
    core.set_cand_filter(False)
    try:
        with Tray(tray, phi) as t:
            # (results per array are asked for: no closed form for an empty tray)
            per = (Res * len(items))()
            its = [np.ascontiguousarray(i, np.int32) for i in items]
            ptrs = (ctypes.c_void_p * len(its))(*[i.ctypes.data for i in its])
            dims = np.array([i.shape for i in its], np.int32).ravel()
            r = Res()
            t.check(t.lib.psb_tray_search(t.h, ptrs, dims.ctypes.data, len(its), flags, ctypes.byref(r),
                                          ctypes.byref(per)))
            return (r.found, r.x, r.y, r.z, r.orientation, r.score)
    finally:
        core.set_cand_filter(True)


@pytest.mark.parametrize("flags", [SCAN, BLOCK, BLOCK | INTERLOCK])
def test_empty_tray_takes_the_best_array(gpu_core, flags):
    """Arrays of different sums on an empty tray: the lightest wins wherever it
    stands, the first of equal ones, and none that does not fit or scores too
    high for the scan."""
    empty = np.zeros((20, 18, 16), np.int32)
    big, one, flat = np.ones((2, 2, 2), np.int32), np.ones((1, 1, 1), np.int32), np.ones((4, 2, 1), np.int32)
    wide, heavy = np.ones((30, 1, 1), np.int32), np.full((2, 2, 2), 1 << 24, np.int32)
    for items in ([big, one], [one, big], [big, flat], [wide, big, flat, one, one], [heavy, big], [heavy], [wide]):
        with Tray(empty) as t:
            assert t.search(items, flags) == by_transforms(gpu_core, empty, None, items, flags), items


@pytest.mark.parametrize("shape", [(20, 18, 16), (90, 80, 70), (300, 280, 210)])
def test_tray_set_source_may_be_reused_on_return(gpu_core, shape):
    """Page-locked arrays, overwritten as soon as psb_tray_set has returned:
    below the staged sizes, staged, and above a staging block."""
    import torch
    rng = np.random.default_rng(5)
    tray = torch.zeros(shape, dtype=torch.int32).pin_memory().numpy()
    phi = torch.zeros(shape, dtype=torch.int32).pin_memory().numpy()
    with Tray(np.zeros(shape, np.int32)) as t:
        for _ in range(3):
            want_tray, want_phi = (rng.integers(0, 9, shape, dtype=np.int32) for _ in range(2))
            tray[...], phi[...] = want_tray, want_phi
            t.check(t.lib.psb_tray_set(t.h, tray.ctypes.data, phi.ctypes.data))
            tray[...] = 3
            phi[...] = -1
            got_tray, got_phi = t.get()
            assert np.array_equal(got_tray, want_tray) and np.array_equal(got_phi, want_phi)


@pytest.mark.parametrize("flags", [SCAN, BLOCK, BLOCK | INTERLOCK])
def test_negative_values_anywhere_are_refused(gpu_core, flags):
    """Negative voxels beyond the positive ones, or no positive ones at all:
    an error that names the first such array, and the tray stays usable."""
    tray = np.zeros((20, 18, 16), np.int32)
    tray[:6, :6, :6] = 1
    ok = np.ones((2, 3, 4), np.int32)
    only = np.full((12, 12, 12), -1, np.int32)
    beyond = np.zeros((12, 11, 10), np.int32)
    beyond[0, 0, 0] = 2
    beyond[11, 10, 9] = -3
    with Tray(tray) as t:
        want = t.search([ok], flags)
        for items, bad in (([only], 0), ([ok, beyond], 1), ([ok, ok, only, beyond], 2)):
            st, _ = t.search_status(items, flags)
            assert st == PSB_ERR_ARG and "orientation %d holds negative" % bad in t.err()
            assert t.search([ok], flags) == want


def _boxes(rng, shape, n):
    tray = np.zeros(shape, np.int32)
    for k in range(n):
        e = [int(rng.integers(2, s // 3)) for s in shape]
        o = [int(rng.integers(0, s - ee + 1)) for s, ee in zip(shape, e)]
        tray[o[0]:o[0] + e[0], o[1]:o[1] + e[1], o[2]:o[2] + e[2]] = 1 + k % 3
    return tray


@pytest.mark.parametrize("flags", [BLOCK, BLOCK | INTERLOCK])
@pytest.mark.parametrize("top", [1, 1 << 20, 1 << 26, (1 << 31) - 1])
def test_search_with_heavy_items(gpu_core, monkeypatch, top, flags):
    """Item values whose bounds stay below 2^53 and such that pass it, against
    the oracle's exact sums (not the transforms: in FP32 their collision counts
    are not exact at such weights).  The oracle's FP64 correlations are exact up
    to about 2^30, so they take the values' halves one by one."""
    corr = O.corr_exact
    monkeypatch.setattr(O, "corr_exact", lambda t, i, linear=True:
                        (corr(t, np.asarray(i) >> 16, linear) << 16) + corr(t, np.asarray(i) & 0xffff, linear))
    rng = np.random.default_rng(top % 1000 + flags)
    shape = (60, 50, 44)
    for trial in range(4):
        tray = _boxes(rng, shape, 3 + 4 * trial)
        items = []
        for e in ((14, 12, 10), (18, 18, 18), (9, 21, 11)):
            it = rng.integers(top - top // 3, top, e, endpoint=True, dtype=np.int64).astype(np.int32)
            it[rng.random(e) < 0.2] = 0
            items.append(it)
        phi = O.calculate_distance(tray)
        pos, found, score, o = O.fft_search_batch(items, tray, phi, 1, interlock=flags != BLOCK)
        for handed_in in (None, phi):
            with Tray(tray, handed_in) as t:
                assert t.search(items, flags) == (int(found),) + tuple(pos) + (o, score)


def test_heavy_items_far_from_a_corner_source(gpu_core):
    """One source in the tray's corner, where a bound equals the proximity it
    bounds, and proximities of 2^53 and more: a bound that is rounded up must
    not rule its own translation out.  The free space takes an item in twelve
    places at the far end, the lowest of which (a column of the seed lattice)
    wins."""
    rng = np.random.default_rng(1)
    i, j, k = np.indices((32, 32, 32))
    for trial in range(40):
        tray = np.full((300, 40, 40), 2, np.int32)
        tray[0, 0, 0] = 1
        at = (260, trial % 4, 3 + trial % 5)
        tray[at[0]:at[0] + 34, at[1]:at[1] + 33, at[2]:at[2] + 33] = 0
        item = rng.integers((1 << 31) - (1 << 22), 1 << 31, (32, 32, 32), dtype=np.int64)
        prox = int((item * (i + j + k)).sum()) + int(item.sum()) * sum(at)
        assert prox > 1 << 53
        with Tray(tray) as t:
            assert t.search([item], BLOCK) == (1,) + at + (0, O.score_block(float(prox), at[2], 40)), trial


@pytest.mark.parametrize("flags", [BLOCK, BLOCK | INTERLOCK])
@pytest.mark.parametrize("shift", [-(1 << 30), -(1 << 23) + 200, -5000, 5000, (1 << 23) - 200, 1 << 23, 1 << 30])
def test_search_with_shifted_distances(gpu_core, shift, flags):
    """A distance field handed in whose values are far from the tray's, up to
    where a run's sum passes 32 bits."""
    rng = np.random.default_rng(abs(shift) % 1000 + flags)
    shape = (36, 40, 70)
    for trial in range(4):
        tray = _boxes(rng, shape, 2 + 3 * trial)
        phi = gpu_core.calculate_distance(tray) + np.int32(shift)
        items = [np.ones((3, 4, 30), np.int32), np.ones((5, 6, 7), np.int32)]
        with Tray(tray, phi) as t:
            assert t.search(items, flags) == by_transforms(gpu_core, tray, phi, items, flags)


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("length", [30, 32767, 32768, 65536, 100_001])
def test_place_arrays_longer_than_the_tray(gpu_core, length, axis):
    """Long arrays whose last cells reach into the tray, and such that meet a
    filled cell there: the tray's part is written, or nothing is."""
    rng = np.random.default_rng(length)
    shape = (20, 18, 16)
    tray = np.zeros(shape, np.int32)
    tray[tuple(slice(8, 10) if a == axis else slice(None) for a in range(3))] = 3   # met by the longer reach only
    e = [3, 4, 5]
    e[axis] = length
    item = (rng.random(e) < 0.7).astype(np.int32)
    at = [1, 2, 3]
    for inside in (6, 15):
        at[axis] = inside - length
        want = tray.copy()
        lo = [max(0, a) for a in at]
        hi = [min(s, a + m) for s, a, m in zip(shape, at, e)]
        box = tuple(slice(p, q) for p, q in zip(lo, hi))
        part = item[tuple(slice(p - a, q - a) for p, q, a in zip(lo, hi, at))] > 0
        overlap = bool((want[box][part] > 0).any())
        if not overlap:
            want[box][part] = 7
        with Tray(tray) as t:
            st = t.lib.psb_tray_place(t.h, item.ctypes.data, *e, *at, 7)
            assert st == (PSB_ERR_OVERLAP if overlap else 0), t.err()
            np.testing.assert_array_equal(t.get()[0], want)


def test_search_of_many_large_arrays(gpu_core):
    """Arrays that are counted before they are staged (above 2^24 cells, and too
    large to be pinned as a whole) find what each finds on its own, and the tray
    does not keep the memory they took (20 bytes per cell with room for a run
    per cell; the tray's pool keeps 1 GiB)."""
    import torch
    rng = np.random.default_rng(8)
    shape = (190, 185, 181)
    tray = np.zeros(shape, np.int32)
    tray[100:110, 5:25, 5:25] = 1
    tray[60:90, 40:90, 30:60] = 2
    items = []
    for k in range(24):
        it = np.zeros((180, 180, 180 - k), np.int32)
        for _ in range(8):
            it[tuple(slice(int(v), int(v) + 4) for v in rng.integers(0, 150, 3))] = 1 + k % 2
        it[0, 0, 0] = it[-1, -1, -1] = 1
        items.append(it)
    with Tray(tray) as t:
        alone = [t.search([i], BLOCK) for i in items]
        free0 = torch.cuda.mem_get_info()[0]
        got = t.search(items, BLOCK)
        assert free0 - torch.cuda.mem_get_info()[0] < 3 << 29
    found = [(r[5], o) for o, r in enumerate(alone) if r[0]]
    assert found
    score, o = min(found)
    assert got == alone[o][:4] + (o, score)


def test_search_after_a_run_that_failed(gpu_core):
    """Packing runs on an empty tray that fail at one of their allocations: a
    search then answers for what the tray holds, be it empty or not."""
    from psacking_b200 import workloads
    from psacking_b200.rotations import orientation_maps
    items = [np.ascontiguousarray(i, np.int32) for i in workloads.config1_items(5)[:6]]
    ptrs = (ctypes.c_void_p * len(items))(*[i.ctypes.data for i in items])
    dims = np.array([i.shape for i in items], np.int32).ravel()
    maps = np.ascontiguousarray(orientation_maps(4), np.int32)
    small = np.ones((2, 3, 2), np.int32)
    filled = failed = 0
    for k in range(1, 64):
        with Tray(np.zeros((40, 36, 30), np.int32)) as t:
            t.lib.psb_pack.argtypes = [ctypes.c_void_p] * 3 + [ctypes.c_int, ctypes.c_void_p, ctypes.c_int, ctypes.c_int,
                                                               ctypes.c_int32, ctypes.c_void_p, ctypes.c_void_p]
            t.lib.psb_debug_fail_alloc(k)
            st = t.lib.psb_pack(t.h, ptrs, dims.ctypes.data, len(items), maps.ctypes.data, 4, 0, 0, (Res * len(items))(),
                                None)
            t.lib.psb_debug_fail_alloc(0)
            tray, _ = t.get()
            got = t.search([small], BLOCK)
            pos = tuple(slice(p, p + e) for p, e in zip(got[1:4], small.shape))
            assert got[0] and not tray[pos].any(), (k, st, got)
            if st == 0:
                break
            failed += 1
            filled += bool(tray.any())
    assert failed >= 3 and filled >= 1


@pytest.mark.parametrize("hole", ["sealed", "bent", "straight"])
def test_search_reports_its_flood_fill(gpu_core, hole):
    """A crowded tray whose best free place lies in a cavity: the flood-fill bit
    of the result is set when that place has no straight way out, by the search
    without transforms as by the transforms' form that floods only then."""
    tray = np.full((24, 24, 100), 2, np.int32)   # tall: the height penalty is small at z = 1
    tray[16:, 16:, :] = 0
    tray[4:14, 4:14, 1:12] = 0
    tray[8, 8, 1] = 1
    if hole == "bent":
        tray[4:9, 9:14, 12:] = 0
    elif hole == "straight":
        tray[4:14, 4:14, 12:] = 0
    item = np.ones((4, 4, 5), np.int32)
    FLOOD, DIRECT = 0x400, 0x800
    with Tray(tray) as t:
        got, r = t.search([item], BLOCK | INTERLOCK), t.search_status([item], BLOCK | INTERLOCK)[1]
        assert r.diag & DIRECT and bool(r.diag & FLOOD) == (hole != "straight")
        gpu_core.set_cand_filter(False)
        gpu_core.set_plane_variant(2)
        try:
            assert t.search([item], BLOCK | INTERLOCK) == got
            assert t.search_status([item], BLOCK | INTERLOCK)[1].diag & FLOOD == r.diag & FLOOD
        finally:
            gpu_core.set_plane_variant(3)
            gpu_core.set_cand_filter(True)


def test_failed_streamed_runs_leave_other_trays_alone(gpu_core):
    """Runs staged in two parts that fail at each of their allocations, their
    trays destroyed at once: the next tray, whose buffers come from the same
    pool, packs as it does on its own."""
    from psacking_b200 import BinPacker, workloads
    from psacking_b200.rotations import orientation_maps
    items = [np.ascontiguousarray(i, np.int32) for s in range(4) for i in workloads.config1_items(s)][:70]
    ptrs = (ctypes.c_void_p * len(items))(*[i.ctypes.data for i in items])
    dims = np.array([i.shape for i in items], np.int32).ravel()
    maps = np.ascontiguousarray(orientation_maps(4), np.int32)
    packer = BinPacker((50, 44, 60), num_orientations=4, interlocking_free=True)
    want = packer.pack_voxels(items[:30]).tray
    failed = 0
    for k in range(1, 100):
        with Tray(np.zeros((64, 64, 40), np.int32)) as t:
            t.lib.psb_pack.argtypes = [ctypes.c_void_p] * 3 + [ctypes.c_int, ctypes.c_void_p, ctypes.c_int, ctypes.c_int,
                                                               ctypes.c_int32, ctypes.c_void_p, ctypes.c_void_p]
            t.lib.psb_debug_fail_alloc(k)
            st = t.lib.psb_pack(t.h, ptrs, dims.ctypes.data, len(items), maps.ctypes.data, 4, 1, 0, (Res * len(items))(),
                                None)
            t.lib.psb_debug_fail_alloc(0)
        np.testing.assert_array_equal(packer.pack_voxels(items[:30]).tray, want)
        if st == 0:
            break
        failed += 1
    assert failed >= 3
