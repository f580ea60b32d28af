"""The voxelizer where a triangle's pixel box crosses the size at which it is
cut into chunks (256 pixels): two-triangle faces spanning 15 to 33 voxels, next
to many small triangles, equal to the CPU oracle."""
import numpy as np
import pytest

from oracle import psb_voxel_oracle as V
from tests import meshes

pytestmark = pytest.mark.gpu


def _turn(tris, seed):
    q, _ = np.linalg.qr(np.random.default_rng(seed).normal(size=(3, 3)))
    return (tris.reshape(-1, 3) @ q.T).reshape(-1, 3, 3).astype(np.float32)


@pytest.mark.parametrize("res", [1, 2, 15, 16, 17, 18, 33, 35])
def test_voxelize_chunk_edges(gpu_core, res):
    from psacking_b200.voxelize import voxelize_mesh
    for tris in (_turn(meshes.box(hi=(1.0, 0.9, 0.8)), res),
                 np.concatenate([_turn(meshes.box(), 3), meshes.icosphere(1) * np.float32(0.2) - np.float32(0.0)])):
        try:
            want = V.voxelize(tris, res)
        except RuntimeError:
            with pytest.raises(RuntimeError, match="occupied"):
                voxelize_mesh(tris, res)
            continue
        got = voxelize_mesh(tris, res)
        assert got.shape == want.shape and np.array_equal(got, want)
