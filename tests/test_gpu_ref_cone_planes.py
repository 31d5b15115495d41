"""Version-1 cone forward where a slab ends exactly on a plane of voxels."""
import numpy as np
import pytest

import oracle as O
from framelab_gb300 import geometry as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
def test_gao_forward_non_finite_voxels_beside_a_met_plane(value):
    """One view along x, a detector column on the axis and rows that rise or fall by
    a quarter of a voxel per slab: every fourth slab ends on a z plane, in an
    unchanged in-plane cell. A term of weight zero then reads the voxel beyond the
    plane. Every voxel of the rays' xz plane in turn is not finite."""
    import torch
    from framelab_gb300.projector import Plan
    n, nz = 8, 10
    p = G.cone_para(n, n, nz, 3, 5, 1, L=(8.0, 8.0, 10.0), SO=8.0, OD=8.0, Ly=3.0, Lz=20.0)
    assert p["scale"] == 1.0 and 0.0 in p["y_det"] and 4.0 in p["z_det"] and -4.0 in p["z_det"]
    P = Plan(p)
    base = np.random.default_rng(1).standard_normal((nz, n, n)).astype(np.float32)
    for iz in range(nz):
        for ix in range(n):
            x = base.copy()
            x[iz, n // 2, ix] = value
            y, yn = P.forward_gao(torch.from_numpy(x).cuda())
            want, wantn = O.cone_gao_f32(x.reshape(-1), p)
            assert np.array_equal(y.cpu().numpy().reshape(-1), want, equal_nan=True), (iz, ix)
            assert np.array_equal(yn.cpu().numpy().reshape(-1), wantn, equal_nan=True), (iz, ix)
