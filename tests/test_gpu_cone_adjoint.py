"""General and z-mirror backprojections of cone plans at edge sizes."""
import os

import numpy as np
import pytest

import oracle as O
from framelab_gb300 import geometry as G

pytestmark = pytest.mark.gpu


def _circle(nx, ny, nz, na, nb, nv):
    m = max(nx, ny)
    return G.cone_para(nx, ny, nz, na, nb, nv, L=(2.0 * nx, 2.0 * ny, 2.0 * nz), SO=6.0 * m,
                       OD=6.0 * m, Ly=6.0 * m, Lz=4.4 * nz)


def _helix(n, nz, na, nb, nv):
    return G.cone_para(n, n, nz, na, nb, L=(2.0, 2.0, 2.0 * nz / n), SO=6.0, OD=6.0, Ly=5.6,
                       Lz=5.6 * nb / na, scan="helix", zmax=2.0 * nz / n, rps=3.0, vtab=2.0,
                       fps=(nv - 1) * n / nz)


# heights below, at and off a multiple of the 32 lanes and with 16 and 8 lanes
# per block; odd sizes; more views than a warp's lanes; detectors
# so fine that a block's shadow holds more than 8 or 32 columns
@pytest.mark.parametrize("geom", [
    (7, 5, 3, 12, 9, 33), (13, 13, 33, 30, 41, 9), (12, 9, 64, 25, 70, 65),
    (81, 83, 16, 120, 20, 5), (161, 159, 8, 240, 12, 4), (9, 9, 40, 400, 50, 6),
    (80, 79, 16, 1300, 21, 3), ("helix", 16, 16, 24, 10, 40), ("helix", 9, 41, 20, 7, 70)])
@pytest.mark.parametrize("mirror", [False, True])
def test_cone_backprojection_of_any_size(geom, mirror):
    """Against the FP64 transpose (5e-6, the bound of the forms' other tests),
    FP32, and FP16 storage in and out."""
    import torch
    from framelab_gb300.projector import Plan
    if geom[0] == "helix":
        p = _helix(*geom[1:])
    else:
        nx, ny, nz, na, nb, nv = geom
        if mirror:
            nz, nb = nz + nz % 2, nb + nb % 2
        p = _circle(nx, ny, nz, na, nb, nv)
    P = Plan(p)
    P.rot_mirror = False
    if mirror and not P.z_mirror:
        pytest.skip("no mirror in this scan")
    P.z_mirror = mirror
    r = np.random.default_rng(5).standard_normal(P.n_rays).astype(np.float32)
    want = O.exact_adjoint(r, p, threads=os.cpu_count() or 1).reshape(-1)
    x = P.adjoint(torch.from_numpy(r).cuda()).cpu().numpy().reshape(-1)
    assert np.linalg.norm(x - want) < 5e-6 * np.linalg.norm(want)
    h = P.adjoint(torch.from_numpy(r).cuda().half(), out_dtype=torch.float16)
    h = h.float().cpu().numpy().reshape(-1)
    assert np.linalg.norm(h - want) < 2e-3 * np.linalg.norm(want)


def test_cone_backprojection_of_frames():
    """Two frames with interleaved views: each sums its own views."""
    import torch
    from framelab_gb300.projector import Plan
    p = dict(_circle(14, 11, 9, 30, 15, 13))
    ids = (np.arange(13) % 2).astype(np.uint32)
    p.update(nt=np.uint32(2), id_X=ids)
    for k in ("id_Y", "Nv", "tmp_size"):
        p.pop(k)
    P = Plan(p)
    y = np.random.default_rng(6).standard_normal(P.n_rays).astype(np.float32)
    x = P.adjoint(torch.from_numpy(y).cuda()).cpu().numpy().reshape(2, -1)
    one = _circle(14, 11, 9, 30, 15, 13)
    for f in range(2):
        m = y.reshape(13, -1) * (ids == f)[:, None]
        want = O.exact_adjoint(m.reshape(-1), one, threads=4).reshape(-1)
        assert np.linalg.norm(x[f] - want) < 5e-6 * np.linalg.norm(want)
