"""Detectors so fine that most of the volume's shadow lies more than 2^31 columns
beside them: the lanes of the backprojections that share such a window with a
view or an image that meets the detector must not leave the tables."""
import os

import numpy as np
import pytest

import oracle as O
from framelab_gb300 import geometry as G

pytestmark = pytest.mark.gpu

PITCH = 2e-9                       # of a voxel, six columns


def _check(P, p):
    """Against the FP64 transpose (5e-6, the bound of the forms' other tests)."""
    import torch
    r = np.random.default_rng(4).standard_normal(P.n_rays).astype(np.float32)
    x = P.adjoint(torch.from_numpy(r).cuda()).cpu().numpy().reshape(-1)
    want = O.exact_adjoint(r, p, threads=os.cpu_count() or 1).reshape(-1)
    assert np.any(want)
    e = np.linalg.norm(x - want) / np.linalg.norm(want)
    assert e < 5e-6, e


def _para(n, nz, nv):
    return dict(G.cone_para(n, n, nz, 6, 14, nv, L=(1.0 * n, 1.0 * n, 1.0 * nz), SO=30.0, OD=30.0,
                            Ly=6 * PITCH, Lz=2.6 * nz))


# one and 2 x 2 columns per warp (with few and many heights), general and z-mirror
@pytest.mark.parametrize("nz", [8, 640])
@pytest.mark.parametrize("mirror", [False, True])
def test_cone_backprojection(nz, mirror):
    from framelab_gb300.projector import Plan
    p = _para(19, nz, 40)
    phi = (0.3 + 0.15 * np.arange(40)).astype(np.float32)     # no view along an axis
    p.update(sd_phi=phi, cos_phi=np.cos(phi.astype(np.float64)).astype(np.float32),
             sin_phi=np.sin(phi.astype(np.float64)).astype(np.float32))
    P = Plan(p)
    P.z_mirror = mirror
    assert not P.reflect and P.rotations == 1 and P.z_mirror == mirror
    _check(P, p)


@pytest.mark.parametrize("run", [1, 2])
def test_reflection_backprojection(run):
    from framelab_gb300.projector import Plan
    from oracle import parity as PAR
    p = _para(20, 8, 24)
    P = Plan(p)
    assert P.reflect and P.rotations == 4
    P.set_tuning("adj_run", run)
    _check(P, PAR.snapped(p, 4, True))


# the source outside the volume and inside it (windows of negative width)
@pytest.mark.parametrize("SO", [30.0, 3.0])
def test_version_1_backprojection(SO):
    """Bit for bit the reference's (its window's conversions to int saturate)."""
    import torch
    from framelab_gb300.projector import Plan
    p = G.cone_para(12, 12, 20, 6, 14, 40, L=(12.0, 12.0, 20.0), SO=SO, OD=30.0, Ly=6 * PITCH,
                    Lz=40.0)
    P = Plan(p)
    y = np.random.default_rng(6).standard_normal(P.n_rays).astype(np.float32)
    x = P.adjoint(torch.from_numpy(y).cuda(), model="chord_ref").cpu().numpy().reshape(-1)
    want = O.cone_adj_f32(y, p, threads=os.cpu_count() or 1)
    assert np.any(want)
    assert np.array_equal(x, want)
