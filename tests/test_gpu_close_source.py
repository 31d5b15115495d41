"""Backprojection with the source within a voxel of the grid's corner: blocks of
2 x 2 columns that reach past an odd grid must not reach the source."""
import os

import numpy as np
import pytest

import oracle as O
from framelab_gb300 import geometry as G

pytestmark = pytest.mark.gpu

# the nearest source the matched model takes, beside the grid's far corner
PHI = (1.25 * np.pi + np.linspace(-0.04, 0.04, 16)).astype(np.float32)


def _source(n):
    return np.sqrt(0.5 * n * n) + 1.0 + 0.01


def _check(P, p):
    """Against the FP64 transpose (5e-6, the bound of the forms' other tests)."""
    import torch
    r = np.random.default_rng(2).standard_normal(P.n_rays).astype(np.float32)
    x = P.adjoint(torch.from_numpy(r).cuda()).cpu().numpy().reshape(-1)
    want = O.exact_adjoint(r, p, threads=os.cpu_count() or 1).reshape(-1)
    e = np.linalg.norm(x - want) / np.linalg.norm(want)
    assert e < 5e-6, e


# a block size that is set, and a grid that takes 2 x 2 by itself
@pytest.mark.parametrize("n,block", [(19, 1), (19, 2), (183, 0)])
def test_fan_blocks_past_the_grid(n, block):
    from framelab_gb300.projector import Plan
    SO = _source(n)
    p = G.fan_para(n, n, 200, 16, L=(1.0 * n, 1.0 * n), SO=SO, OD=SO, Ly=4.0 * SO * np.tan(0.8),
                   sd_phi=PHI)
    P = Plan(p)
    assert not P.reflect and P.rotations == 1
    if block:
        P.set_tuning("fan_block", block)
    else:
        assert P.tuning("fan_block") == 2
    _check(P, p)


# heights that take 2 x 2 columns per warp, and one
@pytest.mark.parametrize("nz", [160, 20])
def test_cone_blocks_past_the_grid(nz):
    from framelab_gb300.projector import Plan
    n = 35
    SO = _source(n)
    p = dict(G.cone_para(n, n, nz, 200, 12, 16, L=(1.0 * n, 1.0 * n, 1.0 * nz), SO=SO, OD=SO,
                         Ly=4.0 * SO * np.tan(0.8), Lz=1.5 * nz))
    p.update(sd_phi=PHI, cos_phi=np.cos(PHI.astype(np.float64)).astype(np.float32),
             sin_phi=np.sin(PHI.astype(np.float64)).astype(np.float32))
    P = Plan(p)
    P.z_mirror = False
    assert not P.reflect and P.rotations == 1
    _check(P, p)
