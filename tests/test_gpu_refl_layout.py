"""Folded volume of the reflection forms: orbits of the eight flips."""
import numpy as np
import pytest

from framelab_gb300 import geometry as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nz,nv", [(4, 4, 2, 8), (4, 8, 2, 6), (36, 36, 10, 16),
                                         (20, 12, 6, 10), (12, 68, 34, 12)])
def test_fold_and_unfold_of_orbits_are_inverse(nx, ny, nz, nv):
    """A solve of no iterations folds u0 and unfolds it again: the same bits,
    on square plans (quarter turns) and rectangular ones (half turn)."""
    import torch
    from framelab_gb300.projector import Plan
    from framelab_gb300.solvers import NativeCGLS
    p = G.cone_para(nx, ny, nz, 2 * max(nx, ny), 2 * nz, nv, L=(2.0 * nx, 2.0 * ny, 2.0 * nz),
                    SO=8.0 * max(nx, ny), OD=8.0 * max(nx, ny), Ly=6.0 * max(nx, ny), Lz=4.0 * nz)
    P = Plan(p)
    assert P.reflect and P.rotations == (4 if nx == ny else 2)
    g = torch.Generator().manual_seed(nx + nz)
    u0 = torch.randn(P.n_vox, generator=g).cuda()
    u = NativeCGLS(P, "graph").solve(torch.ones_like(u0), u0, iters=0)
    assert np.array_equal(u.cpu().numpy(), u0.cpu().numpy())
