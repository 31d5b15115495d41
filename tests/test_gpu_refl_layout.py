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


# (nx, ny, nz, na, nb, nv): half heights below, at and off a multiple of the 32
# lanes and with 16 and 8 lanes per block of columns (the two 160-wide grids),
# odd counts of 2 x 2 blocks, and detectors so fine that a column's shadow holds
# more candidates than the 4, 8, 16 or 32 of one pass
@pytest.mark.parametrize("nx,ny,nz,na,nb,nv", [
    (12, 12, 6, 24, 10, 8), (12, 20, 64, 40, 70, 6), (20, 20, 70, 44, 60, 16),
    (16, 16, 8, 200, 12, 8), (16, 16, 8, 640, 60, 8), (8, 24, 8, 1024, 16, 10),
    (160, 160, 32, 320, 40, 6), (160, 160, 16, 1920, 24, 6)])
def test_reflection_backprojection_of_any_size(nx, ny, nz, na, nb, nv):
    """Against the FP64 transpose of the snapped scan (5e-6, the bound of the
    form's other tests), and the same bits with one or 2 x 2 columns per warp
    and in view chunks."""
    import os
    import torch
    import oracle as O
    from oracle import parity as PAR
    from framelab_gb300.projector import Plan
    m = max(nx, ny)
    p = G.cone_para(nx, ny, nz, na, nb, nv, L=(2.0 * nx, 2.0 * ny, 2.0 * nz), SO=6.0 * m,
                    OD=6.0 * m, Ly=6.0 * m, Lz=4.4 * nz)
    P = Plan(p)
    NR = 4 if nx == ny and nv % 8 == 0 else 2
    assert P.reflect and P.rotations == NR
    r = np.random.default_rng(nx + nz).standard_normal(P.n_rays).astype(np.float32)
    rd = torch.from_numpy(r).cuda()
    want = O.exact_adjoint(r, PAR.snapped(p, NR, True), threads=os.cpu_count() or 1)
    got = {}
    for run in (1, 2):
        for chunks in (1, 2):
            P.set_tuning("adj_run", run)
            P.set_tuning("adj_chunks", chunks)
            got[run, chunks] = P.adjoint(rd).cpu().numpy().reshape(-1)
    x = got[1, 1]
    assert all(np.array_equal(x, g) for g in got.values())
    e = np.linalg.norm(x - want.reshape(-1)) / np.linalg.norm(want)
    assert e < 5e-6, e
