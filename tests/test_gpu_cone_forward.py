"""The cone forwards' batched walk, in every form a scan allows."""
import os

import numpy as np
import pytest

from framelab_gb300 import geometry as G

pytestmark = pytest.mark.gpu


# (nx, ny, nz, na, nb, nv): rays of fewer steps than a batch, sides below and
# above a segment of 128 planes, flat and tall boxes, square grids (quarter
# turns) and rectangles (half turn), blocks of rays with a ragged end
@pytest.mark.parametrize("nx,ny,nz,na,nb,nv", [
    (4, 4, 2, 8, 4, 8), (36, 36, 10, 50, 14, 16), (132, 132, 4, 150, 6, 8), (20, 20, 70, 34, 62, 8),
    (12, 140, 6, 46, 10, 6), (260, 8, 4, 70, 6, 10)])
def test_forward_of_every_form(nx, ny, nz, na, nb, nv):
    """Reflection, turns, half turn, z mirror and general: each against the FP64
    forward of the scan it projects (5e-6, the bound of the forms' other tests)."""
    import torch
    import oracle as O
    from oracle import parity as PAR
    from framelab_gb300.projector import Plan
    m = max(nx, ny)
    p = G.cone_para(nx, ny, nz, na, nb, nv, L=(2.0 * nx, 2.0 * ny, 2.0 * nz), SO=6.0 * m,
                    OD=6.0 * m, Ly=6.0 * m, Lz=4.4 * nz)
    P = Plan(p)
    x = np.random.default_rng(nx + nz).uniform(0, 1, P.n_vox).astype(np.float32)
    xd = torch.from_numpy(x).cuda()
    forms = set()
    for off in (None, "reflect", "quarter_turn", "rot_mirror", "z_mirror"):
        if off:
            setattr(P, off, False)
        form = (P.z_mirror, P.rotations, P.reflect)
        if form in forms:
            continue
        forms.add(form)
        y = P.forward(xd).cpu().numpy().reshape(-1)
        want = O.exact_forward(x, PAR.snapped(p, P.rotations, P.reflect),
                               threads=os.cpu_count() or 1).reshape(-1)
        e = np.linalg.norm(y - want) / np.linalg.norm(want)
        assert e < 5e-6, (form, e)
    assert len(forms) >= 4
