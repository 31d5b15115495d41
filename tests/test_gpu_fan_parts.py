"""The general fan forward's four parts per ray."""
import os

import numpy as np
import pytest

from framelab_gb300 import geometry as G

pytestmark = pytest.mark.gpu


# images of fewer segments (16 planes) than parts, one plane beside a segment's
# end, of as many as parts, of more (odd, so that no ray runs along a plane); rays in counts beside a block's 32
@pytest.mark.parametrize("nx,ny,nd,nv", [
    (1, 1, 1, 1), (3, 3, 5, 3), (15, 17, 31, 1), (17, 15, 33, 3), (33, 31, 63, 5), (65, 63, 97, 3),
    (65, 49, 31, 7), (21, 201, 65, 3), (131, 5, 127, 5)])
def test_general_fan_forward_of_any_size(nx, ny, nd, nv):
    """Against the FP64 forward (5e-6, the bound of the form's other tests)."""
    import torch
    import oracle as O
    from framelab_gb300.projector import Plan
    m = max(nx, ny)
    p = G.fan_para(nx, ny, nd, nv, L=(1.0 * nx, 1.0 * ny), SO=2.0 * m, OD=2.0 * m, Ly=3.0 * m)
    P = Plan(p)
    assert not P.reflect and P.rotations == 1
    x = np.random.default_rng(nx + nd).standard_normal(nx * ny).astype(np.float32)
    y = P.forward(torch.from_numpy(x).cuda()).cpu().numpy().reshape(-1)
    want = O.exact_forward(x, p, threads=os.cpu_count() or 1).reshape(-1)
    assert np.any(want)
    e = np.linalg.norm(y - want) / np.linalg.norm(want)
    assert e < 5e-6, e
