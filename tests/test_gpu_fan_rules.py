"""Default launch variants of fan turn and reflection plans over sizes and view counts."""
import numpy as np
import pytest

from framelab_gb300 import geometry as G

pytestmark = pytest.mark.gpu


def _plan(n, nv, reflect):
    from framelab_gb300.projector import Plan
    P = Plan(G.fan_para(n, n, 2 * n, nv, L=(1.0 * n, 1.0 * n), SO=2.0 * n, OD=2.0 * n, Ly=3.0 * n))
    P.reflect = reflect
    assert P.views_per_walk > 1
    return P


# thread rows of the backprojection: few blocks; blocks beyond the GPU with few and
# with many views; far beyond (152 multiprocessors)
@pytest.mark.parametrize("n,nv,reflect,rows", [
    (64, 90, False, 16), (256, 16, False, 16), (384, 32, False, 16), (512, 32, False, 8),
    (512, 180, False, 16), (1024, 360, False, 8), (256, 64, True, 16), (384, 64, True, 8),
    (384, 360, True, 16), (512, 18, True, 8), (512, 182, True, 16), (384, 17, True, 8)])
def test_thread_rows(n, nv, reflect, rows):
    """The rule's choice, and the bits of the other one."""
    import torch
    P = _plan(n, nv, reflect)
    assert P.tuning("fan_groups") == rows
    y = torch.from_numpy(np.random.default_rng(n + nv).standard_normal(P.n_rays).astype(np.float32)).cuda()
    x = P.adjoint(y)
    P.set_tuning("fan_groups", 24 - rows)
    assert torch.equal(x, P.adjoint(y))
