"""Version-1 cone backprojector's scratch: not needed, and given back."""
import numpy as np
import pytest

import oracle as O
from framelab_gb300 import geometry as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("values", ["finite", "inf", "nan", "all nan"])
@pytest.mark.parametrize("nx,nz,na,nb,nv", [(15, 21, 31, 27, 13), (6, 9, 400, 12, 3)])
def test_chord_backprojection_while_no_memory_can_be_had(nx, nz, na, nb, nv, values):
    """The reference's bits with the next allocation armed to fail, with windows of few
    columns and of more than a warp's lanes."""
    import torch
    from framelab_gb300 import _lib
    from framelab_gb300.projector import Plan
    p = G.cone_para(nx, nx, nz, na, nb, nv, L=(2.0, 2.0, 2.0 * nz / nx), SO=3.0, OD=3.0, Ly=3.0,
                    Lz=4.4 * nz / nx)
    P = Plan(p)
    y = np.random.default_rng(7).standard_normal(P.n_rays).astype(np.float32)
    if values == "all nan":
        y[:] = np.nan
    elif values != "finite":
        y[[0, P.n_rays // 3, P.n_rays // 2 + 5]] = np.float32(values)
    yd, want = torch.from_numpy(y).cuda(), O.cone_adj_f32(y, p, threads=4)
    out = torch.full((P.n_vox,), float("nan"), device="cuda")
    L = _lib.load()
    L.fl_debug_fail_alloc(1)
    try:
        x = P.adjoint(yd, model="chord_ref", out=out).cpu().numpy().reshape(-1)
    finally:
        L.fl_debug_fail_alloc(0)
    assert np.array_equal(x, want, equal_nan=True)


def test_chord_backprojection_gives_its_scratch_back():
    """A sinogram of 201 MB: after the calls the plan keeps no more than a small part of
    a copy of it."""
    import torch
    from framelab_gb300.projector import Plan
    p = G.cone_para(8, 8, 8, 2048, 1536, 16, L=(2.0, 2.0, 2.0), SO=8.0, OD=8.0, Ly=800.0, Lz=800.0)
    P = Plan(p)
    y = torch.zeros(P.sino_shape, device="cuda")
    x = torch.empty(P.vol_shape, device="cuda")
    P.forward_gao(x.zero_())                     # modules loaded
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    for _ in range(2):
        P.adjoint(y, model="chord_ref", out=x)
        torch.cuda.synchronize()
    assert free - torch.cuda.mem_get_info()[0] <= 96 << 20
