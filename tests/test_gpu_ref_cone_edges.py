"""Version-1 cone pair at edge sizes: bit for bit the reference's CPU kernels
(oracle restatement)."""
import os

import numpy as np
import pytest

import oracle as O
from framelab_gb300 import geometry as G

pytestmark = pytest.mark.gpu
TH = os.cpu_count() or 1


def _circle(nx, ny, nz, na, nb, nv, dz=1.0, SO=3.0, Ly=3.0, Lz=None, **kw):
    L = (2.0, 2.0 * ny / nx, 2.0 * nz / nx * dz)
    return G.cone_para(nx, ny, nz, na, nb, nv, L=L, SO=SO, OD=SO, Ly=Ly,
                       Lz=Lz or 2.2 * L[2], **kw)


def _case(name):
    return {
        # heights of 8, 16, 32 and off a multiple; one voxel column
        "low": _circle(20, 17, 5, 40, 14, 9), "half": _circle(18, 18, 16, 30, 40, 40),
        "odd": _circle(21, 19, 45, 33, 51, 35), "one": _circle(1, 1, 33, 5, 41, 3),
        # non-cubic voxels (the chord box is a unit cube all the same)
        "flat": _circle(16, 16, 12, 36, 30, 12, dz=0.4),
        "tall": _circle(16, 16, 12, 36, 31, 12, dz=2.7),
        # windows of more than 8, and of more than 32 columns
        "fine": _circle(12, 12, 10, 150, 20, 5), "finer": _circle(6, 6, 9, 400, 12, 3),
        # a far source (slopes and offsets up to 1e5: the wider margin; above:
        # every ray is evaluated), a steep panel, a helix
        "far": _circle(16, 16, 16, 34, 32, 8, SO=3000.0), "farther": _circle(16, 16, 16, 34, 32, 8, SO=3e4),
        "steep": _circle(16, 16, 40, 34, 60, 8, SO=1.6, Ly=4.0, Lz=14.0),
        "helix": G.cone_para(18, 18, 30, 30, 9, L=(2.0, 2.0, 3.4), SO=4.0, OD=4.0, Ly=3.5, Lz=1.0,
                             scan="helix", zmax=3.0, rps=2.0, vtab=2.0, fps=30),
    }[name]


CASES = ["low", "half", "odd", "one", "flat", "tall", "fine", "finer", "far", "farther", "steep",
         "helix"]


@pytest.mark.parametrize("values", ["finite", "inf", "nan"])
@pytest.mark.parametrize("name", CASES)
def test_chord_backprojection_edges_bit_exact(name, values):
    """Rays the reference gives a chord of zero are skipped unless a value is
    not finite; both ways the sums are the reference's."""
    import torch
    from framelab_gb300.projector import Plan
    p = _case(name)
    P = Plan(p)
    y = np.random.default_rng(7).standard_normal(P.n_rays).astype(np.float32)
    if values != "finite":
        y[[0, P.n_rays // 3, P.n_rays // 2 + 5]] = np.float32(values)
    x = P.adjoint(torch.from_numpy(y).cuda(), model="chord_ref").cpu().numpy().reshape(-1)
    assert np.array_equal(x, O.cone_adj_f32(y, p, threads=TH), equal_nan=True)


def test_chord_backprojection_irregular_rows_and_axis_rays():
    """Rows on no uniform grid, one at zero; views along the axes, whose
    central rays have a zero direction component."""
    import torch
    from framelab_gb300.projector import Plan
    p = dict(_circle(14, 14, 20, 29, 21, 8))
    z = np.sort(np.random.default_rng(3).uniform(-14, 14, 21)).astype(np.float32)
    z[10] = 0.0
    p["z_det"] = np.sort(z)
    P = Plan(p)
    y = np.random.default_rng(8).standard_normal(P.n_rays).astype(np.float32)
    x = P.adjoint(torch.from_numpy(y).cuda(), model="chord_ref").cpu().numpy().reshape(-1)
    assert np.array_equal(x, O.cone_adj_f32(y, p, threads=TH))


def test_chord_backprojection_can_be_captured_and_overlap():
    """Its scratch comes from a stream-ordered pool: a captured call replays to
    the same bits, and calls of one plan on two streams do not disturb each
    other."""
    import torch
    from framelab_gb300.projector import Plan
    p = _case("odd")
    P = Plan(p)
    g = torch.Generator().manual_seed(4)
    ys = [torch.randn(P.sino_shape, generator=g).cuda() for _ in range(2)]
    want = [P.adjoint(y, model="chord_ref") for y in ys]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(2)]
    outs = [torch.zeros_like(want[0]) for _ in range(2)]
    for _ in range(3):
        for k in range(2):
            P.adjoint(ys[k], model="chord_ref", out=outs[k], stream=streams[k])
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(outs, want))
    y, x = ys[0].clone(), torch.zeros_like(want[0])
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        P.adjoint(y, model="chord_ref", out=x)
    for k in range(2):
        y.copy_(ys[k])
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(x, want[k])


@pytest.mark.parametrize("name", CASES)
def test_gao_forward_edges_bit_exact(name):
    import torch
    from framelab_gb300.projector import Plan
    p = _case(name)
    P = Plan(p)
    x = np.random.default_rng(9).standard_normal(P.n_vox).astype(np.float32)
    x[P.n_vox // 2] = np.inf
    y, yn = P.forward_gao(torch.from_numpy(x).cuda())
    want, wantn = O.cone_gao_f32(x, p, threads=TH)
    assert np.array_equal(y.cpu().numpy().reshape(-1), want, equal_nan=True)
    assert np.array_equal(yn.cpu().numpy().reshape(-1), wantn, equal_nan=True)
