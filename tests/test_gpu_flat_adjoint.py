"""Cone backprojections of volumes with few heights: a column per thread where that is
faster, with the bits of the forms that put lanes along z."""
import os

import numpy as np
import pytest

import oracle as O
from framelab_gb300 import geometry as G

pytestmark = pytest.mark.gpu


def _para(n, nz, na, nb, nv, **kw):
    return dict(G.cone_para(n, n, nz, na, nb, nv, L=(1.0 * n, 1.0 * n, 1.0 * nz), SO=3.0 * n, OD=3.0 * n,
                            Ly=3.2 * n, Lz=2.6 * nz, **kw))


# the most heights at each size that takes them, one more, and an odd last run
@pytest.mark.parametrize("n,h", [(256, 1), (256, 3), (256, 4), (364, 5), (364, 6), (364, 7), (512, 2)])
@pytest.mark.parametrize("nv", [16, 18])          # quarter turns, half turn
@pytest.mark.parametrize("dtype", ["float32", "float16"])
def test_reflection_has_the_bits_of_lanes_along_z(n, h, nv, dtype):
    """FL_TUNE_ADJ_CHUNKS above one takes the lanes along z (FP32 output)."""
    import torch
    from framelab_gb300.projector import Plan
    P = Plan(_para(n, 2 * h, n, 4 * h + 2, nv))
    assert P.reflect and P.rotations == (4 if nv == 16 else 2)
    g = torch.Generator(device="cuda").manual_seed(n + h)
    y = torch.randn(P.sino_shape, device="cuda", generator=g)
    x = torch.empty(P.vol_shape, device="cuda", dtype=getattr(torch, dtype))
    P.adjoint(y, out=x)
    P.set_tuning("adj_chunks", 2)
    assert torch.equal(x, P.adjoint(y).to(x.dtype))


def _check(P, p):
    """Against the FP64 transpose (5e-6, the bound of the forms' other tests)."""
    import torch
    r = np.random.default_rng(2).standard_normal(P.n_rays).astype(np.float32)
    x = P.adjoint(torch.from_numpy(r).cuda()).cpu().numpy().reshape(-1)
    want = O.exact_adjoint(r, p, threads=os.cpu_count() or 1).reshape(-1)
    e = np.linalg.norm(x - want) / np.linalg.norm(want)
    assert e < 5e-6, e


@pytest.mark.parametrize("n,h", [(128, 1), (182, 3), (183, 2), (257, 5), (257, 4), (257, 6), (257, 7), (127, 1), (130, 2)])
@pytest.mark.parametrize("mirror", [False, True])
def test_general_and_mirror_forms(n, h, mirror):
    from framelab_gb300.projector import Plan
    p = _para(n, 2 * h if mirror else h, n, 4 * h + 2, 5)
    P = Plan(p)
    P.z_mirror = mirror
    assert not P.reflect and P.rotations == 1 and P.z_mirror == mirror
    _check(P, p)


def test_frames():
    """Three frames of one height, their views interleaved."""
    from framelab_gb300.projector import Plan
    n, nv, nt = 96, 14, 3
    p = _para(n, 1, n, 7, nv)
    views = [list(range(t, nv, nt)) for t in range(nt)]
    ids = np.array([v % nt for v in range(nv)], np.uint32)
    idY = np.zeros((len(views[0]), nt), np.uint32)
    for t, v in enumerate(views):
        idY[:len(v), t] = v
    p.update(nt=np.uint32(nt), id_X=ids, id_Y=idY, Nv=np.array([len(v) for v in views], np.uint32),
             tmp_size=np.uint32(len(views[0])))
    import torch
    P = Plan(p)
    r = np.random.default_rng(5).standard_normal(P.n_rays).astype(np.float32)
    x = P.adjoint(torch.from_numpy(r).cuda()).cpu().numpy().reshape(nt, -1)
    q = _para(n, 1, n, 7, nv)
    y = r.reshape(nv, -1)
    for t in range(nt):                            # one frame's views alone, the others' rays 0
        one = np.where((ids == t)[:, None], y, 0.0).astype(np.float32)
        want = O.exact_adjoint(one.reshape(-1), q, threads=os.cpu_count() or 1).reshape(-1)
        e = np.linalg.norm(x[t] - want) / np.linalg.norm(want)
        assert e < 5e-6, (t, e)


def test_more_frames_than_two_runs_each_fit_a_grid():
    """5 heights are two runs a frame; 32768 frames of one view, their sum is one frame's."""
    import torch
    from framelab_gb300.projector import Plan
    n, nv = 8, 32768
    q = _para(n, 5, n, 6, nv)
    p = dict(q, nt=np.uint32(nv), id_X=np.arange(nv, dtype=np.uint32),
             id_Y=np.arange(nv, dtype=np.uint32).reshape(1, nv), Nv=np.ones(nv, np.uint32),
             tmp_size=np.uint32(1))
    P = Plan(p)
    r = np.random.default_rng(7).standard_normal(P.n_rays).astype(np.float32)
    x = P.adjoint(torch.from_numpy(r).cuda()).double().reshape(nv, -1).sum(0).cpu().numpy()
    want = O.exact_adjoint(r, q, threads=os.cpu_count() or 1).reshape(-1)
    e = np.linalg.norm(x - want) / np.linalg.norm(want)
    assert e < 5e-6, e
