"""View chunks of the reflection backprojection: the default rule, and the mixed
solve's FP16 input."""
import pytest

from framelab_gb300 import geometry as G

pytestmark = pytest.mark.gpu


def _para(n, nz, na, nb, nv):
    return G.cone_para(n, n, nz, na, nb, nv, L=(2.0 * n, 2.0 * n, 2.0 * nz), SO=6.0 * n, OD=6.0 * n,
                       Ly=6.0 * n, Lz=4.4 * nz)


# one per half gigabyte of packed input, 1 to 16 (a plan holds no input)
@pytest.mark.parametrize("na,nb,nv,want", [(64, 32, 24, 1), (1024, 1024, 248, 1), (1024, 1024, 256, 2),
                                           (1024, 768, 720, 4), (2048, 2048, 720, 16)])
def test_default_chunk_count(na, nb, nv, want):
    from framelab_gb300.projector import Plan
    P = Plan(_para(16, 8, na, nb, nv))
    assert P.reflect and P.tuning("adj_chunks") == want


def test_default_chunks_continue_the_sums():
    """2^28 rays take two chunks by default: the bits of one launch."""
    import torch
    from framelab_gb300.projector import Plan
    P = Plan(_para(16, 8, 1024, 1024, 256))
    assert P.tuning("adj_chunks") == 2
    g = torch.Generator(device="cuda").manual_seed(3)
    y = torch.randn(P.sino_shape, device="cuda", generator=g)
    a = P.adjoint(y)
    P.set_tuning("adj_chunks", 1)
    assert torch.equal(a, P.adjoint(y))


@pytest.mark.parametrize("n,nv", [(24, 24), (20, 40)])
def test_mixed_solve_in_view_chunks(n, nv):
    """FP16 input, FP32 output: the same bits in one launch and in several."""
    import torch
    from framelab_gb300.projector import Plan
    from framelab_gb300.solvers import NativeCGLS
    P = Plan(_para(n, 12, 2 * n, 20, nv))
    assert P.reflect and P.rotations == 4
    g = torch.Generator(device="cuda").manual_seed(5)
    b = P.adjoint(P.forward(torch.rand(P.vol_shape, device="cuda", generator=g))).reshape(-1)
    u = {}
    for chunks in (1, 2, 16):
        P.set_tuning("adj_chunks", chunks)
        u[chunks] = NativeCGLS(P, "mixed").solve(b, iters=5, refresh=3)
    assert torch.equal(u[1], u[2]) and torch.equal(u[1], u[16])


def test_rows_option_is_accepted_and_read_back():
    """FL_TUNE_ADJ_ROWS selects nothing; its range stays checked."""
    from framelab_gb300 import _lib
    from framelab_gb300.projector import Plan
    P = Plan(_para(16, 8, 32, 16, 24))
    for rows in (1, 2, 3):
        P.set_tuning("adj_rows", rows)
        assert P.tuning("adj_rows") == rows
    for rows in (0, 4):
        with pytest.raises(_lib.FLError):
            P.set_tuning("adj_rows", rows)
