"""The launch autotuner of cone plans whose backprojection has no block shape."""
import pytest

from framelab_gb300 import geometry as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mirror", [False, True])
def test_autotune_tries_no_shapes_where_the_kernel_has_none(mirror):
    """General and z-mirror backprojections take no block shape: the built-in one
    is reported, not the fastest of equal launches."""
    from framelab_gb300.projector import Plan
    P = Plan(G.cone_para(16, 16, 8, 32, 16, 24, L=(32.0, 32.0, 16.0), SO=96.0, OD=96.0, Ly=96.0,
                         Lz=35.2))
    P.rot_mirror = False
    P.z_mirror = mirror
    for _ in range(6):
        assert P.autotune()["adjoint"] == (8, 16)
