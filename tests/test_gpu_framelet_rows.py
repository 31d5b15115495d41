"""The z-streaming framelet levels at the edges of their rows and segments."""
import pytest

pytestmark = pytest.mark.gpu


# rows of one thread, at and beside a warp, at and beside the longest whole row,
# and of several parts with a short last one; planes shorter than the dilation;
# depths of one slice per class and beside the segments' ends
@pytest.mark.parametrize("nx,ny,nz,levels", [
    (1, 3, 2, 2), (2, 9, 5, 4), (31, 7, 9, 3), (32, 8, 33, 1), (33, 17, 12, 4), (129, 5, 70, 2),
    (255, 3, 6, 2), (512, 4, 9, 3), (513, 6, 10, 4), (769, 5, 9, 2), (1029, 2, 7, 4)])
@pytest.mark.parametrize("bank", ["linear", "haar"])
def test_streamed_levels_equal_the_pass_kernels(nx, ny, nz, levels, bank):
    """Every value is the same chain of multiply-adds in both forms: the same bits."""
    import torch
    from framelab_gb300.transforms import FrameletSystem
    g = torch.Generator().manual_seed(nx + ny + nz)
    W = FrameletSystem((nz, ny, nx), bank, levels)
    u, base = (torch.randn((nz, ny, nx), generator=g).cuda() for _ in range(2))
    v0 = torch.randn(W.ncoef, generator=g).cuda()
    out = []
    for fused in (True, False):
        W.fused = fused
        c = W.forward(u)
        v, t, b = v0.clone(), torch.zeros_like(v0), torch.empty_like(u)
        W.bregman(u, v, t, base, 0.7, 0.2, b)
        out.append((c, W.adjoint(c), v, t, b))
    for a, b in zip(*out):
        assert torch.equal(a, b)
