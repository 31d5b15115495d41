"""The z-streaming framelet levels on rows of several tiles, and on rows that are no
multiple of the memory sector, in volumes below and far above the L2."""
import pytest

pytestmark = pytest.mark.gpu


# tiles of 192, 224 and 256 columns with short and full last ones; rows off 32 and off
# 16 bytes (the last two: coefficients of more than 400 MB)
@pytest.mark.parametrize("nx,ny,nz,levels", [
    (520, 5, 9, 3), (600, 3, 12, 2), (672, 3, 5, 4), (768, 4, 6, 2), (1100, 2, 9, 3), (36, 9, 40, 2),
    (34, 9, 40, 2), (161, 160, 160, 2), (164, 160, 160, 1)])
@pytest.mark.parametrize("bank", ["linear", "haar"])
def test_tiled_levels_equal_the_pass_kernels(nx, ny, nz, levels, bank):
    """Every value is the same chain of multiply-adds in both forms: the same bits."""
    import torch
    from framelab_gb300.transforms import FrameletSystem
    g = torch.Generator(device="cuda").manual_seed(nx + ny + nz)
    W = FrameletSystem((nz, ny, nx), bank, levels)
    u, base = (torch.randn((nz, ny, nx), generator=g, device="cuda") for _ in range(2))
    v0 = torch.randn(W.ncoef, generator=g, device="cuda")
    out = []
    for fused in (True, False):
        W.fused = fused
        c = W.forward(u)
        v, t, b = v0.clone(), torch.zeros_like(v0), torch.empty_like(u)
        W.bregman(u, v, t, base, 0.7, 0.2, b)
        out.append((c, W.adjoint(c), v, t, b))
    for a, b in zip(*out):
        assert torch.equal(a, b)
