"""Deposit tiles whose sums need two words per cell (csrc/pm_deposit.cuh: TileSum).

A background of one particle per eight cells and clusters of thousands in one cell, at the edges of
tiles, row bins and the box: the fused deposit leaves the clusters' tiles to a kernel of its
own, the separate deposit takes them half their planes at a time.  Both make the same integer
sums, so a step that fuses the deposit equals one that writes the density, bit for bit; and the
density is the oracle's up to the rounding of the weights (three float32 roundings of a weight
and a quantisation of 2^-21 of a particle at most: 2e-6 in relative L2).
"""
import numpy as np
import pytest

from oracle import pm_oracle as O

pytestmark = pytest.mark.gpu


def clustered(torch, n, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    back = n ** 3 // (8 if n < 768 else 64)
    parts = [torch.rand((3, back), generator=g, device="cuda") * n]
    # (cell x, y, z): box corner, tile and bin edges, an inner cell
    for c in ((n - 1, n - 1, n - 1), (0, 3, 4), (n // 2 - 1, 4, n - 1), (min(127, n - 1), 7, 7), (5, 9, 10)):
        off = torch.tensor(c, device="cuda", dtype=torch.float32)[:, None]
        parts.append((off + 0.001 + 0.998 * torch.rand((3, 3000), generator=g, device="cuda")))
    pos = torch.cat(parts, dim=1).clamp_(max=n * (1 - 2 ** -20))
    return pos[:, torch.randperm(pos.shape[1], generator=g, device="cuda")].contiguous()


@pytest.mark.parametrize("n", [32, 48, 64, 96, 128, 192, 256, 384, 512, 768, 1024])
def test_two_word_tiles(cuda, n):
    torch = cuda
    from pmgpu.config import Config
    from pmgpu.context import PMContext
    pos = clustered(torch, n, n)
    npart = pos.shape[1]
    vel = torch.zeros_like(pos)
    mass = n ** 3 / npart
    ctx = PMContext(Config(n_parts=n // 2, n_cells=n, box_size=100.0))
    p1, v1, p2, v2 = pos.clone(), vel.clone(), pos.clone(), vel.clone()
    rho = ctx.grid()
    ctx.step(p1, v1, mass, 0.02, 0.00098)
    ctx.step(p2, v2, mass, 0.02, 0.00098, rho_out=rho)
    ctx.check_device()
    assert torch.equal(p1, p2) and torch.equal(v1, v2)
    assert abs(float(rho.double().sum()) / (npart * mass) - 1) < 1e-6
    if n <= 128:
        ref = O.density(pos.cpu().numpy(), mass, n)
        assert np.linalg.norm(rho.cpu().numpy() - ref) < 2e-6 * np.linalg.norm(ref)
    ctx.close()
