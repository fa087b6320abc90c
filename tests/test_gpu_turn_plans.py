"""The z pass with the Green function runs plans and launch shapes of its own on the larger grids
(csrc/pm_fft.cuh: TurnPlan): the Poisson solve of a log-normal density with a red spectrum
against float64, with the built-in and with a caller's Green table, at the repository's gate
for potentials (1e-5 in relative L2; gross errors of a plan are of order one)."""
import math

import pytest

pytestmark = pytest.mark.gpu


def density(torch, n):
    g = torch.Generator(device="cuda").manual_seed(n)
    dk = torch.fft.rfftn(torch.randn((n, n, n), generator=g, device="cuda"))
    f = torch.fft.fftfreq(n, device="cuda") * (2 * math.pi)
    k2 = f[:, None, None] ** 2 + f[None, :, None] ** 2 + f[None, None, : n // 2 + 1] ** 2 + 1e-4
    d = torch.fft.irfftn(dk / k2, s=(n, n, n))
    return torch.exp(d / d.std())


@pytest.mark.parametrize("n", [192, 256, 384, 512, 768])
@pytest.mark.parametrize("table", [False, True])
def test_potential_against_float64(cuda, n, table):
    torch = cuda
    from oracle import torch64
    from pmgpu.config import Config
    from pmgpu.context import PMContext
    ctx = PMContext(Config(n_parts=n // 2, n_cells=n, box_size=100.0))
    rho = density(torch, n)
    green = torch64.green(n, "cuda")
    fgrid = None
    if table:  # the reference's full table: the half spectrum and its mirror image
        fgrid = torch.empty((n, n, n), device="cuda")
        fgrid[:, :, : n // 2 + 1] = green
        fgrid[:, :, n // 2 + 1:] = green[:, :, 1: n // 2].flip(2)
    phi = ctx.potential(rho, fgrid, 0.5)
    ref = torch64.potential(rho.double(), 0.5, 0.3, green)
    assert float((phi.double() - ref).norm() / ref.norm()) < 1e-5
    ctx.check_device()
    ctx.close()
