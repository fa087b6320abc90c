"""Paths of the large grids: spectra in blocks of rows from 768 cells on (csrc/pm_common.cuh: spec_row)
and the z passes with plans of their own (csrc/pm_fft.cuh: TurnPlan), where the other tests end
at smaller grids."""
import dataclasses

import numpy as np
import pytest

from test_gpu_turn_plans import density

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("table", [False, True])
def test_potential_1024_against_float64(cuda, table):
    """As test_gpu_turn_plans does for the smaller grids, at the same gate."""
    torch = cuda
    from oracle import torch64
    from pmgpu.config import Config
    from pmgpu.context import PMContext
    n = 1024
    ctx = PMContext(Config(n_parts=n // 2, n_cells=n, box_size=100.0))
    rho = density(torch, n)
    green = torch64.green(n, "cuda")
    fgrid = None
    if table:
        fgrid = torch.empty((n, n, n), device="cuda")
        fgrid[:, :, : n // 2 + 1] = green
        fgrid[:, :, n // 2 + 1:] = green[:, :, 1: n // 2].flip(2)
    phi = ctx.potential(rho, fgrid, 0.5)
    ref = torch64.potential(rho.double(), 0.5, 0.3, green)
    assert float((phi.double() - ref).norm() / ref.norm()) < 1e-5
    ctx.check_device()
    ctx.close()


@pytest.mark.parametrize("n", [768, 1024])
def test_power_spectrum_against_float64(cuda, n):
    """Every shell within 1e-4, the gate of the evolved grids up to 512 cells."""
    torch = cuda
    from oracle import torch64
    from pmgpu.config import Config
    from pmgpu.context import PMContext
    g = torch.Generator(device="cuda").manual_seed(n)
    rho = torch.rand((n, n, n), generator=g, device="cuda")
    ctx = PMContext(Config(n_parts=n // 2, n_cells=n, box_size=100.0))
    k, p, modes = ctx.power_spectrum(rho)
    k2, p2, modes2 = torch64.power_spectrum(rho, 100.0)
    assert np.array_equal(modes, modes2) and np.allclose(k, k2, rtol=1e-12)
    assert np.abs(p / p2 - 1).max() < 1e-4
    ctx.check_device()
    ctx.close()


@pytest.mark.parametrize("n", [192, 256, 384, 512, 768, 1024])
def test_spectral_gradient_matches_central_differences(cuda, n):
    """The gate of test_gpu_gradient: the kick's error is the potential's rounding over the difference of
    neighbouring values, about 6e-8 n / 2 pi, 1e-5 at 1024."""
    torch = cuda
    from pmgpu.config import Config
    from pmgpu.context import PMContext
    g = torch.Generator(device="cuda").manual_seed(n)
    p = 64
    q = torch.arange(p, device="cuda", dtype=torch.float32) * (n / p)
    pos = torch.stack(torch.meshgrid(q, q, q, indexing="ij")).reshape(3, -1)
    pos = (pos + torch.rand(pos.shape, generator=g, device="cuda") * (2 * n / p)).remainder_(n)
    pos.clamp_(max=n * (1 - 2 ** -20))
    cfg = Config(n_parts=p, n_cells=n, box_size=150.0)
    out = []
    for c in (cfg, dataclasses.replace(cfg, spectral_gradient=True)):
        ctx = PMContext(c)
        x, v = pos.clone(), torch.zeros_like(pos)
        ctx.step(x, v, cfg.mass, 0.02, 0.00098)
        ctx.check_device()
        ctx.close()
        out.append((x, v))
    (x1, v1), (x2, v2) = out
    assert float((v2 - v1).norm() / v1.norm()) < 1e-4
    d = (x2 - x1).abs()
    assert float(torch.minimum(d, n - d).max()) < 1e-4
