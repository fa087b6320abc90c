"""Initial conditions of the large lattices, whose displacements are made one direction at a time
(csrc/pm_ics.cu: ic_together) and, from 768 on, from spectra in blocks of rows (spec_row)."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def pairs(torch, p, seed):
    """Uniform points of the unit disc."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    r = torch.rand(p ** 3, generator=g, device="cuda").mul_(0.999).add_(5e-4).sqrt_()
    t = torch.rand(p ** 3, generator=g, device="cuda") * (2 * math.pi)
    return r * torch.cos(t), r * torch.sin(t)


def frequencies(torch, p):
    f = torch.fft.fftfreq(p, dtype=torch.float64, device="cuda") * p
    return f[:, None, None], f[None, :, None], f[None, None, :]


def field(torch, cfg, u, v):
    """gaussian_random_field.py:9-123 in float64."""
    p = cfg.n_parts
    u, v = u.double(), v.double()
    s = u * u + v * v
    t = torch.sqrt(-2.0 * torch.log(s) / s)
    rho = torch.complex(u * t, v * t).view(p, p, p)
    fz, fy, fx = frequencies(torch, p)
    k = 2 * math.pi / cfg.box_size * (fz ** 2 + fy ** 2 + fx ** 2).sqrt_()
    om, ob = cfg.omega_m0, cfg.omega_b0
    q = k / (om * cfg.h0 * math.exp(-ob - ob / om))
    x = torch.where(q > 0, 2.34 * q, 1.0)
    tr = (torch.log(1 + x) / x) ** 2 / torch.sqrt(1 + 3.89 * q + (16.1 * q) ** 2 + (5.46 * q) ** 3 + (6.71 * q) ** 4)
    shape = torch.where(k > 0, k ** cfg.power * tr, 0.0)
    del q, x, tr, k
    power = 64.0 * cfg.h0 ** 2 * float(p) ** 6 / shape.sum() * shape
    growth = 2.5 / om / (om ** (4 / 7) - cfg.omega_lambda0 + (1 + om / 2) * (1 + cfg.omega_lambda0 / 70)) * cfg.a_init
    rho *= torch.sqrt(power) * growth
    return torch.fft.ifftn(rho).real, growth


@pytest.mark.parametrize("p", [256, 384, 768])
def test_field_and_displacements(cuda, p):
    """The field against float64, and its divergence relation: -i sum_d l_d fft(disp_d) is the field's
    transform times the resolutions, off the Nyquist planes.  Positions carry the same displacements,
    the lattice and the generator's jitter, axis by axis."""
    torch = cuda
    from pmgpu.config import Config
    from pmgpu.device_ics import DeviceICs
    cfg = Config(n_parts=p, n_cells=2 * p if p < 768 else p, box_size=1.3 * p, random_seed=p, steps=100)
    g = DeviceICs(p)
    uv = pairs(torch, p, p)
    pos, vel, grf = g.generate(cfg, uv=uv, want_grf=True)
    g.close()
    ref, growth = field(torch, cfg, *uv)
    assert float((grf.double() - ref).norm() / ref.norm()) < 1e-5
    del ref
    om, ol, a0, n = cfg.omega_m0, cfg.omega_lambda0, cfg.a_init, cfg.n_cells
    fa = 1 / math.sqrt((om + ol * a0 ** 3) / a0)
    hh = math.sqrt(cfg.h0 ** 2 * (om / a0 ** 3 + ol))
    res, fres = n / p, n / cfg.box_size
    freq = frequencies(torch, p)
    div = torch.zeros((p, p, p), dtype=torch.complex128, device="cuda")
    lattice = torch.linspace(0, n - res, p, dtype=torch.float64, device="cuda") + 0.5
    draws = np.random.Generator(np.random.PCG64(cfg.random_seed))
    for d in range(3):
        disp = (vel[d].double() / (a0 * fa * hh * growth)).view(p, p, p)
        jitter = torch.from_numpy(draws.uniform(-2, 2, p ** 3)).cuda().view(p, p, p)
        at = [1, 1, 1]
        at[d] = p
        diff = (pos[d].double().view(p, p, p) - (lattice.view(at) + growth * disp + jitter)).remainder_(n)
        assert float(torch.minimum(diff, n - diff).max()) < 1e-4
        del jitter, diff
        div += torch.fft.fftn(disp) * (-2j * math.pi / cfg.box_size * freq[d])
    rk = torch.fft.fftn(grf.double()) * (res * fres)
    keep = ((freq[0] != -p // 2) & (freq[1] != -p // 2) & (freq[2] != -p // 2)).expand(p, p, p).clone()
    keep[0, 0, 0] = False
    assert float((div - rk)[keep].norm() / rk[keep].norm()) < 1e-5


@pytest.mark.parametrize("p", [384, 512])
def test_scratch(cuda, p):
    """Two spectra and one grid, and tables."""
    torch = cuda
    from pmgpu.device_ics import DeviceICs
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    g = DeviceICs(p)
    held = before - torch.cuda.mem_get_info()[0]
    g.close()
    pitch = (p // 2 + 1 + 15) // 16 * 16
    assert held < 2 * 8 * p * p * pitch + 4 * p ** 3 + (64 << 20)
