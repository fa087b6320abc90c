"""The order in which the drop-in step takes its particles (csrc/pm_particles.cu: ParticleOrder), and the
pairs (k, M - k) of the x rows (csrc/pm_spectral.cuh)."""
import math

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side", [1, 3, 4, 15, 16, 17, 33])
def test_lattice_order_equals_plain_order(cuda, side):
    """side^3 particles are taken in boxes of the lattice by a context for side^3 particles and in
    plain order by any other: integer deposits and one force per particle, so the same bits."""
    torch = cuda
    from pmgpu.config import Config
    from pmgpu.context import PMContext
    n, out = 32, []
    g = torch.Generator(device="cuda").manual_seed(side)
    pos = torch.rand((3, side ** 3), generator=g, device="cuda") * n
    vel = torch.randn((3, side ** 3), generator=g, device="cuda") * 0.01
    for n_parts in (side, side + 1):
        ctx = PMContext(Config(n_parts=n_parts, n_cells=n, box_size=100.0))
        p, v = pos.clone(), vel.clone()
        ctx.step(p, v, n ** 3 / side ** 3, 0.02, 0.00098)
        ctx.check_device()
        out.append((p, v))
        ctx.close()
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])


@pytest.mark.parametrize("n", [32, 48, 64, 96, 128, 192, 256, 384, 512, 768, 1024])
def test_rows_of_x_against_float64(cuda, n):
    """A density that depends on x alone has its whole spectrum in one row, which both ends of
    every row plan take apart: the Poisson solve against the closed form in float64, at the repository's
    gate for potentials (1e-5 in relative L2; a wrong pair is of order one)."""
    torch = cuda
    from pmgpu.config import Config
    from pmgpu.context import PMContext
    g = torch.Generator(device="cuda").manual_seed(n)
    f = torch.randn(n, generator=g, device="cuda")
    ctx = PMContext(Config(n_parts=n // 2, n_cells=n, box_size=100.0))
    phi = ctx.potential(f.expand(n, n, n).contiguous(), None, 0.5)
    k = torch.fft.rfft(f.double())
    s = torch.sin(math.pi * torch.arange(n // 2 + 1, device="cuda", dtype=torch.float64) / n) ** 2
    k[1:] *= -3 * 0.3 / 8 / 0.5 / s[1:]
    k[0] = 0
    ref = torch.fft.irfft(k, n=n)
    for row in (phi[0, 0], phi[n - 1, 1], phi[n // 2, n - 1]):
        assert float((row.double() - ref).norm() / ref.norm()) < 1e-5
    ctx.check_device()
    ctx.close()
