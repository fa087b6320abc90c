"""The drop-in step takes a whole lattice of particles in boxes when their positions say that they are in
lattice order, and in plain order else (csrc/pm_particles.cu: lattice_vote): the same bits, whatever
the order and the vote."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side,n", [(5, 32), (127, 128), (128, 192), (130, 192), (131, 64), (143, 256), (145, 192)])
@pytest.mark.parametrize("order", ["lattice", "reversed", "shuffled"])
def test_orders(cuda, side, n, order):
    torch = cuda
    from pmgpu.config import Config
    from pmgpu.context import PMContext
    g = torch.Generator(device="cuda").manual_seed(side)
    q = torch.arange(side, device="cuda", dtype=torch.float32) * (n / side)
    pos = torch.stack(torch.meshgrid(q, q, q, indexing="ij"))
    pos = (pos + torch.rand(pos.shape, generator=g, device="cuda") * 0.5).clamp_(max=n * (1 - 2 ** -20))
    vel = torch.randn((3, side ** 3), generator=g, device="cuda") * 0.01
    if order == "reversed":
        pos = pos.permute(0, 3, 2, 1)
    pos = pos.reshape(3, -1)
    if order == "shuffled":
        pos = pos[:, torch.randperm(side ** 3, generator=g, device="cuda")]
    pos = pos.contiguous()
    mass, out = n ** 3 / side ** 3, []
    for n_parts in (side, side + 1):  # (a context for side + 1 takes side^3 particles in plain order)
        ctx = PMContext(Config(n_parts=n_parts, n_cells=n, box_size=100.0))
        p, v = pos.clone(), vel.clone()
        rho = ctx.density(p, mass)
        ctx.step(p, v, mass, 0.02, 0.00098)
        hp, hv = pos.cpu().pin_memory(), vel.cpu().pin_memory()
        ctx.step_host(hp, hv, mass, 0.02, 0.00098)
        torch.cuda.synchronize()
        ctx.check_device()
        assert torch.equal(hp.cuda(), p) and torch.equal(hv.cuda(), v)
        out.append((rho, p, v))
        ctx.close()
    assert all(torch.equal(a, b) for a, b in zip(*out))
