"""Deposit tiles of 4096 and more source entries, whose sums are held at 2^-26 in two words per cell
(csrc/pm_deposit.cuh: TileSum)."""
import pytest

pytestmark = pytest.mark.gpu

TWO_WORDS = 4096  # source entries from which on a tile sums in two words


def tile_entries(torch, pos, n):
    """Source entries of every tile (4 x 4 rows, and the row and plane below them, periodic)."""
    c = pos.floor().long() % n
    own = torch.bincount(c[2] * n + c[1], minlength=n * n).view(n, n)
    ext = torch.cat([own[-1:], own], 0)
    ext = torch.cat([ext[:, -1:], ext], 1).double()
    p = torch.zeros((n + 2, n + 2), dtype=torch.float64, device=pos.device)
    p[1:, 1:] = ext.cumsum(0).cumsum(1)
    i = torch.arange(0, n, 4, device=pos.device)
    return p[i + 5][:, i + 5] - p[i][:, i + 5] - p[i + 5][:, i] + p[i][:, i]


def uniform(torch, n, per_cell):
    g = torch.Generator(device="cuda").manual_seed(n)
    pos = torch.rand((3, int(per_cell * n ** 3)), generator=g, device="cuda") * (n * (1 - 2 ** -20))
    assert float(tile_entries(torch, pos, n).min()) >= TWO_WORDS
    return pos


@pytest.mark.parametrize("n,per_cell", [(32, 8), (64, 4), (96, 3), (128, 2), (192, 2), (256, 1), (384, 1), (512, 0.5)])
def test_dense_tiles(cuda, n, per_cell):
    """Density against float64: quantisation at 2^-26 (2^-26 / sqrt(12) a corner), the float32
    roundings of the weights and of the sum make about 3e-8 in relative L2 at one particle per cell
    and 4e-8 at a half (sums at 2^-21: 3.9e-7).  A step that deposits straight into the
    spectrum makes the same sums, so it equals the one that writes its density, bit for bit."""
    torch = cuda
    from oracle import torch64
    from pmgpu.config import Config
    from pmgpu.context import PMContext
    pos = uniform(torch, n, per_cell)
    mass = n ** 3 / pos.shape[1]
    ctx = PMContext(Config(n_parts=n // 2, n_cells=n, box_size=100.0))
    rho = ctx.density(pos, mass)
    ref = torch64.density(pos.double(), mass, n)
    assert float((rho.double() - ref).norm() / ref.norm()) < 6e-8
    p1, p2, out = pos.clone(), pos.clone(), ctx.grid()
    v1, v2 = torch.zeros_like(pos), torch.zeros_like(pos)
    ctx.step(p1, v1, mass, 0.02, 0.00098)
    ctx.step(p2, v2, mass, 0.02, 0.00098, rho_out=out)
    ctx.check_device()
    assert torch.equal(out, rho) and torch.equal(p1, p2) and torch.equal(v1, v2)
    ctx.close()


@pytest.mark.parametrize("n", [16, 32, 48, 64, 128, 192, 256, 512, 768, 1024])
def test_around_the_threshold(cuda, n):
    """Particles on grid points, all of a tile in one cell: the sums are whole numbers, and the cells
    of tiles just below and just above the threshold hold them exactly."""
    torch = cuda
    from pmgpu.config import Config
    from pmgpu.context import PMContext
    counts = (TWO_WORDS - 1, TWO_WORDS, TWO_WORDS + 1, 4 * TWO_WORDS, 1, 2048)
    cells = [(n - 1, 1, 1), (0, 5, 2), (n // 2 - 1, n - 3, n - 2), (min(127, n - 1), 9, 10), (5, 13, 1), (7, 2, 14)]
    pos = torch.cat([torch.tensor(c, dtype=torch.float32, device="cuda")[:, None].expand(3, k)
                     for c, k in zip(cells, counts)], dim=1)
    g = torch.Generator(device="cuda").manual_seed(n)
    pos = pos[:, torch.randperm(pos.shape[1], generator=g, device="cuda")].contiguous()
    e = tile_entries(torch, pos, n)
    for c, k in zip(cells, counts):
        assert int(e[c[2] // 4, c[1] // 4]) == k
    ctx = PMContext(Config(n_parts=n // 2, n_cells=n, box_size=100.0))
    rho = ctx.density(pos, 1.0)
    want = torch.zeros_like(rho)
    for c, k in zip(cells, counts):
        want[c[2], c[1], c[0]] = k
    assert torch.equal(rho, want)
    p1, p2, out = pos.clone(), pos.clone(), ctx.grid()
    v1, v2 = torch.zeros_like(pos), torch.zeros_like(pos)
    ctx.step(p1, v1, 1.0, 0.02, 0.00098)
    ctx.step(p2, v2, 1.0, 0.02, 0.00098, rho_out=out)
    ctx.check_device()
    assert torch.equal(out, want) and torch.equal(p1, p2) and torch.equal(v1, v2)
    ctx.close()


def test_dense_ensemble(cuda):
    """Eight particles a cell: every tile of every simulation takes two words, two sizes at once and
    on each of the deposit's schedules; each ends as it does alone and untuned."""
    torch = cuda
    from pmgpu.batch import Batch
    from pmgpu.config import Config
    sims = []
    for n, seed in ((32, 1), (48, 2), (32, 3)):
        p = 2 * n
        g = torch.Generator(device="cuda").manual_seed(seed)
        q = torch.arange(p, device="cuda", dtype=torch.float32) * 0.5
        grid = torch.stack(torch.meshgrid(q, q, q, indexing="ij")).reshape(3, -1)
        pos = (grid + torch.rand(grid.shape, generator=g, device="cuda") * 0.5).clamp_(max=n * (1 - 2 ** -20))
        assert float(tile_entries(torch, pos, n).min()) >= TWO_WORDS
        vel = torch.randn(pos.shape, generator=g, device="cuda") * 0.01
        sims.append((Config(n_parts=p, n_cells=n, box_size=100.0, random_seed=seed, steps=1000), pos, vel))

    torch.cuda.synchronize()  # (admission reads complete arrays)

    def run(sel, tune):
        b = Batch(autotune=tune)
        ids = [b.add(*sims[i]) for i in sel]
        b.step(5)
        b.check_device()
        out = [b.get(i, device=True)[:2] for i in ids]
        torch.cuda.synchronize()
        b.close()
        return out

    mixed, tuned = run((0, 1, 2), False), run((0, 1, 2), True)
    for i in range(3):
        alone = run((i,), False)[0]
        for got in (mixed[i], tuned[i]):
            assert torch.equal(got[0], alone[0]) and torch.equal(got[1], alone[1])


@pytest.mark.parametrize("n", [16, 64, 256])
@pytest.mark.parametrize("count", [300_000, 2 ** 20 - 1])
def test_a_million_particles_in_a_cell(cuda, n, count):
    """Two words hold a cell's sum up to 2^20 particles (2^46), exactly."""
    torch = cuda
    from pmgpu.config import Config
    from pmgpu.context import PMContext
    pos = torch.tensor([n - 1.0, 5.0, 6.0], device="cuda")[:, None].expand(3, count).contiguous()
    ctx = PMContext(Config(n_parts=n // 2, n_cells=n, box_size=100.0))
    want = torch.zeros((n, n, n), device="cuda")
    want[6, 5, n - 1] = count
    assert torch.equal(ctx.density(pos, 1.0), want)
    p1, p2, out = pos.clone(), pos.clone(), ctx.grid()
    v1, v2 = torch.zeros_like(pos), torch.zeros_like(pos)
    ctx.step(p1, v1, 1.0, 0.02, 0.00098)
    ctx.step(p2, v2, 1.0, 0.02, 0.00098, rho_out=out)
    ctx.check_device()
    assert torch.equal(out, want) and torch.equal(p1, p2) and torch.equal(v1, v2)
    ctx.close()


@pytest.mark.parametrize("n", [768, 1024])
def test_dense_slab(cuda, n):
    """The largest grids with dense tiles in a slab of 64 planes, more than there are CTAs: whole tiles of
    768 cells, halves of 1024 (gates as test_dense_tiles; 0.3 particles per cell: 5e-8)."""
    torch = cuda
    from oracle import torch64
    from pmgpu.config import Config
    from pmgpu.context import PMContext
    g = torch.Generator(device="cuda").manual_seed(n)
    pos = torch.rand((3, int(0.3 * 64 * n * n)), generator=g, device="cuda")
    pos[:2] *= n * (1 - 2 ** -20)
    pos[2] *= 64
    assert int((tile_entries(torch, pos, n) >= TWO_WORDS).sum()) > 1000
    ctx = PMContext(Config(n_parts=n // 2, n_cells=n, box_size=100.0))
    rho = ctx.density(pos, 1.0)
    ref = torch64.density(pos.double(), 1.0, n)
    assert float((rho.double() - ref).norm() / ref.norm()) < 7e-8
    del ref
    p1, p2, out = pos.clone(), pos.clone(), ctx.grid()
    v1, v2 = torch.zeros_like(pos), torch.zeros_like(pos)
    ctx.step(p1, v1, 1.0, 0.02, 0.00098)
    ctx.step(p2, v2, 1.0, 0.02, 0.00098, rho_out=out)
    ctx.check_device()
    assert torch.equal(out, rho) and torch.equal(p1, p2) and torch.equal(v1, v2)
    ctx.close()
