"""Launches of a resident step, and the row scan that they depend on (csrc/pm_sort.cu: row_scan)."""
import pytest

pytestmark = pytest.mark.gpu


def config(i, parts, cells):
    from pmgpu.config import Config
    return Config(n_parts=parts, n_cells=cells, box_size=100.0, random_seed=i % 5, steps=100)


def batch(cfgs):
    from pmgpu import ics
    from pmgpu.batch import Batch
    b = Batch(graphs=False, autotune=False)
    return b, [b.add(c, *ics.initial_conditions(c)) for c in cfgs]


# one block of 4096 row bins; more than one; and more blocks than a block adds up by itself (8192)
@pytest.mark.parametrize("sizes", [[(8, 16)], [(16, 32)], [(32, 64)], [(32, 64)] * 2, [(24, 96)], [(16, 192)],
                                   [(16, 32), (24, 48)], [(16, 512)] * 33])
def test_launches_per_step(cuda, sizes):
    """launches_per_step counts the kernels of a step."""
    torch = cuda
    from torch.profiler import ProfilerActivity, profile
    b, _ = batch([config(i, *s) for i, s in enumerate(sizes)])
    b.step(2)
    torch.cuda.synchronize()
    for _ in range(2):  # (a process's first profile may hold no device events)
        with profile(activities=[ProfilerActivity.CUDA, ProfilerActivity.CPU]) as p:
            b.step(1)
            torch.cuda.synchronize()
    names = [e.name for e in p.events() if e.device_type == torch.autograd.DeviceType.CUDA]
    if not names:
        pytest.skip("the profiler records no device events here")
    kernels = [n for n in names if not n.startswith(("Memset", "Memcpy"))]
    assert len(kernels) == b.launches_per_step(), kernels
    b.close()


def test_scan_of_many_bins(cuda):
    """33 simulations of 512^3 cells have 34.6 M row bins: each runs as it does alone."""
    import numpy as np
    cfgs = [config(i, 16, 512) for i in range(33)]
    b, ids = batch(cfgs)
    b.step(3)
    b.check_device()
    for i in (0, 1, 7, 32):
        got = b.get(ids[i])[:2]
        alone, (sid,) = batch([cfgs[i]])
        alone.step(3)
        ref = alone.get(sid)[:2]
        alone.close()
        assert np.array_equal(got[0], ref[0]) and np.array_equal(got[1], ref[1])
    b.close()


def test_launches_of_the_noalloc_deposit(cuda):
    """Descriptor, keys, three kernels for each of the two digits of an 18-bit key, row starts, deposit:
    the bin maxima of the deposit's bound take no launch of their own."""
    import ctypes

    torch = cuda
    from pmgpu import _lib
    from torch.profiler import ProfilerActivity, profile
    lib, n = _lib.load(), 64
    pos = torch.rand((3, 10000), device="cuda") * n
    rho = torch.empty((n, n, n), device="cuda")
    for _ in range(3):
        with profile(activities=[ProfilerActivity.CUDA, ProfilerActivity.CPU]) as p:
            assert lib.pm_density_noalloc(ctypes.c_void_p(pos.data_ptr()), 10000, n, 1.0, ctypes.c_void_p(rho.data_ptr()),
                                          ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
            torch.cuda.synchronize()
    names = [e.name for e in p.events() if e.device_type == torch.autograd.DeviceType.CUDA]
    if not names:
        pytest.skip("the profiler records no device events here")
    assert len([k for k in names if not k.startswith(("Memset", "Memcpy"))]) == 10, names
