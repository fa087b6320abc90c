"""Device memory that admission charges for a simulation (csrc/pm_batch.cu: footprint)."""
import os
import shutil

import pytest


@pytest.fixture(scope="module", autouse=True)
def built():
    if shutil.which("nvcc") is None and not os.path.exists("/usr/local/cuda/bin/nvcc"):
        pytest.skip("nvcc not available")
    import pmgpu
    pmgpu.build()


@pytest.mark.parametrize("keep", [False, True])
@pytest.mark.parametrize("parts,n", [(8, 16), (32, 64), (96, 192), (16, 384), (256, 512), (512, 1024), (8, 1024)])
def test_footprint_counts_every_array(parts, n, keep):
    from pmgpu.batch import Batch
    from pmgpu.config import Config
    np_, bins = parts ** 3, n * n * -(-n // (128 if n <= 512 else 256))  # row bins of 128 or 256 cells
    pitch = (n // 2 + 1 + 15) // 16 * 16
    want = (2 if keep else 1) * 4 * n ** 3 + 8 * n * n * pitch    # potential, density, spectrum
    want += np_ * (2 * (6 * 4 + 4 + 16) + 2 * 4 + 6 * 4)          # two states, sort keys and order, final state
    want += 4 * (3 * bins + bins // 16)                           # bin starts, counts, cursors, group maxima
    want += 4 * 2 * (n // 4) ** 2                                 # tile order, list of two-word tiles
    assert 0 <= Batch.footprint(Config(n_parts=parts, n_cells=n, keep_density=keep)) - want <= 4096
