"""The remainder of float32 pairs that wraps the initial positions (csrc/pm_pair.cuh), compiled for the
host and compared with exact arithmetic."""
import os
import shutil
import subprocess
from fractions import Fraction

import numpy as np
import pytest

from conftest import PKG

PROGRAM = """
#include <cstdio>
#include "pm_pair.cuh"
int main() {
  float hi, lo, n;
  while (std::scanf("%a %a %a", &hi, &lo, &n) == 3) std::printf("%a\\n", pm::pair_mod(make_float2(hi, lo), n));
}
"""


@pytest.fixture(scope="module")
def pair_mod(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    d = tmp_path_factory.mktemp("pair")
    (d / "main.cu").write_text(PROGRAM)
    subprocess.run([nvcc, "-std=c++17", "-O2", "-Xcompiler", "-ffp-contract=off", "-I", os.path.join(PKG, "csrc"),
                    str(d / "main.cu"), "-o", str(d / "main")], check=True, capture_output=True)

    def run(hi, lo, n):
        text = "".join(f"{float(a).hex()} {float(b).hex()} {float(n).hex()}\n" for a, b in zip(hi, lo))
        out = subprocess.run([str(d / "main")], input=text, capture_output=True, text=True, check=True).stdout
        return np.array([float.fromhex(t) for t in out.split()])
    return run


@pytest.mark.parametrize("n", [16, 96, 1024])
def test_pair_mod(pair_mod, n):
    """Inside [0, n], and as far from the exact remainder (periodically) as two float32 roundings."""
    f32 = np.float32
    rng = np.random.default_rng(n)
    edges = []
    for e in (-2 * n, -n, 0, n, 2 * n, 3 * n):
        for v in (np.nextafter(f32(e), f32(-9999)), f32(e), np.nextafter(f32(e), f32(9999))):
            edges += [v] * 3
    hi = np.array(edges + list(rng.uniform(-4 * n, 4 * n, 2000)), dtype=f32)
    half = np.spacing(np.abs(hi)).astype(np.float64) / 2
    lo = (half * rng.uniform(-0.49, 0.49, hi.size)).astype(f32)
    for k in range(len(edges)):  # above, below and at each edge
        lo[k] = (0.4 * half[k] * (k % 3 - 1)) if edges[k] != 0 else 1e-9 * (k % 3 - 1)
    got = pair_mod(hi, lo, n)
    for h, l, g in zip(hi, lo, got):
        assert 0 <= g <= n, (h, l, g)
        exact = (Fraction(float(h)) + Fraction(float(l))) % n
        d = abs(Fraction(float(g)) - exact)
        assert min(d, n - d) <= Fraction(float(np.spacing(f32(n)))), (h, l, g)
