"""The autotuner takes no device memory of its own: a batch that fits steps, tuned or not."""
import os
import subprocess
import sys

import pytest

from conftest import PKG, ROOT

pytestmark = pytest.mark.gpu

# (a process of its own: schedules that were timed once are kept for the process)
PROGRAM = """
import torch
from torch.profiler import ProfilerActivity, profile
from pmgpu import ics
from pmgpu.batch import Batch
from pmgpu.config import Config
cfg = Config(n_parts=32, n_cells=64, box_size=100.0, random_seed=1, steps=100)
b = Batch(graphs=False)
b.add(cfg, *ics.initial_conditions(cfg))
for _ in range(2):
    with profile(activities=[ProfilerActivity.CUDA, ProfilerActivity.CPU]) as p:
        b.step(1)
        torch.cuda.synchronize()
x = torch.empty(1 << 24, device="cuda")
with profile(activities=[ProfilerActivity.CUDA, ProfilerActivity.CPU]) as p:
    b.step(1)
    torch.cuda.synchronize()
    y = torch.empty(1 << 26, device="cuda")  # an allocation that the profile has to show
b.check_device()
names = [e.name for e in p.events()]
tuned = [e["tuned"] for e in b.schedule() if "tuned" in e]
print("RESULT", tuned == [True], sum(n.startswith("k_kick") or "k_kick" in n for n in names), names.count("cudaMalloc"))
"""


def test_tuning_allocates_nothing(cuda):
    env = dict(os.environ, PYTHONPATH=os.pathsep.join([ROOT, PKG]))
    r = subprocess.run([sys.executable, "-c", PROGRAM], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    line = [t for t in r.stdout.splitlines() if t.startswith("RESULT")][0].split()
    if int(line[2]) == 0:
        pytest.skip("the profiler records no device events here")
    assert line[1] == "True" and int(line[2]) > 4, line  # the kick was timed in this step
    assert int(line[3]) == 1, line
