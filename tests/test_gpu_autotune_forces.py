"""What clsph_gpu_autotune times for the forces' block size is the kernel that has that size.

Small handles run the forces with several lanes per particle; the block size is the learned step's feature kernel's,
which has one lane per particle as the timed form has. (Trials of the form with eight lanes would all show its time.)
"""

import re

import pytest

from libclsph_gb300 import workloads as W
from libclsph_gb300.gpu import GpuSolver

pytestmark = pytest.mark.gpu


def test_forces_trials_time_the_tuned_form(gpu_lib):
    sc = W.small_block(16, seed=77, velocity_sigma=0.1)
    with GpuSolver(sc.params, sc.terms, sc.n, sc.mesh) as g:
        g.upload(sc.particles)
        report = g.autotune(10)
        g.set_persistent(False)
        g.set_profiling(True)
        g.step(20)
        g.sync()
        total, count = g.kernel_times()["forces"]
    trials = [float(t) for t in re.findall(r"forces block \d+: ([0-9.]+) ms", report)]
    assert len(trials) == 3
    assert min(trials) > 1.3 * total / count  # 1.9 times at 4,096 particles
