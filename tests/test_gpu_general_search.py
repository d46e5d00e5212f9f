"""A smoothing radius outside the cell search's range: another search in its place, not a warp per particle."""

import numpy as np
import pytest

from libclsph_gb300 import workloads as W
from libclsph_gb300.gpu import SEARCH_CELL_WARPS, SEARCH_WINDOW, GpuSolver
from test_gpu_general_forces import _block

pytestmark = pytest.mark.gpu


def test_radius_out_of_range_takes_another_search(gpu_lib):
    side, times, out = 64, [], []
    p, t, pos, vel, mesh, _ = _block(side, 0.99 * 2.0 ** -20 / float(W.water_settings(side ** 3).params["h"]))
    parts = W.particles_from_arrays(pos, vel, vel)
    for mode, persistent in ((SEARCH_WINDOW, False), (SEARCH_CELL_WARPS, False), (SEARCH_CELL_WARPS, True)):
        with GpuSolver(p, t, len(pos), mesh) as g:
            g.set_neighbour_search(mode)
            g.set_persistent(persistent)
            g.upload(parts)
            g.step(2)
            out.append(g.download())
            g.set_profiling(True)
            for _ in range(5):
                g.upload(parts)
                g.step(1)
            g.sync()
            total, count = g.kernel_times()["density"]
            times.append(total / count)
    assert np.array_equal(out[0].view(np.uint8), out[1].view(np.uint8))
    assert np.array_equal(out[0].view(np.uint8), out[2].view(np.uint8))
    assert times[1] < 1.5 * times[0]  # (the same kernel; a warp per particle takes four times as long)


def test_radius_leaves_and_enters_the_range(gpu_lib):
    """Replayed graphs follow a parameter change in both directions."""
    p, t, pos, vel, mesh, _ = _block(32)
    p2, t2, pos2, vel2, _, _ = _block(32, 0.99 * 2.0 ** -20 / float(p["h"]))
    a, b = W.particles_from_arrays(pos, vel, vel), W.particles_from_arrays(pos2, vel2, vel2)
    want = []
    for params, terms, parts in ((p, t, a), (p2, t2, b)):
        with GpuSolver(params, terms, len(pos), mesh) as g:
            g.upload(parts)
            g.step(2)
            want.append(g.download())
    with GpuSolver(p, t, len(pos), mesh) as g:
        g.set_graph(True)
        for k in (0, 1, 0):
            g.set_parameters(*((p, t), (p2, t2))[k])
            g.upload((a, b)[k])
            g.step(2)
            assert np.array_equal(g.download().view(np.uint8), want[k].view(np.uint8))


def test_autotune_offers_no_persistent_form(gpu_lib):
    """Out of range the persistent form is not run: a report would compare the launched one with itself."""
    p, t, pos, vel, mesh, _ = _block(12, 0.99 * 2.0 ** -20 / float(W.water_settings(12 ** 3).params["h"]))
    with GpuSolver(p, t, len(pos), mesh) as g:
        g.upload(W.particles_from_arrays(pos, vel, vel))
        report = g.autotune(2)
    assert "whole substep" not in report and "launched substeps" in report
