"""A handle whose fluid is replaced runs the cell search that the new fluid gets in a handle of its own."""

import numpy as np
import pytest

from libclsph_gb300 import workloads as W
from libclsph_gb300.gpu import SEARCH_CELL_WARPS, GpuSolver

pytestmark = pytest.mark.gpu


def _packed(n):
    """Water with 60 particles within the radius, 115 to a 2h cell at rest."""
    st = W.water_settings(n, particles_inside_influence_radius=60)
    h = float(st.params["h"])
    rng = np.random.default_rng(8)
    side = round(n ** (1 / 3))
    pos = W.lattice((side,) * 3, (4.19 / 60) ** (1 / 3) * h, (0.0, 0.0, 0.0), 0.2, rng)
    vel = rng.normal(0.0, 0.1, pos.shape).astype(np.float32)
    return st, W.particles_from_arrays(pos, vel, vel), W.box_mesh((-9, -9, -9), (9, 9, 9))


def _density_ms(g, parts):
    g.upload(parts)
    g.step(1)
    g.set_profiling(True)
    for _ in range(5):
        g.upload(parts)
        g.step(1)
    g.sync()
    total, count = g.kernel_times()["density"]
    g.set_profiling(False)
    return total / count


def test_lists_follow_the_fluid(gpu_lib):
    n = 45 ** 3
    water = W.water_settings(n)
    st, parts, mesh = _packed(n)
    with GpuSolver(st.params, st.terms, n, mesh) as g:
        own = _density_ms(g, parts)
        g.upload(parts)
        g.step(4)
        want = g.download()
    with GpuSolver(water.params, water.terms, n, mesh) as g:
        g.set_graph(True)
        g.upload(parts)
        g.step(4)  # captured with the first fluid's lists
        g.set_parameters(st.params, st.terms)
        replaced = _density_ms(g, parts)
        g.upload(parts)
        g.step(4)
        got = g.download()
    assert replaced < 1.25 * own
    assert np.array_equal(got.view(np.uint8), want.view(np.uint8))


def test_set_shapes_stay(gpu_lib):
    """The team that a program has set is not replaced with the fluid."""
    n = 45 ** 3
    water = W.water_settings(n)
    st, parts, mesh = _packed(n)
    times = []
    for params in (st, water):
        with GpuSolver(params.params, params.terms, n, mesh) as g:
            g.set_neighbour_search(SEARCH_CELL_WARPS)
            g.set_launch_shape(256, 128, 8)
            g.set_parameters(st.params, st.terms)
            times.append(_density_ms(g, parts))
    assert max(times) < 1.25 * min(times)
