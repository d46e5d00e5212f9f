"""GPU parity of the density kernel's cell search at the edges of its candidate lists.

Every field bit for bit against the oracle, for the three team sizes, on clouds whose cells hold from one
to 200 particles: cells that a warp per particle does (up to 4), cells whose neighbours are chosen by their
windows (up to 32), lists that span one to four and more words of the bit planes, lists that fill a team's
shared memory and lists that do not fit it, octants with more chunks than mask words. On the CPU, the half-
precision cull against exact distances.
"""

import numpy as np
import pytest

from libclsph_gb300 import workloads as W
from libclsph_gb300.gpu import SEARCH_CELL_WARPS, STAGE_FORCES, GpuSolver

PACKED = {"particles_inside_influence_radius": 40, "fluid_density": 1000, "dynamic_viscosity": 36, "k": 5}


def _cloud(n, per_cell, seed, **fluid):
    """n particles at random with a mean of per_cell in a 2h cell, a few far apart."""
    st = W.water_settings(n, **fluid)
    h = float(st.params["h"])
    rng = np.random.default_rng(seed)
    side = (n / per_cell) ** (1.0 / 3.0) * 2.0 * h
    pos = 0.3 + rng.uniform(0.0, side, (n, 3))
    pos[:12] = 0.3 + side + h * np.arange(1, 13)[:, None]  # one to a cell
    pos[12:17] = 0.3 - 7 * h + rng.uniform(0.0, 0.5 * h, (5, 3))  # five in a cell of their own
    vel = rng.normal(0.0, 0.2, (n, 3)).astype(np.float32)
    parts = W.particles_from_arrays(pos.astype(np.float32), vel, vel)
    return W.Scene(f"cloud_{n}", st.params, st.terms, parts, W.box_mesh((-9, -9, -9), (9, 9, 9)), 10, {"h": h})


@pytest.mark.gpu
@pytest.mark.parametrize("density_block", [64, 128, 256])
@pytest.mark.parametrize("n, per_cell, fluid", [(60, 0.5, {}), (2001, 3.0, {}), (2500, 18.0, {}), (4097, 50.0, {}),
                                                (5000, 90.0, {}), (5000, 125.0, {}), (6000, 200.0, {}),
                                                (4097, 76.0, PACKED), (6001, 150.0, PACKED)])
def test_cell_lists_match_oracle(gpu_lib, oracle, n, per_cell, fluid, density_block):
    scene = _cloud(n, per_cell, seed=n + density_block, **fluid)
    ref = oracle.step(scene.params, scene.terms, scene.particles, scene.mesh)
    with GpuSolver(scene.params, scene.terms, scene.n, scene.mesh) as g:
        g.set_neighbour_search(SEARCH_CELL_WARPS)
        g.set_launch_shape(density_block, 128, 8)
        g.upload(scene.particles)
        g.step_until(STAGE_FORCES)
        assert g.sync() == 0
        rho, prs, acc = g.fields()
    assert np.array_equal(rho, ref.forces["density"])
    assert np.array_equal(prs, ref.forces["pressure"])
    assert np.array_equal(acc, ref.forces["acceleration"][:, :3])


def test_half_precision_cull_keeps_every_neighbour():
    """The cull's packed test, in numpy's half precision (FMAs rounded once, through float64), accepts every
    candidate within h of a particle of the cell and few beyond 1.03 h."""
    rng = np.random.default_rng(3)
    n = 400000
    p = rng.uniform(-1.0, 1.0, (n, 3))
    p[: n // 4] = np.sign(p[: n // 4]) * rng.uniform(0.98, 1.0, (n // 4, 3))  # near the cell's corners
    d = rng.normal(size=(n, 3))
    q = p + d / np.linalg.norm(d, axis=1)[:, None] * rng.uniform(0.97, 1.03, (n, 1))
    p, q = p.astype(np.float32), q.astype(np.float32)
    half = lambda x: np.asarray(x, np.float64).astype(np.float16).astype(np.float64)  # noqa: E731
    s = half(-(q.astype(np.float64) ** 2).sum(1))
    for a in (2, 1, 0):
        s = half(half(2.0 * p[:, a]) * half(q[:, a]) + s)
    t = (p.astype(np.float64) ** 2).sum(1) - np.float32(1.015)
    t16 = t.astype(np.float16)
    t16 = np.where(t16.astype(np.float64) > t, np.nextafter(t16, np.float16(-np.inf)), t16)  # rounded down
    r = np.linalg.norm(p.astype(np.float64) - q.astype(np.float64), axis=1)
    hit = s >= t16.astype(np.float64)
    assert hit[r <= 1.0].all()
    assert hit[r > 1.02].mean() < 0.05
