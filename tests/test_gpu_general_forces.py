"""The forces' general evaluation: a tiny coordinate, or h outside the short quotients' range.

Bit for bit against the oracle at the sizes of the three forms of the kernel (eight, four and one lane per particle)
and in the persistent kernel; the feature-gathering form against itself. One tiny coordinate anywhere sends every
particle of the handle there, so it must cost about what the quotients cost, not a new search.
"""

import numpy as np
import pytest

from libclsph_gb300 import learned as Lm
from libclsph_gb300 import workloads as W
from libclsph_gb300.gpu import SEARCH_MODES, STAGE_FORCES, GpuSolver

pytestmark = pytest.mark.gpu

SIDES = [10, 32, 36]  # 1,000, 32,768 and 46,656 particles


def _block(side, h_factor=1.0, seed=3):
    """side^3 particles at half of h; at other scales than water's, with terms that keep every sum finite."""
    n = side ** 3
    st = W.water_settings(n)
    p, t = st.params.copy(), st.terms.copy()
    h = np.float32(float(p["h"]) * h_factor)
    if h_factor != 1.0:
        p["h"], p["particle_mass"], p["fluid_density"] = h, 1.0, 100.0
        p["max_velocity"] = 0.8 * h * 60
        p["surface_tension_threshold"] = 1e-3
        t["poly_6"], t["poly_6_gradient"], t["poly_6_laplacian"] = 10 / h ** 6, -1 / h ** 5, -1 / h ** 4
        t["spiky"], t["viscosity"] = -1 / h ** 2, 1 / h
    rng = np.random.default_rng(seed)
    pos = W.lattice((side,) * 3, 0.5 * h, (0.0, 0.0, 0.0), 0.2, rng)
    vel = (h * rng.normal(0.0, 3.0, pos.shape)).astype(np.float32)
    mesh = W.box_mesh((-99 * h,) * 3, (99 * h,) * 3)
    return p, t, pos, vel, mesh, h


def _check(gpu_lib, oracle, p, t, parts, mesh):
    ref = oracle.step(p, t, parts, mesh)
    assert np.isfinite(ref.forces["acceleration"]).all() and np.isfinite(ref.forces["density"]).all()
    for persistent in (False, True):
        with GpuSolver(p, t, len(parts), mesh) as g:
            g.set_persistent(persistent)
            g.upload(parts)
            if persistent:
                g.step(1)
            else:
                g.step_until(STAGE_FORCES)
            assert g.sync() == 0
            rho, prs, acc = g.fields()
        assert np.array_equal(rho, ref.forces["density"])
        assert np.array_equal(prs, ref.forces["pressure"])
        assert np.array_equal(acc, ref.forces["acceleration"][:, :3])


@pytest.mark.parametrize("tiny", [2.0 ** -77, 1e-30, 3e-39])
@pytest.mark.parametrize("side", SIDES)
def test_tiny_coordinates_match_oracle(gpu_lib, oracle, side, tiny):
    p, t, pos, vel, mesh, h = _block(side)
    pos -= np.float32(0.25 * side) * h
    pos[::5, 0] = np.float32(tiny) * np.random.default_rng(1).integers(-3, 4, len(pos[::5]))
    pos[1::7, 1] = np.float32(tiny)
    pos[3] = pos[2]
    _check(gpu_lib, oracle, p, t, W.particles_from_arrays(pos, vel, vel), mesh)


@pytest.mark.parametrize("h", [0.999 * 2.0 ** -20, 2.0 ** -20])
@pytest.mark.parametrize("side", SIDES)
def test_radius_at_the_low_end_matches_oracle(gpu_lib, oracle, side, h):
    p, t, pos, vel, mesh, _ = _block(side, h / float(W.water_settings(side ** 3).params["h"]))
    _check(gpu_lib, oracle, p, t, W.particles_from_arrays(pos, vel, vel), mesh)


@pytest.mark.parametrize("h", [2.0 ** 20, 1.001 * 2.0 ** 20])
@pytest.mark.parametrize("side", SIDES)
def test_radius_at_the_high_end_is_the_same_in_every_search(gpu_lib, side, h):
    """(The oracle's sums hold 0 times infinity there, for particles out of reach.)"""
    p, t, pos, vel, mesh, _ = _block(side, h / float(W.water_settings(side ** 3).params["h"]))
    out = []
    for mode in SEARCH_MODES:
        with GpuSolver(p, t, len(pos), mesh) as g:
            g.set_neighbour_search(mode)
            g.upload(W.particles_from_arrays(pos, vel, vel))
            g.step_until(STAGE_FORCES)
            assert g.sync() == 0
            out.append(g.fields())
    assert all(np.isfinite(a).all() for a in out[0])
    for other in out[1:]:
        assert all(np.array_equal(a, b) for a, b in zip(out[0], other))


def test_features_with_a_tiny_coordinate(gpu_lib):
    p, t, pos, vel, mesh, h = _block(20)
    out = []
    for x in (0.0, 1e-30):
        pos[0] = (x, 60 * h, 60 * h)  # out of everyone's reach
        with GpuSolver(p, t, len(pos), mesh) as g:
            g.upload(W.particles_from_arrays(pos, vel, vel))
            g.step_until(STAGE_FORCES)
            out.append((g.ids(), g.fields()[2], Lm.read_features(g)))
    assert np.array_equal(out[0][0], out[1][0])
    others = out[0][0] != 0
    for a, b in zip(out[0][1:], out[1][1:]):
        assert np.array_equal(a[others], b[others])


def test_a_tiny_coordinate_costs_no_search(gpu_lib):
    p, t, pos, vel, mesh, _ = _block(64)
    ms = []
    for x in (0.0, 1e-30):
        pos[7, 0] = x
        parts = W.particles_from_arrays(pos, vel, vel)
        with GpuSolver(p, t, len(pos), mesh) as g:
            g.upload(parts)
            g.step(1)
            g.set_profiling(True)
            for _ in range(5):
                g.upload(parts)
                g.step(1)
            g.sync()
            total, count = g.kernel_times()["forces"]
            ms.append(total / count)
    assert ms[1] < 4 * ms[0]  # (1.4 times; rescanning every window took 20)
