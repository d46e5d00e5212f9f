"""GPU parity of the force evaluation's short quotients at the edge of their range, bit for bit against the oracle.

The quotients d / r of a pair share one reciprocal; their residuals are exact when every coordinate is zero or at
least 2^-76 in size. A state with a smaller coordinate takes the general evaluation. Coincident particles and
pairs closer than the reference's 1e-7 floor are in both.
"""

import numpy as np
import pytest

from libclsph_gb300 import workloads as W
from libclsph_gb300.gpu import STAGE_FORCES, GpuSolver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_side", [6, 25])  # a warp per particle; cell teams
@pytest.mark.parametrize("tiny", [0.0, 2.0 ** -76, 2.0 ** -77, 1e-30, 3e-39])
def test_small_coordinates_match_oracle(gpu_lib, oracle, tiny, n_side):
    n = n_side ** 3
    st = W.water_settings(n)
    h = float(st.params["h"])
    rng = np.random.default_rng(5)
    pos = W.lattice((n_side,) * 3, h * 0.5, (-0.25 * n_side * h,) * 3, 0.2, rng)
    pos[::5, 0] = np.float32(tiny) * rng.integers(-3, 4, len(pos[::5]))
    pos[1::7, 1] = np.float32(tiny)
    pos[3] = pos[2]
    pos[5] = pos[4] + np.float32(3e-8)
    vel = rng.normal(0.0, 0.2, pos.shape).astype(np.float32)
    parts = W.particles_from_arrays(pos, vel, vel)
    mesh = W.box_mesh((-4, -4, -4), (4, 4, 4))
    ref = oracle.step(st.params, st.terms, parts, mesh)
    with GpuSolver(st.params, st.terms, n, mesh) as g:
        g.upload(parts)
        g.step_until(STAGE_FORCES)
        assert g.sync() == 0
        rho, _, acc = g.fields()
    assert np.array_equal(rho, ref.forces["density"])
    assert np.array_equal(acc, ref.forces["acceleration"][:, :3])
