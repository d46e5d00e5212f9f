"""GPU parity of the forces kernels around the sizes where their lanes per particle change, bit for bit against the
oracle: eight lanes up to 18,000 particles, four up to 40,000, one above; particles with more neighbours than a list
holds (96) among them."""

import numpy as np
import pytest

from libclsph_gb300.gpu import STAGE_FORCES, GpuSolver
from test_gpu_cell_lists import _cloud

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n, per_cell", [(21, 30.0), (4099, 230.0), (18000, 60.0), (18001, 60.0), (19003, 230.0),
                                         (40000, 60.0), (40001, 60.0)])
def test_forces_match_oracle(gpu_lib, oracle, n, per_cell):
    scene = _cloud(n, per_cell, seed=n)
    ref = oracle.step(scene.params, scene.terms, scene.particles, scene.mesh)
    with GpuSolver(scene.params, scene.terms, scene.n, scene.mesh) as g:
        g.upload(scene.particles)
        g.step_until(STAGE_FORCES)
        assert g.sync() == 0
        acc = g.fields()[2]
    assert np.array_equal(acc, ref.forces["acceleration"][:, :3])
