"""A mesh that cannot be set leaves the scene without one: no step reads what the failed call has freed."""

import numpy as np
import pytest

from libclsph_gb300 import workloads as W
from libclsph_gb300.gpu import ClsphError, GpuSolver

pytestmark = pytest.mark.gpu

CLSPH_ERR_TOO_LARGE = 4096
EMPTY = {"vertices": np.zeros(0, np.float32), "indices": np.zeros(0, np.uint32),
         "face_normals": np.zeros(0, np.float32)}


def test_failed_mesh_leaves_no_mesh(gpu_lib):
    sc = W.small_block(8, seed=91, velocity_sigma=2.0)
    faces = (1 << 22) + 1  # one more than the face lists hold
    big = {"vertices": sc.mesh["vertices"], "face_normals": np.tile(np.float32([0, 1, 0]), faces),
           "indices": np.tile(np.uint32([0, 1, 2]), faces)}
    with GpuSolver(sc.params, sc.terms, sc.n, EMPTY) as g:
        g.upload(sc.particles)
        g.step(5)
        assert g.sync() == 0
        want = g.download()
    with GpuSolver(sc.params, sc.terms, sc.n, sc.mesh) as g:
        with pytest.raises(ClsphError) as err:
            g.set_mesh(big)
        assert err.value.code == CLSPH_ERR_TOO_LARGE
        g.upload(sc.particles)
        g.step(5)
        assert g.sync() == 0
        got = g.download()
    assert np.array_equal(got["position"], want["position"])
