"""GPU parity of the collision test's early rejections, bit for bit against the oracle.

Faces whose normals are not of unit length (down to where the reference's quotient dot(n, d) / (|n| |d|)
underflows and up to large ones), turned, zero or not a number, degenerate faces, particles at rest, particles
that move along a face or end exactly on it.
"""

import numpy as np
import pytest

from libclsph_gb300 import workloads as W
from libclsph_gb300.gpu import GpuSolver

pytestmark = pytest.mark.gpu


CAP = 6


def _scene(scale, seed):
    n = 3000
    st = W.water_settings(n, restitution=0.25)
    rng = np.random.default_rng(seed)
    mesh = W.merge_meshes(W.box_mesh((0, 0, 0), (1, 1, 1)), W.heightfield_mesh((0.0, 0.0), (1.0, 1.0), 12, 0.3, 0.1, 2))
    normals = mesh["face_normals"].reshape(-1, 3).copy()
    normals[::2] *= -1.0
    normals[::3] *= np.float32(scale)
    normals[5] = 0.0
    normals[17] = np.nan
    mesh["face_normals"] = normals.ravel()
    idx = mesh["indices"].reshape(-1, 3)
    idx[40] = idx[40, 0]  # a point
    idx[51, 2] = idx[51, 1]  # a segment
    mesh["indices"] = idx.ravel()
    pos = rng.uniform(0.001, 0.999, (n, 3))
    pos[: n // 2] = np.round(pos[: n // 2] * 12) / 12 + rng.uniform(-2e-4, 2e-4, (n // 2, 3))
    pos[n // 2:: 3, 1] = rng.uniform(0.0, 4e-4, len(pos[n // 2:: 3]))
    vel = rng.normal(0.0, 2.0, (n, 3))
    vel[::7] = 0.0
    vel[1::7, 1] = 0.0
    parts = W.particles_from_arrays(pos.astype(np.float32), vel.astype(np.float32), vel.astype(np.float32))
    return st, parts, mesh


@pytest.mark.parametrize("scale", [1.0, 1e-6, 1e-18, 1e-30, 1e-42, 1e6])
def test_odd_normals_match_oracle(gpu_lib, oracle, scale):
    st, parts, mesh = _scene(scale, seed=int(abs(np.log10(scale))))
    ref = oracle.step(st.params, st.terms, parts, mesh, max_iters=CAP)
    with GpuSolver(st.params, st.terms, len(parts), mesh) as g:
        g.set_collision_cap(CAP)  # odd normals push some particles from face to face without end
        g.upload(parts)
        g.step(1)
        g.sync()
        out = g.download()
    for f in ("position", "velocity", "intermediate_velocity"):
        assert np.array_equal(out[f][:, :3], ref.final[f][:, :3], equal_nan=True)
