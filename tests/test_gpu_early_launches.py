"""Kernels whose blocks are placed while the kernel before them still runs: substeps enqueued back to back, plain and
as graphs, equal substeps that are each waited for (where nothing can overlap), bit for bit, in both forms of the
neighbour search and on both sides of the size where the default form changes (14,000 particles)."""

import numpy as np
import pytest

from libclsph_gb300.gpu import GpuSolver
from test_gpu_cell_lists import _cloud

pytestmark = pytest.mark.gpu

STEPS = 18  # a graph of 16 substeps and one of 2


@pytest.mark.parametrize("n", [33, 4099, 14000, 14001, 40961])
def test_back_to_back_equals_waited(gpu_lib, n):
    scene = _cloud(n, 40.0, seed=n)
    with GpuSolver(scene.params, scene.terms, scene.n, scene.mesh) as g:
        g.upload(scene.particles)
        for _ in range(STEPS):
            g.step(1)
            assert g.sync() == 0
        want = g.download().tobytes()
        for graph in (False, True):
            g.set_graph(graph)
            g.upload(scene.particles)
            g.step(STEPS)
            assert g.sync() == 0
            assert g.download().tobytes() == want, f"graph={graph}"
