"""The sort and the search on a grid of more than 1,023 cells, which is flagged and whose coordinates wrap.

One particle lies 1,028 cells beyond a cloud of 100 x 20 x 20 cells: the wrapped grid size (7 or 8) needs fewer
bits than the cloud's own coordinates. No record may be lost, and since the far particle is out of everyone's
reach, all others move as the oracle moves them without it, bit for bit. The same in a batch, whose other scenes
keep their key range to themselves.
"""

import numpy as np
import pytest

from libclsph_gb300 import workloads as W
from libclsph_gb300.gpu import SEARCH_MODES, WARN_GRID_OVERFLOW, GpuSolver

pytestmark = pytest.mark.gpu

FIELDS = ("position", "velocity", "intermediate_velocity")


def _cloud(n, cells, seed):
    """n particles over a floor of the given cells, half of them in a block; the last one far away."""
    st = W.water_settings(n)
    h = float(st.params["h"])
    rng = np.random.default_rng(seed)
    pos = rng.uniform(0.0, 1.0, (n, 3)) * np.array(cells) * 2 * h
    pos[0], pos[1] = 0.0, np.array(cells) * 2 * h
    block = np.arange(2, n // 2)
    pos[block] = 5 * h + rng.uniform(0.0, 1.0, (len(block), 3)) * 0.5 * h * len(block) ** (1 / 3)
    pos[-1] = (1028 * 2 * h, h, h)
    vel = rng.normal(0.0, 0.2, (n, 3)).astype(np.float32)
    parts = W.particles_from_arrays(pos.astype(np.float32), vel, vel)
    return st, parts, W.box_mesh((-9 * h, -9 * h, -9 * h), (1100 * 2 * h, 99 * h, 99 * h))


def _by_id(out, ids):
    back = np.empty(len(ids), dtype=out.dtype)
    back[ids] = out
    return back


def _want(oracle, st, parts, mesh, steps):
    """The oracle's records after `steps` without the far particle, in input order."""
    ids = np.arange(len(parts) - 1)
    cur = parts[:-1]
    for _ in range(steps):
        ref = oracle.step(st.params, st.terms, cur, mesh)
        ids, cur = ids[ref.perm], ref.final
    return _by_id(cur, ids)


@pytest.mark.parametrize("form", [*(("search", m) for m in SEARCH_MODES), ("persistent", 0), ("graph", 0)])
@pytest.mark.parametrize("n", [4000, 20001])
def test_overflowed_grid_keeps_every_particle(gpu_lib, oracle, n, form):
    st, parts, mesh = _cloud(n, (100, 20, 20), seed=n)
    want = _want(oracle, st, parts, mesh, 2)
    with GpuSolver(st.params, st.terms, n, mesh) as g:
        if form[0] == "search":
            g.set_neighbour_search(form[1])
        elif form[0] == "persistent":
            g.set_persistent(True)
        else:
            g.set_graph(True)
        g.upload(parts)
        g.step(2)
        assert g.sync() == WARN_GRID_OVERFLOW
        ids, out = g.ids(), g.download()
    assert np.array_equal(np.sort(ids), np.arange(n))
    out = _by_id(out, ids)
    for f in FIELDS:
        assert np.array_equal(out[f][:-1, :3], want[f][:, :3]), f
    assert np.array_equal(out["density"][:-1], want["density"])


@pytest.mark.parametrize("scenes", [3, 200])  # the scenes take two and eight bits of a key
def test_overflowed_scene_leaves_the_others_alone(gpu_lib, oracle, scenes):
    st, parts, mesh = _cloud(1500, (100, 20, 20), seed=7)
    others = [W.small_block(4 + k % 3, seed=k, velocity_sigma=0.3) for k in range(scenes - 1)]
    with GpuSolver.batched([st.params] + [o.params for o in others], [st.terms] + [o.terms for o in others],
                           [len(parts)] + [o.n for o in others], [mesh] + [o.mesh for o in others]) as g:
        g.upload(np.concatenate([parts] + [o.particles for o in others]))
        g.step(1)
        assert g.sync() == WARN_GRID_OVERFLOW
        ids, out, first = g.ids(), g.download(), g.first
    assert np.array_equal(np.sort(ids), np.arange(len(ids)))
    assert np.array_equal(np.sort(ids[:len(parts)]), np.arange(len(parts)))
    for k, o in enumerate(others):
        ref = oracle.step(o.params, o.terms, o.particles, o.mesh).final
        part = out[first[k + 1]:first[k + 2]]
        for f in FIELDS:
            assert np.array_equal(part[f][:, :3], ref[f][:, :3]), (k, f)
        assert np.array_equal(part["density"], ref["density"]), k
