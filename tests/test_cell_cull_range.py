"""The cell search's half-precision cull over the whole range of coordinates that it serves.

The constants are read from the kernel. On the CPU: the sum of the worst roundings of every step stays below the
cull's margin, and the packed test in numpy's half precision keeps every neighbour. On the GPU: a cloud so far from
the origin that the centres of its cells are rounded by a good part of h, bit for bit against the oracle.
"""

import re
from pathlib import Path

import numpy as np
import pytest

from libclsph_gb300 import workloads as W
from libclsph_gb300.gpu import SEARCH_CELL_WARPS, STAGE_FORCES, GpuSolver

KERNELS = Path(__file__).resolve().parents[1] / "libclsph_gb300" / "csrc" / "clsph_kernels.cuh"


def _constant(name):
    return float(re.search(rf"constexpr float {name} = ([0-9.]+)f;", KERNELS.read_text())[1])


def _pairs(rng, n, gate):
    """Particles up to the gate, many of them at its corners, and candidates within 1 of them."""
    p = rng.uniform(-gate, gate, (n, 3))
    p = np.where(rng.random((n, 3)) < 0.5, np.sign(p) * rng.uniform(0.97 * gate, gate, (n, 3)), p)
    p = np.where(rng.random((n, 3)) < 0.1, np.sign(p) * gate, p)
    d = rng.normal(size=(n, 3))
    out = rng.random(n) < 0.5
    d[out] = np.abs(d[out]) * np.sign(p[out])
    return p, p + d / np.linalg.norm(d, axis=1)[:, None] * rng.uniform(0.9, 1.0, (n, 1))


def _half_ulp(v):
    return 2.0 ** (np.floor(np.log2(np.maximum(np.abs(v), 2.0 ** -14))) - 11)


def test_worst_roundings_stay_below_the_margin():
    gate, margin = _constant("kCellGate"), _constant("kCellCullR2") - 1.0
    rng = np.random.default_rng(11)
    for _ in range(10):
        p, q = _pairs(rng, 200000, gate)
        up, uq = _half_ulp(2 * p), _half_ulp(q)
        error = (up * np.abs(q) + 2 * np.abs(p) * uq + up * uq).sum(1)
        s = -(q * q).sum(1)
        error += _half_ulp(s * 1.01)
        for a in (2, 1, 0):
            s = s + 2 * p[:, a] * q[:, a]
            error += _half_ulp(s * 1.01)  # (the rounded sums can lie in the next binade)
        assert error.max() < margin


def test_cull_keeps_every_neighbour_up_to_the_gate():
    gate, r2 = _constant("kCellGate"), np.float32(_constant("kCellCullR2"))
    rng = np.random.default_rng(12)
    half = lambda x: np.asarray(x, np.float64).astype(np.float16).astype(np.float64)  # noqa: E731
    for _ in range(5):
        p, q = _pairs(rng, 200000, gate)
        p = np.clip(p.astype(np.float32), -np.float32(gate), np.float32(gate)).astype(np.float64)
        q = q.astype(np.float32).astype(np.float64)
        s = half(-(q ** 2).sum(1))
        for a in (2, 1, 0):
            s = half(half(2.0 * p[:, a]) * half(q[:, a]) + s)
        t = (p ** 2).sum(1) - r2
        t16 = t.astype(np.float16)
        t16 = np.where(t16.astype(np.float64) > t, np.nextafter(t16, np.float16(-np.inf)), t16)  # rounded down
        near = np.linalg.norm(p - q, axis=1) <= 1.0
        assert near.sum() > 100000
        assert (s >= t16.astype(np.float64))[near].all()


@pytest.mark.gpu
@pytest.mark.parametrize("density_block", [64, 128, 256])
@pytest.mark.parametrize("far", [2.0 ** 11, 2.0 ** 13, 2.0 ** 15])  # in units of 64 h: centres off by up to h/128 ... h/8
def test_cloud_far_from_the_origin_matches_oracle(gpu_lib, oracle, far, density_block):
    n = 4001
    st = W.water_settings(n)
    st = W.water_settings(n, mass=0.05 * (1.0 / 64.0 / float(st.params["h"])) ** 3)
    h = float(st.params["h"])
    rng = np.random.default_rng(13)
    side = (n / 40.0) ** (1.0 / 3.0) * 2.0 * h
    pos = (64 * h * far + rng.uniform(0.0, side, (n, 3))).astype(np.float32)
    vel = rng.normal(0.0, 0.2, (n, 3)).astype(np.float32)
    parts = W.particles_from_arrays(pos, vel, vel)
    mesh = W.box_mesh((64 * h * far - 9,) * 3, (64 * h * far + 9,) * 3)
    ref = oracle.step(st.params, st.terms, parts, mesh)
    with GpuSolver(st.params, st.terms, n, mesh) as g:
        g.set_neighbour_search(SEARCH_CELL_WARPS)
        g.set_launch_shape(density_block, 128, 8)
        g.upload(parts)
        g.step_until(STAGE_FORCES)
        assert g.sync() == 0
        rho, prs, acc = g.fields()
    assert np.array_equal(rho, ref.forces["density"])
    assert np.array_equal(prs, ref.forces["pressure"])
    assert np.array_equal(acc, ref.forces["acceleration"][:, :3])
