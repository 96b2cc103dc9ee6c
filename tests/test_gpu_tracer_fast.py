"""Slots with slow and fast flows in one batch: whichever way their particles are traced, the same bits."""
import numpy as np
import pytest

from parallelspectralfluids3d_b200 import _lib as L
from parallelspectralfluids3d_b200.batch import Batch
from parallelspectralfluids3d_b200.fixture import initial_coefficients, initial_particles
from test_gpu_particle_order import toy_basis

pytestmark = pytest.mark.gpu

# Displacement of the faces in voxels per step (root mean square); a flow is fast from 0.12 on.
STEPS = [0.0, 1e-3, 0.11, 0.13, 1.0, 7.0, 0.5]


@pytest.mark.parametrize("integrator", [L.PSF_RK1, L.PSF_RK4])
@pytest.mark.parametrize("fused", [True, False])
def test_fast_slots(small_bases, integrator, fused):
    b = small_bases["sphere12x10x9"]
    dt = 0.01
    params = L.make_params(dt=dt, integrator=integrator, lifetime=5.0, seed=6, precision=L.PSF_PRECISION_BF16X2)
    count = int(0.6 * b.n_voxels)
    out = []
    for capacity in (40 * b.n_voxels, count):  # pairs: lists and straight through; faces once: straight through
        with Batch([b], len(STEPS), capacity, autotune=False, fused=fused, particle_pool=1024 * len(STEPS)) as bt:
            for s, step in enumerate(STEPS):
                w0 = initial_coefficients(b.n_modes, s)
                w0 *= step * b.h * np.sqrt(b.n_active) / (dt * np.linalg.norm(w0))
                p = initial_particles(b, 1 if s == 1 else count, 9 + s)
                p[:, 3] = np.where(np.arange(len(p)) % 4, np.inf, np.arange(len(p)) % 7)
                bt.set_instance(0, s, w0, params, p, steps=4 if s == 5 else 0)
            bt.step(9)
            assert bt.device_status() == 0
            out.append([(bt.get_state(0, s), bt.get_particles(0, s)) for s in range(len(STEPS))])
    for x, y in zip(*out):
        assert np.array_equal(x[0], y[0], equal_nan=True)
        assert np.array_equal(x[1], y[1], equal_nan=True)
    moved = [np.isfinite(p).any() for _, p in out[0]]
    assert all(moved)


@pytest.mark.parametrize("integrator", [L.PSF_RK1, L.PSF_RK4])
@pytest.mark.parametrize("count", [30000, 60000])  # three slots: below and above a particle per thread of the grid
def test_slow_and_fast_with_lists(integrator, count):
    b = toy_basis((64, 48, 48))
    dt = 0.01
    params = L.make_params(dt=dt, integrator=integrator, lifetime=6.0, seed=2, precision=L.PSF_PRECISION_BF16X2)
    rng = np.random.default_rng(count)
    size = np.asarray(b.aabb_max) - b.aabb_min
    start = []
    for s in range(3):
        p = np.full((count - 7 * s, 4), np.inf, np.float32)
        p[:, :3] = b.aabb_min + size * rng.random((len(p), 3), dtype=np.float32)
        p[::9, 3] = np.arange(len(p[::9])) % 8
        start.append(p)
    out = []
    for capacity in (3 * b.n_voxels, count):  # pairs, faces once
        with Batch([b], 3, capacity, autotune=False, particle_pool=3 * count + 1024) as bt:
            for s, step in enumerate((0.02, 0.6, 0.119)):
                w0 = np.array([1.0, -2.0, 0.5])
                w0 *= step * b.h * np.sqrt(b.n_active) / (dt * np.linalg.norm(w0))
                bt.set_instance(0, s, w0, params, start[s])
            bt.step(10)
            out.append([bt.get_particles(0, s) for s in range(3)])
    for x, y in zip(*out):
        assert np.array_equal(x, y)
    moved = np.abs(out[0][1][:, :3] - start[1][:, :3]).max(axis=1) / b.h
    assert np.median(moved) > 1.0
