"""A batch of a centred and an off-centre box: its tracer takes each slot's own form of the interpolant."""
import dataclasses

import numpy as np
import pytest

from oracle import oracle as O
from parallelspectralfluids3d_b200 import _lib as L
from parallelspectralfluids3d_b200.batch import Batch
from parallelspectralfluids3d_b200.fixture import initial_coefficients, initial_particles

from conftest import rel_err

pytestmark = pytest.mark.gpu

W_TOL, P_TOL_VOX = 1e-4, 2e-3  # as for every batch (BF16 hi/lo products)


@pytest.mark.parametrize("integrator", [L.PSF_RK1, L.PSF_RK4])
@pytest.mark.parametrize("count", [301, 4000])  # 0.3 and 4 particles per voxel
def test_mixed_boxes(small_bases, integrator, count):
    b = small_bases["sphere12x10x9"]
    off = np.array([0.3, -0.2, 0.1], dtype=b.aabb_min.dtype)
    moved = dataclasses.replace(b, aabb_min=b.aabb_min + off, aabb_max=b.aabb_max + off)
    steps = 20
    params = L.make_params(dt=0.02, integrator=integrator, lifetime=6.0, seed=4, precision=L.PSF_PRECISION_BF16X2)
    w0 = initial_coefficients(b.n_modes, 21)

    def particles(basis):
        p = initial_particles(basis, count, 22)
        p[:, 3] = np.where(np.arange(count) % 3, np.inf, 1.0 + np.arange(count) % 11)
        return p

    with Batch([b, moved], 3, count, autotune=False) as bt:
        for i, basis in enumerate((b, moved)):
            bt.set_instance(i, 1, w0, params, particles(basis))
        bt.step(steps)
        got = [(bt.get_state(i, 1), bt.get_particles(i, 1)) for i in range(2)]
    # The centred box gives the bits that it gives in a batch of its own.
    with Batch([b], 3, count, autotune=False) as bt:
        bt.set_instance(0, 1, w0, params, particles(b))
        bt.step(steps)
        assert np.array_equal(got[0][0], bt.get_state(0, 1))
        assert np.array_equal(got[0][1], bt.get_particles(0, 1))
    ref = O.OracleRollout(moved, w0, particles(moved), dt=0.02, integrator=integrator, seed=4, lifetime=6.0).step(steps)
    assert rel_err(got[1][0], ref.w) <= W_TOL
    assert np.array_equal(got[1][1][:, 3], ref.life)
    # With the index and the weight coordinate apart the interpolant jumps at cell boundaries: a
    # particle on one may take the other side in FP32.
    err = np.abs(got[1][1][:, :3] - ref.pos).max(axis=1) / b.h
    assert np.mean(err > P_TOL_VOX) <= 0.01, (np.percentile(err, 99), err.max())
