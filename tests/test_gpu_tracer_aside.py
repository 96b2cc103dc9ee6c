"""Particles the batch's tracer puts aside: the same bits as particles that go straight through."""
import numpy as np
import pytest

from parallelspectralfluids3d_b200 import _lib as L
from parallelspectralfluids3d_b200.batch import Batch
from parallelspectralfluids3d_b200.fixture import initial_coefficients, initial_particles

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("speed", [1.0, 30.0, 300.0])  # few lanes put aside, some, nearly all
@pytest.mark.parametrize("count", [1, 31, 32, 33, 129, 20001])  # under and over a warp, a block, many rounds
@pytest.mark.parametrize("integrator", [L.PSF_RK1, L.PSF_RK4])
def test_aside_equals_straight(small_bases, speed, count, integrator):
    b = small_bases["sphere12x10x9"]
    slots, few = 3, 256  # 256 particles on 1,080 voxels: faces stored once, no particle is put aside
    params = L.make_params(dt=0.01, integrator=integrator, lifetime=3.0, seed=5, precision=L.PSF_PRECISION_BF16X2)
    p = initial_particles(b, count, 11)
    p[:, 3] = np.inf
    p[:few, 3] = np.arange(len(p[:few])) % 5  # some lives end; a respawn depends on the particle's index
    parts = [(0, min(few, count))] + ([(count // 2, count // 2 + few), (count - few, count)] if count > 3 * few else [])
    w0 = [initial_coefficients(b.n_modes, s) * speed for s in range(slots)]
    with Batch([b], slots, 40 * b.n_voxels, autotune=False, particle_pool=slots * (count + 512)) as bt:
        for s in range(slots):
            bt.set_instance(0, s, w0[s], params, p, steps=2 if s == 1 else 0)
        bt.step(4)
        dense = [bt.get_particles(0, s) for s in range(slots)]
    for lo, hi in parts:
        with Batch([b], slots, few, autotune=False) as bt:
            for s in range(slots):
                bt.set_instance(0, s, w0[s], params, p[lo:hi], steps=2 if s == 1 else 0)
            bt.step(4)
            for s in range(slots):
                assert np.array_equal(bt.get_particles(0, s), dense[s][lo:hi])
