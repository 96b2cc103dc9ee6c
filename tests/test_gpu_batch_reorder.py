"""Particles put back in order during a rollout: the same bits as steps that never reorder them."""
import numpy as np
import pytest

from parallelspectralfluids3d_b200 import _lib as L
from parallelspectralfluids3d_b200.batch import Batch
from parallelspectralfluids3d_b200.fixture import initial_coefficients, initial_particles

pytestmark = pytest.mark.gpu

# Windows hold up to 3,968 particles and up to 128 windows are dealt out together.
MANY = [0, 1, 31, 3968, 3969, 7937, 100003, 3968 * 128, 3968 * 128 + 1, 600000]
FEW = [0, 1, 31, 33, 300]  # stored with every face once


@pytest.mark.parametrize("counts", [MANY, FEW], ids=["many", "few"])
@pytest.mark.parametrize("integrator", [L.PSF_RK1, L.PSF_RK4])
def test_reordered_rollout_keeps_its_bits(small_bases, counts, integrator):
    bases = [small_bases["box576"], small_bases["sphere12x10x9"]]
    params = L.make_params(dt=0.01, integrator=integrator, lifetime=40.0, seed=3, precision=L.PSF_PRECISION_BF16X2)
    steps = 150
    out = []
    for reorder in (True, False):
        with Batch(bases, len(counts), max(counts), autotune=False,
                   particle_pool=2 * sum(c + 256 for c in counts)) as bt:
            for i, b in enumerate(bases):
                for s, n in enumerate(counts):
                    p = initial_particles(b, n, 7 + s) if n else np.zeros((0, 4), np.float32)
                    p[:, 3] = np.inf
                    p[::7, 3] = 1.0 + np.arange(len(p[::7])) % 90  # lives that end and begin again
                    # One slot stops between two reorderings, one exactly at the first.
                    limit = {len(counts) - 1: 100, len(counts) - 2: 64}.get(s, 0) if i else 0
                    bt.set_instance(i, s, initial_coefficients(b.n_modes, s) * 100.0, params, p, steps=limit)
            if reorder:
                bt.step(steps)
            else:
                for _ in range(steps):
                    bt.profile_step()  # single steps, no reordering
            out.append([bt.get_particles(i, s) for i in range(2) for s in range(len(counts))])
    for x, y in zip(*out):
        assert np.array_equal(x, y)
