"""The two forms of the batch's face fields give the same bits: the form depends on the slots' capacity only."""
import numpy as np
import pytest

from parallelspectralfluids3d_b200 import _lib as L
from parallelspectralfluids3d_b200.batch import Batch
from parallelspectralfluids3d_b200.fixture import initial_coefficients, initial_particles

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["box576", "sphere12x10x9"])
@pytest.mark.parametrize("slots", [1, 33, 70])  # one chunk of 32 columns, a second, a third
@pytest.mark.parametrize("integrator", [L.PSF_RK1, L.PSF_RK4])
def test_field_forms_agree(small_bases, name, slots, integrator):
    b = small_bases[name]
    few = max(8, int(0.3 * b.n_voxels))
    params = L.make_params(dt=0.01, integrator=integrator, lifetime=3.0, precision=L.PSF_PRECISION_BF16X2)
    out = []
    for capacity in (few, 40 * b.n_voxels):  # below and above the density where the form changes
        with Batch([b], slots, capacity, autotune=False, particle_pool=512 * slots) as bt:
            for s in sorted({0, slots // 2, slots - 1}):
                p = initial_particles(b, few, 7 + s)
                p[:, 3] = np.arange(few) % 5
                bt.set_instance(0, s, initial_coefficients(b.n_modes, s) * 30.0, params, p, steps=4 if s else 0)
            bt.step(6)  # the limited slots stop: their fields keep the last step's values
            out.append([(bt.get_state(0, s), bt.get_particles(0, s), bt.get_velocity(0, s), bt.get_steps(0, s))
                        for s in sorted({0, slots // 2, slots - 1})])
    for x, y in zip(*out):
        assert all(np.array_equal(u, v) for u, v in zip(x, y))
    assert np.abs(out[0][0][2]).max() > 0
