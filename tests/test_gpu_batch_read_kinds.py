"""Grouped read-back into one array that is page-locked in parts: a copy must not join the parts."""
import numpy as np
import pytest

from parallelspectralfluids3d_b200 import _lib as L
from parallelspectralfluids3d_b200.batch import Batch
from parallelspectralfluids3d_b200.fixture import initial_coefficients, initial_particles
from test_gpu_batch_read import read

pytestmark = pytest.mark.gpu
COUNT = 512  # two pages of particles per slot


# Registrations (first slot, slots) of an array of six slots' particles.
@pytest.mark.parametrize("locked", [[], [(0, 6)], [(0, 1)], [(5, 1)], [(2, 2)], [(0, 2), (2, 1)], [(1, 1), (2, 1), (4, 1)]])
def test_partly_registered(small_bases, locked):
    import torch

    rt = torch.cuda.cudart()
    b = small_bases["box576"]
    params = L.make_params(dt=0.01, precision=L.PSF_PRECISION_BF16X2)
    raw = np.zeros(6 * COUNT * 4 + 1024, np.float32)
    skip = -raw.ctypes.data % 4096 // 4
    flat = raw[skip:skip + 6 * COUNT * 4].reshape(6 * COUNT, 4)
    p = [flat[k * COUNT:(k + 1) * COUNT] for k in range(6)]
    held = []
    with Batch([b], 6, COUNT, autotune=False) as bt:
        try:
            for first, n in locked:
                at = p[first].ctypes.data
                assert int(rt.cudaHostRegister(at, n * COUNT * 16, 0)) == 0
                held.append(at)
            for s in range(6):
                bt.set_instance(0, s, initial_coefficients(b.n_modes, s), params, initial_particles(b, COUNT, s))
            bt.step(2)
            want = [bt.get_particles(0, s) for s in range(6)]
            for _ in range(3):
                flat[:] = -7.0
                w = [np.zeros(b.n_modes) for _ in range(6)]
                L.check(read(bt, [(0, s) for s in range(6)], w, p))
                for s in range(6):
                    assert np.array_equal(p[s], want[s])
                    assert np.array_equal(w[s], bt.get_state(0, s))
        finally:
            for at in held:
                rt.cudaHostUnregister(at)
