"""Grouped read-back: any set of slots and host buffers gives what the single reads give."""
import ctypes as ct

import numpy as np
import pytest

from parallelspectralfluids3d_b200 import _lib as L
from parallelspectralfluids3d_b200.batch import Batch
from parallelspectralfluids3d_b200.fixture import initial_coefficients, initial_particles

pytestmark = pytest.mark.gpu


def read(bt, where, w, p):
    n = len(where)
    basis = np.array([x[0] for x in where], np.int32)
    slot = np.array([x[1] for x in where], np.int32)
    wp = (ct.c_void_p * n)(*[None if a is None else a.ctypes.data for a in w])
    pp = (ct.c_void_p * n)(*[None if a is None else a.ctypes.data for a in p])
    return bt.lib.psf_batch_read_instances(bt.handle, n, L.ptr(basis, ct.c_int32), L.ptr(slot, ct.c_int32), wp, pp)


@pytest.mark.parametrize("together", [True, False])
@pytest.mark.parametrize("counts", [(300, 0, 257, 1, 4096, 33), (1300000, 700, 1500000, 1400000)])  # below, above the staging
def test_read_instances(small_bases, together, counts):
    bases = [small_bases["box576"], small_bases["sphere12x10x9"]]
    params = L.make_params(dt=0.01, precision=L.PSF_PRECISION_BF16X2)
    with Batch(bases, 4, max(counts), autotune=False, particle_pool=sum(counts) + 256 * len(counts)) as bt:
        where = []
        for k, count in enumerate(counts):
            i, s = k % 2, k // 2 + (k % 2)
            b = bases[i]
            bt.set_instance(i, s, initial_coefficients(b.n_modes, k), params,
                            initial_particles(b, count, k) if count else None, n_modes=b.n_modes)
            where.append((i, s))
        bt.step(3)
        want = [(bt.get_state(i, s), bt.get_particles(i, s)) for i, s in where]
        gap = 0 if together else 3
        flat = np.full((sum(counts) + gap * len(counts), 4), -7.0, np.float32)
        p, at = [], 0
        for c in counts:
            p.append(flat[at:at + c])
            at += c + gap
        w = [np.zeros(bases[i].n_modes) for i, _ in where]
        w[1], p[-1] = None, None  # not wanted
        for _ in range(2):
            flat[:] = -7.0
            L.check(read(bt, where, w, p))
            for k, (sw, sp) in enumerate(want):
                assert w[k] is None or np.array_equal(w[k], sw)
                assert p[k] is None or np.array_equal(p[k], sp)
            written = sum(c for k, c in enumerate(counts) if p[k] is not None)
            assert np.count_nonzero(flat[:, 0] != -7.0) == written  # nothing beside the wanted buffers
        assert read(bt, [where[0], (0, 3)], [None, None], [None, None]) == -5  # an empty slot
