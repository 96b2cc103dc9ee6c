"""Grouped read-back of every size, and states to one place or several, from buffers made with the batch."""
import numpy as np
import pytest

from parallelspectralfluids3d_b200 import _lib as L
from parallelspectralfluids3d_b200.batch import Batch
from parallelspectralfluids3d_b200.fixture import initial_coefficients, initial_particles
from test_gpu_batch_read import read

pytestmark = pytest.mark.gpu


# Slots of two bases with counts below the staging, above it, and one slot that fills it.
@pytest.mark.parametrize("counts", [(300, 0, 257, 1, 4096, 33, 512, 2), (1300000, 700, 1500000, 1400000), (40, 5000000)])
def test_reads_of_every_size(small_bases, counts):
    bases = [small_bases["box576"], small_bases["sphere12x10x9"]]
    params = L.make_params(dt=0.01, precision=L.PSF_PRECISION_BF16X2)
    n = len(counts)
    with Batch(bases, (n + 1) // 2, max(counts), autotune=False, particle_pool=sum(counts) + 256 * n) as bt:
        where = [(k % 2, k // 2) for k in range(n)]
        for k, (i, s) in enumerate(where):
            b = bases[i]
            bt.set_instance(i, s, initial_coefficients(b.n_modes, k), params,
                            initial_particles(b, counts[k], k) if counts[k] else None)
        bt.step(3)
        want = [(bt.get_state(i, s), bt.get_particles(i, s)) for i, s in where]
        flat = np.empty((sum(counts), 4), np.float32)
        ends = np.cumsum(counts)
        p = [flat[e - c:e] for c, e in zip(counts, ends)]
        w = [np.empty(len(x[0])) for x in want]
        sizes = [bt.info()["device_bytes"]]
        asked = 0
        while asked < 132:
            m = 2 + asked % (n - 1)  # reads of every size
            flat[:] = -7.0
            for a in w:
                a[:] = -7.0
            L.check(read(bt, where[:m], w[:m], p[:m]))
            asked += m
            sizes.append(bt.info()["device_bytes"])
            for k in range(n):
                assert np.array_equal(w[k], want[k][0] if k < m else np.full(len(w[k]), -7.0))
                assert np.array_equal(p[k], want[k][1]) if k < m else np.all(p[k] == -7.0)
        assert len(set(sizes)) == 1  # no read allocates
        # States that follow one another in page-locked memory, all or some of them wanted.
        import torch
        row = torch.empty(sum(len(x[0]) for x in want), dtype=torch.float64, pin_memory=True).numpy()
        ends = np.cumsum([len(x[0]) for x in want])
        w = [row[e - len(x[0]):e] for x, e in zip(want, ends)]
        for left_out in (None, 0, n - 1):
            row[:] = -7.0
            L.check(read(bt, where, [None if k == left_out else a for k, a in enumerate(w)], [None] * n))
            for k in range(n):
                assert np.array_equal(w[k], want[k][0]) if k != left_out else np.all(w[k] == -7.0)
        # The same slot more often than there are slots.
        twice = [where[0]] * (2 * bt.slots[0] + 1)
        q = [np.empty((counts[0], 4), np.float32) for _ in twice]
        L.check(read(bt, twice, [None] * len(twice), q))
        assert all(np.array_equal(a, want[0][1]) for a in q)
