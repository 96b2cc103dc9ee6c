"""Particles put back in order on a grid whose keys span more than the sort's buckets."""
import numpy as np
import pytest

from parallelspectralfluids3d_b200 import _lib as L
from parallelspectralfluids3d_b200.batch import Batch
from test_gpu_particle_order import toy_basis

pytestmark = pytest.mark.gpu

# 3 x 12 x 12 bricks of 256 keys, 110,592 in all against 8,192 buckets.  One window, two and
# several, one more than is dealt out together, and a slot that stops at the first look.
COUNTS = [3000, 7000, 100003, 3968 * 128 + 1, 60000]


@pytest.mark.parametrize("integrator", [L.PSF_RK1, L.PSF_RK4])
def test_reorder_large_grid(integrator):
    b = toy_basis((48, 24, 24))
    params = L.make_params(dt=0.01, integrator=integrator, lifetime=70.0, seed=3, precision=L.PSF_PRECISION_BF16X2)
    rng = np.random.default_rng(8)
    size = np.asarray(b.aabb_max) - b.aabb_min
    start = []
    for n in COUNTS:
        p = np.full((n, 4), np.inf, np.float32)
        p[:, :3] = b.aabb_min + size * rng.random((n, 3), dtype=np.float32)
        p[::5, 3] = 1.0 + np.arange(len(p[::5])) % 120  # lives that end and begin again elsewhere
        start.append(p)
    out = []
    for reorder in (True, False):
        with Batch([b], len(COUNTS), max(COUNTS), autotune=False, particle_pool=sum(c + 256 for c in COUNTS)) as bt:
            for s, p in enumerate(start):
                bt.set_instance(0, s, np.array([1.0, -2.0, 0.5]) * 300.0, params, p,
                                steps=64 if s == len(COUNTS) - 1 else 0)
            assert bt.get_reordered() == 0
            if reorder:
                bt.step(64)
                assert bt.get_reordered() == len(COUNTS) - 1  # not the slot that has stopped
                bt.step(70)
                assert bt.get_reordered() == len(COUNTS) - 1
                bt.step(3)
            else:
                for _ in range(137):
                    bt.profile_step()  # single steps, no reordering
                assert bt.get_reordered() == 0
            out.append([bt.get_particles(0, s) for s in range(len(COUNTS))])
    moved = np.abs(out[0][2][:, :3] - start[2][:, :3]).max(axis=1) / b.h
    assert np.median(moved) > 2.0  # the flow mixes voxels
    for x, y in zip(*out):
        assert np.array_equal(x, y)
