"""The centred-box tracer at the edges of its half-cells, one step against the FP64 oracle, in both engines."""
import numpy as np
import pytest

from oracle import oracle as O
from parallelspectralfluids3d_b200 import _lib as L
from parallelspectralfluids3d_b200.batch import Batch
from parallelspectralfluids3d_b200.fixture import initial_coefficients
from parallelspectralfluids3d_b200.solver import Context

pytestmark = pytest.mark.gpu


def edge_particles(b):
    """Every corner, wall, voxel and half-voxel boundary of the grid, exactly and an ulp to either side."""
    axes = []
    for q in range(3):
        lo, hi = np.float32(b.aabb_min[q]), np.float32(b.aabb_max[q])
        n = b.dims[q]
        k = np.unique(np.concatenate([[0, 1, 2, n, n + 1, 2 * n - 2, 2 * n - 1, 2 * n]]))
        x = (lo + (hi - lo) * (k / (2.0 * n))).astype(np.float32)
        x = np.concatenate([x, np.nextafter(x, lo), np.nextafter(x, hi)])
        axes.append(np.unique(np.clip(x, lo, hi)))
    g = np.stack(np.meshgrid(*axes, indexing="ij"), -1).reshape(-1, 3)
    p = np.full((len(g), 4), np.inf, np.float32)
    p[:, :3] = g
    return p


@pytest.mark.parametrize("name", ["box576", "sphere12x10x9"])
@pytest.mark.parametrize("integrator", [L.PSF_RK1, L.PSF_RK4])
@pytest.mark.parametrize("voxels", [0.02, 0.8])  # per step: stages in one half-cell, and across several
def test_edges_match_oracle(small_bases, name, integrator, voxels):
    b = small_bases[name]
    p = edge_particles(b)
    dt = 0.01
    w0 = initial_coefficients(b.n_modes, 3)
    u = np.abs(b.phi @ w0).max()
    speed = voxels * b.h / (dt * u)
    w0 = w0 * speed
    ref = O.OracleRollout(b, w0, p, dt=dt, integrator=integrator).step(1)
    params = L.make_params(dt=dt, integrator=integrator)
    with Context(b, params) as ctx:
        ctx.set_state(w0)
        ctx.set_particles(p)
        ctx.step(1)
        plain = ctx.get_particles()[:, :3].astype(np.float64)
    with Batch([b], 3, len(p), autotune=False) as bt:
        bt.set_instance(0, 1, w0, L.make_params(dt=dt, integrator=integrator, precision=L.PSF_PRECISION_BF16X2), p)
        bt.step(1)
        batch = bt.get_particles(0, 1)[:, :3].astype(np.float64)
    # FP32: positions and coordinates to a few ulp of the box, velocities to a
    # few ulp of the largest sample; a stage's error moves the next stage's
    # position, whose velocity changes by at most 2 u per voxel on each axis.
    eps, ext = 2.0 ** -24, float((b.aabb_max - b.aabb_min).max())
    move = voxels * b.h
    bound = (4 * eps * ext + 64 * eps * move) * (1 + 6 * voxels) ** 3
    assert np.abs(plain - ref.pos).max() <= bound
    # BF16 hi/lo products drop lo * lo (2^-18 relative per product).
    assert np.abs(batch - ref.pos).max() <= bound + 2.0 ** -17 * move * (1 + 6 * voxels) ** 3 * np.sqrt(b.n_modes)
