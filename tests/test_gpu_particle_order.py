"""The particles' storage order at grid shapes that do not fill its bricks: nothing of it shows."""
import numpy as np
import pytest

from parallelspectralfluids3d_b200 import _lib as L
from parallelspectralfluids3d_b200.batch import Batch
from parallelspectralfluids3d_b200.domain import box_domain
from parallelspectralfluids3d_b200.fixture import Basis
from parallelspectralfluids3d_b200.solver import Context

pytestmark = pytest.mark.gpu


def toy_basis(dims, n=3):
    """Random modes on a box: the order of particles does not depend on the flow."""
    dom = box_domain(dims).build()
    rng = np.random.default_rng(sum(dims))
    F = len(dom.interior_faces)
    return Basis(dom.dims, dom.h, dom.aabb_min, dom.aabb_max, dom.interior_faces.astype(np.int32), np.ones(n),
                 np.zeros(n), rng.standard_normal((F, n)) / np.sqrt(F), rng.standard_normal((n, n, n)) * 1e-3,
                 dom.sign_bits, dom.inside.ravel().astype(np.uint8), name="toy")


@pytest.mark.parametrize("dims", [(1, 2, 1), (17, 3, 5), (16, 2, 2), (1023, 1, 2), (2, 1, 700)])
def test_order_does_not_show(dims):
    b = toy_basis(dims)
    rng = np.random.default_rng(5)
    lo, hi = b.aabb_min, b.aabb_max
    p = np.full((2000, 4), 50.0, np.float32)
    p[:, :3] = lo + (hi - lo) * rng.random((2000, 3), dtype=np.float32)
    p[:8, :3] = [[(lo, hi)[k >> a & 1][a] for a in range(3)] for k in range(8)]  # corners
    p[8:12, 0] = [lo[0] - 1, hi[0] + 1, np.nan, np.inf]                          # outside, and not a number
    back = rng.permutation(len(p))
    w0 = np.array([1.0, -2.0, 0.5]) * 0.05
    with Context(b, L.make_params(dt=0.01)) as ctx:
        out = []
        for q in (p, p[back]):
            ctx.set_state(w0)
            ctx.set_particles(q)
            assert np.array_equal(ctx.get_particles(), q, equal_nan=True)
            ctx.step(2)
            out.append(ctx.get_particles())
        assert np.array_equal(out[0][back], out[1], equal_nan=True)
    with Batch([b], 2, len(p), autotune=False) as bt:
        for s, q in enumerate((p, p[back])):
            bt.set_instance(0, s, w0, L.make_params(dt=0.01, precision=L.PSF_PRECISION_BF16X2), q)
            assert np.array_equal(bt.get_particles(0, s), q, equal_nan=True)
        bt.step(2)
        assert np.array_equal(bt.get_particles(0, 0)[back], bt.get_particles(0, 1), equal_nan=True)
