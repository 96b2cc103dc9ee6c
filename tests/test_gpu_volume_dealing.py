"""The ray march in nearly empty, half filled, filled and opaque volumes, bit for bit against the oracle."""
import numpy as np
import pytest

from oracle import volume_oracle as VO
from parallelspectralfluids3d_b200 import volume

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("res,width,height,count,size,eye", [
    (64, 163, 91, 0, 1.0, (1.2, 0.9, 1.0)),        # no density
    (64, 163, 91, 2, 1.0, (1.2, 0.9, 1.0)),        # hardly a cell: warps hold 32 rays
    (64, 41, 37, 300, 1.0, (0.1, 0.05, 0.2)),      # just above that share
    (48, 45, 31, 12000, 1.0, (0.8, -0.6, 0.9)),    # most cells: walks without look-ups, and back
    (33, 31, 45, 2500, 1.0, (0.8, -0.6, 0.9)),     # fewer than half, R above 32
    (32, 31, 45, 60, 1.0, (0.8, -0.6, 0.9)),       # few cells of eight steps
    (16, 161, 131, 150000, 0.1, (0.01, 0.02, 0.0)),  # filled and opaque, camera inside: larger hands
    (16, 161, 131, 150000, 0.1, (0.1, -0.05, 0.12)), # ... and outside
    (16, 19, 13, 30000, 1.0, (0.1, 0.2, 0.1)),        # filled, long shadow rays
])
def test_dealing(res, width, height, count, size, eye):
    rng = np.random.default_rng(res + count)
    p = np.ones((count, 4), np.float32)
    p[:, :3] = size * (rng.random((count, 3)) - 0.5)
    mn, mx = np.full(3, -0.5 * size, np.float32), np.full(3, 0.5 * size, np.float32)
    view = volume.make_view(width, height, eye=eye, light=(0.7, 2.0, -1.5))
    vol = volume.Volume(res)
    try:
        vol.splat(p, mn, mx)
        want = VO.render(VO.density(VO.histogram(p, mn, mx, res)), view, mn, mx)
        assert np.array_equal(vol.render(view), want, equal_nan=True)
        assert np.array_equal(vol.render(view), want, equal_nan=True)
    finally:
        vol.close()
