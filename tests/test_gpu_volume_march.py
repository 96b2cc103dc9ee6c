"""The ray march's pool, occupancy words and pixel dealing at their edges, bit for bit against the oracle."""
import numpy as np
import pytest

from oracle import volume_oracle as VO
from parallelspectralfluids3d_b200 import volume

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("res,width,height,count,lo,hi,eye", [
    (2, 1, 1, 3, -0.5, 0.5, (0.2, 0.1, 1.5)),          # smallest volume and image
    (31, 9, 5, 4000, -0.5, 0.5, (0.9, -0.4, 1.2)),     # a row of texels and of cells fits one word
    (32, 8, 4, 4000, -0.5, 0.5, (-1.1, 0.3, 0.6)),     # ... its cells need two
    (33, 65, 3, 60, -0.5, 0.5, (0.3, 1.4, 0.2)),       # nearly empty: long steps over cells
    (24, 17, 33, 200000, -0.5, 0.5, (0.1, 0.2, 0.1)),  # every cell has density, camera inside: full pools
    (24, 33, 17, 3000, -2.0, 3.0, (4.0, 5.0, 3.0)),    # a large box: steps of many cells
    (16, 12, 7, 2000, -1e-17, 1e-17, (1e-17, 2e-17, 4e-17)),  # the voxel volume underflows to zero
])
def test_march_matches_oracle(res, width, height, count, lo, hi, eye):
    rng = np.random.default_rng(res * 1000 + width)
    p = np.ones((count, 4), np.float32)
    p[:, :3] = lo + (hi - lo) * rng.random((count, 3))
    mn, mx = np.full(3, lo, np.float32), np.full(3, hi, np.float32)
    view = volume.make_view(width, height, eye=eye, light=(0.7, 2.0, -1.5))
    vol = volume.Volume(res)
    try:
        for keep in (1, 3):  # the second splat of fewer particles leaves nothing of the first
            vol.splat(p[::keep], mn, mx)
            want = VO.render(VO.density(VO.histogram(p[::keep], mn, mx, res)), view, mn, mx)
            assert np.array_equal(vol.render(view), want, equal_nan=True)
    finally:
        vol.close()
