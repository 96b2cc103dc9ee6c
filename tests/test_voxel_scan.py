"""The blocked scan of a mesh's vertices against NumPy, at counts around its block (no device)."""
import numpy as np
import pytest

from parallelspectralfluids3d_b200 import _lib as L
from parallelspectralfluids3d_b200 import voxel


@pytest.mark.parametrize("count", [1, 2, 15, 16, 17, 31, 32, 33, 100, 4097])
def test_grid_of_any_vertex_count(count):
    rng = np.random.default_rng(count)
    v = (rng.standard_normal((count, 3)) * [1.0, 2.0, 0.5] + [0.5, -1.0, 3.0]).astype(np.float32)
    res = np.float32(0.02)  # at 0.01 the larger meshes span more than the 1023 voxels a grid may have
    dims, lo, hi = voxel.grid(v, res)
    want_lo, want_hi = np.minimum(v.min(0), 0), np.maximum(v.max(0), 0)  # the box starts at the origin
    assert np.array_equal(lo, want_lo) and np.array_equal(hi, want_hi)
    assert dims == tuple(int(np.ceil(e / res)) for e in want_hi - want_lo)
    for at in (0, count // 2, count - 1):
        for bad in (np.nan, np.inf, -np.inf):
            w = v.copy()
            w[at, at % 3] = bad
            with pytest.raises(L.PSFError) as e:
                voxel.grid(w, res)
            assert e.value.code == -1
