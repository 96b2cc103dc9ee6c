"""The density volume's memory, and what a frame leaves for the next one."""
import numpy as np
import pytest

from oracle import volume_oracle as VO
from parallelspectralfluids3d_b200 import volume

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("res", [128, 256, 512])
def test_memory(res):
    """Counts (4 bytes) and FP16 density (2) per texel are enough; a volume takes no more."""
    import torch

    free = lambda: torch.cuda.mem_get_info(0)[0]  # noqa: E731
    one = np.zeros((1, 4), np.float32)
    vol = volume.Volume(32)
    vol.splat(one, (-1, -1, -1), (1, 1, 1))  # loads the kernels
    vol.close()
    before = free()
    vol = volume.Volume(res)
    vol.splat(one, (-1, -1, -1), (1, 1, 1))
    taken = before - free()
    vol.close()
    assert taken <= 6 * res ** 3 + (4 << 20)  # allocations are whole pages of 2 MB


@pytest.mark.parametrize("res", [2, 3, 31, 32, 33, 63, 64, 65, 97])
def test_frames(res):
    """Frames of many, few, no and other particles, edges and corners among them, bit for bit."""
    rng = np.random.default_rng(res)
    mn, mx = np.full(3, -0.5, np.float32), np.full(3, 0.5, np.float32)
    many = rng.random((3 * res ** 3 // 2, 3)) - 0.5
    few = rng.random((max(1, res * res // 40), 3)) - 0.5
    edge = np.where(rng.random((40, 3)) < 0.7, np.where(rng.random((40, 3)) < 0.5, 0.4999, -0.5), rng.random((40, 3)) - 0.5)
    view = volume.make_view(24, 17, eye=(0.9, -0.4, 1.1), light=(0.7, 2.0, -1.5))
    vol = volume.Volume(res)
    assert not vol.density().view(np.uint16).any()
    for p3 in (many, edge, np.zeros((0, 3)), few, many[::7], edge + 2.0, few):
        p = np.ones((len(p3), 4), np.float32)
        p[:, :3] = p3
        vol.splat(p, mn, mx)
        want = VO.density(VO.histogram(p, mn, mx, res))
        assert np.array_equal(vol.density().view(np.uint16), want.view(np.uint16))
        assert np.array_equal(vol.render(view), VO.render(want, view, mn, mx), equal_nan=True)
    vol.close()
