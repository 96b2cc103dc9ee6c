"""The advection tensor's workspace is no larger than with all columns of every mode (host arithmetic)."""
import ctypes as ct

import pytest

from parallelspectralfluids3d_b200 import _lib as L
from parallelspectralfluids3d_b200._lib_pre import WedgeDesc


def up(a, b):
    return -(-a // b)


def all_columns(edges, ldn, kb):
    """W with ldn columns per mode, and partial sums over about two 128 x 128 tiles per SM."""
    chunks, ldc = up(edges, 16), kb * ldn
    tiles = (ldn // 128) * (ldc // 128)
    splits = max(1, min(up(296, tiles), 64, max(1, chunks)))
    per = max(1, up(chunks, splits))
    return 8 * (chunks * 16 * ldc + max(1, up(chunks, per)) * ldn * ldc)


@pytest.mark.parametrize("modes", [1, 2, 25, 64, 65, 128, 200, 256, 384, 512])
def test_workspace(modes):
    lib = L.load()
    ldn = up(modes, 128) * 128
    for edges in (0, 1, 15, 100, 1000, 5000, 11280, 40000, 400000):
        for kb in {1, 2, 3, 8, 16, 33, 64}:
            if kb > modes:
                continue
            d = WedgeDesc(edges, modes, ldn, 16, 16, 16, 16, 1, 16)  # the pointers are not followed
            need = ct.c_int64()
            L.check(lib.psf_pre_advection_workspace(ct.byref(d), kb, ct.byref(need)))
            # The parts may each be rounded up to 256 bytes.
            assert 0 < need.value <= all_columns(edges, ldn, kb) + 1024, (edges, kb)
