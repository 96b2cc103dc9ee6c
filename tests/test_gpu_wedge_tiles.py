"""The tensor's GEMM tiles, antisymmetric columns and mode batches at their edges, against FP64 NumPy."""
import ctypes as ct

import numpy as np
import pytest

from parallelspectralfluids3d_b200 import _lib as L
from parallelspectralfluids3d_b200._lib_pre import WedgeDesc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,E,kb", [
    (1, 5, 1), (2, 16, 1),          # no pair, one pair of modes
    (7, 1, 3), (31, 17, 31),        # one edge; one chunk and a row
    (63, 200, 20), (64, 200, 64),   # just under and exactly one row tile; a short last batch
    (65, 333, 64), (129, 150, 50),  # a second row tile with one row; three row tiles, ldn 256
    (16, 0, 16),                    # no edges: zeros
])
def test_tensor_matches_numpy(N, E, kb):
    import torch

    rng = np.random.default_rng(N * 7 + E)
    F, ldn = 40, (N + 127) // 128 * 128
    faces = np.full((E, 8), F, np.int32)  # row F of phi is the zero row
    for e in range(E):
        n = int(rng.integers(2, 9))
        faces[e, rng.permutation(8)[:n]] = rng.permutation(F)[:n]
    S = rng.integers(-2, 3, (E, 8, 8)).astype(np.float64) / 4
    S = S - S.transpose(0, 2, 1)
    phi = np.zeros((F + 1, ldn))
    phi[:F, :N] = rng.standard_normal((F, N))
    psi = np.zeros((max(E, 1), ldn))
    psi[:E, :N] = rng.standard_normal((E, N))
    lam = 0.5 + rng.random(N)

    def dev(a):
        return torch.from_numpy(np.ascontiguousarray(a)).cuda()

    d = [dev(faces if E else np.zeros((1, 8), np.int32)), dev(S if E else np.zeros((1, 8, 8))), dev(psi), dev(phi),
         dev(lam)]
    desc = WedgeDesc(E, N, ldn, d[0].data_ptr(), d[1].data_ptr(), d[2].data_ptr(), d[3].data_ptr(), F,
                     d[4].data_ptr())
    lib = L.load()
    need = ct.c_int64()
    L.check(lib.psf_pre_advection_workspace(ct.byref(desc), kb, ct.byref(need)))
    # Whatever the workspace and the output held must not matter.
    ws = torch.full(((need.value + 7) // 8,), float("nan"), dtype=torch.float64, device="cuda")
    C = torch.full((N, N, N), float("nan"), dtype=torch.float64, device="cuda")
    L.check(lib.psf_pre_advection_tensor(ct.byref(desc), kb, ws.data_ptr(), need.value, C.data_ptr(), None))
    torch.cuda.synchronize()
    pf = phi[faces][:, :, :N]  # [E][8][N]
    W = np.einsum("efg,efk,egj->ekj", S, pf, pf, optimize=True)
    want = np.einsum("ea,ekj->kaj", psi[:E, :N], W, optimize=True) / lam[:, None, None]
    # Forward bound: every element is a sum of at most 64 E products, in any order.
    Wa = np.einsum("efg,efk,egj->ekj", np.abs(S), np.abs(pf), np.abs(pf), optimize=True)
    size = np.einsum("ea,ekj->kaj", np.abs(psi[:E, :N]), Wa, optimize=True) / lam[:, None, None]
    assert np.all(np.abs(C.cpu().numpy() - want) <= 2 * (64 + E + 4) * np.finfo(np.float64).eps * size)
