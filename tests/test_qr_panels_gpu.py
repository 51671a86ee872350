"""The panel QR (csrc/tsqr.cu) at the edges of its chunks: through the
recompression of U V^T, whose QRs of U and V run panel by panel.  Rows around
one warp (32), one chunk (256) and several levels of chunks, last panels of
any width, more columns than rows, zero and repeated columns.

Householder QR of an m x s factor is backward stable, so U' V'^T differs from
U V^T by a small multiple of sqrt(m s) eps ||U|| ||V|| (m s <= 9000 * 70 here:
2e-13), and the kept columns of V' are orthonormal to the same order; 1e-12
holds both."""
import ctypes as C

import numpy as np
import pytest
import torch

from hmat_lib_b200 import abi

pytestmark = pytest.mark.gpu


def recompress(lib, u, v, tol):
    m, s = u.shape
    n = v.shape[0]
    cap = max(s, min(m, n))
    du = torch.from_numpy(np.ascontiguousarray(u.T)).cuda()
    dv = torch.from_numpy(np.ascontiguousarray(v.T)).cuda()
    uo = torch.zeros(cap, m, dtype=torch.float64, device="cuda")
    vo = torch.zeros(cap, n, dtype=torch.float64, device="cuda")
    rank = C.c_int(0)
    torch.cuda.synchronize()
    st = lib.hodlr_b200_recompress_dev(m, n, s, C.c_void_p(du.data_ptr()), m,
                                       C.c_void_p(dv.data_ptr()), n, tol, 0,
                                       C.c_void_p(uo.data_ptr()), C.c_void_p(vo.data_ptr()),
                                       C.byref(rank), None)
    assert st == abi.SUCCESS
    r = rank.value
    return uo[:r].cpu().numpy().T, vo[:r].cpu().numpy().T


@pytest.mark.parametrize("m,n,s", [(1, 1, 1), (3, 5, 2), (31, 33, 32), (32, 32, 31), (33, 64, 33),
                                   (255, 257, 32), (256, 256, 64), (257, 300, 40), (512, 2049, 5),
                                   (2050, 511, 70), (9000, 40, 37), (20, 700, 45)])
@pytest.mark.parametrize("deficient", [False, True])
def test_recompress_panel_edges(m, n, s, deficient):
    lib = abi.load()
    rng = np.random.default_rng(m * 1000 + n + s)
    u, v = rng.standard_normal((m, s)), rng.standard_normal((n, s))
    if deficient:
        u[:, s // 2] = 0.0
        u[:, -1] = u[:, 0]
        v[:, 0] = 0.0
    want = u @ v.T
    scale = np.linalg.norm(u) * np.linalg.norm(v)
    up, vp = recompress(lib, u, v, 1e-13 * scale)
    assert np.linalg.norm(up @ vp.T - want) <= 1e-12 * scale
    if np.linalg.norm(want) > 0.0:
        assert np.abs(vp.T @ vp - np.eye(vp.shape[1])).max() <= 1e-12
