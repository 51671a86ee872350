"""The build's sketch products (blocks of 1024 columns and more by the Hadamard
kernel, narrower ones by the GEMM) at the edges of the tiles and of that rule:
a remainder of one row or column, odd leading dimensions and a base off 16
bytes (8-byte copies), columns split among several items, blocks of a few
non-zero columns, constant blocks and blocks of full rank.  The decaying blocks
have known singular values with the tolerance half way (in logarithm) between
two of them, so the ranks are known and the error is the discarded tail."""
import numpy as np
import pytest
import torch

from hmat_lib_b200.hodlr import DeviceTree

pytestmark = pytest.mark.gpu


def _build(a, lda, shift, tol):
    n = a.shape[0]
    buf = torch.zeros(lda * n + shift, dtype=torch.float64, device="cuda")
    view = buf[shift:].view(n, lda)
    view[:, :n] = torch.from_numpy(np.ascontiguousarray(a.T))
    torch.cuda.synchronize()
    t = DeviceTree.build(buf.data_ptr() + 8 * shift, n, lda, 1, tol, ms=[n // 2, n - n // 2])
    e = torch.eye(n, dtype=torch.float64, device="cuda")
    y = torch.zeros_like(e)
    torch.cuda.synchronize()
    t.matmat(e.data_ptr(), n, n, y.data_ptr(), n)
    torch.cuda.synchronize()
    ranks = np.array(t.ranks())
    t.free()
    return ranks, y.cpu().numpy().T


# height 1: two leaves, blocks of (n // 2) x (n - n // 2) and back
@pytest.mark.parametrize("n,pad,shift,ratio,keep", [
    (258, 0, 0, 0.5, 20),       # 129 x 129: rounds of 64, 64 and 1 columns
    (2046, 0, 0, 0.7, 40),      # the widest blocks of the GEMM
    (2048, 0, 0, 0.7, 40),      # whole tiles
    (2048, 2, 1, 0.7, 40),      # base off 16 bytes
    (2049, 0, 0, 0.5, 20),      # 1024 x 1025 and back, odd leading dimension
    (2178, 1, 0, 0.9, 130),     # several rounds, remainders of one
    (8320, 0, 0, 0.8, 60),      # columns of a row tile split among items
])
def test_decaying_blocks(n, pad, shift, ratio, keep):
    rng = np.random.default_rng(n)
    a = np.zeros((n, n))
    h = n // 2
    sig = ratio ** np.arange(min(h, 4 * keep))
    for rows, cols in ((slice(0, h), slice(h, n)), (slice(h, n), slice(0, h))):
        m, k = rows.stop - rows.start, cols.stop - cols.start
        u = np.linalg.qr(rng.standard_normal((m, sig.size)))[0]
        v = np.linalg.qr(rng.standard_normal((k, sig.size)))[0]
        a[rows, cols] = (u * sig) @ v.T
    # the tolerance between sigma_keep and sigma_{keep + 1}; the sketch stops at
    # a hundredth of it, which moves no singular value across
    tol = sig[keep] ** 0.5 * sig[keep - 1] ** 0.5
    ranks, got = _build(a, n + pad, shift, tol)
    assert list(ranks) == [keep, keep]
    tail = np.sqrt(2 * (sig[keep:] ** 2).sum())
    assert np.linalg.norm(got - a) <= 1.05 * tail + 1e-13 * np.linalg.norm(a)


@pytest.mark.parametrize("n", [300, 2049, 2051])
def test_sparse_and_constant_blocks(n):
    rng = np.random.default_rng(n)
    a = np.zeros((n, n))
    h = n // 2
    # eight non-zero columns, neighbours and 64 apart among them
    cols = h + np.array([0, 1, 2, 63, 64, 65, 127, 128])
    a[:h, cols] = rng.standard_normal((h, cols.size))
    a[h + 1:, :h] = 3.0
    ranks, got = _build(a, n, 0, 1e-9)
    assert list(ranks) == [8, 1]
    assert np.linalg.norm(got - a) <= 1e-12 * np.linalg.norm(a)


@pytest.mark.parametrize("n", [258, 512, 2050])
def test_full_rank_blocks(n):
    """Nothing to compress: every column of the sketch has to be independent."""
    a = np.random.default_rng(n).standard_normal((n, n))
    ranks, got = _build(a, n, 0, 1e-9)
    assert list(ranks) == [n // 2, n // 2]
    assert np.linalg.norm(got - a) <= 1e-11 * np.linalg.norm(a)


@pytest.mark.parametrize("n,h,band", [(1024, 1, 64), (1024, 1, 129), (4096, 2, 64), (4096, 2, 129)])
def test_steep_end_of_the_singular_values(n, h, band):
    """Random banded matrices: a block is a triangular corner, whose singular
    values fall off a cliff inside a panel (to 1e-12 and below within a few
    columns).  Columns of the basis at that level are not orthogonal to the
    rest and must not stay in it.  What the truncation drops is at most
    sqrt(band) 1e-8 of a block's norm, far less of the matrix's."""
    import torch
    r = np.random.default_rng(band)
    i = np.arange(n)
    a = np.where(np.abs(i[:, None] - i[None, :]) <= band, r.standard_normal((n, n)), 0.0)
    d = torch.from_numpy(np.ascontiguousarray(a.T)).cuda()      # column-major
    torch.cuda.synchronize()
    t = DeviceTree.build(d.data_ptr(), n, n, h, 1e-8)
    e = torch.eye(n, dtype=torch.float64, device="cuda")
    y = torch.zeros_like(e)
    torch.cuda.synchronize()
    t.matmat(e.data_ptr(), n, n, y.data_ptr(), n)
    torch.cuda.synchronize()
    assert float((y - d).norm() / d.norm()) <= 1e-8
    t.free()
