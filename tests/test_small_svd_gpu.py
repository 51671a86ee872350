"""The shared-memory SVD of small blocks (csrc/jacobi.cu, pivoted QR then
Jacobi) at the edges of its sizes: one row or column, sizes around a chunk of
16 rows, the 128-row variant and the last size that fits a CTA, W in shared
and in global memory, past it the general kernel; both orientations, graded,
rank-deficient, zero and extremely scaled blocks.

The block is the top-right one of a height-1 tree.  Householder QR and Jacobi
are backward stable: singular values within about C eps sigma_0 of LAPACK's
(ranks are compared where no singular value lies that near the threshold),
U V^T within tol sqrt(C) + C eps of the block relative to sigma_0, V
orthonormal to C eps."""
import numpy as np
import pytest

from hmat_lib_b200.hodlr import Tree

pytestmark = pytest.mark.gpu


def svd_of(blk, tol):
    m, n = blk.shape
    a = np.zeros((m + n, m + n), order="F")
    a[:m, m:] = blk
    a[np.arange(m + n), np.arange(m + n)] = 1.0
    t = Tree.from_dense(a, 1, tol, [m, n])
    u, v = t.data().blocks[(0, 0, 1)]
    u, v = u.copy(), v.copy()
    t.free()
    return u, v


def check(blk, tol):
    u, v = svd_of(blk, tol)
    s = np.linalg.svd(blk, compute_uv=False)
    C = min(blk.shape)
    eps = 2.3e-16
    slack = 8 * C * eps * s[0]
    lo = max(1, int(np.sum(s >= tol * s[0] + slack))) if s[0] > tol else 1
    hi = max(1, int(np.sum(s >= tol * s[0] - slack))) if s[0] > tol else 1
    assert lo <= u.shape[1] <= hi
    kept = s[u.shape[1]:].max() if u.shape[1] < C else 0.0
    assert np.linalg.norm(u @ v.T - blk, 2) <= 1.01 * kept + 1e-3 * tol * s[0] + slack
    got = np.linalg.norm(u / (s[0] or 1.0), axis=0) * s[0]
    assert np.abs(got - s[:u.shape[1]]).max() <= 1e-3 * tol * s[0] + slack
    if s[0] > 0:
        assert np.abs(v.T @ v - np.eye(v.shape[1])).max() <= 8 * C * eps + 1e-14


def graded(m, n, decay, seed):
    """Random singular vectors, singular values 10^(-decay i / C)."""
    rng = np.random.default_rng(seed)
    c = min(m, n)
    u = np.linalg.qr(rng.standard_normal((m, c)))[0]
    v = np.linalg.qr(rng.standard_normal((n, c)))[0]
    return (u * 10.0 ** (-decay * (np.arange(c) + 0.37) / c)) @ v.T


SIZES = [(1, 1), (1, 128), (128, 1), (2, 3), (15, 17), (16, 16), (33, 31), (64, 128), (100, 100),
         (127, 128), (128, 128), (129, 128), (128, 129), (160, 100), (100, 176), (177, 100),
         (40, 500)]


@pytest.mark.parametrize("m,n", SIZES)
@pytest.mark.parametrize("decay,tol", [(12.0, 1e-8), (1.0, 1e-8), (14.0, 1e-3)])
def test_graded_blocks(m, n, decay, tol):
    check(graded(m, n, decay, m * 1000 + n), tol)


@pytest.mark.parametrize("m,n", [(16, 16), (100, 128), (128, 100)])
def test_special_blocks(m, n):
    rng = np.random.default_rng(7)
    one = np.zeros((m, n))
    one[m // 2, n // 3] = -0.5
    u, v = svd_of(one, 1e-8)
    sign = 1.0 if m >= n else -1.0   # the longer side's vector carries the entry's sign
    assert u.shape[1] == 1 and u[m // 2, 0] == -0.5 * sign and v[n // 3, 0] == sign
    u, v = svd_of(np.zeros((m, n)), 1e-8)
    assert u.shape[1] == 1 and not u.any() and np.linalg.norm(v) == 1.0
    low = rng.standard_normal((m, 5)) @ rng.standard_normal((5, n))
    low[:, 3] = 0.0
    low[:, 7] = low[:, 6]
    check(low, 1e-8)
    check(np.eye(m, n), 1e-8)
    check(graded(m, n, 12.0, 3) * 1e160, 1e-8)
    u, v = svd_of(graded(m, n, 12.0, 3) * 1e-160, 1e-8)
    assert u.shape[1] == 1    # sigma_0 below the tolerance: one column
    s = np.linalg.svd(graded(m, n, 12.0, 3), compute_uv=False)
    assert abs(np.linalg.norm(u * 1e160) - s[0]) <= 1e-12
    bad = rng.standard_normal((m, n))
    bad[1, 2] = np.nan
    u, v = svd_of(bad, 1e-8)
    assert np.isnan(u @ v.T).any()
