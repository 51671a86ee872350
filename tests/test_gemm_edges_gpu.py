"""The FP64 GEMM's tile shapes, edges and K splits, through products of one
tree: right-hand sides around the 8-column MMA tile, the 64-column shape and
the 128-column tiles; ranks that leave every kind of K tail (odd ones rule out
16-byte copies of the projections); odd leading dimensions; every forced tile
shape; enough tiles of long K that the last wave is split.  Against the CPU
oracle at 1e-12: sums of at most 3000 terms, 3000 eps = 6.7e-13 relative to the
magnitudes added."""
import ctypes as C

import numpy as np
import pytest

from hmat_lib_b200 import abi
from hmat_lib_b200.hodlr import Tree
from hmat_lib_b200.tree import TreeData
from oracle import hodlr_oracle as O

pytestmark = pytest.mark.gpu


def tree(sizes, h, ranks, seed):
    rng = np.random.default_rng(seed)
    td = TreeData(h, list(sizes))
    td.leaves = [rng.standard_normal((m, m)) for m in sizes]
    at = 0
    for d in range(h):
        for j in range(1 << d):
            _, size, top = td.node_range(d, j)
            for c in (1, 2):
                m, n = (top, size - top) if c == 1 else (size - top, top)
                r = min(ranks[at % len(ranks)], m, n)
                at += 1
                td.blocks[(d, j, c)] = (rng.standard_normal((m, r)), rng.standard_normal((n, r)))
    return td


def check(td, k, pad):
    lib = abi.load()
    n = td.n
    t = Tree.from_tree_data(td)
    x = np.asfortranarray(np.random.default_rng(k).standard_normal((n + pad, k)))
    ierr = C.c_int(0)
    for fn, want in ((lib.multiply_hodlr_dense, O.multiply_dense(td, x[:n])),
                     (lib.multiply_hodlr_transpose_dense, O.multiply_transpose_dense(td, x[:n]))):
        y = np.full((n + pad, k), 5.0, order="F")
        fn(t.tp, x.ctypes.data_as(abi.DP), k, n + pad, y.ctypes.data_as(abi.DP), n + pad,
           C.byref(ierr))
        assert ierr.value == abi.SUCCESS
        assert O.rel_fro(y[:n], want) < 1e-12
        assert (y[n:] == 5.0).all()
    xl = np.asfortranarray(x[:n].T)
    assert O.rel_fro(t.matmat(xl, "L"), O.multiply_dense_hodlr(td, xl)) < 1e-12
    t.free()


@pytest.mark.parametrize("k,pad", [(2, 0), (7, 1), (8, 0), (9, 2), (33, 1), (63, 0), (64, 0),
                                   (65, 1), (127, 0), (129, 2)])
def test_columns_and_tails(k, pad):
    check(tree([70, 65, 128, 33], 2, [1, 2, 3, 31, 32, 33], seed=k), k, pad)


@pytest.mark.parametrize("shape", [0, 1, 2, 3, 4])
@pytest.mark.parametrize("k", [20, 100])
def test_forced_shapes(shape, k):
    lib = abi.load()
    td = tree([130, 63, 1, 96], 2, [5, 40, 63, 64], seed=shape)
    for name in (b"product_shape1", b"product_shape2"):
        lib.hodlr_b200_set_option(name, float(shape))
    try:
        check(td, k, 0)
    finally:
        for name in (b"product_shape1", b"product_shape2"):
            lib.hodlr_b200_set_option(name, -1.0)


@pytest.mark.parametrize("sizes,ranks", [([600] * 4, [257, 300]), ([513, 700, 640, 515], [128, 511])])
def test_split_last_wave(sizes, ranks):
    """K of 1100 to 1700 per output tile, far fewer tiles than slots."""
    check(tree(sizes, 2, ranks, seed=9), 70, 0)
