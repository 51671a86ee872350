"""The single-vector kernels (csrc/matvec.cu) at the edges of their work
split: blocks just below and at the height that takes a whole CTA per item
(512 rows), ranks around the columns of an item (4) and the columns a row
strip keeps in flight (128), leaves that are no multiple of a 32-row strip.
Against the CPU oracle at 1e-12: sums of at most 2000 products, whose rounding
is below 2000 eps = 4.4e-13 of the magnitudes added."""
import numpy as np
import pytest

from hmat_lib_b200.hodlr import Tree
from hmat_lib_b200.tree import TreeData
from oracle import hodlr_oracle as O

pytestmark = pytest.mark.gpu


def tree_with_ranks(sizes, h, ranks, seed):
    rng = np.random.default_rng(seed)
    td = TreeData(h, list(sizes))
    for s in sizes:
        td.leaves.append(rng.standard_normal((s, s)))
    at = 0
    for d in range(h):
        for j in range(1 << d):
            _, size, top = td.node_range(d, j)
            for c in (1, 2):
                m, n = (top, size - top) if c == 1 else (size - top, top)
                r = min(ranks[at % len(ranks)], min(m, n))
                at += 1
                td.blocks[(d, j, c)] = (rng.standard_normal((m, r)), rng.standard_normal((n, r)))
    return td


@pytest.mark.parametrize("sizes,h,ranks", [
    ([511, 512], 1, [1, 4]),
    ([513, 511, 33, 31], 2, [5, 3, 0, 127]),
    ([1000, 1000], 1, [128, 129]),
    ([32, 64, 1, 31, 128, 97, 160, 2], 3, [2, 7, 8, 31]),
    ([300, 200, 300, 200], 2, [257, 130, 0, 4]),
])
def test_matvec_work_split(sizes, h, ranks):
    td = tree_with_ranks(sizes, h, ranks, seed=sum(sizes))
    t = Tree.from_tree_data(td)
    x = np.random.default_rng(1).standard_normal(sum(sizes))
    want = O.multiply_dense(td, x[:, None])[:, 0]
    assert O.rel_fro(t.matvec(x), want) < 1e-12
    t.free()
