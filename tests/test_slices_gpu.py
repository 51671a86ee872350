"""The int8 product's operand slices at the edges of their items: right-hand
sides that fill no whole 8-row group, 32-line item or 64-column tile, leading
dimensions that rule out 16-byte copies, leaves that are no multiple of the
64-value item.  Against the FP64 product of the same tree: the slices carry 42
bits relative to the largest entry of a row and column, 2^-42 = 2.3e-13 per
term, summed over at most 800 terms of equal magnitude and both phases; 1e-11
bounds it, as for the library's other mixed products."""
import numpy as np
import pytest
import torch

from hmat_lib_b200.hodlr import DeviceTree, Tree
from hmat_lib_b200.tree import TreeData

pytestmark = pytest.mark.gpu


def tree(sizes, h, rank, seed):
    rng = np.random.default_rng(seed)
    td = TreeData(h, list(sizes))
    td.leaves = [rng.standard_normal((m, m)) for m in sizes]
    for d in range(h):
        for j in range(1 << d):
            _, size, top = td.node_range(d, j)
            for c in (1, 2):
                m, n = (top, size - top) if c == 1 else (size - top, top)
                td.blocks[(d, j, c)] = (rng.standard_normal((m, rank)),
                                        rng.standard_normal((n, rank)))
    return td


@pytest.mark.parametrize("sizes,h,rank", [([32, 32], 1, 1), ([96, 160, 128, 64], 2, 33),
                                          ([128] * 4, 2, 2)])
@pytest.mark.parametrize("k,pad", [(1, 0), (7, 1), (8, 0), (17, 3), (33, 0), (64, 1), (65, 0),
                                   (127, 2), (129, 1)])
def test_mixed_product_edges(sizes, h, rank, k, pad):
    n = sum(sizes)
    ld = n + pad
    t = Tree.from_tree_data(tree(sizes, h, rank, seed=n + k))
    dt = DeviceTree.of_host(t)
    x = torch.randn(k, ld, dtype=torch.float64, device="cuda")
    y = [torch.full((k, ld), 7.0, dtype=torch.float64, device="cuda") for _ in range(2)]
    torch.cuda.synchronize()
    for p in (0, 1):
        dt.matmat(x.data_ptr(), k, ld, y[p].data_ptr(), ld, precision=p)
    torch.cuda.synchronize()
    a, b = y[0][:, :n], y[1][:, :n]
    assert float((a - b).norm() / a.norm()) < 1e-11
    assert bool((y[1][:, n:] == 7.0).all())
    dt.free()
    t.free()
