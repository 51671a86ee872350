"""The blocked Gauss-Jordan inverses of the solver (csrc/solve.cu) at the
edges of their panels: matrices of 1 to 33 rows, around several panels of 32,
taller than a panel that fits shared memory (736 rows), one matrix per
cluster size, and pivots far from the diagonal.

Height-1 trees: leaves are a row-permuted multiple of the identity plus noise
(condition number below 4), so the solve's error is a small multiple of
n eps cond growth < 900 * 2.2e-16 * 4 * 8 = 6.4e-12; 1e-11 is used."""
import numpy as np
import pytest
import torch

from hmat_lib_b200.hodlr import DeviceTree, HodlrError, Tree
from hmat_lib_b200.tree import TreeData

pytestmark = pytest.mark.gpu


def shuffled(m, rng):
    a = rng.standard_normal((m, m)) / (2.0 * np.sqrt(m))
    a[rng.permutation(m), np.arange(m)] += 4.0
    return a


def make(sizes, h, rank, seed):
    rng = np.random.default_rng(seed)
    td = TreeData(h, list(sizes))
    td.leaves = [shuffled(m, rng) for m in sizes]
    for d in range(h):
        for j in range(1 << d):
            _, size, top = td.node_range(d, j)
            for c in (1, 2):
                m, n = (top, size - top) if c == 1 else (size - top, top)
                r = min(rank, m, n)
                u = np.linalg.qr(rng.standard_normal((m, r)))[0]
                v = np.linalg.qr(rng.standard_normal((n, r)))[0]
                td.blocks[(d, j, c)] = (0.5 * u, v)
    return td


@pytest.mark.parametrize("sizes,h,rank", [
    ([1, 2], 1, 1), ([31, 32], 1, 5), ([33, 64], 1, 31), ([65, 127], 1, 33), ([129, 200], 1, 64),
    ([735, 737], 1, 40), ([900, 350], 1, 300), ([40] * 8, 3, 20), ([96] * 32, 5, 48),
    ([17] * 128, 7, 9),
])
def test_solve_panel_edges(sizes, h, rank):
    td = make(sizes, h, rank, seed=sum(sizes) + rank)
    n = sum(sizes)
    t = Tree.from_tree_data(td)
    dt = DeviceTree.of_host(t)
    b = np.random.default_rng(2).standard_normal((n, 3))
    bd = torch.from_numpy(np.ascontiguousarray(b.T)).cuda()
    xd = torch.zeros_like(bd)
    torch.cuda.synchronize()
    f = dt.factorize()
    f.solve(bd.data_ptr(), 3, n, xd.data_ptr(), n)
    torch.cuda.synchronize()
    want = np.linalg.solve(td.to_dense(), b)
    got = xd.cpu().numpy().T
    assert np.linalg.norm(got - want) <= 1e-11 * np.linalg.norm(want)
    f.free()
    dt.free()
    t.free()


@pytest.mark.parametrize("m", [1, 33, 100, 740])
def test_singular_in_a_late_panel(m):
    """A matrix whose last pivot vanishes is reported, whatever its panel."""
    td = make([m, m], 1, 1, seed=m)
    td.leaves[1][:, -1] = td.leaves[1][:, 0] if m > 1 else 0.0
    t = Tree.from_tree_data(td)
    dt = DeviceTree.of_host(t)
    with pytest.raises(HodlrError):
        dt.factorize()
    dt.free()
    t.free()
