"""A build from points forms its kernel matrix when it is small against the
device memory (option kernel_form_frac) and generates the entries it needs
otherwise; both compute every entry with the same function, so the trees have
the same ranks and their products agree to the rounding of split-K sums."""
import numpy as np
import pytest
import torch

from hmat_lib_b200 import abi
from hmat_lib_b200 import workloads as W
from hmat_lib_b200.hodlr import DeviceTree
from oracle import hodlr_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,dim,h,kind,tol", [(1, 1, 1, 0, 1e-8), (257, 1, 2, 0, 1e-10),
                                              (1500, 2, 3, 1, 1e-8), (2049, 3, 4, 2, 1e-6)])
def test_formed_equals_generated(n, dim, h, kind, tol):
    lib = abi.load()
    pts = W.points_1d_sorted(n, 3) if dim == 1 else W.points_morton(n, dim, 3)
    d_pts = torch.from_numpy(np.ascontiguousarray(pts.T)).cuda()
    x = torch.randn(5, n, dtype=torch.float64, device="cuda")
    out = []
    for frac in (0.0, 0.0625):
        lib.hodlr_b200_set_option(b"kernel_form_frac", frac)
        try:
            t = DeviceTree.build_kernel(d_pts.data_ptr(), n, dim, kind, 0.2, 1e-2, h, tol)
        finally:
            lib.hodlr_b200_set_option(b"kernel_form_frac", 0.0625)
        y = torch.zeros_like(x)
        torch.cuda.synchronize()
        t.matmat(x.data_ptr(), 5, n, y.data_ptr(), n)
        torch.cuda.synchronize()
        out.append((t.ranks(), y.cpu().numpy()))
        t.free()
    assert np.array_equal(out[0][0], out[1][0])
    assert O.rel_fro(out[1][1], out[0][1]) < 1e-12
