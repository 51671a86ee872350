"""Trees, factors and batch plans can be freed while work that uses them is
queued: the free waits for it (and only then).  Without a GPU on the stand-in
runtime, which counts every release of stream-ordered memory under queued
work; on the GPU by the results of such work."""
import ctypes as C

import numpy as np
import pytest

import fake_runtime as F
from hmat_lib_b200 import hodlr
from hmat_lib_b200 import workloads as W
from hmat_lib_b200.hodlr import DeviceTree, matmat_batched


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    d = tmp_path_factory.mktemp("fake")
    return F.link(d), d


def _product(lib, t, n, op=0, k=3, precision=0, times=1):
    x = np.zeros(n * k)
    y = np.zeros(n * k)
    ld = k if op == 2 else n
    for _ in range(times):
        t.matmat(x.ctypes.data, k, ld, y.ctypes.data, ld, op=op, precision=precision, stream=64)
    return x, y


CALLS = {
    "matvec": lambda lib, t, n: _product(lib, t, n, k=1),
    "matmat": lambda lib, t, n: _product(lib, t, n),
    "transposed": lambda lib, t, n: _product(lib, t, n, op=1),
    "left": lambda lib, t, n: _product(lib, t, n, op=2),
    "graph": lambda lib, t, n: _product(lib, t, n, times=3),
    "mixed": lambda lib, t, n: _product(lib, t, n, precision=1),
    "mixed_left": lambda lib, t, n: _product(lib, t, n, op=2, precision=1),
}


@pytest.mark.parametrize("call", sorted(CALLS))
def test_tree_free_waits_for_products(fake, call):
    with F.loaded(*fake) as lib:
        t = F.device_tree()
        keep = CALLS[call](lib, t, 128)
        waits = lib.fake_device_waits()
        t.free()
        assert lib.fake_device_waits() > waits
        assert lib.fake_frees_under_work() == 0
        del keep


def test_tree_free_waits_for_the_call_without_allocations(fake):
    with F.loaded(*fake) as lib:
        t, x, y = F.device_tree(), np.zeros(128), np.zeros(128)
        assert lib.hodlr_b200_matvec_noalloc_dev(t.h, x.ctypes.data, y.ctypes.data, 64) == 0
        t.free()
        assert lib.fake_frees_under_work() == 0


@pytest.mark.parametrize("precision", [0, 1])
def test_batch_plans_and_trees_wait(fake, precision):
    with F.loaded(*fake) as lib:
        trees = [F.device_tree() for _ in range(3)]
        x, y = np.zeros((3, 256)), np.zeros((3, 256))
        matmat_batched(trees, [v.ctypes.data for v in x], [2] * 3, [128] * 3,
                       [v.ctypes.data for v in y], [128] * 3, precision=precision, stream=64)
        trees[0].free()
        assert lib.fake_frees_under_work() == 0
        matmat_batched(trees[1:], [v.ctypes.data for v in x[1:]], [2] * 2, [128] * 2,
                       [v.ctypes.data for v in y[1:]], [128] * 2, precision=precision, stream=64)
        lib.hodlr_b200_batched_release()
        assert lib.fake_frees_under_work() == 0
        for t in trees[1:]:
            t.free()
        assert lib.fake_frees_under_work() == 0


@pytest.mark.parametrize("tree_first", [False, True])
def test_factor_free_waits_for_solves(fake, tree_first):
    with F.loaded(*fake) as lib:
        t, b, x = F.device_tree(), np.zeros(256), np.zeros(256)
        f = t.factorize(stream=64)
        f.solve(b.ctypes.data, 2, 128, x.ctypes.data, 128, stream=64)
        for h in (t, f) if tree_first else (f, t):
            h.free()
        assert lib.fake_frees_under_work() == 0


def test_free_of_what_no_queued_work_uses_does_not_wait(fake):
    with F.loaded(*fake) as lib:
        x = np.zeros((128, 128))
        t = DeviceTree.build(x.ctypes.data, 128, 128, 2, 1e-8, stream=64)
        loaded = F.device_tree()
        f = loaded.factorize(stream=64)
        c = loaded.hxh(loaded, 1e-8)                    # waits for its work itself
        host = hodlr.Tree.from_tree_data(F.tree_data(2, 32, 4))
        host.matmat(x)                                  # on host buffers: so does this
        waits, launches = lib.fake_device_waits(), lib.fake_launches()
        for h in (f, c, loaded, t, host):
            h.free()
        assert lib.fake_device_waits() == waits
        assert lib.fake_frees_under_work() == 0 and lib.fake_launches() == launches


def test_of_many_frees_in_a_row_the_first_one_waits(fake):
    with F.loaded(*fake) as lib:
        trees = [F.device_tree() for _ in range(4)]
        keep = [_product(lib, t, 128) for t in trees]
        waits = lib.fake_device_waits()
        for t in trees[:3]:
            t.free()
        assert lib.fake_device_waits() == waits + 1
        keep.append(_product(lib, trees[3], 128))       # used again since
        trees[3].free()
        assert lib.fake_device_waits() == waits + 2
        assert lib.fake_frees_under_work() == 0


def test_waits_are_per_device(fake):
    with F.loaded(*fake) as lib:
        trees, keep = [], []
        for dev in (0, 1):
            lib.fake_set_device(dev)
            trees.append(F.device_tree())
            keep.append(_product(lib, trees[-1], 128))
        lib.fake_set_device(0)
        for t in trees:                                 # the second lives on device 1
            t.free()
        assert lib.fake_frees_under_work() == 0


@pytest.mark.gpu
def test_results_of_queued_work_survive_the_free():
    """Products (one vector, 64 columns, a batch) and a solve queued behind
    other work; their trees and factors freed at once; builds and solves on
    another stream meanwhile.  Bounds: two orders of summation differ by at
    most 2 n eps |A| |x| per entry (taken four times, for the factors' own
    sums); the solve's by cond(A) <= 1 + n times that, relative to x."""
    import torch
    n, h, k = 2048, 4, 64
    eps = 2.0 ** -52
    dev = torch.device("cuda")
    pts = W.points_1d_sorted(n, 7)
    p = torch.from_numpy(np.ascontiguousarray(pts.T)).to(dev)
    build = lambda s=0: DeviceTree.build_kernel(p.data_ptr(), n, 1, 0, 0.2, 1.0, h, 1e-10, stream=s)
    gen = torch.Generator(device="cuda").manual_seed(3)
    x = torch.rand(k, n, dtype=torch.float64, device=dev, generator=gen)
    busy = torch.rand(4096, 4096, dtype=torch.float64, device=dev)
    a, b = torch.cuda.Stream(), torch.cuda.Stream()

    def pieces(stream, free_at_once):
        tree, one, pair = build(), build(), [build(), build()]
        factor = tree.factorize(stream=stream.cuda_stream)
        out = [torch.zeros_like(x) for _ in range(5)]
        torch.cuda.synchronize()
        with torch.cuda.stream(stream):
            if free_at_once:
                for _ in range(4):
                    torch.mm(busy, busy)
        s = stream.cuda_stream
        one.matmat(x.data_ptr(), 1, n, out[0].data_ptr(), n, stream=s)
        one.free() if free_at_once else None
        tree.matmat(x.data_ptr(), k, n, out[1].data_ptr(), n, stream=s)
        factor.solve(x.data_ptr(), k, n, out[2].data_ptr(), n, stream=s)
        if free_at_once:
            tree.free()
            factor.free()
            others = [build(b.cuda_stream) for _ in range(3)]
            z = torch.empty_like(x)
            g = others[0].factorize(stream=b.cuda_stream)
            g.solve(x.data_ptr(), k, n, z.data_ptr(), n, stream=b.cuda_stream)
        matmat_batched(pair, [x.data_ptr()] * 2, [k, 1], [n] * 2, [o.data_ptr() for o in out[3:]],
                       [n] * 2, stream=s)
        if free_at_once:
            for t in pair:
                t.free()
            others += [build(b.cuda_stream) for _ in range(3)]
        torch.cuda.synchronize()
        return out

    want = pieces(a, False)
    got = pieces(a, True)
    d = torch.cdist(p.t(), p.t())
    A = torch.exp(-0.5 * (d / 0.2) ** 2) + torch.eye(n, dtype=torch.float64, device=dev)
    prod = 8 * n * eps * (x @ A)
    for i, cols in ((0, 1), (1, k), (3, k), (4, 1)):
        assert bool(((got[i] - want[i]).abs()[:cols] <= prod[:cols]).all()), i
    assert float((got[2] - want[2]).norm() / want[2].norm()) <= 8 * n * eps * (1 + n)


def test_stand_in_runtime_counts_such_frees(fake):
    """The count the tests above rely on is not always zero."""
    with F.loaded(*fake) as lib:
        rt = C.CDLL(lib._name)
        ptr = C.c_void_p()
        assert rt.cudaMallocAsync(C.byref(ptr), C.c_size_t(64), None) == 0
        graph = C.c_void_p(1)
        assert rt.cudaGraphLaunch(graph, C.c_void_p(64)) == 0
        assert rt.cudaFree(ptr) == 0
        assert lib.fake_frees_under_work() == 1
