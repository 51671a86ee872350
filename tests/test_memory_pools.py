"""Near full device memory the library's two pools make room for each other,
and a large tree is allocated at its exact size when the rounded one does not
fit (the library's own objects on the stand-in runtime, whose pools keep what
is freed)."""
import numpy as np
import pytest

import fake_runtime as F
from hmat_lib_b200 import hodlr
from hmat_lib_b200.hodlr import DeviceTree, matmat_batched

MB = 1 << 20


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    d = tmp_path_factory.mktemp("fake")
    return F.link(d), d


def _fill_scratch_pool(columns=3400):
    """A product on host buffers: 2 x 8 n columns bytes of scratch, kept."""
    host = hodlr.Tree.from_tree_data(F.tree_data(1, 1024, 2))
    x = np.zeros((2048, columns), order="F")
    host.matmat(x)
    host.free()


def test_scratch_gets_what_freed_trees_left(fake):
    with F.loaded(*fake) as lib:
        lib.fake_set_capacity(170 * MB)
        F.device_tree(1, 2048, 1).free()            # 64 MiB and more stay in the default pool
        assert lib.fake_pool_bytes(0, 1) - lib.fake_pool_bytes(0, 0) >= 64 * MB
        _fill_scratch_pool()                        # 2 x 53 MiB


def test_trees_get_what_scratch_left(fake):
    with F.loaded(*fake) as lib:
        _fill_scratch_pool()
        lib.fake_set_capacity(170 * MB)
        assert lib.fake_pool_bytes(1, 1) - lib.fake_pool_bytes(1, 0) >= 100 * MB
        F.device_tree(1, 2048, 1).free()


def _nothing_left(lib):
    """Everything that is not in use lies in the scratch pool."""
    mapped = lib.fake_pool_bytes(1, 1) + lib.fake_pool_bytes(0, 0)
    assert lib.fake_pool_bytes(1, 1) - lib.fake_pool_bytes(1, 0) >= 100 * MB
    lib.fake_set_capacity(mapped)


def _run(t, k, precision=0, op=0):
    x, y = np.zeros(2048 * k), np.zeros(2048 * k)
    t.matmat(x.ctypes.data, k, k if op == 2 else 2048, y.ctypes.data, k if op == 2 else 2048, op=op,
             precision=precision, stream=64)
    return x, y


def _batch(t):
    x, y = np.zeros(2048 * 8), np.zeros(2048 * 8)
    matmat_batched([t], [x.ctypes.data], [8], [2048], [y.ctypes.data], [2048], stream=64)


def _solve(t):
    f = t.factorize(stream=64)
    b, x = np.zeros(2048 * 8), np.zeros(2048 * 8)
    f.solve(b.ctypes.data, 8, 2048, x.ctypes.data, 2048, stream=64)
    f.free()


def _build(t):
    a = np.zeros((2048, 2048))
    DeviceTree.build(a.ctypes.data, 2048, 2048, 4, 1e-8, stream=64).free()


CALLS = {
    "matvec": lambda t: _run(t, 1),
    "matmat": lambda t: _run(t, 64),
    "mixed": lambda t: _run(t, 64, precision=1),
    "mixed_left": lambda t: _run(t, 64, precision=1, op=2),
    "batch": _batch,
    "solve": _solve,
    "hxh": lambda t: t.hxh(t, 1e-8).free(),
    "build": _build,
}


@pytest.mark.parametrize("call", sorted(CALLS))
def test_calls_get_what_scratch_left(fake, call):
    with F.loaded(*fake) as lib:
        t = F.device_tree(5, 64, 8)
        _fill_scratch_pool()
        _nothing_left(lib)
        CALLS[call](t)
        t.free()


def _build_points():
    p = np.zeros(2048)
    return DeviceTree.build_kernel(p.ctypes.data, 2048, 1, 0, 0.1, 1.0, 4, 1e-8, stream=64)


def test_formed_matrix_leaves_the_default_pool_alone_if_it_fits(fake):
    with F.loaded(*fake) as lib:
        F.device_tree(1, 2048, 1).free()
        kept = lib.fake_pool_bytes(0, 1)
        _build_points().free()                      # 32 MiB of 4 GiB
        assert lib.fake_pool_bytes(1, 1) >= 32 * MB
        assert lib.fake_pool_bytes(0, 1) >= kept


def test_formed_matrix_gets_what_freed_trees_left(fake):
    with F.loaded(*fake) as lib:
        lib.hodlr_b200_set_option(b"kernel_form_frac", 0.6)
        F.device_tree(1, 3072, 1).free()
        lib.fake_set_capacity(lib.fake_pool_bytes(0, 1) + 20 * MB)
        _build_points().free()                      # 32 MiB, 20 of them free
        assert lib.fake_pool_bytes(1, 1) >= 32 * MB
        assert lib.fake_pool_bytes(0, 1) < 144 * MB


def test_arena_falls_back_to_its_exact_size(fake):
    with F.loaded(*fake) as lib:
        exact = 8 * (2 * 2048 * 2048 + 2 * 2 * 2048)
        lib.fake_set_capacity(exact + MB)           # rounded: 72 MiB
        t = F.device_tree(1, 2048, 1)
        assert t.info()["arena_bytes"] == exact
        assert lib.fake_pool_bytes(0, 0) < exact + MB
        t.free()


def test_full_is_still_an_error(fake):
    with F.loaded(*fake) as lib:
        lib.fake_set_capacity(32 * MB)
        with pytest.raises(hodlr.HodlrError):
            F.device_tree(1, 2048, 1)
