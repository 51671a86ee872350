"""Kernels that take more than 48 KB of dynamic shared memory are allowed to on
every device, not only on the first one used (the library's own objects on the
stand-in runtime, which has two devices and refuses such launches otherwise)."""
import numpy as np
import pytest

import fake_runtime as F
from hmat_lib_b200 import abi


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    d = tmp_path_factory.mktemp("fake")
    return F.link(d), d


def _product(lib, k, precision=0):
    t = F.device_tree(3, 64, 8)
    x, y = np.zeros(512 * k), np.zeros(512 * k)
    t.matmat(x.ctypes.data, k, 512, y.ctypes.data, 512, precision=precision, stream=64)
    t.free()


def _with_engine(lib, engine):
    lib.hodlr_b200_set_option(b"gemm_f64_engine", engine)
    _product(lib, 100)


def _gradient(lib):
    f = lambda n: np.zeros(n, np.float32)
    p, x, t, g, loss = f(lib.hodlr_b200_rank_model_size()), f(8 * 64), f(64), f(1 << 16), f(1)
    ptr = lambda a: a.ctypes.data_as(abi.FP)
    assert lib.hodlr_b200_rank_model_gradient(ptr(p), ptr(x), ptr(t), 64, ptr(g), ptr(loss)) == 0


CALLS = {
    "product_64_columns": lambda lib: _product(lib, 64),
    "product_100_columns": lambda lib: _product(lib, 100),
    "product_16_deep": lambda lib: _with_engine(lib, 1.0),
    "product_dfma": lambda lib: _with_engine(lib, 0.0),
    "product_mixed": lambda lib: _product(lib, 100, precision=1),
    "rank_model": _gradient,
}


@pytest.mark.parametrize("call", sorted(CALLS))
def test_launches_on_a_second_device(fake, call):
    with F.loaded(*fake) as lib:
        for dev in (0, 1, 0):
            assert lib.fake_set_device(dev) == 0
            before = lib.fake_launches()
            CALLS[call](lib)
            assert lib.fake_launches() > before
        lib.fake_set_device(0)
