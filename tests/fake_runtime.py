"""The library's own objects linked against tests/fake_cudart.cpp instead of
the CUDA runtime: its host code runs on a machine without a GPU, and the tests
see the order of its launches, waits, allocations and frees."""
from __future__ import annotations

import contextlib
import ctypes as C
import glob
import os
import shutil
import subprocess
from concurrent.futures import ThreadPoolExecutor

import numpy as np

from hmat_lib_b200 import abi, build, hodlr
from hmat_lib_b200.tree import TreeData

HERE = os.path.dirname(os.path.abspath(__file__))
CUDA = os.path.dirname(os.path.dirname(build.NVCC))


def link(directory) -> str:
    """Builds the library against the stand-in runtime; its path.  Objects that
    are missing or old are compiled, but the library itself, which this process
    may have loaded, is left alone."""
    os.makedirs(build.BUILD, exist_ok=True)
    header = build._newest_header()
    with ThreadPoolExecutor(max_workers=8) as ex:
        made = list(ex.map(lambda s: build._compile(s, False, header), build._sources()))
    made.append(build._hash_object(False))
    assert not [e for _, e in made if e], made
    objects = [o for o, _ in made]
    out = os.path.join(str(directory), "libhodlr_fake.so")
    cmd = ["g++", "-shared", "-fPIC", "-O1", "-std=c++17", "-I", os.path.join(CUDA, "include"),
           os.path.join(HERE, "fake_cudart.cpp"), *objects, "-Wl,-Bsymbolic", "-lpthread", "-o", out]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    return out


@contextlib.contextmanager
def loaded(path: str, directory):
    """The library behind abi.load() for the time of a test, with fresh state
    (a copy of its own)."""
    n = len(glob.glob(os.path.join(str(directory), "copy*.so")))
    mine = shutil.copy(path, os.path.join(str(directory), f"copy{n}.so"))
    lib = C.CDLL(mine, mode=C.RTLD_LOCAL)
    abi._declare(lib, abi.HMAT_API)
    abi._declare(lib, abi.B200_API)
    abi._declare(lib, {
        "fake_set_capacity": (None, [C.c_ulonglong]),
        "fake_frees_under_work": (C.c_longlong, []),
        "fake_device_waits": (C.c_longlong, []),
        "fake_launches": (C.c_longlong, []),
        "fake_set_device": (C.c_int, [C.c_int]),
        "fake_pool_bytes": (C.c_ulonglong, [C.c_int, C.c_int]),
    })
    before, abi._LIB = abi._LIB, lib
    try:
        yield lib
    finally:
        lib.hodlr_b200_batched_release()
        abi._LIB = before


def tree_data(height: int, leaf: int, rank: int) -> TreeData:
    """A tree of equal leaves and ranks (numbers mean nothing here)."""
    td = TreeData(height, [leaf] * (1 << height), [np.eye(leaf)] * (1 << height))
    for d in range(height):
        size = leaf << (height - d - 1)
        for j in range(1 << d):
            for c in (1, 2):
                td.blocks[(d, j, c)] = (np.ones((size, rank)), np.ones((size, rank)))
    return td


def device_tree(height: int = 2, leaf: int = 32, rank: int = 4) -> hodlr.DeviceTree:
    """A device tree that no host tree refers to any more."""
    host = hodlr.Tree.from_tree_data(tree_data(height, leaf, rank))
    t = hodlr.DeviceTree.of_host(host)
    host.free()
    return t


def buffer(*shape) -> np.ndarray:
    """"Device" memory of the stand-in runtime."""
    return np.zeros(shape)
