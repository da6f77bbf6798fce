"""The grid barrier of evp1d_run_device_noalloc counts arrivals over a whole call,
modulo 2^32: its test against the count in unbounded integers, before, across
and after the wrap (14.5 million subcycles on 148 blocks)."""
import ctypes as C
import os
import subprocess

import pytest

from conftest import PKG, ROOT


@pytest.fixture(scope="module")
def complete(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("barrier") / "barrier_shim.so")
    subprocess.run(["g++", "-O2", "-fPIC", "-shared", "-std=c++17", "-I", os.path.join(PKG, "csrc"),
                    "-I", os.path.join(ROOT, "include"), "-I", "/usr/local/cuda/include",
                    os.path.join(ROOT, "tests", "native", "barrier_shim.cpp"), "-o", out], check=True)
    f = C.CDLL(out).barrier_complete
    f.argtypes = [C.c_uint, C.c_uint]
    return f


@pytest.mark.parametrize("blocks", [2, 145, 148])
def test_barrier_across_the_wrap(complete, blocks):
    first = 2 ** 32 // blocks
    for k in (1, 2, first - 1, first, first + 1, first + 2, 2 * first, 2 ** 31):
        need = k * blocks
        for count in (need - blocks + 1, need - 1, need, need + 1, need + blocks - 1):
            assert bool(complete(count % 2 ** 32, need % 2 ** 32)) == (count >= need), (k, count)
