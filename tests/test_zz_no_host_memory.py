"""A call whose own lists cannot grow (std::bad_alloc) returns EVP1D_ERR_NOMEM: no
exception leaves a C entry point, which would end the process.  In a process of
its own, with an operator new that fails at the n-th call; every n of a call, on
arrays that are staged whole, go in chunks and are page-locked, and gradients.
After each failure the handle gives the same bits."""
import os
import subprocess
import sys

import pytest

from conftest import PKG, ROOT

pytestmark = pytest.mark.gpu

SCRIPT = """
import ctypes as C, sys
import numpy as np
import evp1d
from evp1d import synth

shim = C.CDLL(sys.argv[1])
shim.arm_new.argtypes, shim.new_left.restype = [C.c_long], C.c_long
failed = 0


def every(call, good):
    # call() with each of its allocations failing in turn
    global failed
    for n in range(1, 500):
        shim.arm_new(n)
        try:
            call()
        except evp1d.EVP1DError as e:
            assert e.code == -4, e
            failed += 1
        left = shim.new_left()
        shim.arm_new(0)
        assert good(), n
        if left > 0:
            return
    raise AssertionError("no end")


for nx, ny, pinned in ((64, 48, False), (300, 200, False), (64, 48, True)):
    pr = synth.to_1d(synth.make_grid(nx, ny, seed=7, ndte=4))
    with evp1d.EVP1D.from_problem(pr, ndte=4) as s:
        f = evp1d.FieldSet.from_problem(pr, pinned=pinned)
        for _ in range(40):  # enough for the shared page-locked memory
            f.refill(pr)
            s.run(4, f)
        ref = np.array(f.stress)

        def good():
            f.refill(pr)
            s.run(4, f)
            return np.array_equal(ref.view(np.int64), np.array(f.stress).view(np.int64))
        every(lambda: s.run(4, f), good)
        s.run_checkpointed(4, f, 0)
        s.adjoint_seed(np.ones(pr.na), np.ones(pr.na))
        s.adjoint_sweep()
        g = s.adjoint_gradients(stress=True)

        def same():
            h = s.adjoint_gradients(stress=True)
            return all(np.array_equal(g[k].view(np.int64), h[k].view(np.int64)) for k in g)
        every(lambda: s.adjoint_gradients(stress=True), same)
assert failed > 20, failed
print("all reported:", failed, flush=True)
"""


def test_no_exception_leaves_a_call(tmp_path):
    shim = str(tmp_path / "new_shim.so")
    subprocess.run(["g++", "-O2", "-fPIC", "-shared", "-std=c++17",
                    os.path.join(ROOT, "tests", "native", "new_shim.cpp"), "-o", shim], check=True)
    env = dict(os.environ, PYTHONPATH=os.pathsep.join([PKG, ROOT]), LD_PRELOAD=shim)
    r = subprocess.run([sys.executable, "-c", SCRIPT, shim], capture_output=True, text=True,
                       timeout=300, env=env)
    assert r.returncode == 0 and "all reported" in r.stdout, (r.returncode, r.stdout, r.stderr[-2000:])
