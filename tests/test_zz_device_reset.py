"""A handle made after the device was reset (the process's own context ended and
begun again) under one that was not finalized: the page-locked memory that
handles share went with the reset.  In a process of its own; page-locked and
pageable calls, small (through the shared staging) and in chunks."""
import os
import subprocess
import sys

import pytest

from conftest import PKG, ROOT

pytestmark = pytest.mark.gpu

SCRIPT = """
import ctypes as C, os, sys
import numpy as np
import evp1d
from evp1d import synth

def call(pr):
    s = evp1d.EVP1D.from_problem(pr, ndte=6)
    out = [evp1d.FieldSet.from_problem(pr, pinned=k) for k in (False, True)]
    for f in out:
        for _ in range(40):  # enough for the page-locked memory to be there
            s.run(6, f)
    return s, [np.array(a) for f in out for a in (f.stress, f.uvel, f.vvel, f.Cb)]

kept = []
for nx, ny in ((64, 48), (300, 200)):
    pr = synth.to_1d(synth.make_grid(nx, ny, seed=7, ndte=6))
    s, before = call(pr)
    kept.append(s)
    cu, dev = C.CDLL("libcuda.so.1"), C.c_int()
    assert cu.cuDeviceGet(C.byref(dev), 0) == 0 and cu.cuDevicePrimaryCtxReset_v2(dev) == 0
    for _ in range(2):
        s, after = call(pr)
        assert all(np.array_equal(a.view(np.int64), b.view(np.int64))
                   for a, b in zip(before, after))
        s.finalize()
print("same bits", flush=True)
os._exit(0)  # the handles of the lost contexts are not finalized
"""


def test_handle_after_a_device_reset():
    env = dict(os.environ, PYTHONPATH=os.pathsep.join([PKG, ROOT]))
    r = subprocess.run([sys.executable, "-c", SCRIPT], capture_output=True, text=True, timeout=300, env=env)
    assert r.returncode == 0 and "same bits" in r.stdout, (r.returncode, r.stdout, r.stderr[-2000:])
