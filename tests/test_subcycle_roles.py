"""The subcycle kernel, whose producer, stress and stepu warps go on by
themselves, against the oracle, bit for bit (zero tolerance: the same
operations in the same order).  Sizes: runs of no more than one tile, of two,
three (every table in use once) and five; all 13 stepu inputs read (general)
and ten."""
import os
import re

import numpy as np
import pytest

import evp1d
from evp1d import synth

from conftest import PKG


def test_lane_arrivals_follow_a_warp_sync():
    """Lane 0's arrival on an mbarrier stands for what its whole warp read or
    wrote: the statement before it is a __syncwarp() (a vote orders no memory).
    No execution shows the difference reliably, so the source is read."""
    src = open(os.path.join(PKG, "csrc", "evp_kernels_tma.cu")).read()
    src = re.sub(r"//[^\n]*", "", src)
    arrivals = list(re.finditer(r"if \(lane == 0\)\s*(?:\{\s*const[^;]*;\s*)?mbar_arrive", src))
    assert len(arrivals) >= 5
    for m in arrivals:
        before = src[:m.start()].rstrip()
        assert before.endswith("__syncwarp();"), before[-200:] + m.group()


def test_every_producer_warp_waits_for_its_copies():
    """The waits of the four producer warps can run out one without the other, so
    that a gather warp has copies under way into a slot that the bulk warp
    neither arms nor waits for: each warp waits for its own slots after its
    loop, on every path.  Read in the source: no test may leave copies in
    flight."""
    src = open(os.path.join(PKG, "csrc", "evp_kernels_tma.cu")).read()
    src = re.sub(r"//[^\n]*", "", src)
    tail = re.sub(r"\s+", " ", src[src.index("issued++;"):])
    assert tail.startswith("issued++; } for (int k = issued - kSSlots; k < issued; k++) "
                           "if (k >= 0 && lane == 0) mbar_wait(&S.sfull[k % kSSlots], "
                           "(uint32_t)(k / kSSlots) & 1"), tail[:200]


@pytest.mark.gpu
@pytest.mark.parametrize("general", [False, True])
@pytest.mark.parametrize("runs,nx,ny", [(148, 3, 2), (148, 131, 77), (16, 131, 77), (10, 131, 77),
                                        (6, 131, 77), (148, 531, 377)])
def test_roles_bitwise(oracle_mod, monkeypatch, runs, nx, ny, general):
    from test_gpu_parity import assert_same, gpu_run, oracle_run
    monkeypatch.setenv("EVP1D_RESIDENT", "0")
    monkeypatch.setenv("EVP1D_RUNS", str(runs))
    ndte = 4
    g = synth.make_grid(nx, ny, seed=21, ndte=ndte, curvilinear=True)
    p = evp1d.set_evp_parameters(ndte)
    if general:
        p.revp, p.Ktens, p.capping = 1.0, 0.2, 0.0
        p.cosw, p.sinw = np.cos(0.4), np.sin(0.4)
        rng = np.random.default_rng(6)
        g.f["Tbu"] = np.asfortranarray(rng.uniform(0.0, 5.0, g.f["Tbu"].shape))
    pr = synth.to_1d(g)
    fs = gpu_run(pr, ndte, params=p, explicit_init=general)
    assert_same(fs, oracle_run(oracle_mod, pr, ndte, params=p), pr)
