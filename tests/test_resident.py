"""The resident solver: a call's subcycles in one launch, one point per thread.

CPU: the resident plan's indices against the neighbour vectors, over grids at
the edges of the kernel's width classes, and mistakes planted in a plan.
GPU: the launch against the oracle, bit for bit (zero tolerance: the same
operations in the same order), at sizes around the class edges, over counts
around the smallest it takes, and against the one-launch-per-subcycle form.
"""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

import evp1d
from evp1d import synth

from conftest import PKG, ROOT

NEIGHBOURS = ("ee", "ne", "se", "nw", "sw", "sse")
BLOCKS = 148


@pytest.fixture(scope="module")
def shim(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("resident") / "resident_plan_shim.so")
    csrc = os.path.join(PKG, "csrc")
    subprocess.run(["g++", "-O2", "-fPIC", "-shared", "-std=c++17", "-I", csrc,
                    os.path.join(csrc, "evp_tiles.cpp"), os.path.join(csrc, "evp_resident.cpp"),
                    os.path.join(ROOT, "tests", "native", "resident_plan_shim.cpp"), "-o", out],
                   check=True)
    L = C.CDLL(out)
    L.resident_plan.restype = C.c_longlong
    return L


def plan(L, pr, blocks=BLOCKS, plant=0):
    nb = np.ascontiguousarray(np.stack([pr.idx[k] - 1 for k in NEIGHBOURS]).astype(np.int32))
    st = (C.c_longlong * 6)()
    bad = L.resident_plan(pr.na, pr.navel, nb.ctypes.data_as(C.POINTER(C.c_int32)), blocks, plant, st)
    return bad, list(st)


@pytest.mark.parametrize("nx,ny", [(3, 2), (64, 48), (131, 77), (203, 151), (45, 550), (300, 200),
                                   (330, 250), (400, 300), (416, 312)])
def test_plan_indices(shim, nx, ny):
    pr = synth.to_1d(synth.make_grid(nx, ny, seed=3, ndte=2))
    bad, (nb, threads, cls, most, halo, exported) = plan(shim, pr)
    assert bad == 0
    assert nb <= BLOCKS and most <= threads <= cls
    assert pr.na + halo <= nb * threads


def test_plan_refuses_what_does_not_fit(shim):
    # more points than one per thread, and a graph without a grid layout
    assert plan(shim, synth.to_1d(synth.make_grid(700, 500, seed=3, ndte=2)))[0] == -1
    rng = np.random.default_rng(2)
    pr = synth.to_1d(synth.make_grid(40, 30, seed=3, ndte=2))
    for k in NEIGHBOURS:
        pr.idx[k] = rng.integers(1, pr.navel + 1, pr.na).astype(np.int32)
    assert plan(shim, pr)[0] == -1


@pytest.mark.parametrize("k", NEIGHBOURS)
def test_plan_refuses_one_way_relations(shim, k):
    """One neighbour entry led to a halo slot while the point it named still
    points back: a mask that leaves only the other points active would make one
    block wait for a block that does not wait for it."""
    pr = synth.to_1d(synth.make_grid(64, 48, seed=3, ndte=2))
    assert plan(shim, pr)[0] == 0
    listed = np.flatnonzero(pr.idx[k] <= pr.na)
    for p in listed[[0, len(listed) // 2, -1]]:
        was = pr.idx[k][p]
        pr.idx[k][p] = pr.navel
        assert plan(shim, pr)[0] == -1, (k, p)
        pr.idx[k][p] = was


@pytest.mark.parametrize("plant", [1, 2, 3, 4, 5])
def test_plan_verifier_catches(shim, plant):
    pr = synth.to_1d(synth.make_grid(131, 77, seed=3, ndte=2))
    assert plan(shim, pr, plant=plant)[0] > 0


def _params(ndte, general):
    p = evp1d.set_evp_parameters(ndte)
    if general:
        p.revp, p.Ktens, p.capping = 1.0, 0.2, 0.0
        p.cosw, p.sinw = np.cos(0.4), np.sin(0.4)
    return p


# four lanes per point (mode 1, the smaller sizes; 180 x 140 is near its end), one
# thread per point (mode 2): widths 128, 256, 384, 512 of the kernel and beyond
@pytest.mark.gpu
@pytest.mark.parametrize("general", [False, True])
@pytest.mark.parametrize("nx,ny,ndte,mode", [
    (3, 2, 5, 1), (64, 48, 24, 1), (131, 77, 6, 1), (180, 140, 5, 1), (3, 2, 5, 2), (64, 48, 24, 2),
    (200, 150, 5, 1), (300, 200, 5, 1), (330, 250, 4, 1), (400, 300, 4, 1)])
def test_launch_bitwise(oracle_mod, monkeypatch, nx, ny, ndte, mode, general):
    from test_gpu_parity import assert_same, gpu_run, oracle_run
    monkeypatch.setenv("EVP1D_RESIDENT", str(mode))
    g = synth.make_grid(nx, ny, seed=13, ndte=ndte, curvilinear=True)
    if general:
        rng = np.random.default_rng(5)
        g.f["Tbu"] = np.asfortranarray(rng.uniform(0.0, 5.0, g.f["Tbu"].shape))
    pr = synth.to_1d(g)
    p = _params(ndte, general)
    fs = gpu_run(pr, ndte, params=p, explicit_init=general)
    assert_same(fs, oracle_run(oracle_mod, pr, ndte, params=p), pr)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 2, 3, 7, 101])
@pytest.mark.parametrize("nx,ny", [(64, 48), (203, 151)])
def test_same_as_one_launch_per_subcycle(monkeypatch, nx, ny, n):
    """The same bits as the subcycle kernel in every output, over three calls
    on one handle (mailbox numbers go on, both buffer sets are used), and the
    call that does not end (evp1d_subcycles_inner) between them."""
    pr = synth.to_1d(synth.make_grid(nx, ny, seed=5, ndte=n, curvilinear=True))
    got = []
    for resident in ("1", "0"):
        monkeypatch.setenv("EVP1D_RESIDENT", resident)
        fs = evp1d.FieldSet.from_problem(pr, want_str=True)
        with evp1d.EVP1D.from_problem(pr, ndte=n) as s:
            s.upload(fs)
            s.launch_count(reset=True)
            s.subcycles(n)
            launches = s.launch_count()
            s.subcycles_inner(n)
            s.subcycles(n)
            s.download(fs)
        assert launches == (1 if resident == "1" else n)
        got.append(fs)
    for k in ("stress", "uvel", "vvel", "strintx", "strinty", "Cb", "str"):
        a, b = (np.asarray(getattr(f, k)).view(np.int64) for f in got)
        assert np.array_equal(a, b), k


@pytest.mark.gpu
@pytest.mark.parametrize("mask", ["one point", "half", "sparse"])
@pytest.mark.parametrize("one_way", [False, True])
def test_masked_bitwise(oracle_mod, one_way, mask):
    """Calls that skip most points: on a grid on chip (blocks without an active
    point beside working ones), on a list with a one-way relation by a launch
    per subcycle."""
    from test_gpu_parity import assert_same, oracle_run
    ndte = 6
    pr = synth.to_1d(synth.make_grid(64, 48, seed=3, ndte=ndte))
    w = int(np.flatnonzero((pr.idx["ee"] <= pr.na) & (pr.skipT == 0))[0])
    if one_way:
        pr.idx["ee"][w] = pr.navel
    rng = np.random.default_rng(4)
    keep = {"one point": np.arange(pr.na) == w, "half": np.arange(pr.na) < pr.na // 2,
            "sparse": rng.random(pr.na) < 0.05}[mask]
    pr.skipT[~keep] = 1
    pr.skipU[~keep] = 1
    fs = evp1d.FieldSet.from_problem(pr, want_str=True)
    with evp1d.EVP1D.from_problem(pr, ndte=ndte) as s:
        s.launch_count(reset=True)
        s.run(ndte, fs)
        assert s.launch_count() == (ndte if one_way else 1)
    assert_same(fs, oracle_run(oracle_mod, pr, ndte), pr)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [2, 3])
def test_after_an_exchange(monkeypatch, n):
    """Received velocities are those of the current state: points that a
    subcycle does not write keep others in the second buffer set.  Several
    subcycles after an unpack give what a launch per subcycle gives."""
    import torch
    pr = synth.to_1d(synth.make_grid(64, 48, seed=6, ndte=n, curvilinear=True))
    still = 1 + np.concatenate([np.flatnonzero(pr.skipU), np.arange(pr.na, pr.navel)])
    buf = torch.from_numpy(np.random.default_rng(1).normal(0.0, 0.1, 2 * len(still))).cuda()
    got = []
    for resident in ("1", "0"):
        monkeypatch.setenv("EVP1D_RESIDENT", resident)
        fs = evp1d.FieldSet.from_problem(pr, want_str=True)
        with evp1d.EVP1D.from_problem(pr, ndte=n) as s:
            s.exchange_setup([1], still.tolist())
            s.upload(fs)
            s.subcycles_inner(2)
            s.exchange_unpack(buf.data_ptr())
            s.subcycles_inner(n)
            s.subcycles(n)
            s.download(fs)
            got.append([np.array(getattr(fs, k)) for k in ("stress", "uvel", "vvel", "strintx", "str")])
            s.launch_count(reset=True)
            s.run(n, fs)  # an upload makes the sets equal again
            assert s.launch_count() == (1 if resident == "1" else n)
    for a, b in zip(*got):
        assert np.array_equal(a.view(np.int64), b.view(np.int64))


# widths 128, 256, 384, 512 of the reverse kernel; segments of 1, 2 and more subcycles
@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny,ndte,interval", [(3, 2, 3, 0), (64, 48, 11, 0), (64, 48, 11, 5),
                                                 (64, 48, 7, 1), (203, 151, 6, 4), (330, 250, 4, 0),
                                                 (370, 280, 4, 3)])
def test_reverse_launch_bitwise(monkeypatch, nx, ny, ndte, interval):
    """The reverse sweep in one launch against its two kernels per subcycle:
    the same gradients bit for bit (both add products by the same explicit
    fused multiply-adds), with stress seeds, twice on one recording."""
    g = synth.make_grid(nx, ny, seed=17, ndte=ndte, curvilinear=True)
    rng = np.random.default_rng(8)
    g.f["Tbu"] = np.asfortranarray(rng.uniform(0.0, 5.0, g.f["Tbu"].shape) *
                                   (rng.random(g.f["Tbu"].shape) < 0.3))
    pr = synth.to_1d(g)
    lu, lv = rng.normal(size=pr.na), rng.normal(size=pr.na)
    ls = rng.normal(size=(12, pr.na)) * 1e-6
    got = []
    for resident in ("1", "0"):
        monkeypatch.setenv("EVP1D_RESIDENT", resident)
        with evp1d.EVP1D.from_problem(pr, ndte=ndte) as s:
            s.run_checkpointed(ndte, evp1d.FieldSet.from_problem(pr), interval)
            first = s.adjoint(lu, lv, ls, stress=True)
            again = s.adjoint(lu, lv, ls, stress=True)
            launches = s.adjoint_info()["sweep_launches"]
        for k in first:
            assert np.array_equal(first[k].view(np.int64), again[k].view(np.int64)), k
        got.append(first)
    assert launches > 2 * ndte  # the second handle ran the two kernels
    for k in got[0]:
        assert np.array_equal(got[0][k].view(np.int64), got[1][k].view(np.int64)), k


# four-lane plans whose width is no whole number of warps, on which the reverse
# kernel, a thread per position, polls by warp votes
@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny,width", [(131, 77, 56), (150, 110, 88)])
def test_reverse_launch_bitwise_ragged_width(shim, monkeypatch, nx, ny, width):
    assert plan(shim, synth.to_1d(synth.make_grid(nx, ny, seed=17, ndte=5)))[1][1] == width
    test_reverse_launch_bitwise(monkeypatch, nx, ny, 5, 3)


# blocks wider than a CTA: the positions beyond its 512 threads take four lanes
# each, in one pass (400 x 300) or two (440 x 330, 460 x 345: the kernel's end);
# more than 512 owned points a block (410 x 310 on) take two passes of stepu
WIDE = [(400, 300), (410, 310), (440, 330), (460, 345)]


@pytest.mark.parametrize("nx,ny", WIDE)
def test_wide_plan_indices(shim, nx, ny):
    pr = synth.to_1d(synth.make_grid(nx, ny, seed=3, ndte=2))
    bad, (nb, threads, cls, most, halo, exported) = plan(shim, pr)
    assert bad == 0
    assert 512 < most <= threads <= cls


@pytest.mark.gpu
@pytest.mark.parametrize("general", [False, True])
@pytest.mark.parametrize("nx,ny", WIDE)
def test_wide_launch_bitwise(oracle_mod, nx, ny, general):
    """Against the oracle over calls that keep the resident launch's state
    (stresses of the extra positions included), bit for bit."""
    from test_gpu_parity import assert_same, gpu_run, oracle_run
    ndte = 3
    pr = synth.to_1d(synth.make_grid(nx, ny, seed=3, ndte=ndte, curvilinear=True))
    p = _params(ndte, general)
    fs = gpu_run(pr, ndte, params=p, explicit_init=general)
    assert_same(fs, oracle_run(oracle_mod, pr, ndte, params=p), pr)
    got = []
    for resident in (True, False):
        f = evp1d.FieldSet.from_problem(pr, want_str=True)
        with evp1d.EVP1D.from_problem(pr, ndte=7, params=p) as s:
            s.upload(f)
            s.launch_count(reset=True)
            for n in ((7, 6) if resident else (1,) * 13):
                s.subcycles_inner(n)
            assert s.launch_count() == (2 if resident else 13)
            s.subcycles(2)
            s.download(f)
        got.append(f)
    for k in ("stress", "uvel", "vvel", "strintx", "strinty", "Cb", "str"):
        a, b = (np.asarray(getattr(f, k)).view(np.int64) for f in got)
        assert np.array_equal(a, b), k
