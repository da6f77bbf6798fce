"""Where a call's arrays live in host memory does not change its results.

The transfer kernels go to arrays the GPU can address themselves (page-locked,
the whole range), small pageable calls pass through page-locked staging, large
ones through device staging.  Each mix must give the pageable call's bits
(zero tolerance: the values are only moved); an array of which only a part is
registered must not be addressed."""
import ctypes as C

import numpy as np
import pytest

import evp1d
from evp1d import synth

pytestmark = pytest.mark.gpu

FIELDS = ("stress", "uvel", "vvel", "strintx", "strinty", "Cb", "str")
_D = C.POINTER(C.c_double)


def bits(fs):
    return {k: np.asarray(getattr(fs, k)).view(np.int64).copy() for k in FIELDS}


def problem(nx, ny):
    pr = synth.to_1d(synth.make_grid(nx, ny, seed=2, ndte=3, curvilinear=True))
    rng = np.random.default_rng(1)
    pr.uvel[pr.na:] = rng.normal(0, 0.05, pr.navel - pr.na)  # halo velocities are read
    pr.vvel[pr.na:] = rng.normal(0, 0.05, pr.navel - pr.na)
    return pr


# pageable: page-locked staging (97 x 61), device staging (400 x 300);
# page-locked: the kernels (97 x 61), the copy engine (640 x 480)
@pytest.mark.parametrize("nx,ny", [(97, 61), (400, 300), (640, 480)])
@pytest.mark.parametrize("explicit", [False, True])
def test_page_locked_pageable_and_mixed(oracle_mod, nx, ny, explicit):
    from test_gpu_parity import assert_same, oracle_run
    pr = problem(nx, ny)
    kw = dict(want_str=True, explicit_init=explicit)
    got = []
    with evp1d.EVP1D.from_problem(pr, ndte=3) as s:
        for kind in ("pageable", "pinned", "mixed", "pinned"):
            fs = evp1d.FieldSet.from_problem(pr, pinned=kind != "pageable", **kw)
            if kind == "mixed":
                fs.keep = {}
                for k in ("strength", "Tbu", "uocn"):  # ordinary memory among page-locked
                    fs.keep[k] = np.array(fs.dyn[k])
                    setattr(fs.c, k, fs.keep[k].ctypes.data_as(_D))
            s.run(3, fs)
            got.append(bits(fs))
    for g in got[1:]:
        for k in FIELDS:
            assert np.array_equal(g[k], got[0][k]), k
    assert_same(fs, oracle_run(oracle_mod, pr, 3), pr)


def test_partly_registered_arrays_are_copied():
    import torch
    rt = torch.cuda.cudart()
    pr = problem(131, 77)
    ref = evp1d.FieldSet.from_problem(pr, want_str=True)
    fs = evp1d.FieldSet.from_problem(pr, want_str=True)
    # an array on a page boundary of which the first page alone is registered,
    # and one whose middle is
    big = np.zeros(1 << 16)
    at = (-big.ctypes.data // 8) % 512
    first = big[at:at + pr.na]
    first[:] = pr.f["strength"]
    fs.c.strength = first.ctypes.data_as(_D)
    mid = (fs.uvel.ctypes.data + 4095) // 4096 * 4096
    assert int(rt.cudaHostRegister(first.ctypes.data, 4096, 0)) == 0
    assert int(rt.cudaHostRegister(mid, 4096, 0)) == 0
    try:
        with evp1d.EVP1D.from_problem(pr, ndte=3) as s:
            s.run(3, ref)
            s.run(3, fs)
    finally:
        rt.cudaHostUnregister(first.ctypes.data)
        rt.cudaHostUnregister(mid)
    a, b = bits(ref), bits(fs)
    for k in FIELDS:
        assert np.array_equal(a[k], b[k]), k


def test_partly_registered_arrays_without_the_staging():
    """The same where the staging buffer is not used (device memory among the
    arrays): cudaMemcpyAsync refuses such ranges."""
    import torch
    rt = torch.cuda.cudart()
    pr = problem(131, 77)
    ref = evp1d.FieldSet.from_problem(pr, want_str=True)
    fs = evp1d.FieldSet.from_problem(pr, want_str=True)
    there = torch.from_numpy(fs.dyn["uocn"]).cuda()
    fs.c.uocn = C.cast(C.c_void_p(there.data_ptr()), _D)
    torch.cuda.synchronize()
    big = np.zeros(1 << 16)
    at = (-big.ctypes.data // 8) % 512
    first = big[at:at + pr.na]
    first[:] = pr.f["strength"]
    fs.c.strength = first.ctypes.data_as(_D)
    mid = (fs.uvel.ctypes.data + 4095) // 4096 * 4096
    assert int(rt.cudaHostRegister(first.ctypes.data, 4096, 0)) == 0
    assert int(rt.cudaHostRegister(mid, 4096, 0)) == 0
    try:
        with evp1d.EVP1D.from_problem(pr, ndte=3) as s:
            s.run(3, ref)
            s.run(3, fs)
    finally:
        rt.cudaHostUnregister(first.ctypes.data)
        rt.cudaHostUnregister(mid)
    a, b = bits(ref), bits(fs)
    for k in FIELDS:
        assert np.array_equal(a[k], b[k]), k


@pytest.mark.parametrize("pinned", [False, True])
def test_batched_positions(pinned):
    """A batched call's velocities and str, halo slots between the members."""
    members = [problem(nx, ny) for nx, ny in ((60, 40), (9, 7), (131, 77))]
    ens = synth.concat(members)
    fs = evp1d.FieldSet.from_problem(ens.combined, want_str=True, pinned=pinned)
    if pinned:  # str addressable as well
        fs.str = evp1d.pinned_copy(fs.str)
        for k in range(8):
            fs.c.str[k] = fs.str[k].ctypes.data_as(_D)
    with evp1d.EVP1D.batched(ens, ndte=3) as s:
        s.run(3, fs)
    u, st = ens.split_slots(fs.uvel), ens.split_slots(fs.str)
    for m, pr in enumerate(members):
        one = evp1d.FieldSet.from_problem(pr, want_str=True)
        with evp1d.EVP1D.from_problem(pr, ndte=3) as s:
            s.run(3, one)
        assert np.array_equal(u[m].view(np.int64), one.uvel.view(np.int64))
        assert np.array_equal(np.ascontiguousarray(st[m]).view(np.int64), one.str.view(np.int64))


@pytest.mark.parametrize("nx,ny", [(97, 61), (330, 250), (640, 480)])
def test_gradients_into_any_memory(nx, ny):
    """Gradients gathered by the kernel (page-locked), through page-locked
    staging and in chunks by several host threads: the same bits."""
    from evp1d import _lib
    pr = problem(nx, ny)
    rng = np.random.default_rng(4)
    lu, lv = rng.normal(size=pr.na), rng.normal(size=pr.na)
    names = ("strength", "Cw", "forcex", "forcey", "uvel", "vvel")
    with evp1d.EVP1D.from_problem(pr, ndte=3) as s:
        s.run_checkpointed(3, evp1d.FieldSet.from_problem(pr), 0)
        want = s.adjoint(lu, lv, stress=True)
        g = _lib.Grads()
        out = {k: evp1d.pinned_empty(pr.na) for k in names}
        st = evp1d.pinned_empty((12, pr.na))
        for k in names:
            setattr(g, k, out[k].ctypes.data_as(_D))
        for k in range(12):
            g.stress[k] = st[k].ctypes.data_as(_D)
        s.adjoint_seed(lu, lv)
        s.adjoint_sweep()
        _lib.check(s._L.evp1d_adjoint_gradients(s.h, C.byref(g)), "gradients")
    for k in names:
        assert np.array_equal(out[k].view(np.int64), want[k].view(np.int64)), k
    assert np.array_equal(np.ascontiguousarray(st).view(np.int64), want["stress"].view(np.int64))


def test_pageable_calls_from_two_threads():
    """Two handles' large pageable calls at once: one has the staging buffer,
    the other goes without; both give the serial call's bits."""
    import threading
    pr = problem(400, 300)
    ref = evp1d.FieldSet.from_problem(pr, want_str=True)
    with evp1d.EVP1D.from_problem(pr, ndte=3) as s:
        s.run(3, ref)
    sets = [evp1d.FieldSet.from_problem(pr, want_str=True) for _ in range(2)]
    solvers = [evp1d.EVP1D.from_problem(pr, ndte=3) for _ in range(2)]
    errors = []

    def call(k):
        try:
            for _ in range(3):
                sets[k].refill(pr)
                solvers[k].run(3, sets[k])
        except Exception as e:  # noqa: BLE001
            errors.append(e)
    threads = [threading.Thread(target=call, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for s in solvers:
        s.finalize()
    assert not errors
    for fs in sets:
        for k in FIELDS:
            assert np.array_equal(bits(fs)[k], bits(ref)[k]), k


def test_device_memory_among_the_arrays():
    """Device memory in the place of a host array is copied, never touched by
    host code: the same bits."""
    import torch
    pr = problem(97, 61)
    ref = evp1d.FieldSet.from_problem(pr, want_str=True)
    fs = evp1d.FieldSet.from_problem(pr, want_str=True)
    t = {k: torch.from_numpy(fs.dyn[k]).cuda() for k in ("strength", "uocn")}
    cb = torch.from_numpy(fs.Cb).cuda()
    for k in t:
        setattr(fs.c, k, C.cast(C.c_void_p(t[k].data_ptr()), _D))
    fs.c.Cb = C.cast(C.c_void_p(cb.data_ptr()), _D)
    torch.cuda.synchronize()
    with evp1d.EVP1D.from_problem(pr, ndte=3) as s:
        s.run(3, ref)
        s.run(3, fs)
    fs.Cb[:] = cb.cpu().numpy()
    a, b = bits(ref), bits(fs)
    for k in FIELDS:
        assert np.array_equal(a[k], b[k]), k
