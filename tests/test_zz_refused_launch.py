"""A launch whose blocks must all be resident, refused by the device (less of it
is free to this context than at evp1d_init; here evp1d_debug_refuse_launch):
nothing has been launched, so the call goes on with a launch per subcycle and
gives the same results, bit for bit."""
import numpy as np
import pytest

import evp1d
from evp1d import _lib, synth

from test_zz_no_alloc import DeviceCase, _bits

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _disarm():
    yield
    evp1d.debug_refuse_launch(0)


@pytest.mark.parametrize("nx,ny", [(64, 48), (300, 200), (400, 300)])
def test_refused_run(oracle_mod, nx, ny):
    from test_gpu_parity import assert_same, oracle_run
    ndte = 5
    pr = synth.to_1d(synth.make_grid(nx, ny, seed=23, ndte=ndte))
    ref = oracle_run(oracle_mod, pr, ndte)
    with evp1d.EVP1D.from_problem(pr, ndte=ndte) as s:
        for refused in (False, True, True):  # before, at and after the refusal
            evp1d.debug_refuse_launch(1 if refused else 0)
            fs = evp1d.FieldSet.from_problem(pr, want_str=True)
            s.launch_count(reset=True)
            s.run(ndte, fs)
            assert s.launch_count() == (ndte if refused else 1)
            assert_same(fs, ref, pr)


@pytest.mark.parametrize("interval", [0, 3])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 6])
def test_refused_gradient(n, interval):
    """The n-th of the launches of a recording and its sweep: forward segments,
    recomputed segments, reversed segments."""
    ndte = 8
    pr = synth.to_1d(synth.make_grid(64, 48, seed=24, ndte=ndte, curvilinear=True))
    rng = np.random.default_rng(9)
    lu, lv = rng.normal(size=pr.na), rng.normal(size=pr.na)
    got = []
    for refuse in (0, n):
        with evp1d.EVP1D.from_problem(pr, ndte=ndte) as s:
            evp1d.debug_refuse_launch(refuse)
            fs = evp1d.FieldSet.from_problem(pr)
            s.run_checkpointed(ndte, fs, interval)
            got.append(dict(s.adjoint(lu, lv, stress=True), u=fs.uvel, v=fs.vvel, s=fs.stress))
    for k in got[0]:
        assert np.array_equal(_bits(got[0][k]), _bits(got[1][k])), k


@pytest.mark.parametrize("nx,ny", [(64, 48), (416, 312)])
def test_refused_noalloc(oracle_mod, nx, ny):
    from test_gpu_parity import oracle_run
    ndte = 4
    pr = synth.to_1d(synth.make_grid(nx, ny, seed=25, ndte=ndte, curvilinear=True))
    p = evp1d.set_evp_parameters(ndte)
    dc = DeviceCase(pr)
    evp1d.debug_refuse_launch(1)
    _lib.check(dc.run(ndte, p), "evp1d_run_device_noalloc")
    got, st = dc.host(), oracle_run(oracle_mod, pr, ndte, params=p)
    for k in ("stress", "strintx", "strinty", "Cb"):
        assert np.array_equal(_bits(got[k]), _bits(getattr(st, k))), k
    assert np.array_equal(_bits(got["uvel"][:pr.na]), _bits(st.uvel[:pr.na]))
