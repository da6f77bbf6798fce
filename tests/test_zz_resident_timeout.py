"""The timeout path of the waits between a launch's own blocks: the mailboxes of
a resident launch and the grid barrier of evp1d_run_device_noalloc.  Each runs
out on purpose, with a limit of 50 ms, on something nobody sends or completes;
nothing faults.  The status is reported and cleared, and the next call solves
a problem bit for bit like the oracle."""
import time

import numpy as np
import pytest

import evp1d
from evp1d import _lib, synth

from test_zz_no_alloc import DeviceCase, _bits

pytestmark = pytest.mark.gpu

NS = 50_000_000


@pytest.mark.parametrize("nx,ny", [(60, 40), (300, 200)])
def test_mailbox_waits_run_out(oracle_mod, nx, ny):
    from test_gpu_parity import assert_same, oracle_run
    ndte = 7
    pr = synth.to_1d(synth.make_grid(nx, ny, seed=21, ndte=ndte))
    with evp1d.EVP1D.from_problem(pr, ndte=ndte) as s:
        s.run(ndte, evp1d.FieldSet.from_problem(pr))
        s.synchronize()
        t0 = time.perf_counter()
        s.debug_mail_wait_timeout(NS)
        with pytest.raises(evp1d.EVP1DError) as e:
            s.synchronize()
        assert 0.08 < time.perf_counter() - t0 < 5.0  # the two forms in turn
        assert e.value.code == -5 and "mailbox-wait probe" in str(e.value)
        s.synchronize()
        with pytest.raises(evp1d.EVP1DError) as e:
            s.debug_mail_wait_timeout(10)
        assert e.value.code == -1
        fs = evp1d.FieldSet.from_problem(pr, want_str=True)
        s.run(ndte, fs)
    assert_same(fs, oracle_run(oracle_mod, pr, ndte), pr)


def test_a_handle_without_mailboxes_says_so():
    pr = synth.to_1d(synth.make_grid(700, 500, seed=3, ndte=2))
    with evp1d.EVP1D.from_problem(pr, ndte=2) as s:
        with pytest.raises(evp1d.EVP1DError) as e:
            s.debug_mail_wait_timeout(NS)
    assert e.value.code == -7


def test_grid_barrier_runs_out(oracle_mod):
    from test_gpu_parity import oracle_run
    import torch
    ndte = 5
    pr = synth.to_1d(synth.make_grid(60, 40, seed=22, ndte=ndte))
    st = torch.cuda.current_stream().cuda_stream
    t0 = time.perf_counter()
    rc = _lib.load().evp1d_debug_grid_wait_timeout(NS, st)
    assert 0.04 < time.perf_counter() - t0 < 5.0
    assert rc == -5 and b"barrier over the grid" in _lib.load().evp1d_last_error()
    assert _lib.load().evp1d_debug_grid_wait_timeout(10, st) == -1
    dc = DeviceCase(pr)
    _lib.check(dc.run(ndte, evp1d.set_evp_parameters(ndte)), "evp1d_run_device_noalloc")
    got, ref = dc.host(), oracle_run(oracle_mod, pr, ndte)
    assert np.array_equal(_bits(got["stress"]), _bits(ref.stress))
    assert np.array_equal(_bits(got["uvel"][:pr.na]), _bits(ref.uvel[:pr.na]))
