"""evp1d_run_device_noalloc in one launch: one point per thread (its state on
chip) and several per thread, at the sizes around the line between them, the
general parameters, and uvel_init given as the velocities themselves.  Bit for
bit (zero tolerance: the same operations in the same order) the oracle's
results."""
import numpy as np
import pytest

import evp1d
from evp1d import _lib, synth

from test_zz_no_alloc import DeviceCase, _bits, _dp

pytestmark = pytest.mark.gpu


# 148 x 512 = 75776 points: 400 x 300 has fewer, 416 x 312 and 480 x 360 more
@pytest.mark.parametrize("nx,ny,ndte", [(3, 2, 4), (64, 48, 1), (131, 77, 9), (400, 300, 3),
                                        (416, 312, 3), (480, 360, 3)])
@pytest.mark.parametrize("general", [False, True])
def test_one_launch_matches_the_oracle(oracle_mod, nx, ny, ndte, general):
    from test_gpu_parity import oracle_run
    g = synth.make_grid(nx, ny, seed=19, ndte=ndte, curvilinear=True)
    p = evp1d.set_evp_parameters(ndte)
    if general:
        rng = np.random.default_rng(6)
        g.f["Tbu"] = np.asfortranarray(rng.uniform(0.0, 5.0, g.f["Tbu"].shape))
        p.revp, p.Ktens, p.capping = 1.0, 0.2, 0.0
        p.cosw, p.sinw = np.cos(0.4), np.sin(0.4)
    pr = synth.to_1d(g)
    dc = DeviceCase(pr, explicit_init=general)
    _lib.check(dc.run(ndte, p), "evp1d_run_device_noalloc")
    got, st = dc.host(), oracle_run(oracle_mod, pr, ndte, params=p)
    for k in ("stress", "strintx", "strinty", "Cb"):
        assert np.array_equal(_bits(got[k]), _bits(getattr(st, k))), k
    for k in ("uvel", "vvel"):
        assert np.array_equal(_bits(got[k][:pr.na]), _bits(getattr(st, k)[:pr.na])), k
    assert np.array_equal(_bits(got["str"]), _bits(st.str[:, :pr.navel]))


def test_uvel_init_given_as_uvel(oracle_mod):
    """It then follows the velocities from subcycle to subcycle."""
    ndte = 5
    pr = synth.to_1d(synth.make_grid(60, 40, seed=4, ndte=ndte, curvilinear=True))
    p = evp1d.set_evp_parameters(ndte)
    p.revp = 1.0
    dc = DeviceCase(pr)
    dc.c.uvel_init, dc.c.vvel_init = _dp(dc.uvel), _dp(dc.vvel)
    _lib.check(dc.run(ndte, p), "evp1d_run_device_noalloc")
    op = oracle_mod.OracleParams(**{k: getattr(p, k) for k in _lib.PARAM_FIELDS})
    st = oracle_mod.State1D(pr)
    for _ in range(ndte):
        st.f["uvel_init"][:] = st.uvel[:pr.na]
        st.f["vvel_init"][:] = st.vvel[:pr.na]
        oracle_mod.run_1d(pr, 1, p=op, state=st)
    got = dc.host()
    assert np.array_equal(_bits(got["uvel"][:pr.na]), _bits(st.uvel[:pr.na]))
    assert np.array_equal(_bits(got["stress"]), _bits(st.stress))
