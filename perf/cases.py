"""The work that a user of this framework has it do, as cases to measure.

A case is one call of a public entry point at one size:

* ``run``      -- EVP1D.run: the drop-in for dyn_evp1d_run, once per dynamics time step of a host model.  Fields
                  are host arrays (page-locked, as the integration notes advise, or ordinary), copied in, ndte
                  subcycles, results copied out in place; the next call goes on from there.
* ``ensemble`` -- the same call on a batched handle of several members with uneven domains.
* ``dyn2d``    -- Dyn2D.run: the call on the model's own 2D arrays, conversions included.
* ``adjoint``  -- run_checkpointed, then the gradient of a velocity misfit (one step of a parameter estimation),
                  with checkpoints every `interval` subcycles or (0) the tape sized to device memory.
* ``noalloc``  -- evp1d_run_device_noalloc on arrays that the caller has on the device.

``params``: "evp" is the classic scheme with the reference's parameters (no basal stress); "general" switches every
term on (revised EVP, basal stress, tensile strength, turning angle, uncapped viscosity, explicit starting
velocities).  ``curv``: edge lengths vary from cell to cell instead of a uniform 10 km grid.  About 0.615 of a
grid's cells are list points (20 % land, ice-free water).
"""
import ctypes
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "cice-evp1d_b200"))

import evp1d  # noqa: E402
from evp1d import _lib, dyn, synth  # noqa: E402

ACTIVE = 0.615            # list points per grid cell
GRADS = ("strength", "Cw", "forcex", "forcey", "uvel", "vvel")
NEIGHBOURS = ("ee", "ne", "se", "nw", "sw", "sse")
GEO = ("dxT", "dyT", "HTE", "HTN", "HTEm1", "HTNm1", "uarear")


def _case(name, kind, nx, ny, ndte, params="evp", curv=False, pinned=True, members=1, interval=0):
    c = {"kind": kind, "nx": nx, "ny": ny, "ndte": ndte, "params": params, "curv": curv, "pinned": pinned,
         "members": members, "interval": interval}
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest domains (a regional test set-up, a unit of a column study): latency and launches
        _case("run 64x48 x120", "run", 64, 48, 120),
        # a short call on an odd curvilinear grid, fields in ordinary host memory
        _case("run 131x77 x40 pageable", "run", 131, 77, 40, curv=True, pinned=False),
        # the repository's 400 x 300 configuration, CICE's usual ndte
        _case("run 400x300 x120", "run", 400, 300, 120),
        # every term of the scheme live, ragged size
        _case("run 531x377 x240 general", "run", 531, 377, 240, params="general", curv=True),
        # a regional model at 10 km
        _case("run 800x600 x240", "run", 800, 600, 240, curv=True),
        # the operational-scale configuration with its ndte: the largest
        _case("run 1600x1200 x1000", "run", 1600, 1200, 1000),
        # an ensemble of eight members, 300 rows, 100 to 1300 columns
        _case("ensemble 8 x240", "ensemble", 1300, 300, 240, members=8),
        # the call on 2D arrays, as a host model holds them
        _case("dyn2d 400x300 x120", "dyn2d", 400, 300, 120),
        # the adjoint configuration: checkpoints every 50 subcycles
        _case("adjoint 800x600 x500 every 50", "adjoint", 800, 600, 500, interval=50),
        # a small gradient with everything on the tape
        _case("adjoint 203x151 x120", "adjoint", 203, 151, 120, curv=True),
        # arrays that live on the device with the caller
        _case("noalloc 400x300 x120", "noalloc", 400, 300, 120),
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["run"] * 5 + ["ensemble", "dyn2d", "adjoint", "adjoint", "noalloc"])
    params = "general" if kind not in ("ensemble", "adjoint") and rng.random() < 0.3 else "evp"
    curv, pinned = rng.random() < 0.5, kind != "run" or rng.random() < 0.7
    members, interval = 1, 0
    if kind == "noalloc":      # its scratch holds 262144 points
        nx, ny, most = _log(rng, 40, 640), _log(rng, 30, 480), 3.0e7
    elif kind == "adjoint":
        nx, ny, most = _log(rng, 60, 800), _log(rng, 45, 600), 1.4e8
        interval = rng.choice([0, 0, 20, 50])
    elif kind == "ensemble":
        nx, ny, most = _log(rng, 100, 1300), 300, 4.0e8
        members = rng.randint(2, 8)
    else:
        nx, ny, most = _log(rng, 32, 1600), _log(rng, 24, 1200), 1.0e9
    points = ACTIVE * nx * ny * members
    ndte = _log(rng, 24, max(25, min(500 if kind == "adjoint" else 1000, most / points)))
    return _case(None, kind, nx, ny, ndte, params, curv, pinned, members, interval)


# ---- inputs ------------------------------------------------------------------

def _grid(case, seed, domain=7, nx=None):
    """A state on a domain (land, ice cover, cell sizes) that the case fixes: thickness, velocities, currents and
    wind stress come from the seed."""
    g = synth.make_grid(nx or case["nx"], case["ny"], seed=domain, ndte=case["ndte"], curvilinear=case["curv"])
    rng, f = np.random.default_rng([seed, domain]), g.f
    shp = f["strength"].shape
    thick = rng.uniform(0.5, 1.5, shp)
    new = {k: f[k] * thick for k in ("strength", "umassdti", "fm")}
    for k in ("uvel", "vvel"):
        new[k] = np.where(g.iceU, rng.normal(0.0, 0.05, shp), 0.0)
    for k, sd in (("waterx", 0.2), ("watery", 0.2), ("forcex", 0.1), ("forcey", 0.1)):
        new[k] = rng.normal(0.0, sd, shp)
    new["uocn"], new["vocn"] = new["waterx"], new["watery"]
    if case["params"] == "general":
        new["Tbu"] = rng.uniform(0.0, 5.0, shp) * (rng.random(shp) < 0.5)
        new["fm"] = new["fm"] * np.where(rng.random(shp) < 0.3, -1.0, 1.0)
    f.update({k: np.array(a, order="F") for k, a in new.items()})
    return g


def _members(case, seed):
    """Problems of an ensemble: domains of uneven width, up to the case's nx."""
    rng = np.random.default_rng([case["nx"], case["members"]])
    widths = rng.integers(max(24, case["nx"] // 13), case["nx"] + 1, case["members"])
    return [synth.to_1d(_grid(case, seed, domain=11 + m, nx=int(n))) for m, n in enumerate(widths)]


def _problem(case, seed):
    pr = synth.to_1d(_grid(case, seed))
    if case["params"] == "general":
        rng = np.random.default_rng([seed, 3])
        for k in ("uvel_init", "vvel_init"):
            pr.f[k] = pr.f[k] + rng.normal(0.0, 0.01, pr.na)
    return pr


def _params(case):
    p = evp1d.set_evp_parameters(case["ndte"])
    if case["params"] == "general":
        p.revp, p.Ktens, p.capping = 1.0, 0.2, 0.0
        p.cosw, p.sinw = float(np.cos(0.4)), float(np.sin(0.4))
    return p


def _observations(na, seed):
    rng = np.random.default_rng([seed, 4])
    return rng.normal(0.0, 0.1, na), rng.normal(0.0, 0.1, na)


def _pinned_2d(a):
    """A page-locked Fortran-ordered copy."""
    out = evp1d.pinned_empty(a.shape[::-1], a.dtype).T
    out[...] = a
    return out


def _dp(t):
    return ctypes.cast(ctypes.c_void_p(t.data_ptr()), ctypes.POINTER(ctypes.c_double))


def _ip(t):
    return ctypes.cast(ctypes.c_void_p(t.data_ptr()), ctypes.POINTER(ctypes.c_int32))


def _device_state(case, pr):
    """One problem's arrays on the device and the C structure that names them."""
    def put(a):
        return torch.from_numpy(np.ascontiguousarray(a)).cuda()
    explicit = case["params"] == "general"
    t = {k: put(pr.f[k]) for k in evp1d.FieldSet.DYN}
    t.update(stress=put(pr.stress), uvel=put(pr.uvel), vvel=put(pr.vvel), strintx=put(pr.strintx),
             strinty=put(pr.strinty), Cb=put(pr.Cb), skipT=put(pr.skipT), skipU=put(pr.skipU))
    if explicit:
        t.update(uvel_init=put(pr.f["uvel_init"]), vvel_init=put(pr.f["vvel_init"]))
    f = _lib.Fields()
    f.skipT, f.skipU = _ip(t["skipT"]), _ip(t["skipU"])
    for k in range(12):
        f.stress[k] = _dp(t["stress"][k])
    for k in evp1d.FieldSet.DYN + ("uvel", "vvel", "strintx", "strinty", "Cb") + (
            ("uvel_init", "vvel_init") if explicit else ()):
        setattr(f, k, _dp(t[k]))
    static = [put(pr.idx[k]) for k in NEIGHBOURS] + [put(pr.f[k]) for k in GEO]
    return dict(t=t, f=f, static=static, na=pr.na, navel=pr.navel, lib=_lib.load())


def prepare(case, seed):
    kind = case["kind"]
    s = dict(kind=kind, ndte=case["ndte"], params=_params(case))
    general = case["params"] == "general"
    if kind == "ensemble":
        ens = synth.concat(_members(case, seed))
        s["solver"] = evp1d.EVP1D.batched(ens, params=s["params"])
        s["fields"] = evp1d.FieldSet.from_problem(ens.combined, pinned=case["pinned"])
    elif kind == "dyn2d":
        g = _grid(case, seed)
        s["solver"] = dyn.Dyn2D((g.iceT | g.iceU), g.f["dyT"], g.f["dxT"], g.f["uarear"], g.f["HTE"], g.f["HTN"],
                                s["params"])
        s["fields"] = {k: _pinned_2d(a) for k, a in dyn.fields_from_grid(g).items()}
        s["iceT"], s["iceU"] = (_pinned_2d(m.astype(np.int32)) for m in (g.iceT, g.iceU))
    elif kind == "noalloc":
        s.update(_device_state(case, _problem(case, seed)))
    else:
        pr = _problem(case, seed)
        s["solver"] = evp1d.EVP1D.from_problem(pr, params=s["params"])
        s["fields"] = evp1d.FieldSet.from_problem(pr, pinned=case["pinned"], explicit_init=general)
        s["interval"], s["obs"] = case["interval"], _observations(pr.na, seed)
    return s


def _results(f):
    return dict(stress=f.stress, uvel=f.uvel, vvel=f.vvel, strintx=f.strintx, strinty=f.strinty, Cb=f.Cb)


def run(s):
    kind = s["kind"]
    if kind in ("run", "ensemble"):
        return _results(s["solver"].run(s["ndte"], s["fields"]))
    if kind == "dyn2d":
        f = s["solver"].run(s["ndte"], s["fields"], s["iceT"], s["iceU"])
        return {k: f[k] for k in dyn.STRESS + ("strintxU", "strintyU", "Cb", "uvel", "vvel")}
    if kind == "adjoint":
        f = s["solver"].run_checkpointed(s["ndte"], s["fields"], s["interval"])
        na = f.na
        g = s["solver"].adjoint(2.0 * (f.uvel[:na] - s["obs"][0]), 2.0 * (f.vvel[:na] - s["obs"][1]), want=GRADS,
                                stress=True)
        return dict(forward=_results(f), gradients=g)
    rc = s["lib"].evp1d_run_device_noalloc(
        s["na"], s["navel"], *[ctypes.c_void_p(t.data_ptr()) for t in s["static"]], ctypes.byref(s["params"]),
        s["ndte"], ctypes.byref(s["f"]), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    _lib.check(rc, "evp1d_run_device_noalloc")
    return {k: s["t"][k] for k in ("stress", "uvel", "vvel", "strintx", "strinty", "Cb")}


def work(case):
    """Bytes: the call's fields in and results out once, 47 doubles a point (the adjoint: gradients and
    observations too).  Operations: 374 of stress and 74 of stepu per point and subcycle, +, -, *, /, sqrt each
    counted as one; the adjoint's reverse subcycle about 640."""
    width = 0.54 if case["members"] > 1 else 1.0  # an ensemble's mean width over its largest
    na = ACTIVE * case["nx"] * case["ny"] * case["members"] * width
    if case["kind"] == "dyn2d":
        return {"bytes": 8.0 * 47 * case["nx"] * case["ny"], "flops": 448.0 * na * case["ndte"]}
    if case["kind"] == "adjoint":
        return {"bytes": 8.0 * (47 + 20) * na, "flops": (448.0 + 640.0) * na * case["ndte"]}
    return {"bytes": 8.0 * 47 * na, "flops": 448.0 * na * case["ndte"]}


# ---- the same call in plain 64-bit torch ---------------------------------------

def _root(x):
    """Square root with derivative 0 at 0."""
    pos = x > 0
    return torch.where(pos, torch.sqrt(torch.where(pos, x, torch.ones_like(x))), torch.zeros_like(x))


class _Exact:
    """One problem in torch; nb holds 0-based positions in the velocity arrays (`own`: those of the points)."""

    def __init__(self, pr, nb, own, p):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        put = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)  # noqa: E731
        self.p, self.own = p, put(own)
        self.nb = {k: put(nb[k].astype(np.int64)) for k in NEIGHBOURS}
        self.f = {k: put(np.asarray(v, dtype=np.float64)) for k, v in pr.f.items()}
        self.iceT, self.iceU = put(pr.skipT == 0), put(pr.skipU == 0)
        self.S, self.u, self.v = put(pr.stress), put(pr.uvel), put(pr.vvel)
        self.u0, self.v0 = self.f["uvel_init"], self.f["vvel_init"]
        self.pos = torch.full((self.u.numel(),), -1, dtype=torch.int64, device=dev)
        self.pos[self.own] = torch.arange(self.own.numel(), device=dev)

    def at(self, x, k):
        """A per-point quantity at the neighbours `k`; 0 outside the list."""
        q = self.pos[self.nb[k]]
        return torch.where(q >= 0, x[q.clamp(min=0)], torch.zeros_like(x))

    def subcycle(self, S, u, v, strength, Cw, fx, fy):
        f, p = self.f, self.p
        dx, dy = f["dxT"], f["dyT"]
        cxp, cyp = 1.5 * f["HTN"] - 0.5 * f["HTNm1"], 1.5 * f["HTE"] - 0.5 * f["HTEm1"]
        cxm, cym = -(1.5 * f["HTNm1"] - 0.5 * f["HTN"]), -(1.5 * f["HTEm1"] - 0.5 * f["HTE"])
        dxhy, dyhx = 0.5 * (f["HTE"] - f["HTEm1"]), 0.5 * (f["HTN"] - f["HTNm1"])
        least = p.deltaminEVP * (dx * dy)
        uc, vc = u[self.own], v[self.own]
        ue, ve, un, vn, us, vs = (x[self.nb[k]] for k in ("ee", "ne", "se") for x in (u, v))
        div = (cyp * uc - dy * ue + cxp * vc - dx * vs, cym * ue + dy * uc + cxp * ve - dx * vn,
               cym * un + dy * us + cxm * vn + dx * ve, cyp * us - dy * un + cxm * vs + dx * vc)
        ten = (-cym * uc - dy * ue + cxm * vc + dx * vs, -cyp * ue + dy * uc + cxm * ve + dx * vn,
               -cyp * un + dy * us + cxp * vn - dx * ve, -cym * us - dy * un + cxp * vs - dx * vc)
        shr = (-cym * vc - dy * ve - cxm * uc - dx * us, -cyp * ve + dy * vc - cxm * ue - dx * un,
               -cyp * vn + dy * vs - cxp * un + dx * ue, -cym * vs - dy * vn - cxp * us + dx * uc)
        new = [None] * 12
        for k in range(4):
            delta = _root(div[k] ** 2 + p.e_factor * (ten[k] ** 2 + shr[k] ** 2))
            q = p.capping * (strength / torch.where(delta > least, delta, least)) + (1 - p.capping) * (
                strength / (delta + least))
            z, r = (1 + p.Ktens) * q, (1 - p.Ktens) * q * delta
            e, keep, a, d = p.epp2i * z, 1 - p.arlx1i * p.revp, p.arlx1i, p.denom1
            new[k] = (S[k] * keep + a * (z * div[k] - r)) * d
            new[4 + k] = (S[4 + k] * keep + a * e * ten[k]) * d
            new[8 + k] = (S[8 + k] * keep + a * 0.5 * e * shr[k]) * d
        S1 = torch.where(self.iceT, torch.stack(new), S)
        # str1..str8 from the four corners ne, nw, sw, se of each stress
        sp, sm, s12 = S1[0:4], S1[4:8], S1[8:12]

        def corners(s, c, n, o):  # own corner, the two beside it, the one opposite
            return [c * s[k] + n * (s[(k + 1) % 4] + s[(k + 3) % 4]) + o * s[(k + 2) % 4] for k in range(4)]
        cp, cm = corners(sp, 1 / 9, 1 / 18, 1 / 36), corners(sm, 1 / 9, 1 / 18, 1 / 36)
        c12 = corners(s12, 2 / 9, 1 / 9, 1 / 18)
        side = lambda s: (s[0] + s[1], s[2] + s[3], s[0] + s[3], s[1] + s[2])  # noqa: E731  n, s, e, w
        (pn, ps, pe, pw), (mn, ms, me, mw), (tn, ts, te, tw) = side(sp), side(sm), side(s12)
        mix = lambda a, b: a / 3 + b / 6  # noqa: E731
        ew, we, ns, sn = 0.5 * dx * mix(te, tw), 0.5 * dx * mix(tw, te), 0.5 * dy * mix(tn, ts), 0.5 * dy * mix(ts, tn)
        A, B = 0.25 * dy * mix(pn, ps), 0.25 * dy * mix(mn, ms)
        C, D = 0.25 * dy * mix(ps, pn), 0.25 * dy * mix(ms, mn)
        E, F = 0.25 * dx * mix(pe, pw), 0.25 * dx * mix(me, mw)
        G, H = 0.25 * dx * mix(pw, pe), 0.25 * dx * mix(mw, me)
        st = (-A - B - ew + dxhy * (cm[0] - cp[0]) + dyhx * c12[0], A + B - we + dxhy * (cm[1] - cp[1]) + dyhx * c12[1],
              -C - D + ew + dxhy * (cm[3] - cp[3]) + dyhx * c12[3], C + D + we + dxhy * (cm[2] - cp[2]) + dyhx * c12[2],
              -E + F - ns - dyhx * (cp[0] + cm[0]) + dxhy * c12[0], E - F - sn - dyhx * (cp[3] + cm[3]) + dxhy * c12[3],
              -G + H + ns - dyhx * (cp[1] + cm[1]) + dxhy * c12[1], G - H + sn - dyhx * (cp[2] + cm[2]) + dxhy * c12[2])
        st = [torch.where(self.iceT, x, torch.zeros_like(x)) for x in st]
        sx = f["uarear"] * (st[0] + self.at(st[1], "nw") + self.at(st[2], "sse") + self.at(st[3], "sw"))
        sy = f["uarear"] * (st[4] + self.at(st[5], "sse") + self.at(st[6], "nw") + self.at(st[7], "sw"))
        vrel = f["aiu"] * p.rhow * Cw * _root((f["uocn"] - uc) ** 2 + (f["vocn"] - vc) ** 2)
        Cb = f["Tbu"] / (_root(uc ** 2 + vc ** 2) + p.u0)
        m, fm = f["umassdti"], f["fm"]
        ca = (p.brlx + p.revp) * m + vrel * p.cosw + Cb
        cb = fm + torch.copysign(torch.ones_like(fm), fm) * vrel * p.sinw
        c1 = sx + fx + vrel * f["waterx"] + m * (p.brlx * uc + p.revp * self.u0)
        c2 = sy + fy + vrel * f["watery"] + m * (p.brlx * vc + p.revp * self.v0)
        n = ca ** 2 + cb ** 2
        u1, v1 = torch.where(self.iceU, (ca * c1 + cb * c2) / n, uc), torch.where(self.iceU, (ca * c2 - cb * c1) / n, vc)
        return S1, u.index_copy(0, self.own, u1), v.index_copy(0, self.own, v1), sx, sy, Cb

    def fields(self):
        return [self.f[k] for k in ("strength", "Cw", "forcex", "forcey")]

    def forward(self, ndte, keep=None):
        S, u, v, x = self.S, self.u, self.v, self.fields()
        with torch.no_grad():
            for _ in range(ndte):
                if keep is not None:
                    keep.append((S, u, v))
                S, u, v, sx, sy, Cb = self.subcycle(S, u, v, *x)
        z = torch.zeros_like(sx)
        return dict(stress=S, uvel=u, vvel=v, strintx=torch.where(self.iceU, sx, z),
                    strinty=torch.where(self.iceU, sy, z), Cb=torch.where(self.iceU, Cb, z))

    def gradients(self, ndte, obs):
        states = []
        out = self.forward(ndte, states)
        lam = [torch.zeros_like(self.S), torch.zeros_like(self.u), torch.zeros_like(self.v)]
        for q, k in ((1, "uvel"), (2, "vvel")):
            o = torch.from_numpy(obs[q - 1]).to(self.u)
            lam[q] = lam[q].index_copy(0, self.own, 2.0 * (out[k][self.own] - o))
        total = [torch.zeros_like(x) for x in self.fields()]
        while states:
            x = [t.detach().requires_grad_(True) for t in list(states.pop()) + self.fields()]
            y = self.subcycle(*x)[:3]
            g = torch.autograd.grad(y, x, lam)
            lam, total = list(g[:3]), [a + b for a, b in zip(total, g[3:])]
        g = dict(zip(GRADS[:4], total), uvel=lam[1][self.own], vvel=lam[2][self.own], stress=lam[0])
        return dict(forward=out, gradients=g)


def exact(case, seed):
    kind, ndte = case["kind"], case["ndte"]
    if work(case)["flops"] > 1.2e12:  # keeps it under about 20 seconds
        return None
    p = _params(case)
    if kind == "ensemble":
        ens = synth.concat(_members(case, seed))
        pr, slot = ens.combined, np.concatenate([[0], np.cumsum(ens.navel)])
        own = np.concatenate([slot[m] + np.arange(n) for m, n in enumerate(ens.na)])
        off = np.concatenate([np.full(n, slot[m] - 1) for m, n in enumerate(ens.na)])
        return _Exact(pr, {k: pr.idx[k].astype(np.int64) + off for k in NEIGHBOURS}, own, p).forward(ndte)
    g = _grid(case, seed) if kind == "dyn2d" else None
    pr = synth.to_1d(g) if kind == "dyn2d" else _problem(case, seed)
    e = _Exact(pr, {k: pr.idx[k].astype(np.int64) - 1 for k in NEIGHBOURS}, np.arange(pr.na), p)
    if kind == "adjoint":
        return e.gradients(ndte, _observations(pr.na, seed))
    r = e.forward(ndte)
    if kind != "dyn2d":
        return r
    f, at = dyn.fields_from_grid(g), (pr.indxti - 1, pr.indxtj - 1)
    one = {k: r["stress"][i] for i, k in enumerate(dyn.STRESS)}
    one.update(strintxU=r["strintx"], strintyU=r["strinty"], Cb=r["Cb"], uvel=r["uvel"][:pr.na], vvel=r["vvel"][:pr.na])
    for k, x in one.items():
        f[k][at] = x.cpu().numpy()
    return {k: f[k] for k in one}
