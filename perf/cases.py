"""Timed workloads of the DG hydro step, over the range its users run it in.

Each case is one stretch of a host program's time loop through the public
entry points (``HydroStep``, ``Ensemble``, ``GaugeMisfitProblem``): a number of
time steps and the result read back, on a deck of the synthetic generators in
``dgswem_b200.decks``.  ``prepare`` holds what the program has before the
call -- the deck, the device handle, the state of the flow (drawn from the
seed: long waves and currents over the deck's bathymetry, the shore of a
beach left as the deck has it) and pinned buffers for the result.  ``run``
steps on from wherever the state is, as a time loop does.

``exact`` is the same scheme in plain torch FP64 (``Flow`` below: modal DG of
degree 1 or 2, local Lax-Friedrichs fluxes, slope limiter, wetting and drying,
SSP Runge-Kutta), written from the equations.
"""
import ctypes
import hashlib
import json
import math
import os
import shutil
import tempfile
from pathlib import Path

import numpy as np
import torch

from dgswem_b200 import Deck, Ensemble, HydroStep, decks
from dgswem_b200.adjoint import GaugeMisfitProblem, element_manning, locate_gauges
from dgswem_b200.ensemble import make_members

WIND = (0.1e-3 * math.cos(math.radians(30.0)), 0.1e-3 * math.sin(math.radians(30.0)))  # 0.1 Pa at 30 degrees


def listed():
    return [
        # A harbour-scale tidal run stepped by a host program one time step per
        # call, nodal fields written every 32 steps: launch latency is all.
        dict(name="annulus_1k_calls", kind="annulus", n1=16, n2=32, variant="strict", order=1, steps=32, graph=0,
             out="nodal", limiter=False, wind=False),
        # The same size of problem replayed as whole-step graphs (a long tidal
        # spin-up): quadratic friction, slope limiter.
        dict(name="annulus_3k_graph", kind="annulus", n1=31, n2=51, variant="strict", order=1, steps=64, graph=64,
             out="state", limiter=True, wind=False),
        # An estuary on a small mesh with wetting and drying, odd sizes.
        dict(name="beach_17k_graph", kind="beach", n1=207, n2=41, variant="strict", order=1, steps=64, graph=32,
             out="state"),
        # A regional wet/dry run, the drop-in build called step by step with
        # nodal output.
        dict(name="beach_120k_run", kind="beach", n1=548, n2=110, variant="strict", order=1, steps=32, graph=0,
             out="nodal"),
        # The headline workload: the wet/dry sloping beach with limiter and
        # Manning friction, bit-exact build, state read back.
        dict(name="beach_1m_graph", kind="beach", n1=1581, n2=316, variant="strict", order=1, steps=32, graph=8,
             out="state"),
        # The same physics in the FMA build.
        dict(name="beach_400k_fast", kind="beach", n1=1003, n2=199, variant="fast", order=1, steps=8, graph=8,
             out="state"),
        # An ocean basin under wind at p=1 (no limiter, no wet/dry).
        dict(name="annulus_800k_wind", kind="annulus", n1=500, n2=800, variant="strict", order=1, steps=24, graph=8,
             out="state", limiter=False, wind=True),
        # The same basin at p=2 with SSP-RK(3,3), FP64 and the mixed form.
        dict(name="annulus_250k_p2", kind="annulus", n1=250, n2=500, variant="strict", order=2, steps=16, graph=8,
             out="state", limiter=False, wind=True),
        dict(name="annulus_130k_p2_mixed", kind="annulus", n1=181, n2=361, variant="mixed", order=2, steps=4,
             graph=4, out="state", limiter=False, wind=True),
        # A parameter study: uneven wet/dry members in one handle, mixed
        # precision (the ensemble's default), wind per member.
        dict(name="ensemble_24_mixed", kind="ensemble", n1=24, n2=120000, variant="mixed", order=1, steps=4, graph=4,
             out="state"),
        # One iteration of a Manning / bathymetry inversion: forward run and
        # gradient of a gauge misfit.
        dict(name="gradient_60k", kind="gradient", n1=387, n2=78, variant="strict", order=1, steps=36, graph=0,
             out="gradient"),
    ]


def draw(rng):
    def spread(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["annulus", "annulus", "beach", "beach", "beach", "annulus_p2", "ensemble", "gradient"])
    if kind == "beach":
        ne = spread(4000, 900000)
        n2 = max(3, int(math.sqrt(ne / 10.0) * rng.uniform(0.7, 1.4)))
        variant = rng.choice(["strict", "strict", "fast", "mixed"])
        steps = rng.choice([16, 24, 32]) if variant == "strict" else 4
        return dict(kind="beach", n1=max(5, ne // (2 * n2)), n2=n2, variant=variant, order=1, steps=steps,
                    graph=rng.choice([0, 4, 8]), out=rng.choice(["state", "nodal"]))
    if kind == "annulus":
        ne = spread(600, 900000)
        n1 = max(3, int(math.sqrt(ne / 4.0) * rng.uniform(0.7, 1.4)))
        variant = rng.choice(["strict", "strict", "fast", "mixed"])
        steps = rng.choice([16, 24, 32]) if variant == "strict" else 4
        return dict(kind="annulus", n1=n1, n2=max(3, ne // (2 * n1)), variant=variant, order=1, steps=steps,
                    graph=rng.choice([0, 4, 8]), out=rng.choice(["state", "nodal"]),
                    limiter=rng.random() < 0.3 and variant == "strict", wind=rng.random() < 0.5)
    if kind == "annulus_p2":
        ne = spread(2000, 250000)
        n1 = max(3, int(math.sqrt(ne / 4.0) * rng.uniform(0.7, 1.4)))
        variant = rng.choice(["strict", "fast", "mixed"])
        return dict(kind="annulus", n1=n1, n2=max(3, ne // (2 * n1)), variant=variant, order=2, steps=4,
                    graph=rng.choice([0, 4]), out="state", limiter=False, wind=rng.random() < 0.5)
    if kind == "ensemble":
        return dict(kind="ensemble", n1=rng.randint(3, 20), n2=spread(8000, 100000), variant="mixed", order=1,
                    steps=4, graph=rng.choice([0, 4]), out="state")
    n2 = rng.randint(12, 70)
    return dict(kind="gradient", n1=5 * n2 - rng.randint(0, 9), n2=n2, variant="strict", order=1,
                steps=rng.randint(16, 36), graph=0, out="gradient")


# ---- decks: written once per geometry, read once per process ------------------
def _dt(case):
    """A stable time step: the beach's and the members' own 0.5 s; on the
    annulus a fraction of the shortest cell side over the wave speed."""
    if case["kind"] != "annulus":
        return 0.5
    cell = min(91440.0 / case["n1"], 95756.0 / case["n2"])
    return min(10.0, round((0.1 if case["order"] == 1 else 0.04) * cell / 14.0, 4))


def _write(case, path):
    kind, n1, n2 = case["kind"], case["n1"], case["n2"]
    if kind == "annulus":
        p2 = dict(rk_stage=3, rk_order=3, extra=dict(pl=2, ph=2, px=2)) if case["order"] == 2 else {}
        limiter = dict(slopeflag=5, nolibf=1, cf=0.0025) if case["limiter"] else {}
        decks.quarter_annulus(path, nr=n1, nth=n2, dt=_dt(case), nsteps=100000, nws=1 if case["wind"] else 0, **p2,
                              **limiter)
    elif kind == "beach":
        decks.sloping_beach(path, nx=n1, ny=n2, nsteps=100000, dramp=0.01)
    elif kind == "gradient":  # config of the inversion: the beach on a shorter basin, so that the tide is felt
        decks.sloping_beach(path, nx=n1, ny=n2, lx=20e3, ly=4e3, nsteps=1000, dramp=0.001)
    else:
        specs = decks.ensemble_specs(n1, seed=17, ne_min=max(2000, n2 // 16), ne_max=n2)
        (path / "specs.json").write_text(json.dumps(specs))
        for i, s in enumerate(specs):
            decks.ensemble_member(path / f"member_{i:04d}", s["kind"], s["ne"], s["amp"], s["n_manning"], s["seed"])


_decks = {}


def _geometry(case):
    """(deck, extra) of the case's mesh; for an ensemble (members, met).  The
    files stay in the temporary directory under the geometry's hash."""
    key = {k: case.get(k) for k in ("kind", "n1", "n2", "order", "limiter", "wind")}
    name = hashlib.sha256(json.dumps(key, sort_keys=True).encode()).hexdigest()[:20]
    if name not in _decks:
        path = Path(tempfile.gettempdir()) / f"dgswem_decks_{os.getuid()}" / name
        if not path.exists():
            path.parent.mkdir(parents=True, exist_ok=True)
            part = Path(tempfile.mkdtemp(dir=path.parent))
            _write(case, part)
            try:
                part.rename(path)
            except OSError:  # another process was first
                shutil.rmtree(part, ignore_errors=True)
        if case["kind"] == "ensemble":
            _decks[name] = make_members(path, json.loads((path / "specs.json").read_text()))
        else:
            _decks[name] = (Deck(path), None)
    return _decks[name]


# ---- the state of the flow ---------------------------------------------------
def _waves(rng, x, y, amp):
    """A sum of six long waves of random direction and phase, about `amp`."""
    s = max(np.ptp(x), np.ptp(y))
    f = np.zeros_like(x)
    for _ in range(6):
        k, a, p = rng.uniform(1.0, 9.0) * 2 * math.pi / s, rng.uniform(0, 2 * math.pi), rng.uniform(0, 2 * math.pi)
        f += np.sin(k * (math.cos(a) * x + math.sin(a) * y) + p)
    return amp * f / math.sqrt(3.0)


def _initial(deck, case, seed):
    """(ze, qx, qy, wd), (NE, DOFH) arrays: waves of 0.15 m and currents of
    0.3 m/s where the bed is well under water, the deck's own initial state
    elsewhere."""
    s = deck.s
    ne, npn, dof = s.ne, s.np, s.dofh
    rng = np.random.default_rng([int(seed), 7])
    x, y, dp = (deck.real_array(n, npn) for n in ("x", "y", "dp"))
    nm = deck.int_array("nm", 3 * ne).reshape(3, ne) - 1
    wet = np.clip((dp - 0.05) / 0.5, 0.0, 1.0)
    eta = _waves(rng, x, y, 0.15) * wet
    h = np.maximum(dp + eta, 0.0)
    qx, qy = (_waves(rng, x, y, 0.3) * wet * h for _ in range(2))
    keep = (dp[nm] <= 0.05).any(axis=0)
    out = []
    for name, f in (("ze", eta), ("qx", qx), ("qy", qy)):
        v1, v2, v3 = f[nm[0]], f[nm[1]], f[nm[2]]
        m = np.zeros((ne, dof))
        m[:, 0] = (v1 + v2 + v3) / 3.0
        m[:, 1] = -(v1 + v2) / 6.0 + v3 / 3.0
        m[:, 2] = (v2 - v1) / 2.0
        for k in range(3, dof):
            m[:, k] = 0.02 * _waves(rng, x[nm].mean(0), y[nm].mean(0), 1.0) * m[:, 0]
        m[keep] = deck.real_array(name, dof * ne).reshape(ne, dof)[keep]
        out.append(m)
    return (*out, deck.int_array("wdflg", ne))


def _met(deck, case, extra):
    if case["kind"] == "ensemble":
        return tuple(np.concatenate(f) for f in extra)
    if not case.get("wind"):
        return None
    n = deck.s.np
    return np.full(n, WIND[0]), np.full(n, WIND[1]), np.zeros(n)


def _kw(case):
    return {"strict": {}, "fast": dict(fast=True), "mixed": dict(mixed=True)}[case["variant"]]


def _gauges(deck, seed):
    """16 gauges in the first kilometre off the open boundary and the misfit's
    observations' amplitude."""
    rng = np.random.default_rng([int(seed), 11])
    xy = np.column_stack([rng.uniform(30.0, 900.0, 16), rng.uniform(100.0, 3900.0, 16)])
    elem, phi = locate_gauges(deck, xy)
    return elem, phi, rng


def prepare(case, seed):
    deck, extra = _geometry(case)
    if case["kind"] == "gradient":
        elem, phi, rng = _gauges(deck, seed)
        obs = 0.01 * rng.normal(size=(case["steps"], len(elem)))
        p = GaugeMisfitProblem(deck, elem, phi, case["steps"], obs=obs)
        n = element_manning(deck)
        return dict(case=case, problem=p, nbar=n * (1.0 + 0.1 * rng.uniform(-1.0, 1.0, n.shape)))
    if case["kind"] == "ensemble":
        ens = Ensemble(deck, mixed=case["variant"] == "mixed")
        hs, whole = ens.hs, ens.deck
        ens.set_met(*extra)
    else:
        ens, whole = None, deck
        hs = HydroStep(deck, **_kw(case))
        met = _met(deck, case, extra)
        if met is not None:
            hs.set_met(*met)
    hs.set_state(*_initial(whole, case, seed))
    if case["graph"]:
        hs.set_graph(case["graph"])
    state = dict(case=case, hs=hs, ens=ens, it=1)
    if case["out"] == "state":
        state["buf"] = [torch.empty((hs.ne, hs.dofh), dtype=torch.float64, pin_memory=True).numpy() for _ in range(3)]
        state["buf"].append(torch.empty(hs.ne, dtype=torch.int32, pin_memory=True).numpy())
    return state


def run(state):
    case = state["case"]
    if case["kind"] == "gradient":
        p = state["problem"]
        p.set_params(state["nbar"])
        j = p.forward()
        gn, ghb = p.gradient()
        return dict(misfit=j, eta=p.eta, nbar=gn, hb=ghb)
    hs, n = state["hs"], case["steps"]
    if case["graph"]:
        hs.run(state["it"], n)
    else:
        for it in range(state["it"], state["it"] + n):
            hs.timestep(it)
    state["it"] += n
    if case["out"] == "nodal":
        eta, uu, vv, code = hs.modal2nodal()
        return dict(eta=eta, u=uu, v=vv, code=code)
    hs.download_into(*state["buf"])
    ze, qx, qy, wd = state["buf"]
    return dict(ze=ze, qx=qx, qy=qy, wd=wd)


def _elements(case):
    deck, _ = _geometry(case)
    if case["kind"] == "ensemble":
        return sum(d.s.ne for d in deck)
    return deck.s.ne


def work(case):
    """Per element and Runge-Kutta stage: the state in and out (and the
    step-start state at every stage but the first), bathymetry, geometry, the
    neighbour ids, flags, Manning n, and with the limiter the node ids and
    node bounds; FP64 operations of the fluxes, sources and sums."""
    ne, p2 = _elements(case), case["order"] == 2
    stages = 3 if p2 else 2
    state = 144.0 if p2 else 72.0
    per = state * (2.0 + (stages - 1.0) / stages) + (48.0 if p2 else 24.0) + 52.0
    limited = case["kind"] != "annulus" or case["limiter"]
    if limited:
        per += 52.0
    flops = 3400.0 if p2 else 1500.0 + (250.0 if limited else 0.0)
    n = ne * stages * case["steps"]
    if case["kind"] == "gradient":  # the forward, its repeat, and the reverse sweep's state, cotangents and reads
        return {"bytes": n * (2.0 * per + 6.0 * state), "flops": n * (2.0 * flops + 2.0 * flops)}
    return {"bytes": n * per + ne * (3 * state), "flops": n * flops}


# ---- the scheme in plain FP64 --------------------------------------------------
def _tables(order):
    """Orthogonal modes on the triangle (-1,-1), (1,-1), (-1,1), the edge and
    area rules, as numpy arrays."""
    def phi(x, y):
        s, r = (1 + 2 * x + y) / 2, (1 - y) / 2
        b = [np.ones_like(x), (1 + 3 * y) / 2, s]
        if order == 2:
            b += [(5 * y * y + 2 * y - 1) / 2, s * (3 + 5 * y) / 2, (3 * s * s - r * r) / 2]
        return np.array(b)

    def grad(x, y):
        s, r, z = (1 + 2 * x + y) / 2, (1 - y) / 2, np.zeros_like(x)
        dx, dy = [z, z, z + 1], [z, z + 1.5, z + 0.5]
        if order == 2:
            dx += [z, (3 + 5 * y) / 2, 3 * s]
            dy += [5 * y + 1, (3 + 5 * y) / 4 + 2.5 * s, 1.5 * s + 0.5 * r]
        return np.array(dx), np.array(dy)

    if order == 1:
        t, w = np.array([-1.0, 0.0, 1.0]), np.array([1.0, 4.0, 1.0]) / 3
        bary, wa = np.array([[1, 1, 4], [1, 4, 1], [4, 1, 1]]) / 6.0, np.full(3, 2.0 / 3.0)
    else:
        q = math.sqrt(0.2)
        t, w = np.array([-1.0, -q, q, 1.0]), np.array([1.0, 5.0, 5.0, 1.0]) / 6
        bary, wa = [], []
        for a, wt in ((0.4459484909159648863183292538830519, 0.2233815896780114656950070084331228),
                      (0.0915762135097707434595714634022015, 0.1099517436553218676383263249002105)):
            c = 1 - 2 * a
            bary += [[a, a, c], [a, c, a], [c, a, a]]
            wa += [2 * wt] * 3
        bary, wa = np.array(bary), np.array(wa)
    edge = np.stack([phi(-t, t), phi(np.full_like(t, -1.0), -t), phi(t, np.full_like(t, -1.0))])  # (3, modes, points)
    xa, ya = -bary[:, 0] + bary[:, 1] - bary[:, 2], -bary[:, 0] - bary[:, 1] + bary[:, 2]
    deg = [(0, 0), (0, 1), (1, 0), (0, 2), (1, 1), (2, 0)][: 3 if order == 1 else 6]
    minv = np.array([(2 * i + 1) * (2 * j + 2 * i + 2) / 4 for i, j in deg])
    lin = np.stack([-(xa + ya) / 2, (1 + xa) / 2, (1 + ya) / 2])
    corner = phi(np.array([-1.0, 1.0, -1.0]), np.array([-1.0, -1.0, 1.0]))[:3]
    return dict(t=t, w=w, wa=wa, edge=edge, area=phi(xa, ya), grad=grad(xa, ya), minv=minv, lin=lin, corner=corner)


class Flow:
    """The nonlinear shallow-water equations in modal DG, on torch FP64."""

    def __init__(self, deck, case, met):
        s = deck.s
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        T = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=dev)  # noqa: E731
        ne, npn = s.ne, s.np
        self.order = 2 if s.dofh == 6 else 1
        self.dof, self.nrk = s.dofh, s.nrk
        tb = {k: (tuple(T(x) for x in v) if isinstance(v, tuple) else T(v)) for k, v in _tables(self.order).items()}
        self.tb = tb
        nm = deck.int_array("nm", 3 * ne).reshape(3, ne) - 1
        x, y, dp = (deck.real_array(n, npn) for n in ("x", "y", "dp"))
        X, Y = x[nm], y[nm]
        area2 = (X[0] - X[2]) * (Y[1] - Y[2]) + (X[2] - X[1]) * (Y[0] - Y[2])
        a, b = [1, 2, 0], [2, 0, 1]
        ln = np.hypot(X[b] - X[a], Y[b] - Y[a])
        self.nx, self.ny, self.fac = T((Y[b] - Y[a]) / ln), T((X[a] - X[b]) / ln), T(ln / area2)
        self.drdx, self.dsdx = T(2 / area2 * (Y[2] - Y[0])), T(2 / area2 * (Y[0] - Y[1]))
        self.drdy, self.dsdy = T(2 / area2 * (X[0] - X[2])), T(2 / area2 * (X[1] - X[0]))
        self.nm, self.dpn, self.npn, self.ne = T(nm), T(dp[nm]), npn, ne
        self.hb = T(deck.real_array("hb", s.dofh * ne).reshape(ne, s.dofh).T)
        ned = s.nedges
        nedel = deck.int_array("nedel", 2 * ned).reshape(ned, 2)
        nedsd = deck.int_array("nedsd", 2 * ned).reshape(ned, 2)
        inner = np.nonzero((nedel > 0).all(1))[0]
        self.e_in, self.e_ex = (T(nedel[inner, k].astype(np.int64) - 1) for k in (0, 1))
        self.l_in, self.l_ex = (T(nedsd[inner, k].astype(np.int64) - 1) for k in (0, 1))
        outer = {}
        for kind, n, name in (("ocean", s.needs, "needn"), ("land", s.nleds, "nledn")):
            g = deck.int_array(name, n).astype(np.int64) - 1
            outer[kind] = (T(nedel[g, 0].astype(np.int64) - 1), T(nedsd[g, 0].astype(np.int64) - 1))
        self.ocean, self.land = outer["ocean"], outer["land"]
        nb = s.nbfr
        amp, eq = (np.ctypeslib.as_array(ctypes.cast(p, ctypes.POINTER(ctypes.c_double)),
                                         shape=(2, max(s.needs, 1), max(nb, 1))) for p in (s.emo_dg, s.efa_dg))
        self.amp, self.eq = T(amp.copy()), T(eq.copy())
        arr = lambda n, k: [float(getattr(s, n)[i]) for i in range(k)]  # noqa: E731
        self.tide = list(zip(*(arr(n, nb) for n in ("amig", "ff", "face", "per"))))
        self.g, self.h0, self.dt, self.dramp, self.nramp, self.statim = s.g, s.h0, s.dtdp, s.dramp, s.nramp, s.statim
        self.quadratic, self.wetdry, self.limiter = s.iflinbf == 0, s.nolifa >= 2, s.slopeflag == 5
        self.cf = s.cf
        self.fric = float(s.fric_el[0]) if s.fric_el else s.cf
        self.manning = T(deck.real_array("manning", npn)[nm].mean(0)) if s.load_manning else None
        self.nonlinear = s.ifnlfa != 0
        self.met = None if met is None else [T(f[nm]) for f in met]
        n = self.nrk
        self.a, self.b = (np.array([p[i] for i in range(n * n)]).reshape(n, n) for p in (s.atvd, s.btvd))
        self.d = np.array([s.dtvd[i] for i in range(n)])
        self.T = T

    def llf(self, i, e, hi, he, nx, ny, g):
        """Local Lax-Friedrichs flux of states i, e = (zeta, qx, qy)."""
        def phys(q, h):
            z, u, v = q
            d = z + h
            p = g * z * (0.5 * z + h)
            return (u, u * u / d + p, u * v / d), (v, u * v / d, v * v / d + p), (u * nx + v * ny) / d, d
        fi, gi, ui, di = phys(i, hi)
        fe, ge, ue, de = phys(e, he)
        n2 = nx * nx + ny * ny
        speed = lambda u, d: torch.maximum(u.abs(), u.abs() + torch.nan_to_num(torch.sqrt(g * d * n2)))  # noqa: E731
        lam = torch.maximum(speed(ui, di), speed(ue, de))
        return [0.5 * ((fi[k] + fe[k]) * nx + (gi[k] + ge[k]) * ny) - 0.5 * lam * (e[k] - i[k]) for k in range(3)]

    def rhs(self, q, wd, t, ramp):
        """d/dt of the modes q (3, modes, NE)."""
        tb, m = self.tb, self.dof
        r = torch.zeros_like(q)
        wq = 2 * tb["minv"][:, None] * tb["edge"] * tb["w"]  # (3, modes, points)

        def trace(e, l, flip):
            b = tb["edge"][l]  # (n, modes, points)
            b = b.flip(2) if flip else b
            f = [torch.einsum("kn,nkp->np", q[c][:, e], b) for c in range(3)]
            return f, torch.einsum("kn,nkp->np", self.hb[:, e], b)

        def add(e, l, flip, f, sign):
            w = wq[l] * self.fac[l, e][:, None, None]
            w = w.flip(2) if flip else w
            for c in range(3):
                r[c].index_add_(1, e, sign * torch.einsum("nkp,np->kn", w, f[c]))

        wet = wd == 1
        for kind, (e, l) in (("ocean", self.ocean), ("land", self.land)):
            if not len(e):
                continue
            i, h = trace(e, l, False)
            nx, ny = self.nx[l, e][:, None], self.ny[l, e][:, None]
            if kind == "ocean":
                z = torch.zeros_like(h)
                x = tb["t"]
                for f, (w0, ff, face, per) in enumerate(self.tide):
                    arg = w0 * (t - (int(t / per) if per else 0) * per) + face
                    v = self.amp[:, :, f] * ff * ramp * torch.cos(arg - self.eq[:, :, f])
                    z = z + 0.5 * (v[0] + v[1])[:, None] + 0.5 * (v[1] - v[0])[:, None] * x
                z = torch.where(z * float(self.nonlinear) + h <= 0, h.abs() + self.h0, z)
                ex = [z, i[1], i[2]]
            else:
                qn, qt = i[1] * nx + i[2] * ny, -i[1] * ny + i[2] * nx
                ex = [i[0], -qn * nx - qt * ny, -qn * ny + qt * nx]
            f = self.llf(i, ex, h, h, nx, ny, self.g)
            on = wet[e][:, None]
            add(e, l, False, [torch.where(on, v, torch.zeros_like(v)) for v in f], -1.0)
        a, b = self.e_in, self.e_ex
        i, hi = trace(a, self.l_in, False)
        e, he = trace(b, self.l_ex, True)
        nx, ny = self.nx[self.l_in, a][:, None], self.ny[self.l_in, a][:, None]
        f = self.llf(i, e, hi, he, nx, ny, self.g)
        fi, fe = [f[0], f[1], f[2]], [f[0], f[1], f[2]]
        if self.wetdry:
            wi, we = wet[a][:, None], wet[b][:, None]
            front = (wi ^ we) & (f[0].abs() > 1e-8)
            zero = torch.zeros_like(f[0])
            for dry_in in (True, False):
                at = front & (we if dry_in else wi)
                reflect = at & (f[0] > 0 if dry_in else f[0] < 0)
                slack = at & ~reflect
                w, hw = (e, he) if dry_in else (i, hi)
                qn, qt = w[1] * nx + w[2] * ny, -w[1] * ny + w[2] * nx
                mirror = [w[0], -qn * nx - qt * ny, -qn * ny + qt * nx]
                fr = self.llf(mirror, w, hw, hw, nx, ny, self.g) if dry_in else self.llf(w, mirror, hw, hw, nx, ny, self.g)
                f0 = self.llf(i, e, hi, he, nx, ny, 0.0)
                dry, live = (fi, fe) if dry_in else (fe, fi)
                dry[0] = torch.where(reflect, fr[0], dry[0])
                live[0] = torch.where(reflect, fr[0], live[0])
                for c in (1, 2):
                    live[c] = torch.where(reflect, fr[c], live[c])
                    dry[c] = torch.where(reflect, zero, torch.where(slack, f0[c], dry[c]))
            on = wi | we
            fi, fe = ([torch.where(on, v, zero) for v in k] for k in (fi, fe))
        add(a, self.l_in, False, fi, -1.0)
        add(b, self.l_ex, True, fe, 1.0)
        # area terms
        gr, gs = tb["grad"]
        dx = gr[:, :, None] * self.drdx + gs[:, :, None] * self.dsdx  # (modes, points, NE)
        dy = gr[:, :, None] * self.drdy + gs[:, :, None] * self.dsdy
        for p in range(tb["wa"].numel()):
            ph = tb["area"][:, p]
            z, u, v = (torch.einsum("k,kn->n", ph, q[c]) for c in range(3))
            h = torch.einsum("k,kn->n", ph, self.hb)
            hx, hy = ((self.hb * d[:, p]).sum(0) for d in (dx, dy))
            d = z + h
            tau = torch.full_like(d, self.fric)
            if self.manning is not None:
                tau = torch.clamp(self.g * self.manning ** 2 / torch.sign(d) / d.abs() ** (1.0 / 3.0), min=self.cf)
            if self.quadratic:
                tau = torch.clamp(tau * torch.sqrt(u * u + v * v) / d / d, max=0.9 / self.dt)
            pr = self.g * z * (0.5 * z + h)
            fx, fy = (u, u * u / d + pr, u * v / d), (v, u * v / d, v * v / d + pr)
            sx, sy = -tau * u + self.g * z * hx, -tau * v + self.g * z * hy
            if self.met is not None:
                lin = tb["lin"][:, p]
                wx, wy = (torch.einsum("k,kn->n", lin, ramp * f) for f in self.met[:2])
                n0, n1, n2 = (ramp * f for f in self.met[2])
                px = ((n1 - n0) * self.drdx + (n2 - n0) * self.dsdx) / 2
                py = ((n1 - n0) * self.drdy + (n2 - n0) * self.dsdy) / 2
                sx, sy = sx + wx - self.g * d * px, sy + wy - self.g * d * py
            on = wet.to(q.dtype)
            for k in range(m):
                w = tb["minv"][k] * tb["wa"][p]
                for c, src in ((0, None), (1, sx), (2, sy)):
                    t_ = w * (dx[k, p] * fx[c] + dy[k, p] * fy[c])
                    if src is not None:
                        t_ = t_ + w * ph[k] * src
                    r[c, k] += torch.where(wet, t_, torch.zeros_like(t_)) * on
        return r

    def limit(self, q):
        c = self.tb["corner"]
        nm = self.nm.reshape(-1)
        for var in range(3):
            z = q[var, 0]
            rep = z.repeat(3)
            lo, hi = (torch.full((self.npn,), s, dtype=z.dtype, device=z.device).scatter_reduce(0, nm, rep, op)
                      for s, op in ((99999.0, "amin"), (-99999.0, "amax")))
            lo, hi = lo[self.nm], hi[self.nm]
            v = torch.einsum("ka,kn->an", c, q[var][:3])
            v = torch.maximum(torch.minimum(v, hi), lo)
            for _ in range(3):
                over = ((v[0] + v[1] + v[2]) / 3.0 - z) * 3.0
                sg = torch.where(over < 0, -1.0, 1.0).to(z.dtype)
                up = (v - z) * sg > 0
                left = up.sum(0)
                for k in range(3):
                    red = torch.where(up[k], over * sg / torch.clamp(left, min=1), torch.zeros_like(over))
                    left = left - up[k].long()
                    red = torch.minimum(red, torch.where(sg > 0, v[k] - lo[k], hi[k] - v[k]))
                    over = over - red * sg
                    v[k] = v[k] - red * sg
            q[var, 1] = -(v[0] + v[1]) / 6.0 + v[2] / 3.0
            q[var, 2] = (v[1] - v[0]) / 2.0

    def dry(self, q, wd):
        """Vertex-based wetting and drying, in place."""
        c, h0, zero = self.tb["corner"], self.h0, 1e-6
        zn = torch.einsum("ka,kn->an", c, q[0][:3])
        ht = self.dpn + zn
        nd = (ht <= h0 + zero).sum(0)
        avg = q[0, 0] + self.dpn.mean(0)
        flat = (nd == 3) | ((nd > 0) & (avg <= h0 + zero))
        part = (nd > 0) & ~flat
        top = torch.where(ht.amax(0) > zero, ht.argmax(0), torch.zeros_like(nd))
        # partly wet: lift the shallow vertices to H0 from the others' water
        order = torch.argsort(ht, dim=0, stable=True)
        s = torch.gather(ht, 0, order)
        d0 = torch.clamp(s[0], min=h0) - s[0]
        d1 = torch.clamp(s[1] - 0.5 * d0, min=h0) - s[1]
        hh = ht + torch.zeros_like(ht).scatter(0, order, torch.stack([d0, d1, -d0 - d1]))
        dryv = hh <= h0 + 1e-10
        n2 = dryv.sum(0)
        lifted = hh - self.dpn
        top = torch.where(part, hh.argmax(0), top)
        new = [f.clone() for f in q]
        for var in (1, 2):
            qn = torch.einsum("ka,kn->an", c, q[var][:3])
            share = torch.where(dryv, qn, torch.zeros_like(qn)).sum(0) / torch.clamp(3 - n2, min=1)
            v = torch.where(dryv, torch.zeros_like(qn), qn + share)
            mo = torch.stack([v.mean(0), -(v[0] + v[1]) / 6 + v[2] / 3, (v[1] - v[0]) / 2])
            mo = torch.where(n2 == 3, torch.zeros_like(mo), mo)
            new[var][:3] = torch.where(part, mo, torch.where(flat, torch.zeros_like(mo), q[var][:3]))
        z1 = torch.where(avg < zero, zero - self.dpn.mean(0), q[0, 0])
        zf = torch.stack([z1, -self.hb[1], -self.hb[2]])
        zp = torch.stack([q[0, 0], -(lifted[0] + lifted[1]) / 6 + lifted[2] / 3, (lifted[1] - lifted[0]) / 2])
        new[0][:3] = torch.where(flat, zf, torch.where(part, zp, q[0][:3]))
        zh = torch.where(part, lifted, torch.where(flat, z1.expand(3, -1), zn))
        zt = torch.gather(zh, 0, top[None])[0]
        check = (nd != 3) & ~((nd == 0) & (wd == 1))
        up = zt > -self.dpn.amin(0) + h0
        stop = check & ~up
        for var in (1, 2):
            new[var] = torch.where(stop, torch.zeros_like(new[var]), new[var])
        wd = torch.where(nd == 3, torch.zeros_like(wd), torch.where(check, up.to(wd.dtype), wd))
        for var in range(3):
            q[var] = new[var]
        return wd

    def run(self, ze, qx, qy, wd, it, n):
        q = torch.stack([self.T(f.T) for f in (ze, qx, qy)])
        wd = self.T(wd.astype(np.int64))
        for i in range(it, it + n):
            qs, rs = [q], []
            for k in range(self.nrk):
                t = i * self.dt + self.statim * 86400.0 - self.dt + self.d[k] * self.dt
                ramp = math.tanh(2.0 * ((i - 1) + self.d[k]) * self.dt / 86400.0 / self.dramp) if self.nramp else 1.0
                rs.append(self.rhs(qs[k], wd, t, ramp))
                nxt = sum(self.a[k, j] * qs[j] + self.b[k, j] * self.dt * rs[j] for j in range(k + 1))
                if self.limiter:
                    self.limit(nxt)
                if self.wetdry:
                    wd = self.dry(nxt, wd)
                qs.append(nxt)
            q = qs[-1]
        return q, wd

    def nodal(self, q, wd):
        """Area-weighted nodal elevation and velocity over the wet elements."""
        c = self.tb["corner"]
        z, u, v, h = (torch.einsum("ka,kn->an", c, f[:3]) for f in (q[0], q[1], q[2], self.hb))
        area = 1.0 / (self.drdx * self.dsdy - self.dsdx * self.drdy)
        w = (area * (wd == 1)).expand(3, -1)
        put = lambda f: torch.zeros(self.npn, dtype=z.dtype, device=z.device).index_add_(  # noqa: E731
            0, self.nm.reshape(-1), f.reshape(-1))
        tot = put(w)
        d = z + h
        safe = torch.where(tot > 0, tot, torch.ones_like(tot))
        return [put(torch.where(w > 0, w * f, torch.zeros_like(f))) / safe for f in (z, u / d, v / d)]


def exact(case, seed):
    """run()'s first outputs in plain FP64.  None for the gradient (its
    branches are held at the forward run's, so it is no derivative of a
    function plain arithmetic could differentiate)."""
    if case["kind"] == "gradient":
        return None
    deck, extra = _geometry(case)
    whole = Deck.merge(deck) if case["kind"] == "ensemble" else deck
    flow = Flow(whole, case, _met(whole, case, extra))
    q, wd = flow.run(*_initial(whole, case, seed), 1, case["steps"])
    if case["out"] == "nodal":
        eta, u, v = (f.cpu().numpy() for f in flow.nodal(q, wd))
        return dict(eta=eta, u=u, v=v, code=None)
    ze, qx, qy = (np.ascontiguousarray(f.cpu().numpy().T) for f in q)
    return dict(ze=ze, qx=qx, qy=qy, wd=None)
