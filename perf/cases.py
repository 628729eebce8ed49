"""The work of a user's program on the QG core, as cases that can be timed.

A case is a dict of plain values.  `prepare` makes what the program holds
before the call (handles, states, forcing), `run` is one pass through the
public entry points, `work` the bytes and operations that pass cannot do
without, and `exact` the same pass in 64 bits in plain torch.

Kinds of cases:
  step      QG.step on one basin: the model's time loop (closed boxes and
            periodic channels, FP64 and FP32 storage, 2 to 4 layers, with and
            without entrainment and topography)
  ensemble  Ensemble.step, then every member's state read back
  gradient  QGRun.apply and its backward: a run and its gradients
  coupled   the coupled driver's loop: wind stress, heat fluxes, both mixed
            layers and both basins' steps, all on the device
  exchange  step_qg with host forcing and the layer-1 pressure read back, as
            a host program that keeps its own forcing does every step
"""
import ctypes
import math

import numpy as np
import torch

from openqg_b200 import core
from openqg_b200.adjoint import QGRun, ekei
from openqg_b200.core import QG, AtmosMixedLayer, Ensemble, OceanMixedLayer, ekman_from_tau, init_qg, step_qg
from openqg_b200.params import OQG_FP64, OQG_MIXED, Basin, atmos_channel, double_gyre_tau, ocean_double_gyre
from openqg_b200.radiation import coupled_start, rbal_states

# layer thicknesses (m) and reduced gravities (m/s^2) by number of layers
OCEAN = {2: ([500.0, 3500.0], [0.03]), 3: ([350.0, 750.0, 2900.0], [0.05, 0.025]),
         4: ([300.0, 500.0, 1000.0, 2200.0], [0.05, 0.025, 0.015])}
ATMOS = {2: ([2000.0, 3000.0], [1.2]), 3: ([2000.0, 3000.0, 4000.0], [1.2, 0.4]),
         4: ([2000.0, 3000.0, 4000.0, 4000.0], [1.2, 0.4, 0.3])}
MEMBER_SIZES = (65, 97, 129, 193, 257)


def step(kind, nxp, nyp, precision="fp64", nl=3, nsteps=10, ent=False, topo=False):
    return {"kind": kind, "nxp": nxp, "nyp": nyp, "precision": precision, "nl": nl, "nsteps": nsteps, "ent": ent,
            "topo": topo}


def listed():
    return [
        # the smallest call: one step of a small basin, where launches and
        # latency are everything (a driver that does something each step)
        dict(step("box", 65, 65, nsteps=1), name="box65_fp64_1step"),
        # the small ocean-only configuration, stepped in runs
        dict(step("box", 129, 129, nsteps=16), name="box129_fp64"),
        # the coupled configuration's ocean basin, in both storage types
        dict(step("box", 513, 513), name="box513_fp64"),
        dict(step("box", 513, 513, "fp32"), name="box513_fp32"),
        # a basin of nobody's power of two: two layers, topography and
        # entrainment, as a regional set-up has them
        dict(step("box", 361, 287, nl=2, nsteps=8, ent=True, topo=True), name="box361x287_2layer_fp64"),
        # the eddy-resolving ocean, the largest grid, in both storage types
        dict(step("box", 2049, 2049, nsteps=4), name="box2049_fp64"),
        dict(step("box", 2049, 2049, "fp32", nsteps=4), name="box2049_fp32"),
        # the atmosphere of the coupled configuration, stepped by itself
        dict(step("channel", 193, 97, ent=True), name="channel193x97_fp64"),
        # an ensemble study: members of uneven size stepped together, then
        # every member's state read
        {"kind": "ensemble", "members": 24, "precision": "fp32", "nsteps": 400, "name": "ensemble24_fp32"},
        # a sensitivity study: a run and the gradients of its kinetic energy
        {"kind": "gradient", "nxp": 257, "nyp": 257, "nsteps": 60, "every": 20, "name": "gradient257"},
        # the coupled model's own loop: ten ocean steps of ten atmosphere steps
        {"kind": "coupled", "n": 513, "precision": "fp64", "nocean": 10, "nstr": 10, "name": "coupled513"},
        # a host program that keeps its forcing and reads the pressure each step
        {"kind": "exchange", "nxp": 513, "nyp": 513, "precision": "fp64", "name": "exchange513_fp64"},
    ]


def _smooth(n):
    """Whether n has no prime factor above 5 (the x-transforms' lengths)."""
    for f in (2, 3, 5):
        while n % f == 0:
            n //= f
    return n == 1


LENGTHS = [n for n in range(32, 2049) if _smooth(n)]


def _near(rng, lo, hi, precision="fp64"):
    """A transform length drawn over the logarithm of [lo, hi].  FP32 storage
    is used at multiples of 16, as in all of the repository's configurations."""
    x = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    every = 16 if precision == "fp32" else 1
    return min((n for n in LENGTHS if lo <= n <= hi and n % every == 0), key=lambda n: abs(n - x))


def draw(rng):
    r = rng.random()
    precision = rng.choice(["fp64", "fp64", "fp32"])
    if r < 0.12:
        return {"kind": "ensemble", "members": rng.randint(4, 24), "precision": precision,
                "nsteps": rng.randint(50, 400)}
    if r < 0.24:
        n = _near(rng, 64, 320) + 1
        nsteps = rng.randint(10, 60)
        return {"kind": "gradient", "nxp": n, "nyp": rng.randint(max(33, n // 2), n), "nsteps": nsteps,
                "every": rng.randint(4, 20)}
    if r < 0.34:
        return {"kind": "coupled", "n": rng.choice([129, 193, 257, 321, 385, 513]), "precision": precision,
                "nocean": rng.randint(2, 10), "nstr": rng.randint(4, 10)}
    if r < 0.42:
        n = _near(rng, 64, 1024, precision) + 1
        return {"kind": "exchange", "nxp": n, "nyp": rng.randint(n // 2, n), "precision": precision}
    nl = rng.choice([2, 3, 3, 3, 4])
    if r < 0.62:
        nxp = _near(rng, 64, 768, precision) + 1
        nyp = rng.randint(max(33, nxp // 3), nxp)
        return step("channel", nxp, nyp, precision, nl, rng.randint(1, 16), rng.random() < 0.5, rng.random() < 0.3)
    nxp = _near(rng, 32, 2048, precision) + 1
    nyp = min(2049, max(33, int(nxp * math.exp(rng.uniform(math.log(0.5), math.log(1.6))))))
    most = max(1, int(2049 * 2049 * 3 * 4 / (nxp * nyp * nl)))
    return step("box", nxp, nyp, precision, nl, min(most, rng.randint(1, 16)), rng.random() < 0.4,
                rng.random() < 0.3)


# ------------------------------------------------------------------ inputs
def _rng(case, seed):
    return np.random.default_rng([int(seed) & 0x7FFFFFFF, case.get("nxp", case.get("n", case.get("members", 0)))])


def _smooth_field(rng, b, layers, std):
    """Noise of the first 7 modes of each direction, zero on the solid walls,
    periodic in a channel, with the given standard deviation."""
    y = np.arange(b.nyp)
    sy = np.sin(np.pi * (np.outer(y, np.arange(1, 8)) % (2 * (b.nyp - 1))) / (b.nyp - 1))
    x = np.arange(b.nxp)
    if b.cyclic:
        a = 2.0 * np.pi * (np.outer(x, np.arange(0, 4)) % (b.nxp - 1)) / (b.nxp - 1)
        sx = np.concatenate([np.cos(a), np.sin(a[:, 1:])], axis=1)
    else:
        sx = np.sin(np.pi * (np.outer(x, np.arange(1, 8)) % (2 * (b.nxp - 1))) / (b.nxp - 1))
    f = np.stack([sy @ rng.standard_normal((7, 7)) @ sx.T for _ in range(layers)])
    if not b.cyclic:
        f[:, :, 0] = f[:, :, -1] = 0.0
    f[:, 0] = f[:, -1] = 0.0
    return f * (std / f.std(axis=(1, 2), keepdims=True))


def _stored(case, a):
    """The values as FP32 storage holds them, where the case has it."""
    return a.astype(np.float32).astype(np.float64) if case["precision"] == "fp32" else a


def _basin(case, rng):
    prec = OQG_MIXED if case["precision"] == "fp32" else OQG_FP64
    nxp, nyp, nl = case["nxp"], case["nyp"], case.get("nl", 3)
    if case["kind"] == "channel":
        # the atmosphere's domain length at any resolution
        dx = 15360.0e3 / (nxp - 1)
        b = Basin(nxp=nxp, nyp=nyp, dx=dx, dy=dx, h=ATMOS[nl][0], gp=ATMOS[nl][1], cyclic=True, dz_sign=1,
                  tau_sign=-1, ah4=[2.0e13 * (dx / 80.0e3) ** 4] * nl, ah2=[0.0] * nl, bcco=1.0, delek=0.0, rho=1.0,
                  k_topo=1, precision=prec, suppress_period=100)
        tdt = 360.0 * min(1.0, dx / 80.0e3)
    else:
        n = max(nxp, nyp)
        dx, ah4, tdt = (20.0e3, 2.0e10, 3600.0) if n <= 257 else (10.0e3, 2.0e10, 3600.0) if n <= 1025 else \
            (5.0e3, 1.0e9, 1200.0)
        b = Basin(nxp=nxp, nyp=nyp, dx=dx, dy=dx, h=OCEAN[nl][0], gp=OCEAN[nl][1], ah2=[0.0] * nl, ah4=[ah4] * nl,
                  precision=prec)
    if case.get("topo"):
        k = b.ktopo() - 1
        b.ddyn = _smooth_field(rng, b, 1, 100.0 * b.fnot / b.h[k])[0]
    return b, tdt


def _wind(rng, b):
    """Double-gyre stress of a seeded amplitude, as Ekman pumping."""
    return ekman_from_tau(b, *double_gyre_tau(b, amp=float(rng.uniform(0.05, 0.15)), rho0=b.rho))


def _inputs(case, rng, b):
    p = _stored(case, _smooth_field(rng, b, b.nl, 1.0e3 * b.fnot * (30.0 if b.cyclic else 1.0)))
    w, ts, tn = _wind(rng, b)
    e = _stored(case, _smooth_field(rng, b, b.nl - 1, 1.0e-7)) if case.get("ent") else None
    return p, _stored(case, w), ts, tn, e


def _type(case):
    """The type that holds all that the case's storage knows of a value."""
    return np.float32 if case["precision"] == "fp32" else np.float64


class _Field:
    """A field of a handle as torch sees it, keeping the handle alive."""

    def __init__(self, owner, ptr, shape, pitch, eb):
        self.owner = owner
        self.__cuda_array_interface__ = {
            "shape": shape, "strides": (shape[1] * pitch * eb, pitch * eb, eb), "data": (ptr, False),
            "typestr": "<f%d" % eb, "version": 3}


def _views(g):
    """The handle's four state buffers as tensors, by address."""
    ptrs, pitch, eb = g.device_state()
    return {x: torch.as_tensor(_Field(g, x, g.b.shape3, pitch, eb), device="cuda") for x in ptrs}


def _state(g, views):
    ptrs = g.device_state()[0]
    return [views[x] for x in ptrs]


def _members(case, rng):
    out = []
    for i in range(case["members"]):
        n = MEMBER_SIZES[3 * i % 5]
        b = ocean_double_gyre(n, dx=20.0e3, ah4=float(rng.uniform(1.0e10, 4.0e10)),
                              precision=OQG_MIXED if case["precision"] == "fp32" else OQG_FP64)
        out.append((b,) + _inputs(case, rng, b))
    return out


def prepare(case, seed):
    rng = _rng(case, seed)
    kind = case["kind"]
    if kind in ("box", "channel"):
        b, tdt = _basin(case, rng)
        p, w, ts, tn, e = _inputs(case, rng, b)
        g = init_qg(b)
        g.set_state(p, p)
        g.set_forcing(w, e, ts, tn)
        return {"kind": "step", "g": g, "tdt": tdt, "n": case["nsteps"], "views": _views(g)}
    if kind == "exchange":
        b, tdt = _basin(case, rng)
        p, w, ts, tn, e = _inputs(dict(case, ent=True), rng, b)
        g = init_qg(b)
        g.set_state(p, p)
        return {"kind": kind, "g": g, "tdt": tdt, "w": w, "e": e, "ts": ts, "tn": tn, "views": _views(g),
                "type": _type(case)}
    if kind == "ensemble":
        ms = _members(case, rng)
        ens = Ensemble([m[0] for m in ms])
        for i, (_, p, w, ts, tn, _) in enumerate(ms):
            ens.set_state(i, p, p)
            ens.set_forcing(i, w, None, ts, tn)
        return {"kind": kind, "ens": ens, "n": case["nsteps"], "type": _type(case)}
    if kind == "gradient":
        b, tdt = _basin(dict(case, precision="fp64"), rng)
        p, w, _, _, _ = _inputs(dict(case, precision="fp64"), rng, b)
        dev = lambda a: torch.tensor(a, device="cuda")
        return {"kind": kind, "g": init_qg(b), "b": b, "tdt": tdt, "n": case["nsteps"], "every": case["every"],
                "psi": dev(p / b.fnot), "curl": dev(b.fnot * w.reshape(b.shape2))}
    return _prepare_coupled(case, rng)


def _prepare_coupled(case, rng):
    """The coupled double-gyre set-up with its radiative start-up."""
    prec = OQG_MIXED if case["precision"] == "fp32" else OQG_FP64
    bo = ocean_double_gyre(case["n"], dx=10.0e3, precision=prec)
    ba = atmos_channel(193, 97, dx=80.0e3, precision=prec)
    rad, ak, ok = coupled_start(ba, bo, hm_a=1000.0, fsbar=-210.0, fspamp=80.0, zopt=[200.0, 3.0e4, 3.0e4, 4.0e4],
                                gamma=1.0e-2, xlamda=35.0, tabsat=[330.0, 340.0, 350.0], rho_a=1.0, cp_a=1.0e3,
                                t1_abs_o=278.0, t2_abs_o=268.0, rho_o=1.0e3, cp_o=4.0e3)
    go, ga = QG(bo), QG(ba)
    for g in (go, ga):
        p = _inputs(dict(case, ent=False), rng, g.b)[0]
        g.set_state(p, p)
    oml = OceanMixedLayer(go, hm=100.0, rho_cp=ok["rho_cp"], t1_rel=ok["t1_rel"], dt_12=ok["dt_12"], st2d=380.0,
                          st4d=4.0e10, ycexp=1.0, fluxs=True, sval=ok["sval"], nval=ok["nval"])
    _, sst, ast = rbal_states(ba, bo, rad, ak)
    sst = sst + 0.5 * rng.standard_normal(sst.shape)
    oml.set_sst(sst, sst)
    aml = AtmosMixedLayer(ga, ak["xc1ast"], None, hm=1000.0, rho_cp=ak["rho_cp"], t1_rel=ak["t1_rel"],
                          dt_12=ak["dt_12"], hmamin=100.0, hmadmp=0.15, xcexp=1.0, at2d=5.0e4, at4d=3.0e14,
                          ahmd=2.0e5, aface=ak["aface"], bface=ak["bface"], dface=ak["dface"], cdat=1.3e-3)
    hm = np.full(ast.shape, 1000.0)
    aml.set_state(ast, ast, hm, hm)
    oml.couple(aml, 1.0e-3)
    return {"kind": "coupled", "go": go, "ga": ga, "oml": oml, "aml": aml, "rad": rad.c, "nocean": case["nocean"],
            "nstr": case["nstr"], "vo": _views(go), "va": _views(ga), "type": _type(case)}


# ------------------------------------------------------------------ one pass
def run(s):
    kind = s["kind"]
    if kind == "step":
        s["g"].step(s["tdt"], s["n"])
        return _state(s["g"], s["views"])
    if kind == "exchange":
        step_qg(s["tdt"], s["e"], s["w"], s["ts"], s["tn"], s["g"])
        return [s["g"].p_layer(0).astype(s["type"], copy=False)] + _state(s["g"], s["views"])
    if kind == "ensemble":
        ens = s["ens"]
        ens.step(3600.0, s["n"])
        # p and q of every member
        out = [ens.get_state(i) for i in range(len(ens))]
        return [np.concatenate([f[k].ravel() for f in out]).astype(s["type"], copy=False) for k in (0, 2)]
    if kind == "gradient":
        psi, curl = s["psi"].detach().requires_grad_(), s["curl"].detach().requires_grad_()
        p = QGRun.apply(psi, curl, s["g"], s["n"], s["tdt"], s["every"])
        ekei(s["b"], p)[0].backward()
        return [p.detach(), psi.grad, curl.grad]
    go, ga, oml, aml = s["go"], s["ga"], s["oml"], s["aml"]
    for _ in range(s["nocean"]):
        core.xforc(aml, oml)
        oml.compute_forcing(s["rad"])
        for k in range(s["nstr"]):
            aml.forcing(None, None, None, True, 360.0)
            ga.step(360.0, 1)
            if k == 0:
                oml.forcing(None, None, None, True, 3600.0)
                go.step(3600.0, 1)
    mixed = list(oml.get_sst()) + list(aml.get_state())
    return _state(go, s["vo"]) + _state(ga, s["va"]) + [f.astype(s["type"], copy=False) for f in mixed]


# ------------------------------------------------------------------ what a pass cannot do without
def _step_work(nxp, nyp, nl, size, nsteps, ent=0, topo=0):
    """Bytes: p, pm, q and qm read, p and q written, one word of pumping (and
    entrainment, topography) per column.  Operations per cell and layer: the
    Arakawa sum (27), three Laplacians (7 each), the leapfrog and its terms
    (12), the projections on the modes and back (4 nl), the tridiagonal solve
    (6) and two real sine transforms (2.5 log2 n each)."""
    cells = nxp * nyp
    ops = 60 + 4 * nl + 6 + 5 * math.log2(nxp)
    return cells * nsteps * (size * (6 * nl + 1 + ent + topo)), cells * nl * nsteps * ops


def work(case):
    kind = case["kind"]
    size = 4 if case.get("precision") == "fp32" else 8
    if kind in ("box", "channel"):
        by, fl = _step_work(case["nxp"], case["nyp"], case["nl"], size, case["nsteps"], case["ent"], case["topo"])
    elif kind == "exchange":
        # the host's two forcing planes and the pressure plane besides
        by, fl = _step_work(case["nxp"], case["nyp"], 3, size, 1, 1)
        by += 3 * 8 * case["nxp"] * case["nyp"]
    elif kind == "ensemble":
        n2 = case["members"] * sum(n * n for n in MEMBER_SIZES) // len(MEMBER_SIZES)
        by, fl = _step_work(n2, 1, 3, size, case["nsteps"])
    elif kind == "gradient":
        # the run, and a reversed step for each (p, q read, the adjoint state
        # read and written, about twice the operations)
        by, fl = _step_work(case["nxp"], case["nyp"], 3, 8, case["nsteps"])
        by, fl = by * 2.7, fl * 3
    else:
        bo, fo = _step_work(case["n"], case["n"], 3, size, case["nocean"], 1)
        ba, fa = _step_work(193, 97, 3, size, case["nocean"] * case["nstr"], 1)
        # the mixed layers' fields on the T grids: sst, sstm, the flux; ast,
        # astm, hmixa, hmixam, the flux, read, and the new levels written
        mo, ma = 4 * 8 * (case["n"] - 1) ** 2 * case["nocean"], 7 * 8 * 192 * 96 * case["nocean"] * case["nstr"]
        by, fl = bo + ba + mo + ma, fo + fa
    return {"bytes": float(by), "flops": float(fl)}


# ------------------------------------------------------------------ the same in 64 bits
class _Exact:
    """One basin's step in FP64 torch.  The Helmholtz problems are solved with
    dense sine bases (closed walls) and an FFT (periodic x)."""

    def __init__(self, b, device):
        self.b, self.dev = b, device
        t = self.t = lambda a: torch.as_tensor(np.asarray(a, dtype=np.float64), device=device)
        nl, f0 = b.nl, b.fnot
        A = np.zeros((nl, nl))
        for k in range(nl):
            if k > 0:
                A[k, k - 1] = -1.0 / (b.gp[k - 1] * b.h[k])
            if k < nl - 1:
                A[k, k + 1] = -1.0 / (b.gp[k] * b.h[k])
            A[k, k] = -A[k].sum()
        # modes: A = H^-1 T with T symmetric
        rh = np.sqrt(np.asarray(b.h, dtype=np.float64))
        w, V = np.linalg.eigh(0.5 * ((rh[:, None] * A / rh) + (rh[:, None] * A / rh).T))
        order = np.argsort(np.abs(w))
        w, V = w[order], V[:, order]
        right, left = V / rh[:, None], V * rh[:, None]
        self.A = t(A)
        self.l2m = t(left / (left * right).sum(axis=0))     # [k, m]
        self.m2l = t(right.T.copy())                        # [m, k]
        rd = f0 * f0 * np.abs(w)
        rd[0] = 0.0
        self.rdm2 = t(rd)
        self.y = t(b.yprel)
        self.kt = b.ktopo() - 1
        self.N = b.nxp - 1
        self.bc = b.bcco / (0.5 * b.bcco + 1.0)
        self.dd = None
        if b.ddyn is not None:
            self.dd = self.cut(t(np.asarray(b.ddyn).reshape(b.shape2)))

        def sine(n, h):
            i = np.arange(1, n + 1)
            S = math.sqrt(2.0 / (n + 1)) * np.sin(np.pi * (np.outer(i, i) % (2 * (n + 1))) / (n + 1))
            return t(S), t((-4.0 / (h * h)) * np.sin(0.5 * np.pi * i / (n + 1)) ** 2)

        self.Sy, self.ly = sine(b.nyp - 2, b.dy)
        if b.cyclic:
            self.lx = t((-4.0 / b.dx ** 2) * np.sin(np.pi * np.arange(self.N // 2 + 1) / self.N) ** 2)
            yl = (b.nyp - 1) * b.dy
            up = t(np.arange(b.nyp) / (b.nyp - 1.0))
            self.hbt = 1.0 - up
            h1 = self.mode_one((1.0 - up)[:, None].expand(b.nyp, self.N))[:, :, 0]
            h2 = self.mode_one(up[:, None].expand(b.nyp, self.N))[:, :, 0]
            self.h1, self.h2 = h1, h2                       # [m, y]
            xl, dy, r = self.N * b.dx, b.dy, self.rdm2
            s = lambda h: -xl * (h[:, 1] - h[:, 0]) / dy + 0.5 * dy * r * h[:, 0] * xl
            n = lambda h: xl * (h[:, -1] - h[:, -2]) / dy + 0.5 * dy * r * h[:, -1] * xl
            self.sn = s(h1), s(h2), n(h1), n(h2)
            self.hbsi = yl / xl
        else:
            self.Sx, self.lx = sine(b.nxp - 2, b.dx)
            wx, wy = np.ones(b.nxp), np.ones(b.nyp)
            wx[[0, -1]] = wy[[0, -1]] = 0.5
            self.w = t(np.outer(wy, wx) * b.dx * b.dy)
            self.hom = self.mode_one(torch.ones(b.shape2, dtype=torch.float64, device=device))[1:]
            ai = (self.hom * self.w).sum(dim=(1, 2))
            self.C = (self.m2l[1:, 1:] - self.m2l[1:, :-1]).T * ai[None, :]

    def mode_one(self, f):
        """f + rdm2_m times the mode's solution for f: the homogeneous solution
        that equals f on the walls."""
        return f[None] + self.rdm2[:, None, None] * self.solve(f[None].expand(self.b.nl, *f.shape))

    def cut(self, f):
        """A channel keeps its N distinct columns."""
        return f[..., :self.N] if self.b.cyclic else f

    def full(self, f):
        return torch.cat([f, f[..., :1]], dim=-1) if self.b.cyclic else f

    def solve(self, rhs):
        """(Del^2 - rdm2_m) u_m = rhs_m inside, u_m = 0 on the walls."""
        if self.b.cyclic:
            r = torch.fft.rfft(rhs[:, 1:-1], dim=-1)
            S = self.Sy.to(r.dtype)
            c = (S @ r) / (self.ly[None, :, None] + self.lx[None, None] - self.rdm2[:, None, None])
            return torch.nn.functional.pad(torch.fft.irfft(S @ c, n=self.N, dim=-1), (0, 0, 1, 1))
        den = self.ly[None, :, None] + self.lx[None, None] - self.rdm2[:, None, None]
        u = self.Sy @ ((self.Sy @ rhs[:, 1:-1, 1:-1] @ self.Sx) / den) @ self.Sx
        return torch.nn.functional.pad(u, (1, 1, 1, 1))

    def ew(self, f):
        """The east and west neighbours; zeros beyond a wall."""
        if self.b.cyclic:
            return torch.roll(f, -1, -1), torch.roll(f, 1, -1)
        pad = torch.nn.functional.pad
        return pad(f[..., 1:], (0, 1)), pad(f[..., :-1], (1, 0))

    def lap(self, f):
        b, pad, c = self.b, torch.nn.functional.pad, self.bc
        e, w = self.ew(f)
        x = e + w - 2.0 * f
        if not b.cyclic:
            x = torch.cat([c * (f[..., 1:2] - f[..., :1]), x[..., 1:-1], -c * (f[..., -1:] - f[..., -2:-1])], -1)
        x = pad(x[..., 1:-1, :], (0, 0, 1, 1)) / (b.dx * b.dx)
        y = torch.cat([c * (f[..., 1:2, :] - f[..., :1, :]), f[..., :-2, :] + f[..., 2:, :] - 2.0 * f[..., 1:-1, :],
                       -c * (f[..., -1:, :] - f[..., -2:-1, :])], -2) / (b.dy * b.dy)
        if not b.cyclic:
            y = pad(y[..., 1:-1], (1, 1))
        return x + y

    def dx(self, f):
        e, w = self.ew(f)
        d = e - w
        return d if self.b.cyclic else torch.nn.functional.pad(d[..., 1:-1], (1, 1))

    @staticmethod
    def dy(f):
        return torch.nn.functional.pad(f[..., 2:, :] - f[..., :-2, :], (0, 0, 1, 1))

    def jac(self, p, q):
        px, py, qx, qy = self.dx(p), self.dy(p), self.dx(q), self.dy(q)
        return (qx * py - qy * px + self.dx(q * py) - self.dy(q * px) + self.dy(p * qx) - self.dx(p * qy)) / (
            12.0 * self.b.dx * self.b.dy * self.b.fnot)

    def at_kt(self, f, v):
        """f with v added to the topography's layer."""
        return torch.cat([f[:self.kt], f[self.kt:self.kt + 1] + v, f[self.kt + 1:]])

    def qcomp(self, p):
        q = self.lap(p) / self.b.fnot + self.b.beta * self.y[None, :, None] - \
            self.b.fnot * torch.einsum("kl,lyx->kyx", self.A, p)
        return q if self.dd is None else self.at_kt(q, self.dd)

    def row(self, f, j):
        """x-integral of row j."""
        return f[..., j, :].sum(-1) * self.b.dx

    def start(self, p):
        """The state that set_state(p, p) leaves."""
        b = self.b
        q = self.qcomp(p)
        if b.cyclic:
            f2 = 0.5 * b.dy * b.fnot ** 2
            cs = -(self.row(p, 1) - self.row(p, 0)) / b.dy + f2 * (self.A @ self.row(p, 0))
            cn = (self.row(p, -1) - self.row(p, -2)) / b.dy + f2 * (self.A @ self.row(p, -1))
            return p, p, q, q, (cs, cn, cs, cn)
        ip = (p * self.w).sum(dim=(1, 2))
        d = b.dz_sign * (ip[:-1] - ip[1:])
        return p, p, q, q, (d, d)

    def wall(self, p, q):
        """Wall values of q from p; a corner counts its terms twice."""
        b, pad = self.b, torch.nn.functional.pad
        nyp, nx = p.shape[-2:]
        cnt = torch.zeros(nyp, nx, dtype=p.dtype, device=p.device)
        cnt[0] += 1.0
        cnt[-1] += 1.0
        nbr = pad(p[:, 1:2] - p[:, :1], (0, 0, 0, nyp - 1)) + pad(p[:, -2:-1] - p[:, -1:], (0, 0, nyp - 1, 0))
        if not b.cyclic:
            cnt[:, 0] += 1.0
            cnt[:, -1] += 1.0
            nbr = torch.cat([p[..., 1:2] - p[..., :1], nbr[..., 1:-1], p[..., -2:-1] - p[..., -1:]], -1)
        qw = self.bc / (b.dx * b.dx * b.fnot) * nbr - cnt * b.fnot * torch.einsum("kl,lyx->kyx", self.A, p) + \
            cnt * b.beta * self.y[None, :, None]
        if self.dd is not None:
            qw = self.at_kt(qw, cnt * self.dd)
        return torch.where((cnt > 0)[None], qw, q)

    def step(self, s, tdt, nt, w, e=None, ts=0.0, tn=0.0):
        b, kt, f0 = self.b, self.kt, self.b.fnot
        p, pm, q, qm, con = s
        d2 = self.lap(pm)
        d4 = self.lap(d2)
        c2, c4 = self.t(b.ah2)[:, None, None] / f0, self.t(b.ah4)[:, None, None] / f0
        dq = self.jac(p, q) + c2 * d4 - c4 * self.lap(d4)
        add = [torch.zeros_like(d2[0]) for _ in range(b.nl)]
        add[0] = add[0] + b.tau_sign * f0 / b.h[0] * w
        if e is not None:
            add[0] = add[0] + b.dz_sign * f0 / b.h[0] * e[0]
            add[1] = add[1] - b.dz_sign * f0 / b.h[1] * e[0]
        add[kt] = add[kt] - f0 / b.h[kt] * b.delek / (2.0 * abs(f0)) * d2[kt]
        qn = qm + tdt * (dq + torch.stack(add))
        ql = qn - b.beta * self.y[None, :, None]
        if self.dd is not None:
            ql = self.at_kt(ql, -self.dd)
        u = self.solve(f0 * torch.einsum("km,kyx->myx", self.l2m, ql))
        if b.cyclic:
            cs, cn, csp, cnp = con
            rs, rn = self.strips(p, pm, q, d2, d4, e, ts, tn)
            cs, csp, cn, cnp = csp + tdt * rs, cs, cnp + tdt * rn, cn
            ls = self.l2m.T @ cs + self.row(u, 1) / b.dy
            ln = self.l2m.T @ cn + self.row(u, -2) / b.dy
            p1s, p2s, p1n, p2n = self.sn
            det = p1s * p2n - p2s * p1n
            c1, c2_ = (p2n * ls - p2s * ln) / det, (p1s * ln - p1n * ls) / det
            hom = c1[:, None] * self.h1 + c2_[:, None] * self.h2
            hom[0] = ls[0] * self.hbsi * self.hbt
            u = u + hom[:, :, None]
            con = (cs, cn, csp, cnp)
        else:
            dpi, dpip = con
            xn = (e[0] * self.w).sum() if e is not None else 0.0
            first = torch.zeros_like(dpi)
            first[0] = b.gp[0] * xn
            con = (dpip - tdt * first, dpi)
            ik = self.m2l.T @ (u * self.w).sum(dim=(1, 2))
            al = torch.linalg.solve(self.C, con[0] - (ik[1:] - ik[:-1]))
            u = torch.cat([u[:1], u[1:] + al[:, None, None] * self.hom])
        pn = torch.einsum("mk,myx->kyx", self.m2l, u)
        qn = self.wall(pn, qn)
        if nt % b.suppress_period == 0:
            pn, qn = 0.5 * (pn + p), 0.5 * (qn + q)
            h = len(con) // 2
            con = tuple(0.5 * (x + y) for x, y in zip(con[:h], con[h:])) + con[h:]
        return pn, p, qn, q, con

    def strips(self, p, pm, q, d2, d4, e, ts, tn):
        """The rates of the channel's momentum constraints on both walls."""
        b, f0, kt = self.b, self.b.fnot, self.kt
        px = self.dx(p)
        r = lambda f: f.sum(-1) * b.dx
        zero = torch.zeros(b.nl, dtype=p.dtype, device=p.device)
        rs, rn = zero.clone(), zero.clone()
        if e is not None:
            for k in range(min(2, b.nl - 1)):
                rs[k] -= 0.5 * b.dy * f0 * b.dz_sign * f0 / b.h[0] * self.row(e[k], 0)
                rn[k] += 0.5 * b.dy * f0 * b.dz_sign * f0 / b.h[1] * self.row(e[k], -1)
        rs[0] += b.tau_sign * f0 / b.h[0] * ts
        rn[0] -= b.tau_sign * f0 / b.h[0] * tn
        drag = f0 * b.delek / (2.0 * abs(f0)) * f0 / b.h[-1] / b.dy
        rs[-1] += drag * (self.row(pm[kt], 1) - self.row(pm[kt], 0))
        rn[-1] -= drag * (self.row(pm[kt], -1) - self.row(pm[kt], -2))
        js = (r(q[:, 0] * px[:, 1]) + 2.0 * r(q[:, 1] * px[:, 1])) / (12.0 * b.dx)
        jn = (r(q[:, -1] * px[:, -2]) + 2.0 * r(q[:, -2] * px[:, -2])) / (12.0 * b.dx)
        a2, a4 = self.t(b.ah2) / b.dy, self.t(b.ah4) / b.dy
        up = lambda f: self.row(f, 1) - self.row(f, 0)
        dn = lambda f: self.row(f, -1) - self.row(f, -2)
        return rs + js - a2 * up(d2) + a4 * up(d4), rn - jn + a2 * dn(d2) - a4 * dn(d4)


def _exact_steps(b, p, w, ts, tn, e, tdt, nsteps, dev):
    x = _Exact(b, dev)
    s = x.start(x.cut(x.t(p)))
    wt = x.cut(x.t(w.reshape(b.shape2)))
    et = x.cut(x.t(e)) if e is not None else None
    for n in range(nsteps):
        s = x.step(s, tdt, n, wt, et, ts, tn)
    out = [x.full(f) for f in s[:4]]
    if b.precision == OQG_MIXED:                 # FP32 storage keeps q - beta y
        out[2:] = [f - b.beta * x.y[None, :, None] for f in out[2:]]
    return out


def exact(case, seed):
    rng = _rng(case, seed)
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    kind = case["kind"]
    if kind in ("box", "channel", "exchange"):
        b, tdt = _basin(case, rng)
        p, w, ts, tn, e = _inputs(dict(case, ent=True) if kind == "exchange" else case, rng, b)
        out = _exact_steps(b, p, w, ts, tn, e, tdt, case.get("nsteps", 1), dev)
        return out if kind != "exchange" else [out[0][0].cpu().numpy()] + out
    if kind == "ensemble":
        both = []
        for b, p, w, ts, tn, _ in _members(case, rng):
            f = _exact_steps(b, p, w, ts, tn, None, 3600.0, case["nsteps"], dev)
            q = f[2] + b.beta * torch.as_tensor(b.yprel, device=dev)[None, :, None] if b.precision == OQG_MIXED \
                else f[2]
            both.append((f[0].cpu().numpy().ravel(), q.cpu().numpy().ravel()))
        return [np.concatenate([f[k] for f in both]) for k in (0, 1)]
    if kind == "gradient":
        b, tdt = _basin(dict(case, precision="fp64"), rng)
        p, w, _, _, _ = _inputs(dict(case, precision="fp64"), rng, b)
        x = _Exact(b, dev)
        psi = x.t(p / b.fnot).requires_grad_()
        curl = x.t(b.fnot * w.reshape(b.shape2)).requires_grad_()
        s = x.start(b.fnot * psi)
        for n in range(case["nsteps"]):
            s = x.step(s, tdt, n, curl / b.fnot)
        out = s[0]
        # the upper layer's kinetic energy, with the walls' one-sided differences
        ah, f = 0.5 * b.bcco + 1.0, out[0]
        vx = torch.cat([(f[:, 1:2] - f[:, :1]) / (b.dx * ah), (f[:, 2:] - f[:, :-2]) / (2.0 * b.dx),
                        (f[:, -1:] - f[:, -2:-1]) / (b.dx * ah)], 1)[1:-1]
        uy = torch.cat([(f[1:2] - f[:1]) / (b.dy * ah), (f[2:] - f[:-2]) / (2.0 * b.dy),
                        (f[-1:] - f[-2:-1]) / (b.dy * ah)], 0)[:, 1:-1]
        J = 0.5e3 * b.h[0] * (((vx / b.fnot) ** 2 * x.w[1:-1]).sum() + ((uy / b.fnot) ** 2 * x.w[:, 1:-1]).sum())
        J.backward()
        return [out.detach(), psi.grad, curl.grad]
    return None      # the coupled loop's restatement is a model of its own
