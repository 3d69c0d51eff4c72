"""What a user of this library has it do, as cases that can be timed and compared.

A case goes through the public entry points only: the Python mirror of the C ABI
(unicorn_b200/unichem.py, surrogate.py) and, where the caller's data lives on the GPU,
uc_upload_fields_device and uc_device_view_get of include/unichem.h.

    listed()            the cases
    draw(rng)           one more case of the same ranges
    prepare(case, seed) what the caller has before the call: inputs, context, network
    run(state)          one pass, and its outputs
    work(case)          bytes and operations one pass cannot do without
    exact(case, seed)   the outputs in plain 64-bit torch, written from the mechanism data
"""
from __future__ import annotations

import ctypes
import json
import math
from pathlib import Path

import numpy as np
import torch

from unicorn_b200 import unichem
from unicorn_b200.surrogate import Surrogate, raw_features

LSP, LRX = 52, 544
DT, RELX, TOL, ISOR = 1e-3, 0.99, 1e-8, 100     # the reference's input card; DT = 1e-5 s
ATM = 1.01325e5
F64 = torch.float64
DEV = "cuda"


def F(x):
    """A default-REAL literal of the reference: single precision, promoted."""
    return float(np.float32(x))


# ------------------------------------------------------------------ cases

def listed():
    return [
        # a host program that asks for the source terms of one cell (a 0-D reactor, a point probe)
        dict(name="omega_1", kind="omega", n=1),
        # properties, cp and h along one line of a flame (101 points), on host arrays
        dict(name="props_101", kind="props", n=101),
        # rates and a species update that meets its tolerance, on a small ragged set of hot cells
        dict(name="update_2003", kind="update", n=2003, tol=1e-3),
        # one time step of the 101 x 61 methane jet on the host's own (pinned) arrays: the drop-in call
        dict(name="host_101x61", kind="sweep_host", nz=101, nr=61, fuel=13, precision=0),
        # the same call on the 601 x 301 heptane jet
        dict(name="host_601x301", kind="sweep_host", nz=601, nr=301, fuel=47, precision=0),
        # the heptane jet on the GPU in the mixed form
        dict(name="mixed_601x301", kind="sweep", nz=601, nr=301, fuel=47, precision=1),
        # the benchmark's headline: 1,048,576 heptane cells, 300-2400 K, FP64, state on the GPU
        dict(name="sweep_1m", kind="sweep", nz=0, nr=1 << 20, fuel=47, precision=0),
        # properties and source terms without an update, for a GPU-resident solver; ragged
        dict(name="chem_props_262143", kind="chem_props", n=262143, precision=0),
        # a whole step of a flame on the reference's 131 x 711 grid: faces, sweep, enthalpy equation, density
        dict(name="flame_131x711", kind="flame", lj=131, li=711),
        # stiff integration of independent hot cells over one step
        dict(name="integrate_32768", kind="integrate", n=32768),
        # the learned surrogate of omega, network alone
        dict(name="surrogate_500001", kind="surrogate", n=500001),
        # training the surrogate
        dict(name="train_8192x32", kind="train", n=65536, batch=8192, steps=32),
    ]


def draw(rng):
    def n(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    kind = rng.choice(["omega", "props", "update", "sweep_host", "sweep", "mixed", "chem_props", "flame", "integrate",
                       "surrogate", "train"])
    if kind == "omega":
        return dict(kind=kind, n=n(1, 2048))
    if kind == "props":
        return dict(kind=kind, n=n(16, 65536))
    if kind == "update":
        return dict(kind=kind, n=n(100, 65536), tol=rng.choice([1e-2, 1e-3, 1e-4]))
    if kind == "sweep_host":
        nr = n(17, 301)
        return dict(kind=kind, nz=n(33, 601), nr=nr, fuel=rng.choice([13, 30, 41, 47]), precision=0)
    if kind == "sweep":
        return dict(kind=kind, nz=0, nr=n(3000, 1 << 20), fuel=rng.choice([13, 30, 41, 47]), precision=0)
    if kind == "mixed":
        return dict(kind="sweep", nz=n(65, 601), nr=n(33, 301), fuel=rng.choice([13, 47]), precision=1)
    if kind == "chem_props":
        return dict(kind=kind, n=n(300, 1 << 19), precision=rng.choice([0, 0, 1]))
    if kind == "flame":
        return dict(kind=kind, lj=n(33, 131), li=n(65, 711))
    if kind == "integrate":
        return dict(kind=kind, n=n(200, 40000))
    if kind == "surrogate":
        return dict(kind=kind, n=n(4000, 1 << 20))
    return dict(kind=kind, n=65536, batch=rng.choice([2048, 4096, 8192]), steps=rng.randrange(16, 49))


def cells(case):
    return case["n"] if "n" in case else case["lj"] * case["li"] if "lj" in case else max(1, case["nz"]) * case["nr"]


# ------------------------------------------------------------------ inputs

def _uniform(g, lo, hi, *shape):
    return torch.rand(shape, dtype=F64, device=DEV, generator=g) * (hi - lo) + lo


def _normal(g, sd, *shape):
    return torch.randn(shape, dtype=F64, device=DEV, generator=g) * sd


def _jet(z, r, noise):
    return (torch.exp(-(r / (0.2 + 0.02 * z)) ** 2) + noise).clamp(0.0, 1.0)


def _mix(Z, fuel, g):
    """Fuel and air by mixture fraction, the other species log-uniform in [1e-10, 1e-3], renormalised
    (the composition of the repository's jet and batch generators)."""
    n = Z.shape[0]
    y = 10.0 ** _uniform(g, -10.0, -3.0, LSP, n)
    for k in (2, 6, 10, 52, fuel):
        y[k - 1] = 0.0
    y[fuel - 1] = Z
    y[1] = (1.0 - Z) * 0.233
    y[51] = (1.0 - Z) * 0.767
    return y / y.sum(0)


def _flame(lj, li, g):
    """A burning methane jet: fuel, oxidiser and products of complete burning by mixture fraction, radicals
    and CO in the hot layer, traces elsewhere; r (J) fastest."""
    zst = 0.0552
    z = torch.arange(li, dtype=F64, device=DEV)[:, None]
    r = torch.arange(lj, dtype=F64, device=DEV)[None, :] / (lj - 1)
    Z = _jet(20.0 * z / li, 2.0 * r, _normal(g, 1e-3, li, lj)).reshape(-1)
    hot = torch.where(Z < zst, Z / zst, ((1.0 - Z) / (1.0 - zst)).clamp(min=0.0) ** 4)
    y = 1e-12 * (1.0 + _uniform(g, 0.0, 1.0, LSP, Z.shape[0]))
    fuel = ((Z - zst) / (1.0 - zst)).clamp(min=0.0)
    burnt = Z - fuel
    y[12] = fuel
    y[1] = (0.233 * (1.0 - Z) - burnt * 64.0 / 16.04).clamp(min=0.0)
    y[9] = burnt * 44.01 / 16.04
    y[5] = burnt * 36.04 / 16.04
    y[51] = 0.767 * (1.0 - Z)
    for k, v in ((1, 1e-3), (3, 1e-4), (4, 4e-4), (5, 2e-3), (7, 1e-6), (9, 1e-2), (14, 1e-6)):
        y[k - 1] += v * hot ** 8
    return 300.0 + 1800.0 * hot, torch.full_like(Z, ATM), y / y.sum(0)


def _inputs(case, seed):
    """T (K), p (Pa) and Y [52, n] of a case, on the GPU."""
    g = torch.Generator(device=DEV).manual_seed(int(seed))
    kind, n = case["kind"], cells(case)
    if kind == "flame":
        return _flame(case["lj"], case["li"], g)
    if case.get("nz"):                                   # a jet on a (z, r) grid, r fastest
        z = torch.arange(case["nz"], dtype=F64, device=DEV)[:, None]
        r = torch.arange(case["nr"], dtype=F64, device=DEV)[None, :]
        Z = _jet(z, r, _normal(g, 0.02, case["nz"], case["nr"])).reshape(-1)
        T = 300.0 + 1900.0 * torch.exp(-((Z - 0.055) / 0.08) ** 2)
        return T, torch.full_like(T, ATM), _mix(Z, case["fuel"], g)
    lo = 1000.0 if kind in ("integrate", "update") else 300.0
    hi = 2000.0 if kind == "update" else 2400.0
    if kind == "update":                                 # air, methane and heptane, with traces of the rest
        y = 10.0 ** _uniform(g, -10.0, -3.0, LSP, n)
        y[1], y[51] = _uniform(g, 0.05, 0.23, n), 0.7
        y[12], y[46] = _uniform(g, 0.0, 0.1, n), _uniform(g, 0.0, 0.05, n)
        return _uniform(g, lo, hi, n), torch.full((n,), ATM, dtype=F64, device=DEV), y / y.sum(0)
    side = math.ceil(math.sqrt(n))                       # independent cells
    Z = _jet(_uniform(g, 0.0, side, n), _uniform(g, 0.0, 0.25 * side, n), _normal(g, 0.02, n))
    return _uniform(g, lo, hi, n), _uniform(g, 0.8 * ATM, 1.2 * ATM, n), _mix(Z, case.get("fuel", 47), g)


def _nondimensional(T, p, y, sc):
    tk = T / sc["TSTR"]
    wm = torch.tensor(_mech()["wsp"], dtype=F64, device=DEV) / 1000.0 / sc["WMSTR"]
    return tk, (p / sc["PSTR"]) / (sc["BETA1"] * tk * (y / wm[:, None]).sum(0))


# ------------------------------------------------------------------ state and passes

class _View(ctypes.Structure):
    """uc_device_view"""
    _fields_ = [(k, ctypes.c_void_p) for k in ("tk", "rho", "fsp", "fsp_old", "stmf", "stnd", "rc", "qdsp", "qdot",
                                               "domega_dy", "vmu", "vtc", "vdf", "cp", "h")] + \
               [("n", ctypes.c_int), ("npad", ctypes.c_int), ("stream", ctypes.c_void_p)]


class _Rows:
    """A context's device array as torch sees it; keeps the context alive."""

    def __init__(self, u, ptr, rows, npad):
        self.u = u
        self.__cuda_array_interface__ = dict(shape=(rows, npad) if rows > 1 else (npad,), typestr="<f8",
                                             data=(ptr, False), version=3)


def _device_outputs(u, names):
    v = _View()
    u.lib.uc_device_view_get.argtypes = [ctypes.c_void_p, ctypes.POINTER(_View)]
    u._ck(u.lib.uc_device_view_get(u._h, ctypes.byref(v)))
    many = ("fsp", "qdsp", "domega_dy", "vdf")
    return {k: torch.as_tensor(_Rows(u, getattr(v, k), LSP if k in many else 1, v.npad), device=DEV)[..., :v.n]
            for k in names}


def _pinned(*shape):
    return torch.empty(shape, dtype=F64, pin_memory=True)


class _State:
    def __init__(self, case, **kw):
        self.case = case
        self.__dict__.update(kw)


OUT = dict(qdsp=LSP, qdot=1, domega_dy=LSP, vmu=1, vtc=1, vdf=LSP, cp=1, h=1)


def prepare(case, seed):
    kind, n = case["kind"], cells(case)
    T, p, y = _inputs(case, seed)
    if kind == "train":
        return _prepare_train(case, T, p, y)
    u = unichem.UniChem(n)
    tk, rho = _nondimensional(T, p, y, u.scales)
    s = _State(case, u=u, tk=tk, rho=rho, y=y)
    if kind in ("omega", "props"):
        s.tk, s.rho, s.y = (t.cpu().numpy() for t in (tk, rho, y))
    elif kind == "sweep_host":
        for k, t in (("tk", tk), ("rho", rho), ("y", y)):
            setattr(s, k, _pinned(*t.shape).copy_(t))
        s.out = {k: _pinned(rows, n) if rows > 1 else _pinned(n) for k, rows in OUT.items()}
        s.y_out = _pinned(LSP, n)
        s.np = {k: t.numpy() for k, t in dict(s.out, tk_in=s.tk, rho_in=s.rho, y_in=s.y, y_out=s.y_out).items()}
    elif kind == "flame":
        lj, li = case["lj"], case["li"]
        d = 1.0 / (lj - 1)
        r, z = np.arange(lj)[None, :] * d, np.arange(li)[:, None] * 20.0 / li
        u_ax = (np.exp(-(2.0 * r / (0.2 + 0.02 * z)) ** 2) + 0.05).reshape(-1)
        v_rad = np.random.default_rng(seed).normal(0.0, 0.01, n)
        u.set_grid(lj, li, np.full(li, d), np.full(li, d), np.full(lj, d), np.full(lj, d),
                   np.tile((np.arange(lj) + 0.5) * d, li), isym=1)
        u.set_flow(u_ax, v_rad, 1e-3 * (0.1 + u_ax), 0.9)
        ht = _sensible(T, y, u.scales).cpu().numpy() + 0.5 * (u_ax ** 2 + v_rad ** 2)
        s.ht = ht
    elif kind in ("integrate", "surrogate"):
        u.set_pressure((p / u.scales["PSTR"]).cpu().numpy())
        if kind == "surrogate":
            s.net = Surrogate(capacity=0, seed=1)
            s.net.set_norm(**_norm(T, p, y, tk, rho, u.scales))
    torch.cuda.synchronize()
    return s


def _norm(T, p, y, tk, rho, sc, most=2048):
    """The surrogate's input and output scales from a sample of states, as a training program takes them."""
    m = min(most, T.shape[0])
    pick = lambda t: np.ascontiguousarray(t[..., :m].cpu().numpy())
    with unichem.UniChem(m) as u:
        u.upload(pick(tk), pick(rho), pick(y))
        q = u.omega().qdsp
    feats = raw_features(pick(T), pick(p) / (sc["PBACK"] * sc["PSTR"]), pick(y))
    return Surrogate.norm_from_sample(feats, q)


def _prepare_train(case, T, p, y):
    n = case["n"]
    net = Surrogate(capacity=n, seed=1)
    with unichem.UniChem(n) as u:
        tk, rho = _nondimensional(T, p, y, u.scales)
        torch.cuda.synchronize()
        u.upload_device(tk.data_ptr(), rho.data_ptr(), y.data_ptr())
        u.set_pressure((p / u.scales["PSTR"]).cpu().numpy())
        net.set_norm(**_norm(T, p, y, tk, rho, u.scales))
        net.add_data(u)
        u.sync()
    return _State(case, net=net)


def run(s):
    case, kind = s.case, s.case["kind"]
    if kind == "train":
        loss = s.net.train(steps=case["steps"], batch=case["batch"], lr=1e-3, seed=3)
        return {"loss": loss, "params": s.net.params()}
    u = s.u
    if kind == "omega":
        u.upload(s.tk, s.rho, s.y)
        o = u.omega()
        return {"qdsp": o.qdsp, "qdot": o.qdot, "domega_dy": o.domega_dy}
    if kind == "props":
        u.upload(s.tk, s.rho, s.y)
        mu, lam, d = u.props()
        cp, h = u.cp_h()
        return {"vmu": mu, "vtc": lam, "vdf": d, "cp": cp, "h": h}
    if kind == "sweep_host":
        a = s.np
        passes = u.sweep_host(a["tk_in"], a["rho_in"], a["y_in"], out={k: a[k] for k in OUT}, y_out=a["y_out"], dt=DT,
                              precision=case["precision"], isor=ISOR, relx=RELX, tol=TOL)
        return dict(s.out, fsp=s.y_out, passes=passes)
    u.upload_device(s.tk.data_ptr(), s.rho.data_ptr(), s.y.data_ptr())
    if kind == "update":
        u.ckrates()
        passes = u.solvesp(DT, isor=ISOR, relx=RELX, tol=case["tol"])
        return dict(_device_outputs(u, ["fsp"]), passes=passes)
    if kind == "sweep":
        passes = u.sweep(DT, precision=case["precision"], isor=ISOR, relx=RELX, tol=TOL)
        return dict(_device_outputs(u, list(OUT) + ["fsp"]), passes=passes)
    if kind == "chem_props":
        u.chem_props(case["precision"])
        return _device_outputs(u, OUT)
    if kind == "flame":
        u.set_enthalpy(s.ht)
        passes = u.sweep(DT, isor=ISOR, relx=RELX, tol=TOL)
        h_passes, resdh = u.enthalpy_update(DT, isor=ISOR, relx=RELX, tol=TOL, sigh=0.9)
        u.density()
        return dict(_device_outputs(u, ["tk", "rho", "fsp", "qdot", "vmu", "vtc", "vdf", "cp"]), passes=passes,
                    h_passes=h_passes, resdh=resdh)
    if kind == "integrate":
        u.integrate(DT, isor=ISOR, relx=RELX, tol=TOL)
        return _device_outputs(u, ["tk", "rho", "fsp"])
    s.net.omega(u, tol=float("inf"), stats=False)
    return _device_outputs(u, ["qdsp"])


# ------------------------------------------------------------------ what a pass cannot do without

# operations per cell: the rates, omega and d(omega)/dY (each +, *, / and transcendental one), the transport
# sums of a sub-mixture of about five species, cp and h; per cell and pass of the update, its 2,132 products
# and sums (one multiply-add each) and the 51 closing quotients
RATES, PROPS, CPH, PASS = 9500, 6000, 1100, 2 * 2132 + 51 * 16
# passes and sub-steps taken where the inputs decide them (seen on these inputs)
UPDATE_PASSES, SUBSTEPS, SUBSTEP_PASSES = 30, 60, 4


def work(case):
    kind, n = case["kind"], cells(case)
    row = 8.0 * n
    if kind == "omega":
        return {"bytes": row * (54 + 105), "flops": n * RATES}
    if kind == "props":
        return {"bytes": row * (54 + 56), "flops": n * (PROPS + CPH)}
    if kind == "update":
        return {"bytes": row * (54 + 52), "flops": n * (RATES + UPDATE_PASSES * PASS)}
    if kind in ("sweep", "sweep_host"):
        return {"bytes": row * (54 + 161 + 52), "flops": n * (RATES + PROPS + CPH + ISOR * PASS)}
    if kind == "chem_props":
        return {"bytes": row * (54 + 161), "flops": n * (RATES + PROPS + CPH)}
    if kind == "flame":
        return {"bytes": row * (54 + 5 + 111), "flops": n * (RATES + PROPS + CPH + 2000 + ISOR * PASS)}
    if kind == "integrate":
        return {"bytes": row * (55 + 54), "flops": n * SUBSTEPS * (RATES + SUBSTEP_PASSES * PASS)}
    weights = 64 * 256 + 3 * 256 * 256 + 256 * 64
    if kind == "surrogate":
        return {"bytes": row * (55 + 52), "flops": 2.0 * n * weights}
    return {"bytes": case["steps"] * (case["batch"] * 512.0 + weights * 16), "flops": 6.0 * case["steps"] * case["batch"] * weights}


# ------------------------------------------------------------------ the outputs in plain 64-bit torch

_MECH = {}


def _mech():
    if not _MECH:
        path = Path(unichem.__file__).resolve().parent / "mech" / "sandiego52.json"
        _MECH.update(json.loads(path.read_text()))
    return _MECH


class _Exact:
    """The mechanism's functions of (tk, rho, Y) in 64 bits, from the mechanism data alone: the rate
    expressions, source terms, mixture properties and the point-implicit update as the equations have them."""

    def __init__(self, T, p, y):
        m = self.m = _mech()
        W = np.array(m["wsp"])
        ru, inp = F(8.3144), dict(rtot=0.1, vref=10.0, tref=294.0, pref=1.0133e5, fo2=0.233)
        wref = 1.0 / (inp["fo2"] / W[1] + (1.0 - inp["fo2"]) / W[51]) / 1000.0
        rref = inp["pref"] / (ru / wref) / inp["tref"]
        self.gasc, self.wmstr, self.rstr, self.tstr = ru, wref, rref, inp["tref"]
        self.hstr = inp["vref"] ** 2
        pstr = rref * inp["vref"] ** 2
        self.pback = inp["pref"] / pstr
        self.amref = 5.69428e-07 * inp["tref"] ** F(0.62245)
        acref = 2.78763e-04 * inp["tref"] ** F(0.796783)
        t = inp["tref"]
        self.convrc = F(418.68) * 1.9891e-04 * math.sqrt(t / 1000.0 / wref) / acref
        self.convrm = F(0.1) * 2.6693e-05 * math.sqrt(1000.0 * wref * t) / self.amref
        self.convrd = F(0.02628) * t * math.sqrt(t) / pstr / math.sqrt(wref * 1000.0) / 1.2e-04
        self.c = [0.0] + [inp["rtot"] / inp["vref"] * (rref / wref * 1e-6) ** i for i in range(3)]
        self.rconv = inp["vref"] / wref / inp["rtot"] * 1e-6
        self.wm = W / 1000.0 / wref
        self.poly = torch.tensor(m["poly"], dtype=F64, device=DEV)
        sc = dict(TSTR=t, PSTR=pstr, WMSTR=wref, BETA1=ru * rref * t / pstr / wref)
        self.tk, self.rho = _nondimensional(T, p, y, sc)
        self.T, self.y, self.n = self.tk * t, y.clone(), T.shape[0]
        self.wmt = torch.tensor(self.wm, dtype=F64, device=DEV)[:, None]
        self.low = (self.T <= m["tpol"][0])

    def clip(self):
        self.y[:51].clamp_(min=0.0)
        self.y[51] = 1.0 - self.y[:51].sum(0)

    def nasa(self, k, hot=None):
        """The seven NASA coefficients of species k (0-based) per cell."""
        hot = ~self.low if hot is None else hot
        return torch.where(hot[None, :], self.poly[k, 7:, None], self.poly[k, :7, None])

    def cp_h(self):
        T, cp, h = self.T, torch.zeros_like(self.T), torch.zeros_like(self.T)
        for k in range(LSP):
            a = self.nasa(k)
            cpk = a[0] + T * (a[1] + T * (a[2] + T * (a[3] + T * a[4])))
            cp += cpk / self.wm[k] * self.y[k]
            h += self.henth(k) * self.y[k]
        return cp / self.wmstr * self.gasc * self.tstr / self.hstr, h

    def henth(self, k):
        a, T = self.nasa(k), self.T
        return (T * (a[0] + T * (a[1] / 2 + T * (a[2] / 3 + T * (a[3] / 4 + T * a[4] / 5)))) + a[5]) / self.wm[k] * self.gasc

    def rates(self):
        m, T, y, rho = self.m, self.T, self.y, self.rho
        lnT, cal = torch.log(T), F(1.9872)
        gibbs = []
        for k in range(LSP):
            a = self.nasa(k)
            gibbs.append(a[0] * (lnT - 1.0) + a[1] * T / 2 + a[2] * T ** 2 / 6 + a[3] * T ** 3 / 12 +
                         a[4] * F(1.2) / 24 * T ** 4 - a[5] / T + a[6])
        tb = {"TBODY": (y / self.wmt).sum(0)}
        for name, terms in m["tb"].items():
            if name != "TBODY":
                tb[name] = tb["TBODY"] + sum(s * (1.0 if c is None else c) * y[k - 1] / self.wm[k - 1] for s, k, c in terms[1:])
        mole = rho * self.rstr / self.wmstr * 1e-6
        rc = torch.zeros((LRX, self.n), dtype=F64, device=DEV)
        for f in range(0, LRX, 2):
            R = m["reactions"][f]
            kf = abs(R["akf"]) * torch.exp(R["alf"] * lnT - R["exaf"] / cal / T)
            kr = torch.zeros_like(kf)
            rev = m["reverse"].get(str(f + 2))
            if rev:
                g = sum(gibbs[s - 1] if op == "*" else -gibbs[s - 1] for op, s in rev["q"])
                kr = kf * torch.exp(-g) * (F(82.06) * T) ** rev["rut"]
            if R["akf"] < 0 and R["aklow"] != 0.0:                  # fall-off
                t1, t2, t3, t4 = R["troe"]
                pr = R["aklow"] * torch.exp(R["allow"] * lnT - R["ealow"] / cal / T) * tb[m["dmole"].get(str(f + 1), "TBODY")] * mole / (kf + 1e-20)
                blend = torch.ones_like(pr)
                if t1 > 0.0:
                    fc = (torch.full_like(T, math.log10(t1)) if t2 == 0.0 else
                          torch.log10((1.0 - t1) * torch.exp(-T / t2) + t1 * torch.exp(-T / t3) + torch.exp(-t4 / T)))
                    c = torch.log10(pr) - (F(0.4) + F(0.67) * fc)
                    blend = 10.0 ** (fc / (1.0 + (c / (F(0.75) - F(1.27) * fc - F(0.14) * c)) ** 2))
                elif t1 < 0.0:
                    blend = (-t1 * torch.exp(-t2 / T) + torch.exp(-T / t3)) ** (1.0 / (1.0 + torch.log10(pr) ** 2))
                blend = blend * pr / (1.0 + pr)
                kf, kr = kf * blend, kr * blend
            for r, k in ((f, kf), (f + 1, kr)):
                a = m["rc"].get(str(r + 1))
                if a is None:
                    continue
                v = self.c[a["order"]] * rho ** a["order"] * k
                if a["tb"] is not None:
                    v = v * tb[a["tb"]]
                for op, what, i in a["post"]:
                    v = v * y[i - 1] if what == "Y" else v / self.wm[i - 1]
                rc[r] = v
        self.tbody, self.rc = tb["TBODY"], rc

    def omega(self):
        m, y = self.m, self.y
        ra = self.rc.clone()
        for r in range(LRX):
            sp = m["ra"][str(r + 1)]
            if sp is None:
                ra[r] = 0.0
            for k in sp or ():
                ra[r] *= y[k - 1]
        q, d = torch.zeros_like(y), torch.zeros_like(y)
        qdot = torch.zeros_like(self.T)
        for k in range(LSP):
            acc, loss = torch.zeros_like(self.T), torch.zeros_like(self.T)
            for s, fac in m["prd"][str(k + 1)] or ():
                if fac[-1][0] != "RA":
                    continue
                r = fac[-1][1] - 1
                acc += s * (fac[0][1] if len(fac) > 1 else 1.0) * ra[r]
                if s < 0:
                    sp = list(m["ra"][str(r + 1)])
                    if k + 1 in sp:
                        sp.remove(k + 1)
                    v = self.rc[r]
                    for j in sp:
                        v = v * y[j - 1]
                    loss += v
            q[k] = -self.rconv * self.wm[k] * acc
            d[k] = -self.rconv * self.wm[k] * loss
            qdot += q[k] * self.henth(k)
        return q, qdot, d

    def props(self):
        m, T, y = self.m, self.T, self.y
        hot = T >= m["tpol"][0]
        sub = y >= 1e-3
        sub[51] = True
        x = torch.where(sub, y, torch.zeros_like(y)) / self.wmt
        x[51] = (1.0 - torch.where(sub[:51], y[:51], torch.zeros_like(y[:51])).sum(0)) / self.wm[51]
        mole = x.sum(0)
        w, dia, tlj = self.wm, np.array(m["cdia"]), np.array(m["tlj"])
        om = torch.tensor(m["omega22"], dtype=F64, device=DEV)
        atc, amu = torch.empty_like(y), torch.empty_like(y)
        rt = torch.sqrt(self.tk)
        for k in range(LSP):
            a = self.nasa(k, hot)
            b = torch.where(hot[None, :], om[k, 6:, None], om[k, :6, None])
            eu = F(0.115) + F(0.354) * (a[0] + T * (a[1] + T * (a[2] + T * (a[3] + T * a[4]))))
            si = dia[k] ** 2 * (b[0] + T * (b[1] + T * (b[2] + T * (b[3] + T * (b[4] + T * b[5])))))
            atc[k] = self.convrc * eu * rt / math.sqrt(w[k]) / si
            amu[k] = self.convrm * rt * math.sqrt(w[k]) / si
        col = lambda v: torch.tensor(v, dtype=F64, device=DEV)[:, None]
        ci = torch.tensor(m["ci11"], dtype=F64, device=DEV)
        vtc, vmu, vdf = torch.zeros_like(T), torch.zeros_like(T), torch.empty_like(y)
        base = self.tk * rt / self.pback
        for k in range(LSP):
            t = T[None, :] / col(np.sqrt(tlj[k] * tlj))
            c = ci[(t >= 2.0).to(torch.int64) + (t > 5.0) + (t > 70.0)]
            c = c[..., 0] + t * (c[..., 1] + t * (c[..., 2] + t * (c[..., 3] + t * c[..., 4])))
            ec = 0.5 * (dia[k] + dia)
            inv = c / (col(np.sqrt((w[k] + w) / 2.0 / w[k] / w) / ec / ec) * base)      # 1 / D_kb
            others = x.clone()
            others[k] = 0.0
            wk, dw = col((w[k] / w) ** 0.25), col(F(2.828427125) * np.sqrt(1.0 + w[k] / w))
            phi = (others * (1.0 + torch.sqrt(atc[k] / atc) * wk) ** 2 / dw).sum(0)
            psi = (others * (1.0 + torch.sqrt(amu[k] / amu) * wk) ** 2 / dw).sum(0)
            here = sub[k]
            vtc += torch.where(here, atc[k] * x[k] / (x[k] + F(1.065) * phi), torch.zeros_like(T))
            vmu += torch.where(here, amu[k] * x[k] / (x[k] + psi), torch.zeros_like(T))
            out = mole / (x * inv).sum(0)
            if k < 51:
                alone = torch.where(mole - x[k] <= 1e-10, 1.0 / inv[51], (mole - x[k]) / (others * inv).sum(0))
                out = torch.where(here, alone, out)
            vdf[k] = self.convrd * out
        return vmu, vtc, vdf

    def update(self, isor, tol):
        """The reference's A-term program, pass after pass (no soot at the start, no transport)."""
        y, rc, rho, y0 = self.y, self.rc, self.rho, self.y.clone()
        A, one = {}, torch.zeros_like(self.T)
        A_rc = [rc[r] for r in range(LRX)]
        Y = [y[k].clone() for k in range(LSP)]
        # without soot the only source left is its inception from C2H2
        inception = self.c[1] * rho * 1e4 * torch.exp(-2.0632e4 / self.T) / self.wm[21]
        soot = one

        def chain(fac):
            v, c = None, 1.0
            for f in fac:
                if f[0] == "num":
                    c *= f[1]
                    continue
                if (f[0] == "SOUR" and f[1] != 1) or (f[0] == "A" and A[f[1]] is None):
                    return None
                x = inception if f[0] == "SOUR" else A_rc[f[1] - 1] if f[0] == "RC" else A[f[1]] if f[0] == "A" else y0[f[1] - 1] if f[0] == "Y0" else Y[f[1] - 1]
                v = x if v is None else v * x
            return None if v is None or c == 0.0 else v if c == 1.0 else c * v

        def total(terms):
            acc = one.clone()
            for s, fac in terms:
                v = chain(fac)
                if v is not None:
                    acc.add_(v, alpha=s)
            return acc

        passes = isor + 1
        for it in range(1, isor + 1):
            res, prod = one.clone(), one
            for b in self.m["update"]["blocks"]:
                k = b["species"] - 1
                for r, fac in b["recompute"]:
                    A[r] = chain(fac)
                if b["prod"] is not None:
                    prod = total(b["prod"])
                rhs = rho * y0[k] + DT * self.wm[k] * (prod + total(b["extra"]))
                den = rho if b["loss"] is None else rho + DT * self.wm[k] * total(b["loss"])
                new = (1.0 - RELX) * Y[k] + rhs * RELX / den
                res += (Y[k] - new).abs()
                Y[k] = new.clamp(min=0.0)
                for r in b["multiply"]:
                    if A[r] is not None:
                        A[r] = Y[k] * A[r]
            new = (1.0 - RELX) * soot + DT * (F(0.012011) / self.wmstr) * 2.0 * inception * Y[21] * RELX / rho
            res += (soot - new).abs()
            soot = new
            if float(res.sum()) / (self.n * 51.0) <= tol:
                passes = it
                break
        y = torch.stack(Y)
        total_y = y[:51].sum(0) + soot
        over = total_y > 1.0
        y[:51] = torch.where(over[None, :], y[:51] / total_y, y[:51])
        y[51] = torch.where(over, one, 1.0 - total_y)
        self.y = y
        return passes


def _sensible(T, y, sc):
    """Non-dimensional sensible enthalpy (without formation enthalpies) of a state."""
    wm = np.array(_mech()["wsp"]) / 1000.0 / sc["WMSTR"]
    poly = torch.tensor(_mech()["poly"], dtype=F64, device=DEV)
    out = torch.zeros_like(T)
    for k in range(LSP):
        a = torch.where((T > 1000.0)[None, :], poly[k, 7:, None], poly[k, :7, None])
        h = T * (a[0] + T * (a[1] / 2 + T * (a[2] / 3 + T * (a[3] / 4 + T * a[4] / 5)))) + a[5] - poly[k, 5]
        out += y[k] / wm[k] * h
    return out * sc["GASC"] / sc["WMSTR"] / sc["HSTR"]


def exact(case, seed):
    """None for the whole steps and integrations that only iterate to a tolerance, and for the BF16 network."""
    kind = case["kind"]
    if kind in ("flame", "integrate", "surrogate", "train"):
        return None
    e = _Exact(*_inputs(case, seed))
    out = {}
    if kind in ("props", "chem_props", "sweep", "sweep_host"):
        e.clip()
        out["vmu"], out["vtc"], out["vdf"] = e.props()
        out["cp"], out["h"] = e.cp_h()
    if kind != "props":
        e.rates()
    if kind not in ("props", "update"):
        out["qdsp"], out["qdot"], out["domega_dy"] = e.omega()
    if kind in ("update", "sweep", "sweep_host"):
        out["passes"] = e.update(ISOR, case.get("tol", TOL))
        out["fsp"] = e.y
    return out
