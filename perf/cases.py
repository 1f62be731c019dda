"""What a user of gelios_2d_b200 has it do, as cases whose passes can be timed.

A case is a dict of plain values.  ``kind`` names the call:

``mk2``      one ``Go_5_komponent__MK2`` call of ``steps`` steps on the rail
             grid ``Setka(N1..M4)``, then the new points read back (a driver
             that alternates with the Monte Carlo transport needs both)
``stream``   one-step MK2 calls that take a fresh state from host memory and
             return the result to it (``run_streamed``)
``inner``    ``Go_stationary_5_komponent_inner_MK2`` on the inner region
``k5``       ``Go_5_komponent``: plasma and four hydrogen fluids
``mhd``      ``Go_MHD_pickup``, FP64 or FP32 fluxes, results read back
``sweep``    the batched MHD sweep: instances of uneven size, one call for all
``plain``    ``Go_stationary`` on the polar half-plane grid
``march``    a batch of plain instances marched by
             ``gelios_plain_batch_run_to_residual``
``train``    Adam steps of the warm-start network
``predict``  the network evaluated on every cell of a grid

Grids, states and Monte-Carlo moments come from ``gelios_2d_b200.workloads``
(the rail grids) or from the formulas below (the polar grid), with seeded
variations of the densities.  Every step call restarts dt, as the reference
does, and goes on from the state the call before left.
"""
from __future__ import annotations

import ctypes as C
import functools
import math

import numpy as np
import torch

from gelios_2d_b200 import _native as N
from gelios_2d_b200 import warmstart as WS
from gelios_2d_b200 import workloads as W
from gelios_2d_b200.mesh import Mesh
from gelios_2d_b200.setka import Setka
from gelios_2d_b200.sweep import MIN_DIMS, Sweep, inflow_params

LISM_CELL = 4  # Cell_type C_5: the cells Init_conditions fills with the inflow state


def _grid(dims) -> str:
    return " ".join(str(d) for d in dims)


def _scaled(f: float) -> str:
    """The ~200k-cell rail grid with every count scaled by f."""
    return _grid(max(lo, round(b * f)) for b, lo in zip(W.SETKA_200K, MIN_DIMS))


def listed() -> list[dict]:
    return [
        # small grids while a set-up is tried out: launches and latency count
        {"name": "mk2_8k", "kind": "mk2", "grid": _grid(W.SETKA_SMALL), "steps": 10},
        # the reference driver's main loop at production resolution
        {"name": "mk2_1m", "kind": "mk2", "grid": _grid(W.SETKA_1M), "steps": 20},
        # a host code coupled to every step (the end-to-end benchmark's call)
        {"name": "stream_200k", "kind": "stream", "grid": _grid(W.SETKA_200K), "steps": 4},
        # the inner region's long loop beside the moving grid
        {"name": "inner_200k", "kind": "inner", "grid": _grid(W.SETKA_200K), "steps": 50},
        # the four-fluid run of the same grid
        {"name": "k5_200k", "kind": "k5", "grid": _grid(W.SETKA_200K), "steps": 20},
        # ion MHD + pickup protons, the FP64 form
        {"name": "mhd_200k", "kind": "mhd", "grid": _grid(W.SETKA_200K), "steps": 20, "precision": N.PREC_FP64},
        # the same physics at production resolution with FP32 fluxes
        {"name": "mhd_1m_fp32", "kind": "mhd", "grid": _grid(W.SETKA_1M), "steps": 20,
         "precision": N.PREC_FP32_FLUX},
        # parameter sweep over uneven grids
        {"name": "sweep_8", "kind": "sweep", "instances": 8, "lo": 0.5, "hi": 1.4, "steps": 4},
        # single-fluid runs on the polar grid
        {"name": "plain_180x120", "kind": "plain", "n_theta": 180, "n_r": 120, "steps": 100,
         "precision": N.PREC_FP64},
        # warm-started sweep marched to a steady state
        {"name": "march_32x90x60", "kind": "march", "n_theta": 90, "n_r": 60, "instances": 32, "steps": 200,
         "precision": N.PREC_FP32_WAVES},
        # training and evaluation of the warm-start network
        {"name": "train_8192", "kind": "train", "batch": 8192, "iters": 20, "rows": 86400},
        {"name": "predict_5400", "kind": "predict", "rows": 5400},
    ]


def _between(rng, lo: float, hi: float) -> float:
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng) -> dict:
    kind = rng.choice(["mk2", "mk2", "stream", "inner", "k5", "mhd", "mhd", "sweep", "plain", "march", "train",
                       "predict"])
    if kind == "mk2":
        return {"kind": kind, "grid": _scaled(_between(rng, 0.2, 2.0)), "steps": rng.randint(1, 20)}
    if kind == "stream":
        return {"kind": kind, "grid": _scaled(_between(rng, 0.2, 1.4)), "steps": rng.randint(1, 6)}
    if kind == "inner":
        return {"kind": kind, "grid": _scaled(_between(rng, 0.2, 1.4)), "steps": rng.randint(10, 60)}
    if kind == "k5":
        return {"kind": kind, "grid": _scaled(_between(rng, 0.2, 1.2)), "steps": rng.randint(1, 20)}
    if kind == "mhd":
        return {"kind": kind, "grid": _scaled(_between(rng, 0.2, 1.8)), "steps": rng.randint(1, 20),
                "precision": rng.choice([N.PREC_FP64, N.PREC_FP32_FLUX])}
    if kind == "sweep":
        lo = rng.uniform(0.2, 0.6)
        return {"kind": kind, "instances": rng.randint(2, 10), "lo": lo, "hi": lo + rng.uniform(0.1, 0.7),
                "steps": rng.randint(1, 4)}
    if kind == "plain":
        return {"kind": kind, "n_theta": rng.randint(40, 360), "n_r": rng.randint(30, 240),
                "steps": rng.randint(20, 120),
                "precision": rng.choice([N.PREC_FP64, N.PREC_FP64, N.PREC_FP32_FLUX, N.PREC_FP32_WAVES])}
    if kind == "march":
        return {"kind": kind, "n_theta": rng.randint(40, 120), "n_r": rng.randint(30, 90),
                "instances": rng.randint(4, 40), "steps": 4 * rng.randint(10, 50),
                "precision": rng.choice([N.PREC_FP64, N.PREC_FP32_WAVES])}
    if kind == "train":
        return {"kind": kind, "batch": round(_between(rng, 500, 8192)), "iters": rng.randint(5, 20),
                "rows": round(_between(rng, 5400, 200000))}
    return {"kind": kind, "rows": round(_between(rng, 300, 43200))}


# ---------------------------------------------------------------- inputs
@functools.lru_cache(maxsize=64)
def _rail_mesh(grid: str):
    mesh = Mesh.setka(*(int(d) for d in grid.split()))
    return mesh, W.init_conditions_reference(mesh)


def _modulated(mesh, st, seed: int):
    """st with its density varied by up to 2% with the polar angle."""
    rng = np.random.RandomState(seed % 2**32)
    th = np.arctan2(mesh["y"][mesh["contour"][mesh["contour_start"][:-1]]],
                    mesh["x"][mesh["contour"][mesh["contour_start"][:-1]]])
    out = st.copy()
    out[0] *= 1.0 + 0.02 * rng.uniform(-1, 1) * np.cos(rng.randint(1, 4) * th + rng.uniform(0, 6))
    return out


def _pinned(*shape):
    return torch.empty(shape, dtype=torch.float64, pin_memory=True).numpy()


class _DeviceRows:
    """A state buffer of a context as an array on the GPU."""

    def __init__(self, S: Setka, buf: int):
        p = C.POINTER(C.c_double)()
        N.check(S._L.gelios_state_device_ptr(S._h, buf, C.byref(p)), "gelios_state_device_ptr")
        self.owner = S
        self.__cuda_array_interface__ = {"shape": (5, S.mesh.n_cells), "typestr": "<f8", "version": 2,
                                         "data": (C.cast(p, C.c_void_p).value, False)}


def _rows(S: Setka):
    return [torch.as_tensor(_DeviceRows(S, b), device="cuda") for b in (0, 1)]


def _mhd_inputs(S: Setka, st, mp, seed: int):
    S.set_mhd_params(mp)
    x8 = W.mhd_initial(S.mesh, st, mp)
    S.set_mhd(0, x8)
    S.set_mhd(1, x8)
    S.set_sources(*W.mhd_sources(S.mesh, seed=seed))


def _polar_instance(case, rng):
    """Inflow and inner-wind parameters: the plain workload's, or a sweep's draw."""
    p = W.plain_params() if case["kind"] == "plain" else WS.inflow_params(
        WS.PARAM_LO + rng.uniform(size=5) * (WS.PARAM_HI - WS.PARAM_LO))
    p.precision = case["precision"]
    return p


def _polar_inputs(case, seed: int):
    """Parameters and initial states of the instances of a plain/march case:
    the inner solution inside r = 150, the inflow beyond, 1% density noise."""
    rng = np.random.RandomState(seed % 2**32)
    g = _Polar(case["n_theta"], case["n_r"])
    r = np.sqrt(g.cx**2 + g.cy**2)
    prm, sts = [], []
    for _ in range(case.get("instances", 1)):
        p = _polar_instance(case, rng)
        inner = r < 150.0
        st = np.empty((5,) + r.shape)
        st[0] = np.where(inner, 1.0 / (p.chi * r) ** 2, p.in_ro)
        st[1] = np.where(inner, r ** (-2.0 * p.gamma) / (p.gamma * p.inner_mach**2), p.in_p)
        st[2] = np.where(inner, p.chi * g.cx / r, p.in_u)
        st[3] = np.where(inner, p.chi * g.cy / r, p.in_v)
        st[4] = np.where(inner, st[0], p.in_Q)
        st[0] *= 1.0 + 0.01 * rng.uniform(-1, 1, size=r.shape)
        prm.append(p)
        sts.append(st.reshape(5, -1))
    return prm, sts


def _network_rows(rows: int, seed: int):
    """Raw inputs of `rows` cells (five scaled inflow parameters, scaled log
    radius and polar angle) and standardised smooth targets."""
    rng = np.random.RandomState(seed % 2**32)
    x = rng.uniform(-1, 1, size=(rows, 7)).astype(np.float32)
    a = rng.normal(size=(7, 5))
    t = np.tanh(x @ a) + 0.3 * np.sin(3.0 * x[:, 5:6]) * np.cos(2.0 * x[:, 6:7])
    return x, (t / t.std(axis=0)).astype(np.float32)


def _network_params(seed: int):
    """Flat parameters of the 31 -> 5 x 256 -> 5 network and its layer sizes."""
    rng = np.random.RandomState((seed + 1) % 2**32)
    sizes = [31] + [256] * 5 + [5]
    flat = []
    for i, o in zip(sizes[:-1], sizes[1:]):
        flat += [rng.uniform(-1, 1, size=o * i) / math.sqrt(i), np.zeros(o)]
    return np.concatenate(flat).astype(np.float32), sizes


def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    s = {"case": case}
    if kind in ("mk2", "stream", "inner", "k5", "mhd"):
        mesh, st0 = _rail_mesh(case["grid"])
        st = _modulated(mesh, st0, seed)
        S = s["S"] = Setka(mesh, N.reference_params(precision=case.get("precision", N.PREC_FP64)))
        S.set_par(0, st)
        S.set_par(1, st)
        s["x"], s["y"] = _pinned(mesh.n_points), _pinned(mesh.n_points)
        if kind in ("mk2", "stream", "inner"):
            S.set_mc(*W.mc_fields(mesh, seed=seed))
        if kind == "inner":
            S.build_inner_list()
        if kind == "k5":
            h = W.hydrogen_fields(mesh, seed=seed)
            S.set_hydrogen(0, h)
            S.set_hydrogen(1, h)
            s["extra"] = _pinned(16 * mesh.n_cells)
        if kind == "mhd":
            _mhd_inputs(S, st, W.mhd_params(), seed)
            s["extra"] = _pinned(8 * mesh.n_cells)
        if kind == "stream":
            s["in"] = [_pinned(5, mesh.n_cells) for _ in range(case["steps"])]
            s["out"] = [_pinned(5, mesh.n_cells) for _ in range(case["steps"])]
            for k, a in enumerate(s["in"]):
                a[:] = st
                a[0] *= 1.0 + 0.001 * k
        else:
            s["rows"] = _rows(S)
    elif kind == "sweep":
        rng = np.random.RandomState(seed % 2**32)
        inst, n = [], case["instances"]
        for i in range(n):
            f = case["lo"] + (case["hi"] - case["lo"]) * ((i * 0.618034) % 1.0)
            mesh, st0 = _rail_mesh(_scaled(f))
            inflow = inflow_params(rng.uniform(size=5))
            p = N.reference_params(in_ro=inflow["in_ro"], in_p=inflow["in_p"], in_u=inflow["in_u"],
                                   precision=N.PREC_FP32_FLUX)
            st = st0.copy()
            lism = mesh["cell_type"] == LISM_CELL
            st[0][lism], st[1][lism], st[2][lism], st[3][lism] = p.in_ro, p.in_p, p.in_u, 0.0
            mp = W.mhd_params(b_lism=inflow["b_lism"], b_angle_deg=inflow["b_angle_deg"])
            inst.append((mesh, p, st, (mp, W.mhd_initial(mesh, st, mp), W.mhd_sources(mesh, seed=seed + i))))
        s["sweep"] = Sweep(inst, form=N.FORM_MHD_PUI, batched=True)
        s["rows"] = [_rows(S) for S in s["sweep"].items]
        s["extra"] = [_pinned(8 * S.mesh.n_cells) for S in s["sweep"].items]
    elif kind in ("plain", "march"):
        mesh = Mesh.polar(case["n_theta"], case["n_r"])
        prm, sts = _polar_inputs(case, seed)
        s["items"] = [Setka(mesh, p) for p in prm]
        for S, st in zip(s["items"], sts):
            S.set_par(0, st)
            S.set_par(1, st)
        s["rows"] = [_rows(S) for S in s["items"]]
        if kind == "march":
            n = len(prm)
            s["batch"] = _PlainBatch(s["items"])
            s["done"], s["res"], s["dts"] = np.zeros(n, np.int64), np.zeros(n), np.zeros(n)
    else:
        net = s["net"] = WS.Mlp()
        net.set_params(_network_params(seed)[0])
        x, t = _network_rows(case["rows"], seed)
        s["x"] = x
        if kind == "train":
            net.set_data(x, t)
    return s


class _PlainBatch:
    def __init__(self, items):
        self.L = N.lib()
        self.items = items
        arr = (C.c_void_p * len(items))(*[S._h.value for S in items])
        self.h = C.c_void_p()
        N.check(self.L.gelios_plain_batch_create(C.byref(self.h), arr, len(items)), "gelios_plain_batch_create")

    def __del__(self):
        self.L.gelios_plain_batch_destroy(self.h)


# ---------------------------------------------------------------- one pass
def run(s: dict):
    case = s["case"]
    kind = case["kind"]
    L = N.lib()
    if kind in ("mk2", "inner", "k5", "mhd"):
        S, n = s["S"], case["steps"]
        step = {"mk2": S.Go_5_komponent__MK2, "inner": S.Go_stationary_5_komponent_inner_MK2,
                "k5": S.Go_5_komponent, "mhd": S.Go_MHD_pickup}[kind]
        st = step(n)
        out = {"state": s["rows"][n % 2], "dt": float(st.dt), "flags": int(st.flags)}
        if kind == "k5":
            N.check(L.gelios_download_hydrogen(S._h, n % 2, s["extra"]), "gelios_download_hydrogen")
            out["extra"] = s["extra"]
        if kind == "mhd":
            N.check(L.gelios_download_mhd(S._h, n % 2, s["extra"]), "gelios_download_mhd")
            out["extra"] = s["extra"]
        if kind != "inner":
            N.check(L.gelios_download_points(S._h, s["x"], s["y"]), "gelios_download_points")
            out["x"], out["y"] = s["x"], s["y"]
        return out
    if kind == "stream":
        s["S"].run_streamed(N.FORM_MK2, s["in"], s["out"])
        N.check(L.gelios_download_points(s["S"]._h, s["x"], s["y"]), "gelios_download_points")
        return {"state": s["out"], "x": s["x"], "y": s["y"]}
    if kind == "sweep":
        n = case["steps"]
        st = s["sweep"].batch_step(n, statuses=True)
        for S, e in zip(s["sweep"].items, s["extra"]):
            N.check(L.gelios_download_mhd(S._h, n % 2, e), "gelios_download_mhd")
        return {"state": [r[n % 2] for r in s["rows"]], "extra": s["extra"], "dt": [float(t.dt) for t in st]}
    if kind == "plain":
        st = s["items"][0].Go_stationary(case["steps"])
        return {"state": s["rows"][0][case["steps"] % 2], "dt": float(st.dt)}
    if kind == "march":
        N.check(L.gelios_plain_batch_run_to_residual(s["batch"].h, 0.0, case["steps"], case["steps"] // 2,
                                                     s["done"].ctypes.data, s["res"].ctypes.data,
                                                     s["dts"].ctypes.data), "gelios_plain_batch_run_to_residual")
        return {"state": [r[0] for r in s["rows"]], "steps": s["done"], "residual": s["res"], "dt": s["dts"]}
    if kind == "train":
        hist = s["net"].train(case["iters"], case["batch"], 2e-3, 2e-5, max(1, case["iters"] // 4), 7)
        return {"loss": hist, "params": s["net"].params()}
    return s["net"].predict(s["x"])


# ---------------------------------------------------------------- the least work of a pass
def work(case: dict) -> dict:
    kind = case["kind"]
    if kind in ("train", "predict"):
        params = 31 * 256 + 256 + 4 * (256 * 256 + 256) + 256 * 5 + 5
        rows = case["batch"] * case["iters"] if kind == "train" else case["rows"]
        per = 3 if kind == "train" else 1
        return {"bytes": rows * 12 * 4 + params * 4 * (7 * case["iters"] if kind == "train" else 1),
                "flops": 2.0 * per * rows * params}
    if kind in ("plain", "march"):
        # state in and out, centroid, neighbour indices
        cells = case["n_theta"] * case["n_r"] * case.get("instances", 1)
        return {"bytes": 112 * cells * case["steps"], "flops": 0}
    if kind == "sweep":
        cells = sum(len(_rail_mesh(_scaled(case["lo"] + (case["hi"] - case["lo"]) * ((i * 0.618034) % 1.0)))[0]
                        ["cell_type"]) for i in range(case["instances"]))
        return {"bytes": 288 * cells * case["steps"] + 64 * cells, "flops": 0}
    mesh = _rail_mesh(case["grid"])[0]
    cells, points = mesh.n_cells, mesh.n_points
    if kind == "inner":  # state, moments, centroid, indices of the inner cells
        cells = len(mesh.inner_cells(N.reference_params().R111))
        return {"bytes": 264 * cells * case["steps"], "flops": 0}
    # state in and out, moments or sources, points before and after, indices
    per = {"mk2": 288, "stream": 288 + 80, "k5": 392, "mhd": 288}[kind]
    back = {"mk2": 0, "stream": 0, "k5": 128, "mhd": 64}[kind]
    return {"bytes": per * cells * case["steps"] + back * cells + 16 * points, "flops": 0}


# ---------------------------------------------------------------- the same in plain 64-bit numpy / torch
class _Polar:
    """Geometry of the polar half-plane grid, arrays (n_theta, n_r): rays
    uniform in 0..pi, radii log-spaced 1..600."""

    def __init__(self, nt: int, nr: int):
        th = np.arange(nt + 1) * math.pi / nt
        r = np.exp(math.log(600.0) * np.arange(nr + 1) / nr)
        r[nr] = 600.0
        X, Y = r * np.cos(th)[:, None], r * np.sin(th)[:, None]
        px = [X[:-1, :-1], X[:-1, 1:], X[1:, 1:], X[1:, :-1]]
        py = [Y[:-1, :-1], Y[:-1, 1:], Y[1:, 1:], Y[1:, :-1]]
        cr = [px[i] * py[(i + 1) % 4] - px[(i + 1) % 4] * py[i] for i in range(4)]
        a = 0.5 * sum(cr)
        self.nt, self.nr, self.area = nt, nr, np.abs(a)
        self.cx = sum((px[i] + px[(i + 1) % 4]) * cr[i] for i in range(4)) / (6.0 * a)
        self.cy = sum((py[i] + py[(i + 1) % 4]) * cr[i] for i in range(4)) / (6.0 * a)
        self.rad = np.sqrt(self.cx**2 + self.cy**2)
        # faces across r (nt, nr + 1), normal outwards; across theta (nt + 1, nr), normal to the next ray
        self.rf = self._face(X[:-1], Y[:-1], X[1:], Y[1:])
        self.tf = self._face(X[:, 1:], Y[:, 1:], X[:, :-1], Y[:, :-1])

    @staticmethod
    def _face(xa, ya, xb, yb):
        S = np.sqrt((xb - xa) ** 2 + (yb - ya) ** 2)
        return {"x": (xa + xb) / 2, "y": (ya + yb) / 2, "n1": (yb - ya) / S, "n2": -(xb - xa) / S, "S": S}


def _hllc(g, L, R, n1, n2):
    """HLLC flux (mass, momentum, energy, Q) and the wave-speed bound."""
    u1, v1 = L[2] * n1 + L[3] * n2, L[2] * n2 - L[3] * n1
    u2, v2 = R[2] * n1 + R[3] * n2, R[2] * n2 - R[3] * n1
    c = np.maximum(np.sqrt(g * L[1] / L[0]), np.sqrt(g * R[1] / R[0]))
    SL, SR = np.minimum(u1, u2) - c, np.maximum(u1, u2) + c
    sL, sR = SL - u1, SR - u2
    SM = (sR * R[0] * u2 - sL * L[0] * u1 - R[1] + L[1]) / (sR * R[0] - sL * L[0])
    pt = 0.5 * (R[1] + R[0] * sR * (SM - u2) + L[1] + L[0] * sL * (SM - u1))

    def side(U, u, v, S, s):
        e = U[1] / (g - 1.0) + 0.5 * U[0] * (U[2] ** 2 + U[3] ** 2)
        F = [U[0] * u, U[0] * u * u + U[1], U[0] * u * v, (e + U[1]) * u, U[4] * u]
        k = s / (S - SM)
        star = [U[0] * k, U[0] * k * SM, U[0] * k * v, e * k + (pt * SM - U[1] * u) / (S - SM), U[4] * k]
        base = [U[0], U[0] * u, U[0] * v, e, U[4]]
        return F, [f + S * (a - b) for f, a, b in zip(F, star, base)]

    FL, HL = side(L, u1, v1, SL, sL)
    FR, HR = side(R, u2, v2, SR, sR)
    F = [np.where(SL >= 0, a, np.where(SR <= 0, d, np.where(SM >= 0, b, c))) for a, b, c, d in zip(FL, HL, HR, FR)]
    return ([F[0], n1 * F[1] + n2 * F[2], n2 * F[1] - n1 * F[2], F[3], F[4]],
            np.maximum(np.abs(SL), np.abs(SR)))


def _turn(x1, y1, x2, y2, u, v):
    """A velocity given in the polar frame of point 1, in that of point 2."""
    r1, r2 = np.sqrt(x1**2 + y1**2), np.sqrt(x2**2 + y2**2)
    a, b = (u * x1 + v * y1) / r1, (v * x1 - u * y1) / r1
    return (a * x2 - b * y2) / r2, (a * y2 + b * x2) / r2


def _stationary(g: _Polar, p, st, steps: int):
    """`steps` steps of Go_stationary on the polar grid; state (5, nt, nr), dt."""
    gm, near = p.gamma, g.rad < p.rad_stat
    Ux = st.reshape(5, g.nt, g.nr).copy()

    def scaled(U, x, y, rad, f):
        fr2 = f["x"] ** 2 + f["y"] ** 2
        u, v = _turn(x, y, f["x"], f["y"], U[2], U[3])
        return [U[0] * rad**2 / fr2, U[1] * (rad * rad / fr2) ** gm, u, v, U[4]]

    def dist(f, sl):
        return np.sqrt((g.cx[sl] - f["x"]) ** 2 + (g.cy[sl] - f["y"]) ** 2)

    def cut(f, sl):
        return {k: v[sl] for k, v in f.items()}

    al = slice(None)
    interior = [(cut(g.rf, (al, slice(1, -1))), (al, slice(0, -1)), (al, slice(1, None))),
                (cut(g.tf, slice(1, -1)), slice(0, -1), slice(1, None))]
    dt = p.dt0
    for _ in range(steps):
        cand = [1e7]
        tot = np.zeros((5, g.nt, g.nr))
        for f, a, b in interior:
            A, B = Ux[(al,) + (a if isinstance(a, tuple) else (a,))], Ux[(al,) + (b if isinstance(b, tuple) else (b,))]
            Fp, up = _hllc(gm, A, B, f["n1"], f["n2"])
            Fs, us = _hllc(gm, scaled(A, g.cx[a], g.cy[a], g.rad[a], f), scaled(B, g.cx[b], g.cy[b], g.rad[b], f),
                           f["n1"], f["n2"])
            for sl, sg in ((a, 1.0), (b, -1.0)):
                for k in range(5):
                    tot[k][sl] += sg * np.where(near[sl], Fs[k], Fp[k]) * f["S"]
                cand.append((p.kurant * dist(f, sl) / np.where(near[sl], us, up)).min())

        def boundary(f, sl, sg, own, other):
            F, u = _hllc(gm, own, other, sg * f["n1"], sg * f["n2"])
            for k in range(5):
                tot[k][sl] += F[k] * f["S"]
            cand.append((p.kurant * dist(f, sl) / u).min())

        sl, f = (al, 0), cut(g.rf, (al, 0))
        U, d = [Ux[k][sl] for k in range(5)], np.sqrt(f["x"] ** 2 + f["y"] ** 2)
        ro = 1.0 / (p.chi * d) ** 2
        wind = [ro, ro * p.chi**2 / (gm * p.inner_mach**2), p.chi * f["x"] / d, p.chi * f["y"] / d, ro]
        boundary(f, sl, -1.0, [U[0] * (g.rad[sl] / d) ** 2, U[1] * (g.rad[sl] / d) ** (2 * gm)] + U[2:], wind)
        sl, f = (al, -1), cut(g.rf, (al, -1))
        U = [Ux[k][sl] for k in range(5)]
        inp = 2 * np.arange(g.nt) + 1 < g.nt
        out = [U[0], U[1], np.where(U[2] >= 0, p.extern_u_par, U[2]), U[3], U[4]]
        boundary(f, sl, 1.0, U, [np.where(inp, a, b) for a, b in
                                 zip((p.in_ro, p.in_p, p.in_u, p.in_v, p.in_Q), out)])
        for i, sg in ((0, -1.0), (-1, 1.0)):
            f = cut(g.tf, i)
            U = [Ux[k][i] for k in range(5)]
            tu, _tv = _turn(g.cx[i], g.cy[i], f["x"], f["y"], U[2], U[3])
            U = [U[0], U[1], np.where(near[i], tu, U[2]), 0.0 * U[3], U[4]]
            boundary(f, i, sg, U, U)
        ro, pr, u, v, Q = Ux
        ek = 0.5 * ro * (u * u + v * v)
        n0 = ro - dt * (tot[0] / g.area + ro * v / g.cy)
        n0 = np.where(n0 <= 0, p.ro_floor, n0)
        n2 = (ro * u - dt * (tot[1] / g.area + ro * v * u / g.cy)) / n0
        n3 = (ro * v - dt * (tot[2] / g.area + ro * v * v / g.cy)) / n0
        n4 = Q - dt * (tot[4] / g.area + Q * v / g.cy)
        n1 = (pr / (gm - 1) + ek - dt * (tot[3] / g.area + v * (gm * pr / (gm - 1) + ek) / g.cy)
              - 0.5 * n0 * (n2 * n2 + n3 * n3)) * (gm - 1)
        Ux = np.stack([n0, np.where(n1 <= 0, p.p_floor, n1), n2, n3, n4])
        dt = min(cand)
    return Ux.reshape(5, -1), float(dt)


def _features(x):
    out, pi = [x], math.pi
    for c in (5, 6):
        for f in range(6):
            out += [torch.sin(pi * 2**f * x[:, c:c + 1]), torch.cos(pi * 2**f * x[:, c:c + 1])]
    return torch.cat(out, dim=1)


def _network(flat, sizes, x):
    h, o = _features(x), 0
    for l, (a, b) in enumerate(zip(sizes[:-1], sizes[1:])):
        w, bias = flat[o:o + a * b].reshape(b, a), flat[o + a * b:o + a * b + b]
        o += a * b + b
        h = h @ w.T + bias
        if l + 2 < len(sizes):
            h = torch.nn.functional.gelu(h)
    return h


def _mix(z):
    z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
    z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    return z ^ (z >> np.uint64(31))


def _train(case, seed: int):
    """The Adam steps of a train case in 64 bits (batch rows by the documented hash)."""
    flat0, sizes = _network_params(seed)
    w = torch.tensor(flat0, dtype=torch.float64, device="cuda", requires_grad=True)
    X, T = (torch.tensor(a, dtype=torch.float64, device="cuda") for a in _network_rows(case["rows"], seed))
    m, v, hist, n = torch.zeros_like(w), torch.zeros_like(w), [], case["iters"]
    warm = max(1, n // 4)
    for it in range(n):
        with np.errstate(over="ignore"):
            key = np.uint64(7) * np.uint64(0xD1B54A32D192ED03) + np.uint64(it) * np.uint64(0x8CB92BA72F3D8DD7)
            r = _mix(key + np.arange(case["batch"], dtype=np.uint64) * np.uint64(0x9E3779B97F4A7C15))
        idx = torch.tensor((r % np.uint64(case["rows"])).astype(np.int64), device="cuda")
        loss = ((_network(w, sizes, X[idx]) - T[idx]) ** 2).mean()
        (g,) = torch.autograd.grad(loss, w)
        hist.append(float(loss))
        lr = 2e-3 * (it + 1) / warm if it < warm else \
            2e-5 + 0.5 * (2e-3 - 2e-5) * (1.0 + math.cos(math.pi * (it - warm) / (n - warm)))
        with torch.no_grad():
            m.mul_(0.9).add_(0.1 * g)
            v.mul_(0.999).add_(0.001 * g * g)
            w -= lr * (m / (1 - 0.9 ** (it + 1))) / (torch.sqrt(v / (1 - 0.999 ** (it + 1))) + 1e-8)
    return {"loss": np.array(hist), "params": w.detach().cpu().numpy()}


def exact(case: dict, seed: int):
    """What run() returns, in 64 bits.  None for the steps on rail grids:
    surface tracking, rail motion and exact Riemann solves have no plain
    array form that runs in seconds."""
    kind = case["kind"]
    if kind in ("plain", "march"):
        prm, sts = _polar_inputs(case, seed)
        if case["n_theta"] * case["n_r"] * case["steps"] * len(prm) > 6e7:
            return None
        g = _Polar(case["n_theta"], case["n_r"])
        got = [_stationary(g, p, st, case["steps"]) for p, st in zip(prm, sts)] if kind == "plain" else \
            [_restarted(g, p, st, case["steps"]) for p, st in zip(prm, sts)]
        if kind == "plain":
            return {"state": got[0][0], "dt": got[0][1]}
        return {"state": [a for a, _ in got], "steps": None, "residual": None, "dt": np.array([d for _, d in got])}
    if kind == "train":
        return _train(case, seed)
    if kind == "predict":
        flat, sizes = _network_params(seed)
        x, _t = _network_rows(case["rows"], seed)
        return _network(torch.tensor(flat, dtype=torch.float64), sizes, torch.tensor(x, dtype=torch.float64)).numpy()
    return None


def _restarted(g, p, st, steps: int):
    """A march of `steps` steps checked once on the way: dt restarts there."""
    st, _dt = _stationary(g, p, st, steps // 2)
    return _stationary(g, p, st, steps - steps // 2)
