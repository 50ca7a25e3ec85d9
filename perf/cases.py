"""The performance cases of this library: what its users run, through the
public entry points, over the range of sizes and options they meet.

Three kinds of work:

* ``rk``: explicit multistage steps of a block set resident on the GPU
  (``capi.Handle.rk_steps``), the library's main loop;
* ``nks``: Newton-Krylov steps from the freestream (``set_state`` and
  ``nks``) of one case or of a batch of cases on one handle;
* the warm-start networks: prediction (``forward``), a gradient and
  training (``gradient``, ``train``) of the deep and the shallow network.

``listed()`` names the cases, ``draw()`` gives more of the same ranges,
``prepare()`` makes what a program holds before the call (handle, state,
network, rows), ``run()`` is one pass and returns its outputs, ``work()`` the
bytes and operations a pass cannot do without, and ``exact()`` its outputs in
64-bit torch arithmetic where they have such a value.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from cffc_b200 import capi, cases, warmstart

FP64, FP32, EXACT = 0, 1, 2
PRECISION = {"fp64": FP64, "fp32": FP32, "exact": EXACT}
LIMITER = {"zero": cases.LIMITER_ZERO, "bj": cases.LIMITER_BARTH_JESPERSEN, "venkat": cases.LIMITER_VENKATAKRISHNAN}
FLUX = {"roe": cases.FLUX_ROE, "hlle": cases.FLUX_HLLE, "hllc": cases.FLUX_HLLC, "ausmplus": cases.FLUX_AUSMPLUS}
TIME = {"rk2": (0, 2), "rk4": (cases.TIME_RUNGE_KUTTA, 4), "os4": (cases.TIME_OPTIMAL_SMOOTHING, 4)}
DEEP_NPARAM, SHALLOW_NPARAM = 205840, 20752


def rk(name, grid, nbi, nbj, nci, ncj, steps, precision="fp64", limiter="venkat", flux="roe", time="rk2", local=False):
    c = {"kind": "rk", "grid": grid, "nbi": nbi, "nbj": nbj, "nci": nci, "ncj": ncj, "steps": steps,
         "precision": precision, "limiter": limiter, "flux": flux, "time": time, "local": local}
    return dict(c, name=name) if name else c


def nks(name, nbi, nbj, nci, ncj, newton, max_gmres, ilu=-1, restart=30, mach=1.4, height=0.04, limiter="zero",
        gmres_tol=0.1, cfl0=10.0, batch=1):
    c = {"kind": "nks", "nbi": nbi, "nbj": nbj, "nci": nci, "ncj": ncj, "newton": newton, "max_gmres": max_gmres,
         "ilu": ilu, "restart": restart, "mach": mach, "height": height, "limiter": limiter, "gmres_tol": gmres_tol,
         "cfl0": cfl0, "batch": batch}
    return dict(c, name=name) if name else c


def net(name, kind, rows, steps=0, batch=0):
    c = {"kind": kind, "rows": rows, "steps": steps, "batch": batch}
    return dict(c, name=name) if name else c


def listed():
    return [
        # a small unsteady run (unit box, 16 blocks of 32 x 32): every step is
        # a chain of short kernels, so their latency counts
        rk("rk2_box_16k", "box", 4, 4, 32, 32, 100),
        # the large explicit run: a million cells, the headline workload
        rk("rk2_curvilinear_1m", "curvilinear", 32, 8, 64, 64, 10),
        # the single-precision reconstruction, half that size
        rk("rk2_curvilinear_fp32", "curvilinear", 16, 8, 64, 64, 10, precision="fp32"),
        # the reference's arithmetic bit for bit, for comparisons against it
        rk("rk2_curvilinear_exact", "curvilinear", 12, 6, 48, 48, 10, precision="exact"),
        # a walled channel of odd-sized blocks driven to a steady state with
        # local time steps and a four-stage scheme
        rk("os4_channel_odd", "channel", 6, 5, 37, 29, 20, limiter="bj", flux="hllc", time="os4", local=True),
        # Newton-Krylov on a small supersonic bump, block Jacobi
        nks("nks_jacobi_12k", 6, 2, 32, 32, 5, 200),
        # second order, subsonic, 98 thousand cells
        nks("nks_jacobi_98k", 12, 4, 64, 32, 6, 60, mach=0.5, height=0.1, limiter="venkat", gmres_tol=1e-5, cfl0=1.0),
        # the small bump with the ILU(2) preconditioner
        nks("nks_ilu2_12k", 6, 2, 32, 32, 6, 200, ilu=2),
        # a parameter sweep: eight cases of 8 to 48 blocks as one batch
        nks("nks_ilu2_batch", 0, 0, 32, 32, 4, 200, ilu=2, batch=8),
        # the deep network's prediction over the cells of a sweep
        net("deep_forward_300k", "deep_forward", 300007),
        # its training: minibatches of 8,192 rows from a pool of rows
        net("deep_train_8k", "deep_train", 262144, 100, 8192),
        # the shallow network's full-batch training over the cells of a family
        net("shallow_train_152k", "shallow_train", 151552, 10),
    ]


def log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["rk", "rk", "rk", "rk", "nks", "nks", "nks", "net", "net", "net"])
    if kind == "rk":
        grid = rng.choice(["box", "curvilinear", "curvilinear", "channel"])
        nci = log_int(rng, 8, 64)
        ncj = nci if grid != "channel" else log_int(rng, 8, 64)
        nbi, nbj = log_int(rng, 2, 16), log_int(rng, 2, 8)
        nbi = nbj if grid == "box" else nbi  # the unit box has as many blocks each way
        cells = nbi * nbj * nci * ncj
        precision = rng.choice(["fp64", "fp64", "fp64", "fp32", "exact"])
        most = (3 if precision == "exact" else 6) * 10 ** 6 // cells
        steps = min(log_int(rng, 5, 100), max(5, most))
        if grid == "channel":
            return rk("", grid, nbi, nbj, nci, ncj, steps, precision, rng.choice(["venkat", "bj"]),
                      rng.choice(["roe", "hlle", "hllc", "ausmplus"]), rng.choice(["rk2", "rk4", "os4"]),
                      rng.choice([True, False]))
        return rk("", grid, nbi, nbj, nci, ncj, steps, precision, rng.choice(["venkat", "venkat", "bj"]))
    if kind == "nks":
        batch = rng.choice([1, 1, rng.randint(2, 8)])
        nc = rng.choice([16, 24, 32, 32])
        return nks("", 0 if batch > 1 else rng.randint(3, 12), 0 if batch > 1 else rng.randint(2, 4), nc,
                   nc if batch > 1 else rng.choice([16, 24, 32]), rng.randint(2, 4), rng.choice([60, 100, 200]),
                   rng.choice([-1, 0, 1, 2, 2]), rng.choice([20, 30]), round(rng.uniform(1.35, 1.6), 3),
                   round(rng.uniform(0.02, 0.045), 4), batch=batch)
    kind = rng.choice(["deep_forward", "deep_gradient", "deep_train", "shallow_forward", "shallow_gradient",
                       "shallow_train"])
    if kind == "deep_train":
        return net("", kind, log_int(rng, 8192, 262144), rng.randint(10, 60), log_int(rng, 512, 8192))
    if kind == "shallow_train":
        return net("", kind, log_int(rng, 1000, 151552), rng.randint(2, 10))
    if kind == "deep_gradient":
        return net("", kind, log_int(rng, 100, 65536))
    return net("", kind, log_int(rng, 100, 300000))


# ---- preparation ------------------------------------------------------------

def block_set(case, seed):
    """The explicit case's block set: grid, initial state and scheme."""
    ti, n_stage = TIME[case["time"]]
    sc = cases.Scheme(limiter=LIMITER[case["limiter"]], flux=FLUX[case["flux"]], n_stage=n_stage,
                      time_integration=ti, local_dt=int(case["local"]), precision=PRECISION[case["precision"]], cfl=0.5)
    nbi, nbj, nci, ncj = case["nbi"], case["nbj"], case["nci"], case["ncj"]
    if case["grid"] == "box":
        return cases.periodic_box_bumps(nb=nbi, nbj=nbj, nc=nci, seed=seed, scheme=sc)
    if case["grid"] == "curvilinear":
        return cases.curvilinear_mach2(nbi=nbi, nbj=nbj, nc=nci, seed=seed, scheme=sc)
    return cases.channel(nbi=nbi, nbj=nbj, nci=nci, ncj=ncj, seed=seed, scheme=sc)


def nks_cases(case, seed):
    """The steady case's block sets: one bump channel, or a family of them."""
    rng = np.random.Generator(np.random.PCG64(seed))
    m, h = rng.uniform(-0.02, 0.02), rng.uniform(-0.002, 0.002)  # each seed its own Mach number and bump
    sc = cases.Scheme(limiter=LIMITER[case["limiter"]], local_dt=1, cfl=1.0)
    if case["batch"] > 1:  # the family's layouts in turn, each case its own Mach number and bump
        return [cases.bump_channel(nbi=nbi, nbj=nbj, nci=case["nci"], ncj=case["ncj"], mach=rng.uniform(1.35, 1.6),
                                   h=rng.uniform(0.02, 0.045), scheme=sc)
                for nbi, nbj in cases.LAYOUTS_8_96[:case["batch"]]]
    return [cases.bump_channel(nbi=case["nbi"], nbj=case["nbj"], nci=case["nci"], ncj=case["ncj"],
                               mach=case["mach"] + m, h=case["height"] + h, scheme=sc)]


def rows_of(n, seed, deep):
    """Features in the range the family's cells give, and smooth targets."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    X = torch.zeros((n, 16), device="cuda")
    nf = 5 if deep else 16
    X[:, :nf] = 2.0 * torch.rand((n, nf), generator=g, device="cuda") - 1.0
    mix = torch.randn((nf, 4), generator=g, device="cuda")
    return X, 0.2 * torch.tanh(X[:, :nf] @ mix)


def parameters(kind, seed):
    """Glorot-uniform weights and small biases; inputs past the deep network's
    five features and outputs past the four used ones stay zero."""
    rng, out = np.random.Generator(np.random.PCG64(seed)), []
    layers = _layers(kind)
    for q, (o, i) in enumerate(layers):
        used_in = 5 if kind.startswith("deep") and q == 0 else i
        used_out = 4 if q == len(layers) - 1 else o
        w, b = np.zeros((o, i)), np.zeros(o)
        w[:used_out, :used_in] = rng.uniform(-1.0, 1.0, (used_out, used_in)) * math.sqrt(6.0 / (used_in + used_out))
        b[:used_out] = rng.uniform(-0.05, 0.05, used_out)
        out += [w.ravel(), b]
    return np.concatenate(out).astype(np.float32)


class _Device:
    """A device array of the library for torch (no copy)."""

    def __init__(self, pointer, shape):
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<f8", "data": (pointer, False), "version": 3}


def resident(h, shape):
    """The handle's W and U as torch tensors (e2d_device_state); each keeps
    the handle, which owns the memory."""
    w, u, r = (C.POINTER(C.c_double)() for _ in range(3))
    rc = h.lib.e2d_device_state(h.h, C.byref(w), C.byref(u), C.byref(r))
    if rc:
        raise RuntimeError(f"e2d_device_state: {rc}")
    out = [torch.as_tensor(_Device(C.cast(p, C.c_void_p).value, shape), device="cuda") for p in (w, u)]
    for t in out:
        t.handle = h
    return out


def prepare(case, seed):
    kind = case["kind"]
    if kind == "rk":
        bs = block_set(case, seed)
        h = capi.Handle(bs)
        h.set_state()
        return {"case": case, "h": h, "out": resident(h, bs.cell_shape())}
    if kind == "nks":
        fam = nks_cases(case, seed)
        h = capi.BatchHandle(fam) if case["batch"] > 1 else capi.Handle(fam[0])
        p = capi.nks_params(case["newton"], gmres_restart=case["restart"], max_gmres=case["max_gmres"],
                            overall_tol=1e-10, cfl0=case["cfl0"], gmres_tol=case["gmres_tol"],
                            ilu_level=None if case["ilu"] < 0 else case["ilu"])
        blocks = sum(bs.nblk for bs in fam)
        return {"case": case, "h": h, "p": p, "out": resident(h, (blocks,) + fam[0].cell_shape()[1:])}
    deep = kind.startswith("deep")
    X, T = rows_of(case["rows"], seed, deep)
    torch.cuda.synchronize()
    m = (warmstart.MlpDeep if deep else warmstart.Mlp)()
    m.params(parameters(kind, seed))
    return {"case": case, "net": m, "X": X, "T": T}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "rk":
        rc, hist = state["h"].rk_steps(case["steps"])
        return {"rc": rc, "hist": hist, "W": state["out"][0], "U": state["out"][1]}
    if kind == "nks":
        h = state["h"]
        h.set_state()
        rc, hist = h.nks(state["p"])
        steps = [st for x in hist for st in x] if case["batch"] > 1 else hist
        return {"rc": rc, "iterations": np.array([st["gmres_iters"] for st in steps]),
                "norms": np.array([[st[k] for k in ("l1", "l2", "lmax", "ratio", "cfl")] for st in steps]),
                "W": state["out"][0], "U": state["out"][1]}
    m, X, T = state["net"], state["X"], state["T"]
    if kind.endswith("forward"):
        return {"Y": m.forward(X)}
    if kind.endswith("gradient"):
        loss, g = m.gradient(X, T)
        return {"loss": loss, "gradient": g}
    if kind == "deep_train":
        hist = m.train(X, T, case["steps"], case["batch"], 1e-3)
    else:
        hist = m.train(X, T, case["steps"], 1e-3)
    return {"losses": hist, "params": m.params()}


# ---- what a pass cannot do without ---------------------------------------------

def work(case):
    kind = case["kind"]
    if kind == "rk":
        # per stage the state in and out (32 B each), the nodes (16 B) and,
        # past the first stage, the base state (32 B); about 900 operations a
        # cell and stage (least squares 130, limiter 150, two Roe faces 400, update
        # and time step 100, with their square roots and reciprocals)
        n = TIME[case["time"]][1]
        cells = case["nbi"] * case["nbj"] * case["nci"] * case["ncj"]
        return {"bytes": case["steps"] * cells * (80.0 * n + 32.0 * (n - 1)),
                "flops": case["steps"] * cells * n * 900.0}
    if kind == "nks":
        # per GMRES iteration (about 25 a Newton step) a residual, the
        # preconditioner's blocks (16 doubles a cell and entry) and, for the
        # orthogonalisation, the earlier vectors read once (about 12)
        blocks = case["nbi"] * case["nbj"] or sum(i * j for i, j in cases.LAYOUTS_8_96[:case["batch"]])
        cells = blocks * case["nci"] * case["ncj"]
        entries = {-1: 1.0, 0: 4.9, 1: 6.8, 2: 8.7}.get(case["ilu"], 16.0)
        its = case["newton"] * 25.0
        return {"bytes": its * cells * (112.0 + 128.0 * entries + 12 * 32.0),
                "flops": its * cells * (900.0 + 32.0 * entries + 12 * 16.0)}
    deep = kind.startswith("deep")
    params = DEEP_NPARAM if deep else SHALLOW_NPARAM
    passes, rows = 1, case["rows"]
    if kind.endswith("train"):
        passes, rows = case["steps"], case["batch"] or case["rows"]
    per_row = 2.0 * params * (1 if kind.endswith("forward") else 3)
    return {"bytes": passes * (rows * (16 * 4 + 4 * 4) + 4.0 * params * (1 if kind.endswith("forward") else 7)),
            "flops": passes * rows * per_row}


# ---- the same in 64-bit torch ----------------------------------------------------

def exact(case, seed):
    kind = case["kind"]
    if kind == "rk":
        if case["grid"] == "channel" or case["time"] != "rk2" or case["flux"] != "roe" or case["local"]:
            return None
        return exact_rk2(case, block_set(case, seed))
    if kind == "nks":
        return None  # the Krylov history depends on the rounding of its sums
    return exact_net(case, seed)


class _Periodic:
    """The wired periodic block set as arrays over its blocks, float64."""

    def __init__(self, bs, nbi, nbj):
        self.nbi, self.nbj, self.nci, self.ncj = nbi, nbj, bs.nci, bs.ncj
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        X, Y = (torch.from_numpy(a).to(dev) for a in (bs.node_x, bs.node_y))
        self.X, self.Y = X, Y
        # cell area and centroid from the nodes (SW, SE, NE, NW), taken about
        # the cell's own corner
        ox, oy = X[:, :-1, :-1], Y[:, :-1, :-1]
        x = [a - ox for a in (X[:, :-1, :-1], X[:, :-1, 1:], X[:, 1:, 1:], X[:, 1:, :-1])]
        y = [a - oy for a in (Y[:, :-1, :-1], Y[:, :-1, 1:], Y[:, 1:, 1:], Y[:, 1:, :-1])]
        A2, xt, yt = 0.0, 0.0, 0.0
        for a in range(4):
            b = (a + 1) % 4
            cr = x[a] * y[b] - x[b] * y[a]
            A2, xt, yt = A2 + cr, xt + (x[a] + x[b]) * cr, yt + (y[a] + y[b]) * cr
        self.A = 0.5 * A2
        self.xc, self.yc = ox + xt / (3.0 * A2), oy + yt / (3.0 * A2)

    def ghosts(self, I):
        """Interior cells [nblk][v][ncj][nci] with two layers of ghosts."""
        v = I.shape[1]
        G = I.view(self.nbj, self.nbi, v, self.ncj, self.nci).permute(2, 0, 3, 1, 4)
        G = G.reshape(v, self.nbj * self.ncj, self.nbi * self.nci)
        G = torch.nn.functional.pad(G[None], (2, 2, 2, 2), mode="circular")[0]
        out = G.unfold(1, self.ncj + 4, self.ncj).unfold(2, self.nci + 4, self.nci)
        return out.permute(1, 2, 0, 3, 4).reshape(self.nbi * self.nbj, v, self.ncj + 4, self.nci + 4).contiguous()

    def edge(self, ax, ay, cx, cy):
        """Normal, length and midpoint of the edges a -> c."""
        dx, dy = ax - cx, ay - cy
        ln = torch.sqrt(dx * dx + dy * dy)
        return dy / ln, -dx / ln, ln, 0.5 * (ax + cx), 0.5 * (ay + cy)


def _prim(U, g):
    d = U[:, 0]
    u, v = U[:, 1] / d, U[:, 2] / d
    return torch.stack([d, u, v, (g - 1.0) * (U[:, 3] - 0.5 * d * (u * u + v * v))], 1)


def _roe(l, r, nx, ny, g):
    """Roe's flux with Harten's fix through faces of normal (nx, ny)."""
    def turn(w):
        return w[:, 0], w[:, 1] * nx + w[:, 2] * ny, -w[:, 1] * ny + w[:, 2] * nx, w[:, 3]

    def fx(d, u, v, p):
        return d * u, d * u * u + p, d * u * v, u * (g / (g - 1.0) * p + 0.5 * d * (u * u + v * v))

    L, R = turn(l), turn(r)
    (dl, ul, vl, pl), (dr, ur, vr, pr) = L, R
    hl = g * pl / ((g - 1.0) * dl) + 0.5 * (ul * ul + vl * vl)
    hr = g * pr / ((g - 1.0) * dr) + 0.5 * (ur * ur + vr * vr)
    sl, sr = torch.sqrt(dl), torch.sqrt(dr)
    ua, va, ha = (sl * ul + sr * ur) / (sl + sr), (sl * vl + sr * vr) / (sl + sr), (sl * hl + sr * hr) / (sl + sr)
    ca2 = (g - 1.0) * (ha - 0.5 * (ua * ua + va * va))
    ca, da = torch.sqrt(ca2), sl * sr
    cl, cr = torch.sqrt(g * pl / dl), torch.sqrt(g * pr / dr)

    def harten(la, a, b):
        delta = torch.clamp(2.0 * (b - a), min=0.0)
        fix = 0.5 * (la * la / torch.where(delta < 1e-7, torch.ones_like(delta), delta) + delta) - la.abs()
        return torch.where((la.abs() > delta) | (delta < 1e-7), torch.zeros_like(fix), fix)

    up = ua >= 0
    la0, la3 = ua - ca, ua + ca
    d0, d3 = harten(la0, ul - cl, ur - cr), harten(la3, ul + cl, ur + cr)
    w0 = torch.where(up, 0.5 * (la0 - la0.abs() - d0), 0.5 * (la0 + la0.abs() + d0))
    w3 = torch.where(up, 0.5 * (la3 - la3.abs() - d3), 0.5 * (la3 + la3.abs() + d3))
    zero = torch.zeros_like(w0)
    w0 = torch.where(up, torch.minimum(w0, zero), -torch.maximum(w0, zero))
    w3 = torch.where(up, torch.minimum(w3, zero), -torch.maximum(w3, zero))
    k0 = w0 * (-0.5 * da / ca * (ur - ul) + 0.5 / ca2 * (pr - pl))
    k3 = w3 * (0.5 * da / ca * (ur - ul) + 0.5 / ca2 * (pr - pl))
    F = [torch.where(up, a, b) for a, b in zip(fx(*L), fx(*R))]
    F = [F[0] + k0 + k3, F[1] + k0 * (ua - ca) + k3 * (ua + ca), F[2] + (k0 + k3) * va,
         F[3] + k0 * (ha - ua * ca) + k3 * (ha + ua * ca)]
    return torch.stack([F[0], F[1] * nx - F[2] * ny, F[1] * ny + F[2] * nx, F[3]], 1)


def _residual(P, W, limiter, g):
    """Flux divergence of the interior cells from the state with ghosts."""
    X, Y = P.X, P.Y
    c = (slice(None), slice(1, -1), slice(1, -1))
    cv = (slice(None), slice(None), slice(1, -1), slice(1, -1))
    nj, ni = W.shape[2], W.shape[3]
    w0, xc, yc = W[cv], P.xc[c], P.yc[c]
    sx, sy, xx, xy, yy = 0.0, 0.0, 0.0, 0.0, 0.0
    lo, hi = w0.clone(), w0.clone()
    for dj in (-1, 0, 1):
        for di in (-1, 0, 1):
            if di or dj:
                s = (slice(1 + dj, nj - 1 + dj), slice(1 + di, ni - 1 + di))
                dx, dy = P.xc[:, s[0], s[1]] - xc, P.yc[:, s[0], s[1]] - yc
                w = W[:, :, s[0], s[1]]
                sx, sy = sx + (w - w0) * dx[:, None], sy + (w - w0) * dy[:, None]
                xx, xy, yy = xx + dx * dx, xy + dx * dy, yy + dy * dy
                lo, hi = torch.minimum(lo, w), torch.maximum(hi, w)
    det = (xx * yy - xy * xy)[:, None]
    gx, gy = (sx * yy[:, None] - sy * xy[:, None]) / det, (sy * xx[:, None] - sx * xy[:, None]) / det
    x00, x10, x01, x11 = X[:, 1:-2, 1:-2], X[:, 1:-2, 2:-1], X[:, 2:-1, 1:-2], X[:, 2:-1, 2:-1]
    y00, y10, y01, y11 = Y[:, 1:-2, 1:-2], Y[:, 1:-2, 2:-1], Y[:, 2:-1, 1:-2], Y[:, 2:-1, 2:-1]
    phi = torch.ones_like(w0)
    for ax, ay, bx, by in ((x10, y10, x11, y11), (x00, y00, x01, y01), (x01, y01, x11, y11), (x00, y00, x10, y10)):
        d = gx * (0.5 * (ax + bx) - xc)[:, None] + gy * (0.5 * (ay + by) - yc)[:, None]
        y = torch.where(d > 0, hi - w0, lo - w0) / torch.where(d.abs() > 1e-7, d, torch.ones_like(d))
        f = (y * y + 2.0 * y) / (y * y + y + 2.0) if limiter == "venkat" else y.clamp(max=1.0)
        phi = torch.minimum(phi, torch.where(d.abs() > 1e-7, f, torch.ones_like(f)))
    gx, gy = phi * gx, phi * gy

    def at(j, i, mx, my):  # the limited state of ring cells [j, i] at the points (mx, my)
        return (w0[:, :, j, i] + gx[:, :, j, i] * (mx - xc[:, j, i])[:, None] +
                gy[:, :, j, i] * (my - yc[:, j, i])[:, None])

    inner, every, left, right = slice(1, -1), slice(None), slice(0, -1), slice(1, None)
    # faces between columns: nodes (i, j+1) -> (i, j); between rows: (i, j) -> (i+1, j)
    nx, ny, ln, mx, my = P.edge(X[:, 3:-2, 2:-2], Y[:, 3:-2, 2:-2], X[:, 2:-3, 2:-2], Y[:, 2:-3, 2:-2])
    Fi = _roe(at(inner, left, mx, my), at(inner, right, mx, my), nx, ny, g) * ln[:, None]
    nx, ny, ln, mx, my = P.edge(X[:, 2:-2, 2:-3], Y[:, 2:-2, 2:-3], X[:, 2:-2, 3:-2], Y[:, 2:-2, 3:-2])
    Fj = _roe(at(left, inner, mx, my), at(right, inner, mx, my), nx, ny, g) * ln[:, None]
    A = P.A[:, 2:-2, 2:-2][:, None]
    return (Fi[:, :, every, :-1] - Fi[:, :, every, 1:] + Fj[:, :, :-1] - Fj[:, :, 1:]) / A


def _time_step(P, W, g):
    """The smallest CFL-one step of the interior cells."""
    X, Y = P.X[:, 2:-2, 2:-2], P.Y[:, 2:-2, 2:-2]

    def edge(a, c):
        return P.edge(X[a], Y[a], X[c], Y[c])[:3]

    sw, se = (slice(None), slice(0, -1), slice(0, -1)), (slice(None), slice(0, -1), slice(1, None))
    nw, ne = (slice(None), slice(1, None), slice(0, -1)), (slice(None), slice(1, None), slice(1, None))
    (ex, ey, le), (wx, wy, lw), (nx, ny, lN), (sx, sy, ls) = edge(ne, se), edge(sw, nw), edge(nw, ne), edge(se, sw)
    A = P.A[:, 2:-2, 2:-2]
    d, u, v, p = W[:, 0], W[:, 1], W[:, 2], W[:, 3]
    a = torch.sqrt(g * p / d)
    vi, vj = 0.5 * (u * (ex - wx) + v * (ey - wy)), 0.5 * (u * (nx - sx) + v * (ny - sy))
    return float(torch.minimum(2.0 * A / (le + lw) / (a + vi.abs()), 2.0 * A / (lN + ls) / (a + vj.abs())).min())


def exact_rk2(case, bs):
    """The two-stage scheme with one global time step on a periodic set."""
    g, cfl = bs.scheme.gamma, bs.scheme.cfl
    P = _Periodic(bs, case["nbi"], case["nbj"])
    W = torch.from_numpy(bs.W).to(P.X.device)[:, :, 2:-2, 2:-2]
    U = torch.from_numpy(cases.U_of_W(bs.W)).to(P.X.device)[:, :, 2:-2, 2:-2].contiguous()
    hist, res = [], torch.zeros_like(U)
    for _ in range(case["steps"]):
        dt = _time_step(P, W, g)
        r = res[:, 0]
        hist.append([dt, float(r.abs().sum()), float(r.square().sum().sqrt()), float(r.abs().max())])
        r1 = cfl * dt * _residual(P, P.ghosts(W.contiguous()), case["limiter"], g)
        U1 = U + r1
        G1 = P.ghosts(U1)
        res = r1 + cfl * dt * _residual(P, _prim(G1, g), case["limiter"], g)
        U = U + 0.5 * res
        W = _prim(U, g)
    # after a step the ghost cells hold what its last stage read
    W1 = _prim(G1, g)
    W1[:, :, 2:-2, 2:-2], G1[:, :, 2:-2, 2:-2] = W, U
    return {"rc": None, "hist": np.array(hist), "W": W1.cpu().numpy(), "U": G1.cpu().numpy()}


def _layers(kind):
    """(outputs, inputs) of each layer."""
    if kind.startswith("deep"):
        return [(256, 16), (256, 256), (256, 256), (256, 256), (16, 256)]
    return [(128, 16), (128, 128), (16, 128)]


def _net_loss(flat, sizes, X, T, act):
    h, k = X, 0
    for q, (o, i) in enumerate(sizes):
        Wt, b = flat[k:k + o * i].view(o, i), flat[k + o * i:k + o * i + o]
        k += o * i + o
        h = h @ Wt.T + b
        h = act(h) if q < len(sizes) - 1 else h
    y = h[:, :4]
    return y, None if T is None else (y - T).square().sum() / X.shape[0]


def _minibatches(n, batch, steps, seed):
    """The rows of each training step: PCG32 draws, a shuffle per epoch."""
    s, inc, mask = seed * 2 + 1, (seed << 1) | 1, (1 << 64) - 1
    perm, pos = list(range(n)), n
    for _ in range(steps):
        rows = []
        while len(rows) < batch:
            if pos >= n:
                for i in range(n - 1, 0, -1):
                    old, s = s, (s * 6364136223846793005 + inc) & mask
                    x, r = (((old >> 18) ^ old) >> 27) & 0xFFFFFFFF, old >> 59
                    x = ((x >> r) | (x << ((32 - r) & 31))) & 0xFFFFFFFF
                    j = x % (i + 1)
                    perm[i], perm[j] = perm[j], perm[i]
                pos = 0
            take = min(batch - len(rows), n - pos)
            rows += perm[pos:pos + take]
            pos += take
        yield torch.tensor(rows)


def exact_net(case, seed):
    kind = case["kind"]
    X, T = (a.double() for a in rows_of(case["rows"], seed, kind.startswith("deep")))
    flat = torch.from_numpy(parameters(kind, seed)).to(X.device).double().requires_grad_(True)
    sizes = _layers(kind)
    act = (lambda z: torch.nn.functional.gelu(z, approximate="tanh")) if kind.startswith("deep") else torch.tanh
    if kind.endswith("forward"):
        with torch.no_grad():
            return {"Y": torch.cat([_net_loss(flat, sizes, x, None, act)[0] for x in X.split(65536)])}

    def gradient(x, t):
        loss = _net_loss(flat, sizes, x, t, act)[1]
        return loss.item(), torch.autograd.grad(loss, flat)[0]

    if kind.endswith("gradient"):
        loss, g = gradient(X, T)
        return {"loss": loss, "gradient": g}
    m, v, losses = torch.zeros_like(flat), torch.zeros_like(flat), []
    batch = min(case["batch"] or case["rows"], case["rows"])
    picks = _minibatches(case["rows"], batch, case["steps"], 7) if case["batch"] else iter([None] * case["steps"])
    for k, rows in enumerate(picks, 1):
        x, t = (X, T) if rows is None else (X[rows.to(X.device)], T[rows.to(X.device)])
        loss, g = gradient(x, t)
        losses.append(loss)
        with torch.no_grad():
            m.mul_(0.9).add_(g, alpha=0.1)
            v.mul_(0.999).addcmul_(g, g, value=0.001)
            flat -= 1e-3 * (m / (1 - 0.9 ** k)) / ((v / (1 - 0.999 ** k)).sqrt() + 1e-8)
    return {"losses": np.array(losses), "params": flat.detach()}
