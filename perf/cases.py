"""Performance cases: what a host of the solver core runs, through the public
entry points of the Python binding (``ec2d.gpu.Solver``, ``WarmStartNet``).

A marching case is what a host does between two outputs: it puts a state on
the device (``upload_U`` from page-locked memory, ``bc`` for the ghost cells,
as after a restart), takes the iterations to the next output (``step``), reads
the residual norms and reads U of every block back.  The residual case is one
residual evaluation of a given state.  The network cases are the learned warm
start's training steps and its predictions.
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "opencfd-ec2d_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from ec2d import cases as workloads  # noqa: E402
from ec2d import gpu, grids, learn  # noqa: E402
from ec2d.inputs import (FLUX, RECON, SCHEME, TIME_EULER1, TIME_LUSGS, TIME_RK3, TURB_NONE, TURB_SA,  # noqa: E402
                         TURB_SST, Params)

TIME = {"lusgs": TIME_LUSGS, "rk3": TIME_RK3, "euler": TIME_EULER1}


def listed():
    return [
        # the smallest case a host steps: a coarse inviscid airfoil grid, as
        # used to check a set-up before the real run; latency is all there is
        dict(name="euler_65x17", kind="march", flow="airfoil", nx=65, ny=17, blocks=1, flux="ROE", recon="ORIGINAL",
             scheme="MUSCL3", time="lusgs", mesh=1, steps=20, bits=64),
        # the inviscid airfoil workload, single block, single grid, LU-SGS
        dict(name="euler_257x65", kind="march", flow="airfoil", nx=257, ny=65, blocks=1, flux="ROE", recon="ORIGINAL",
             scheme="MUSCL3", time="lusgs", mesh=1, steps=10, bits=64),
        # the laminar flat plate, two blocks, 3-level V-cycle: the workload
        # the headline metric is quoted on
        dict(name="plate_97x97_v", kind="march", flow="plate", nx=97, ny=97, blocks=2, flux="AUSM", recon="ORIGINAL",
             scheme="MUSCL3", time="lusgs", mesh=3, steps=10, bits=64),
        # the same with the FP32 LU-SGS sweeps (mixed precision)
        dict(name="plate_97x97_v32", kind="march", flow="plate", nx=97, ny=97, blocks=2, flux="AUSM",
             recon="ORIGINAL", scheme="MUSCL3", time="lusgs", mesh=3, steps=10, bits=32),
        # RANS with the SA model on four blocks, WENO5 patch, 3-level V-cycle
        dict(name="rans_sa_513x129", kind="march", flow="sa", nx=513, ny=129, blocks=4, flux="ROE", recon="ORIGINAL",
             scheme="MUSCL3", time="lusgs", mesh=3, steps=5, bits=64),
        # the same airfoil with the SST model
        dict(name="rans_sst_513x129", kind="march", flow="sst", nx=513, ny=129, blocks=4, flux="ROE",
             recon="ORIGINAL", scheme="MUSCL3", time="lusgs", mesh=3, steps=5, bits=64),
        # a batched polar: SA cases of uneven grids in one context, mixed
        # precision, coarse levels keeping the eddy viscosity
        dict(name="polar_16", kind="polar", cases=16, grids=20261203, steps=4, bits=32),
        # a grid far larger than the caches, explicit third-order Runge-Kutta
        dict(name="plate_1025x513_rk3", kind="march", flow="plate", nx=1025, ny=513, blocks=2, flux="AUSM",
             recon="ORIGINAL", scheme="MUSCL3", time="rk3", mesh=1, steps=4, bits=64),
        # odd sizes with the other reconstruction path and flux in use:
        # characteristic WENO3, HLLC, explicit Runge-Kutta
        dict(name="plate_131x59_char", kind="march", flow="plate", nx=131, ny=59, blocks=2, flux="HLLC",
             recon="CHARACTERISTIC", scheme="WENO3", time="rk3", mesh=1, steps=5, bits=64),
        # one residual evaluation of a given state (a host with its own
        # iteration around the core)
        dict(name="residual_513x129", kind="residual", nx=513, ny=129, flux="ROE", scheme="MUSCL3"),
        # training steps of the warm-start network at its working batch
        dict(name="net_train", kind="train", cases=2, batch=16384, steps=10),
        # predictions for a ragged number of cells from host features
        dict(name="net_predict", kind="predict", rows=300007),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["airfoil", "plate", "plate", "vcycle", "vcycle", "rans", "polar", "residual", "train", "predict"])
    if kind == "airfoil":
        nx = 2 * _log(rng, 24, 200) + 1
        while (nx - 2 * ((nx - 1) // 8)) < 9:
            nx += 2
        return dict(kind="march", flow="airfoil", nx=nx, ny=_log(rng, 13, 140), blocks=1,
                    flux=rng.choice(["ROE", "VANLEER", "HLLC"]), recon=rng.choice(["ORIGINAL", "CONSERVATIVE"]),
                    scheme=rng.choice(["MUSCL3", "NND2"]), time=rng.choice(["lusgs", "lusgs", "euler"]), mesh=1,
                    steps=rng.randint(5, 20), bits=rng.choice([64, 64, 32]))
    if kind == "plate":
        n = _log(rng, 33, 800)
        return dict(kind="march", flow="plate", nx=n, ny=_log(rng, 33, 500) if n > 200 else _log(rng, 25, 160),
                    blocks=2, flux=rng.choice(["AUSM", "ROE", "HLLC"]),
                    recon=rng.choice(["ORIGINAL", "ORIGINAL", "CHARACTERISTIC"]),
                    scheme=rng.choice(["MUSCL3", "WENO3"]), time=rng.choice(["lusgs", "rk3"]), mesh=1,
                    steps=rng.randint(3, 6), bits=64)
    if kind == "vcycle":
        return dict(kind="march", flow="plate", nx=4 * _log(rng, 8, 48) + 1, ny=4 * _log(rng, 8, 48) + 1, blocks=2,
                    flux="AUSM", recon="ORIGINAL", scheme="MUSCL3", time="lusgs", mesh=rng.choice([2, 3]),
                    steps=rng.randint(5, 10), bits=rng.choice([64, 32]))
    if kind == "rans":
        return dict(kind="march", flow=rng.choice(["sa", "sst"]), nx=32 * rng.randint(10, 16) + 1,
                    ny=4 * rng.randint(16, 32) + 1, blocks=rng.choice([1, 4]), flux="ROE", recon="ORIGINAL",
                    scheme="MUSCL3", time="lusgs", mesh=3, steps=rng.randint(3, 5), bits=rng.choice([64, 32]))
    if kind == "polar":
        return dict(kind="polar", cases=rng.randint(3, 16), grids=rng.randint(1, 10 ** 6), steps=rng.randint(2, 5),
                    bits=rng.choice([32, 64]))
    if kind == "residual":
        nx = 8 * _log(rng, 8, 120) + 1
        return dict(kind="residual", nx=nx, ny=_log(rng, 17, 257), flux=rng.choice(["ROE", "AUSM"]), scheme="MUSCL3")
    if kind == "train":
        return dict(kind="train", cases=rng.randint(1, 3), batch=256 * _log(rng, 4, 64), steps=rng.randint(4, 10))
    return dict(kind="predict", rows=_log(rng, 500, 300007))


# ---- what a host has in hand ------------------------------------------------
def _problem(case, rng):
    """(Params, blocks, FDM blocks) of a marching or residual case; the flow
    conditions vary a little with the seed."""
    common = dict(Iflag_flux=FLUX[case["flux"]], Iflag_Scheme=SCHEME[case["scheme"]],
                  IFlag_Reconstruction=RECON[case.get("recon", "ORIGINAL")])
    nx, ny, flow = case["nx"], case["ny"], case.get("flow", "airfoil")
    if flow == "airfoil":
        p, blocks = workloads.euler_naca0012(nx, ny)
        p = p.replace(Ma=p.Ma * rng.uniform(0.9, 1.0), AoA=p.AoA * rng.uniform(0.8, 1.2))
        fdm = []
    elif flow == "plate":
        # the wall-normal stretching keeps the far field within some plate
        # lengths on tall grids
        p, _ = workloads.laminar_flat_plate(9, 9, num_mesh=case["mesh"])
        ratio = 1.1 if ny <= 100 else 1.0 + 9.5 / (ny - 1)
        blocks = grids.flat_plate(nx, ny, first=1.0e-4, ratio=ratio, x_lead=0.5, plate=1.0)
        p = p.replace(Re=p.Re * rng.uniform(0.9, 1.1))
        fdm = []
    else:
        p, blocks, fdm = workloads.rans_naca2412(nx, ny, nblocks=case["blocks"],
                                                 turb=TURB_SA if flow == "sa" else TURB_SST)
        p = p.replace(Ma=p.Ma * rng.uniform(0.95, 1.0), AoA=p.AoA * rng.uniform(0.8, 1.2))
    p = p.replace(Num_Mesh=case.get("mesh", 1), Time_Method=TIME[case.get("time", "lusgs")], **common)
    if p.Time_Method != TIME_LUSGS:
        p = p.replace(CFL=0.5)
    return p, blocks, fdm


def _start_state(p, b, rng):
    """U(NVAR,-1:nx+1,-1:ny+1) of a block: a uniform stream with a wall layer
    (viscous cases) and smooth disturbances of some per cent."""
    nv, g = p.nvar(), p.gamma
    ni, nj = b.nx + 2, b.ny + 2
    i = np.arange(ni + 1)[:, None]
    j = np.arange(nj + 1)[None, :]
    ph = rng.uniform(0.0, 2.0 * math.pi, 12)

    def wave(k):
        return (np.sin(0.31 * i + ph[k]) * np.cos(0.17 * j + ph[k + 1]) + 0.5 * np.sin(0.09 * (i + j) + ph[k + 2])) / 1.5

    a = math.radians(p.AoA)
    layer = 1.0
    if p.If_viscous:
        # distance of the cell from the grid line j = 1, cell by cell
        ic = np.clip(i - 2, 0, b.nx - 2)
        jc = np.clip(j - 2, 0, b.ny - 2)
        x = 0.25 * (b.x[ic, jc] + b.x[ic + 1, jc] + b.x[ic, jc + 1] + b.x[ic + 1, jc + 1])
        y = 0.25 * (b.y[ic, jc] + b.y[ic + 1, jc] + b.y[ic, jc + 1] + b.y[ic + 1, jc + 1])
        xw = 0.5 * (b.x[ic, 0] + b.x[ic + 1, 0])
        yw = 0.5 * (b.y[ic, 0] + b.y[ic + 1, 0])
        layer = np.tanh(np.hypot(x - xw, y - yw) / 0.02)
    amp = 0.02
    rho = 1.0 + amp * wave(0)
    u = (math.cos(a) + amp * wave(3)) * layer
    v = (math.sin(a) + amp * wave(6)) * layer
    pr = (1.0 + amp * wave(9)) / (g * p.Ma ** 2)
    U = torch.empty(nv * (ni + 1) * (nj + 1), dtype=torch.float64, pin_memory=True).numpy()
    U = U.reshape((nv, ni + 1, nj + 1), order="F")
    U[0], U[1], U[2] = rho, rho * u, rho * v
    U[3] = pr / (g - 1.0) + 0.5 * rho * (u * u + v * v)
    if nv == 5:
        U[4] = p.vt_inf / p.Re * (1.0 + 0.1 * wave(0))
    elif nv == 6:
        U[4] = 10.0 * p.Kt_inf * (1.0 + 0.1 * wave(0))
        U[5] = p.Wt_inf * (1.0 + 0.1 * wave(3))
    return U


def _march_state(s, problems, rng, steps):
    start = [(c, k, _start_state(p, b, rng)) for c, (p, blocks) in enumerate(problems, start=1)
             for k, b in enumerate(blocks, start=1)]
    # the host's buffer for the result: every block's U side by side
    out = torch.empty(sum(U.size for _, _, U in start), dtype=torch.float64, pin_memory=True)
    flat, back, at = out.numpy(), [], 0
    for c, k, U in start:
        back.append((c, k, flat[at:at + U.size].reshape(U.shape, order="F")))
        at += U.size
    return dict(kind="march", solver=s, ncase=len(problems), start=start, back=back, out=out, steps=steps)


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    if case["kind"] == "march":
        p, blocks, fdm = _problem(case, rng)
        s = gpu.Solver([(p, blocks)], fdm_blocks=[fdm])
        s.set_lusgs_precision(case["bits"])
        s.init_flow()
        return _march_state(s, [(p, blocks)], rng, case["steps"])
    if case["kind"] == "polar":
        problems = [(p.replace(Ma=p.Ma * rng.uniform(0.95, 1.0), AoA=p.AoA * rng.uniform(0.9, 1.1)), b)
                    for p, b in workloads.polar_cases(case["cases"], seed=case["grids"], max_size=(385, 97))]
        s = gpu.Solver(problems)
        s.set_lusgs_precision(case["bits"])
        s.mg_eddy_viscosity(1)
        s.init_flow()
        return _march_state(s, problems, rng, case["steps"])
    if case["kind"] == "residual":
        p, blocks, _ = _problem(case, rng)
        s = gpu.Solver([(p, blocks)])
        s.init_flow()
        st = _march_state(s, [(p, blocks)], rng, 0)
        st["kind"] = "residual"
        return st
    net = gpu.WarmStartNet(hidden=6, width=256, seed=seed % 65521 + 1)
    if case["kind"] == "train":
        chunk = learn.warmstart_cases(case["cases"], seed=seed)
        s = gpu.Solver([(p, b) for p, b, _ in chunk])
        s.init_flow()
        for c, (p, blocks, tc) in enumerate(chunk, start=1):
            s.set_case_shape(c, tc)
            for k, b in enumerate(blocks, start=1):
                s.upload_U(c, 1, k, _start_state(p, b, rng))
        net.add_samples(s)
        s.close()
        net.fit_normalization()
        return dict(kind="train", net=net, batch=case["batch"], steps=case["steps"])
    feat = np.empty((case["rows"], net.NIN), np.float32)
    lo = np.array([-0.5, -1.0, -6.0, 0.3, -2.0, 6.0, 0.09], np.float32)
    hi = np.array([2.0, 1.0, 1.3, 0.8, 8.0, 7.0, 0.15], np.float32)
    feat[:] = lo + (hi - lo) * rng.random(feat.shape, dtype=np.float32)
    mid, half = 0.5 * (lo + hi), (hi - lo) / math.sqrt(12.0)
    net.set_normalization(np.concatenate([mid, half, np.zeros(net.NOUT), np.full(net.NOUT, 0.1)]).astype(np.float32))
    return dict(kind="predict", net=net, feat=feat)


def run(st):
    if st["kind"] == "train":
        loss = st["net"].train(st["steps"], batch=st["batch"], lr=1e-3)
        return {"loss": loss, "weights": [list(st["net"].get_weights(l)) for l in range(st["net"].nlin)]}
    if st["kind"] == "predict":
        return st["net"].predict(st["feat"])
    s = st["solver"]
    for c, k, U in st["start"]:
        s.upload_U(c, 1, k, U)
    if st["kind"] == "residual":
        s.residual(1)
        norms = s.norms(1)
        return {"res": [s.field(c, 1, k, gpu.F_RES) for c, k, _ in st["start"]], "max": norms[0], "rms": norms[1]}
    s.bc(1)
    s.step(st["steps"])
    norms = [s.norms(c)[:2] for c in range(1, st["ncase"] + 1)]
    for c, k, view in st["back"]:
        s.download_U(c, 1, k, view)
    return {"U": st["out"], "max": np.array([n[0] for n in norms]), "rms": np.array([n[1] for n in norms])}


# ---- the work a pass cannot do without -----------------------------------------
def _cells(case):
    if case["kind"] == "polar":
        return case["cases"] * 26000.0  # the mean of the two grid sizes drawn
    per = (case["nx"] - 1) * (case["ny"] - 1)
    return per * (2 if case.get("flow") == "plate" else 1)


def work(case):
    if case["kind"] in ("train", "predict"):
        macs = 7 * 256 + 5 * 256 * 256 + 256 * 5
        if case["kind"] == "predict":
            return {"bytes": case["rows"] * (7 + 5) * 4, "flops": 2.0 * macs * case["rows"]}
        rows = case["steps"] * case["batch"]
        return {"bytes": rows * (7 + 5) * 4 + 2 * 4 * macs, "flops": 6.0 * macs * rows}
    # FP64 operations of one residual evaluation of a cell (primitives, two
    # faces, time step), of the turbulence model, the WENO5 patch and LU-SGS
    flow = "sa" if case["kind"] == "polar" else case.get("flow", "airfoil")
    n = _cells(case)
    nv = {"sa": 5, "sst": 6}.get(flow, 4)
    io = n * 8.0 * (2 * nv + 2)
    res = 600.0 if flow == "airfoil" else 950.0
    turb = {"sa": 350.0, "sst": 500.0}.get(flow, 0.0) + (1200.0 if case["kind"] == "march" and flow in ("sa", "sst")
                                                          else 0.0)
    if case["kind"] == "residual":
        return {"bytes": n * 8.0 * (nv + 2 + nv), "flops": n * res}
    sweep = 400.0
    mesh = 3 if case["kind"] == "polar" else case["mesh"]
    if mesh == 1:
        evals = 3.0 if case["time"] == "rk3" else 1.0
        step = evals * (res + turb) + (sweep if case["time"] == "lusgs" else 0.0)
    else:
        step = 2.0 * (res + turb) + sweep + 0.25 * (2.0 * res * (mesh - 1) / 2.0 + sweep)
    return {"bytes": io, "flops": case["steps"] * n * step}


# ---- the same in plain numpy, in 64 bits ------------------------------------------
def _muscl(q, axis):
    """van Albada-limited states on both sides of every face along an axis:
    q has two ghost layers, the result one entry per face."""
    q = np.moveaxis(q, axis, 0)
    ep, k3 = 1.0e-6, 1.0 / 3.0
    d = q[1:] - q[:-1]
    um, mid, up = d[:-2], d[1:-1], d[2:]
    s = (2.0 * mid * um + ep) / (mid * mid + um * um + ep)
    left = q[1:-2] + 0.25 * s * ((1.0 - k3 * s) * um + (1.0 + k3 * s) * mid)
    s = (2.0 * up * mid + ep) / (up * up + mid * mid + ep)
    right = q[2:-1] - 0.25 * s * ((1.0 - k3 * s) * up + (1.0 + k3 * s) * mid)
    return np.moveaxis(left, 0, axis), np.moveaxis(right, 0, axis)


def _roe(L, R, g):
    dl, ul, vl, pl = L
    dr, ur, vr, pr = R
    hl = g / (g - 1.0) * pl / dl + 0.5 * (ul * ul + vl * vl)
    hr = g / (g - 1.0) * pr / dr + 0.5 * (ur * ur + vr * vr)
    t = np.sqrt(dr / dl)
    d = 0.25 * dl * (1.0 + t) ** 2
    u, v, h = (ul + t * ur) / (1.0 + t), (vl + t * vr) / (1.0 + t), (hl + t * hr) / (1.0 + t)
    a = np.sqrt((g - 1.0) * (h - 0.5 * (u * u + v * v)))
    fix = 0.1
    lam = [np.abs(u - a), np.abs(u), np.abs(u + a)]
    lam = [np.where(l < fix, (l * l + fix * fix) / (2.0 * fix), l) for l in lam]
    dp = pr - pl
    a0 = (d * a * (ul - ur) + dp) / (2.0 * a * a)
    a1 = dr - dl - dp / (a * a)
    a2 = d * (vr - vl) / a
    a3 = (d * a * (ur - ul) + dp) / (2.0 * a * a)
    w0, w1, w2, w3 = lam[0] * a0, lam[1] * a1, lam[1] * a2, lam[2] * a3
    F = [dl * ul + dr * ur, dl * ul * ul + pl + dr * ur * ur + pr, dl * ul * vl + dr * ur * vr,
         dl * ul * hl + dr * ur * hr]
    D = [w0 + w1 + w3, w0 * (u - a) + w1 * u + w3 * (u + a), (w0 + w1 + w3) * v + w2 * a / a,
         w0 * (h - u * a) + w1 * 0.5 * (u * u + v * v) + w2 * v + w3 * (h + u * a)]
    return [0.5 * (f - e) for f, e in zip(F, D)]


def _ausm(L, R, g):
    dl, ul, vl, pl = L
    dr, ur, vr, pr = R
    hl = g / (g - 1.0) * pl / dl + 0.5 * (ul * ul + vl * vl)
    hr = g / (g - 1.0) * pr / dr + 0.5 * (ur * ur + vr * vr)
    a = 0.5 * (np.sqrt(g * pl / dl) + np.sqrt(g * pr / dr))
    ml, mr = ul / a, ur / a
    sl, sr = np.abs(ml) >= 1.0, np.abs(mr) >= 1.0
    m4 = np.where(sl, 0.5 * (ml + np.abs(ml)), 0.25 * (ml + 1.0) ** 2 + 0.125 * (ml * ml - 1.0) ** 2)
    p5 = np.where(sl, (ml > 0.0) * 1.0,
                  0.25 * (ml + 1.0) ** 2 * (2.0 - ml) + 3.0 / 16.0 * ml * (ml * ml - 1.0) ** 2)
    n4 = np.where(sr, 0.5 * (mr - np.abs(mr)), -0.25 * (mr - 1.0) ** 2 - 0.125 * (mr * mr - 1.0) ** 2)
    q5 = np.where(sr, 0.5 * (mr - np.abs(mr)) / mr,
                  0.25 * (mr - 1.0) ** 2 * (2.0 + mr) - 3.0 / 16.0 * mr * (mr * mr - 1.0) ** 2)
    m = m4 + n4
    flow = a * (dl * np.maximum(m, 0.0) + dr * np.minimum(m, 0.0))
    dm = a * np.abs(m) * np.where(m >= 0.0, dl, dr)
    return [flow, 0.5 * flow * (ul + ur) - 0.5 * dm * (ur - ul) + pl * p5 + pr * q5,
            0.5 * flow * (vl + vr) - 0.5 * dm * (vr - vl), 0.5 * flow * (hl + hr) - 0.5 * dm * (hr - hl)]


def _exact_residual(case, seed):
    rng = np.random.default_rng(seed)
    p, blocks, _ = _problem(case, rng)
    g = p.gamma
    out = []
    for b in blocks:
        U = np.array(_start_state(p, b, rng))
        rho, u, v = U[0], U[1] / U[0], U[2] / U[0]
        pr = (g - 1.0) * (U[3] - 0.5 * rho * (u * u + v * v))
        q = np.stack([rho, u, v, pr])
        x, y = b.x, b.y
        total = 0.0
        for axis in (0, 1):
            # faces of the interior cells along this axis; their normals point
            # to increasing i (j)
            if axis == 0:
                dx, dy = x[:, 1:] - x[:, :-1], y[:, 1:] - y[:, :-1]
                nx, ny = dy, -dx
                w = q[:, :, 2:-2]
            else:
                dx, dy = x[1:] - x[:-1], y[1:] - y[:-1]
                nx, ny = -dy, dx
                w = q[:, 2:-2, :]
            s = np.hypot(dx, dy)
            nx, ny = nx / s, ny / s
            L, R = _muscl(w, axis + 1)
            turn = [[S[0], S[1] * nx + S[2] * ny, -S[1] * ny + S[2] * nx, S[3]] for S in (L, R)]
            F = (_roe if case["flux"] == "ROE" else _ausm)(turn[0], turn[1], g)
            F = -np.stack([F[0], F[1] * nx - F[2] * ny, F[1] * ny + F[2] * nx, F[3]]) * s
            total = total + np.diff(F, axis=axis + 1)
        out.append(total)
    flat = np.concatenate([r.reshape(4, -1) for r in out], axis=1)
    pad = np.zeros(2)
    return {"res": [r.reshape(-1, order="F") for r in out], "max": np.concatenate([np.abs(flat).max(1), pad]),
            "rms": np.concatenate([np.sqrt((flat ** 2).mean(1)), pad])}


def _exact_predict(case, seed):
    st = prepare(case, seed)
    net, feat = st["net"], st["feat"].astype(np.float64)
    nrm = net.get_normalization().astype(np.float64)
    h = (feat - nrm[:7]) / nrm[7:14]
    for l in range(net.nlin):
        w, b = (a.astype(np.float64) for a in net.get_weights(l))
        w = w[:, :h.shape[1]]
        h = h @ w.T + b
        if l + 1 < net.nlin:
            h = h / (1.0 + np.exp(-h))
    return h[:, :5] * nrm[19:24] + nrm[14:19]


def exact(case, seed):
    if case["kind"] == "residual":
        return _exact_residual(case, seed)
    if case["kind"] == "predict":
        return _exact_predict(case, seed)
    return None
