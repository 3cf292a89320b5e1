"""The workloads whose time is measured: the implicit time step of the
well-mixed film and of the ConcZ model, the linear solve behind them, the
batched ensemble and the training pass of the learned preconditioner, each
through the package's public entry points.

A pass of a step case starts from the same film every time (a host array in
pinned memory, uploaded, one time step, the film read back): that is the call
of a host program that owns the fields, and it keeps the work of a pass the
same however many passes were made before it.  The films are those of
yuzen_b200.cases with their free inputs (front angle, corrugation, noise,
bump centres) drawn from the seed.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import yuzen_b200 as yz
from yuzen_b200 import cases as yc
from yuzen_b200 import cz as ycz
from yuzen_b200 import ensemble as ye
from yuzen_b200 import learned as yl
from yuzen_b200 import step as ys

#: how a step's solves are set: arithmetic, and the solves one AMG set-up serves
ARMS = {"fp64": (yz.PREC_FP64, 0), "fp32": (yz.PREC_FP32_CYCLE, 0), "fp32_reuse": (yz.PREC_FP32_CYCLE, 64),
        "fp32m_reuse": (yz.PREC_FP32_MATRIX, 64)}
#: the adaptive films keep the dt they start with (the controller still tests every step)
KEEP = {"MaxDtFactor": 1.0e10, "MinDt": 1.0e-15, "Criterion": 1e-3, "KeepSteps": 1000000, "ChangeFactor": 0.75,
        "ScaleFloor": 0.0}


def listed():
    return [
        #  one linear solve handed over in host arrays (the solver seam): a small film, whose
        #  hierarchy is its direct level alone, and an ordinary one of several levels
        {"name": "solve_40", "kind": "solve", "N": 40},
        {"name": "solve_300", "kind": "solve", "N": 300},
        #  one time step on the drop-in FP64 path: the smallest film with every term on,
        #  the periodic spinodal film, the full-size film with every term on
        {"name": "step_allphys_64_fp64", "kind": "step", "film": "allphys", "N": 64, "arm": "fp64"},
        {"name": "step_spinodal_224_fp64", "kind": "step", "film": "spinodal", "N": 224, "arm": "fp64"},
        {"name": "step_allphys_512_fp64", "kind": "step", "film": "allphys", "N": 512, "arm": "fp64"},
        #  the FP32 forms: an odd size with a new AMG set-up every solve, the full-size film as
        #  a long run takes it (a kept hierarchy, the float matrix), and a film beyond it
        {"name": "step_bench2d_301_fp32", "kind": "step", "film": "bench2d", "N": 301, "arm": "fp32"},
        {"name": "step_allphys_512_fp32m", "kind": "step", "film": "allphys", "N": 512, "arm": "fp32m_reuse"},
        {"name": "step_bench2d_1024_fp32m", "kind": "step", "film": "bench2d", "N": 1024, "arm": "fp32m_reuse"},
        #  a batch of dewetting and levelling films of uneven size advanced together
        {"name": "ensemble_24", "kind": "ensemble", "count": 24, "steps": 4, "arm": "fp32_reuse"},
        #  the film with its concentration through the thickness: a small one, the full size
        {"name": "cz_64x16_fp64", "kind": "cz", "N": 64, "Nz": 16, "arm": "fp64"},
        {"name": "cz_256x16_fp64", "kind": "cz", "N": 256, "Nz": 16, "arm": "fp64"},
        #  the learned preconditioner's network: one pair's forward and backward pass
        {"name": "unet_grad_512", "kind": "unet", "N": 512},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "step", "step", "step", "step", "ensemble", "cz", "unet"])
    if kind == "solve":
        return {"kind": kind, "N": _log(rng, 24, 400)}
    if kind == "step":
        film = rng.choice(["allphys", "bench2d", "spinodal", "dewetting", "levelling"])
        lo, hi = {"allphys": (40, 640), "bench2d": (64, 800), "spinodal": (40, 512), "dewetting": (40, 512),
                  "levelling": (40, 512)}[film]
        return {"kind": kind, "film": film, "N": _log(rng, lo, hi), "arm": rng.choice(list(ARMS))}
    if kind == "ensemble":
        return {"kind": kind, "count": rng.randint(3, 24), "steps": rng.randint(2, 4),
                "arm": rng.choice(["fp64", "fp32_reuse"])}
    if kind == "cz":
        return {"kind": kind, "N": _log(rng, 16, 192), "Nz": rng.randint(6, 16),
                "arm": rng.choice(["fp64", "fp32_reuse"])}
    return {"kind": kind, "N": _log(rng, 48, 512)}


# ----------------------------------------------------------------------
#  inputs
# ----------------------------------------------------------------------
def _film(name, N, seed):
    rng = np.random.default_rng(seed)
    if name == "allphys":
        #  the oblique film edge at a seeded angle and place
        c = yc.allphys(N)
        dx = 5.0 / 512.0
        xs = (np.arange(N) + 0.5) * dx - 0.5 * N * dx
        X, Y = np.meshgrid(xs, xs)
        a = math.pi / 6.0 + rng.uniform(-0.15, 0.15)
        s = X * math.cos(a) + Y * math.sin(a) - rng.uniform(-0.1, 0.1) * N * dx
        c.h_init = 0.01 + 0.99 * 0.5 * (1.0 - np.tanh(s / (4.0 * dx)))
        return c
    if name == "bench2d":
        #  the substrate step under a film with a seeded long corrugation
        c = yc.bench2d_512(N)
        i = (np.arange(N) + 0.5) / N
        mode = np.outer(np.cos(math.pi * rng.integers(1, 4) * i), np.cos(math.pi * rng.integers(1, 4) * i))
        c.h_init = c.h_init * (1.0 + rng.uniform(0.01, 0.03) * mode)
        return c
    if name == "spinodal":
        c = yc.dewetting(N, 10.0, 1e-3, seed)
    elif name == "dewetting":
        c = yc.dewetting(N, rng.uniform(5.0, 20.0), 10.0 ** rng.uniform(-4.0, -2.0), seed)
    else:
        c = yc.levelling(N, 10.0 ** rng.uniform(-2.0, -1.0), int(rng.integers(1, 5)), seed)
    c.dtc = dict(KEEP)
    return c


def _batch(count, seed):
    """The ensemble's instances: the sizes and kinds of the benchmark's batch,
    the films' contact angles, amplitudes and noise from the seed."""
    rng = np.random.default_rng(seed)
    out = []
    for c in yc.batch(count):
        s = int(rng.integers(1 << 30))
        if c.name.startswith("dewetting"):
            out.append(yc.dewetting(c.Nx, rng.uniform(5.0, 20.0), 10.0 ** rng.uniform(-4.0, -2.0), s))
        else:
            out.append(yc.levelling(c.Nx, 10.0 ** rng.uniform(-2.0, -1.0), int(rng.integers(1, 5)), s))
    return out


def _pinned(a):
    p = torch.empty(a.size, dtype=torch.float64, pin_memory=True).numpy()
    p[:] = a
    return p


def _step(film, N, seed, arm):
    c = _film(film, N, seed)
    s0 = c.state()
    st = ys.Step(ys.params_from_state(s0), s0["field_h0"], s0["field_c0"], s0["field_s0"])
    precision, reuse = ARMS[arm]
    st.set_precision(precision)
    st.set_amg_reuse(reuse)
    return st, s0


def prepare(case, seed):
    kind = case["kind"]
    if kind == "solve":
        st, s0 = _step("allphys", case["N"], seed, "fp64")
        rowptr, col, _ = st.pattern()
        values, rhs = st.system(s0["field_h0"], s0["field_h0"], s0["dt"])
        st.close()
        #  the column-sorted mirror of the pattern and where its entries come from
        row = np.repeat(np.arange(rowptr.size - 1), np.diff(rowptr))
        src = np.lexsort((col, row)).astype(np.int32)
        pat = yz.CrsPattern(rowptr, col, col[src], src)
        be = yz.MakeLinearSolverBackend("b200")
        be.SetPattern(pat)
        return {"kind": kind, "be": be, "pat": pat, "values": values, "rhs": rhs, "nx": s0["nx"],
                "set": yz.LinearSolverSettings(precondition=2, scaling=True, maxIteration=8000, epsilon=1e-11)}
    if kind == "step":
        st, s0 = _step(case["film"], case["N"], seed, case["arm"])
        n = st.n
        return {"kind": kind, "st": st, "h0": _pinned(s0["field_h0"]), "c0": _pinned(s0["field_c0"]),
                "h": _pinned(np.zeros(n)), "c": _pinned(np.zeros(n))}
    if kind == "ensemble":
        batch = _batch(case["count"], seed)
        precision, reuse = ARMS[case["arm"]]
        ens = ye.Ensemble(batch, precision=precision, amg_reuse=reuse)
        return {"kind": kind, "ens": ens, "steps": case["steps"], "start": [s.state() for s in ens.steps]}
    if kind == "cz":
        r = yc.cz_bumps(case["N"], case["Nz"], seed=seed).record()
        m = ycz.CzModel(ycz.params_from_record(r), r["xc"], r["xf"], r["yc"], r["yf"], r["h0"], r["s"], r["c0"])
        precision, reuse = ARMS[case["arm"]]
        m.set_precision(precision)
        m.set_amg_reuse(reuse)
        return {"kind": kind, "m": m, "h0": _pinned(r["h0"]), "c0": _pinned(r["c0"]), "h": _pinned(r["h0"]),
                "c": _pinned(r["c0"])}
    N = case["N"] + 4
    net = yl.UNet(N, N, capacity=4, seed=1)
    params, feat, target = _unet_inputs(N, net.param_count(), seed)
    net.set_params(params)
    return {"kind": kind, "net": net, "feat": feat, "target": target}


def run(state):
    kind = state["kind"]
    if kind == "solve":
        x = np.zeros(state["rhs"].size)
        ret, it, res = state["be"].Solve(state["set"], state["pat"], state["values"], state["rhs"], x)
        return {"ret": ret, "x": x}
    if kind == "step":
        st = state["st"]
        st.set_fields(state["h0"], state["c0"])
        r = st.advance(1)
        st.fields_into(state["h"], state["c"])
        return {"h": state["h"], "c": state["c"], "time_steps": r["steps"]}
    if kind == "ensemble":
        ens = state["ens"]
        for st, s0 in zip(ens.steps, state["start"]):
            st.set_state(s0)
        r = ens.advance(state["steps"])
        return {"films": [ens.fields(k)[0] for k in range(len(ens))], "time": np.array([x["time"] for x in r])}
    if kind == "cz":
        m = state["m"]
        m.set_fields(state["h0"], state["c0"])
        r = m.advance(1)
        m.fields_into(state["h"], state["c"])
        return {"h": state["h"], "c": state["c"], "time_steps": r["steps"]}
    loss, grad = state["net"].loss_grad(state["feat"], state["target"])
    return {"loss": np.float32(loss), "grad": grad}


# ----------------------------------------------------------------------
#  what a pass cannot do without
# ----------------------------------------------------------------------
#: (cin, cout, level) of the network's seven 3x3 convolutions
CONVS = [(16, 16, 0), (16, 32, 1), (32, 64, 2), (64, 64, 3), (128, 64, 2), (96, 32, 1), (48, 16, 0)]


def work(case):
    kind = case["kind"]
    if kind == "solve":
        n = (case["N"] + 4) ** 2
        #  the matrix's values and columns, the right-hand side, the answer
        return {"bytes": 13 * 12 * n + 16 * n, "flops": 2 * 13 * n}
    if kind == "step":
        n = (case["N"] + 4) ** 2
        #  h, c, s in, h and c out, and the Newton matrix of one pass written and read
        return {"bytes": 40 * n + 2 * 13 * 12 * n, "flops": 1000 * n}
    if kind == "ensemble":
        n = sum((c.Nx + 4) ** 2 for c in yc.batch(case["count"]))
        return {"bytes": (40 + 2 * 13 * 12) * n * case["steps"], "flops": 1000 * n * case["steps"]}
    if kind == "cz":
        n = (case["N"] + 4) ** 2
        m = n * (case["Nz"] + 4)
        #  the film's system twice (predictor, corrector), the concentration's once
        return {"bytes": 2 * 2 * 13 * 12 * n + 2 * 21 * 12 * m + 32 * (n + m), "flops": 2000 * n + 1000 * m}
    N = case["N"] + 4
    px = [N * N / 4 ** k for k in range(4)]
    flops = sum(3 * 2 * 9 * ci * co * px[lv] for ci, co, lv in CONVS)
    #  the feature maps and the target, every layer's activations written and read forward and
    #  backward in 16 bits, the parameters and their gradient
    acts = sum((ci + co) * px[lv] for ci, co, lv in CONVS)
    return {"bytes": 16 * N * N + 2 * 3 * acts, "flops": flops}


# ----------------------------------------------------------------------
#  64-bit values, where plain torch gives them
# ----------------------------------------------------------------------
def _unet_inputs(N, np_, seed):
    """Weights of variance 1 / fan-in, the residual a rough field, the two
    feature maps smooth ones, the target a smoothed residual."""
    rng = np.random.default_rng(seed)
    p = np.zeros(np_, np.float32)
    at = 0
    for ci, co, _ in CONVS:
        p[at:at + 9 * ci * co] = rng.normal(0.0, math.sqrt(1.0 / (9 * ci)), 9 * ci * co)
        at += 9 * ci * co + co
    p[at:at + 16] = rng.normal(0.0, 0.25, 16)
    i = np.arange(N) / N
    f1 = 0.3 + 0.2 * np.outer(np.cos(math.pi * rng.integers(1, 4) * i), np.cos(math.pi * i))
    f2 = 0.5 + 0.4 * np.tanh((i[:, None] + i[None, :] - 1.0 + rng.uniform(-0.2, 0.2)) * 8.0)
    r = rng.standard_normal((N, N))
    r /= math.sqrt(np.mean(r * r))
    t = 0.25 * (r + np.roll(r, 1, 0) + np.roll(r, 1, 1) + np.roll(r, (1, 1), (0, 1)))
    feat = np.stack([r, f1, f2]).reshape(3, -1).astype(np.float32)
    return p, feat, t.reshape(-1).astype(np.float32)


def _exact_solve(state):
    """The grid's rows taken two at a time make the matrix block tridiagonal
    (13-point rows reach two grid rows; the mirrored ghost rows their
    neighbours): block elimination in 64 bits."""
    pat, nx = state["pat"], state["nx"]
    n = pat.n
    b = 2 * nx
    nb = -(-n // b)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    row = torch.from_numpy(np.repeat(np.arange(n), np.diff(pat.rowptr))).to(dev)
    col = torch.from_numpy(pat.col.astype(np.int64)).to(dev)
    val = torch.from_numpy(state["values"]).to(dev)
    rhs = torch.zeros(nb * b, dtype=torch.float64, device=dev)
    rhs[:n] = torch.from_numpy(state["rhs"]).to(dev)
    D = torch.zeros(nb, 3, b, b, dtype=torch.float64, device=dev)
    if nb * b > n:
        k = torch.arange(n - (nb - 1) * b, b, device=dev)
        D[nb - 1, 1, k, k] = 1.0
    D.index_put_((row // b, col // b - row // b + 1, row % b, col % b), val, accumulate=True)
    y = rhs.reshape(nb, b, 1).clone()
    up = [None] * nb
    for k in range(nb):
        A = D[k, 1]
        if k:
            A = A - D[k, 0] @ up[k - 1]
            y[k] -= D[k, 0] @ y[k - 1]
        sol = torch.linalg.solve(A, torch.cat([D[k, 2], y[k]], 1))
        up[k], y[k] = sol[:, :b], sol[:, b:]
    for k in range(nb - 2, -1, -1):
        y[k] -= up[k] @ y[k + 1]
    return y.reshape(-1)[:n].cpu().numpy()


def _exact_unet(N, params, feat, target):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    F = torch.nn.functional
    p = torch.from_numpy(params).double().to(dev).requires_grad_(True)
    W, at = [], 0
    for ci, co, _ in CONVS:
        W.append(p[at:at + 9 * ci * co].reshape(co, 3, 3, ci).permute(0, 3, 1, 2))
        at += 9 * ci * co + co
    r, f1, f2 = (torch.from_numpy(feat[k]).double().to(dev).reshape(1, 1, N, N) for k in range(3))
    x = torch.cat([r, r * f1, r * f2, r * f1 * f1, r * f2 * f2, r * f1 * f2] + [torch.zeros_like(r)] * 10, 1)

    def conv(v, k):
        return F.conv2d(v, W[k], padding=1)

    def pool(v):
        return F.avg_pool2d(F.pad(v, (0, v.shape[3] % 2, 0, v.shape[2] % 2)), 2)

    def up(v, like):
        return F.interpolate(v, scale_factor=2, mode="nearest")[:, :, :like.shape[2], :like.shape[3]]

    e0 = conv(x, 0)
    e1 = conv(pool(e0), 1)
    e2 = conv(pool(e1), 2)
    b3 = conv(pool(e2), 3)
    d2 = conv(torch.cat([e2, up(b3, e2)], 1), 4)
    d1 = conv(torch.cat([e1, up(d2, e1)], 1), 5)
    d0 = conv(torch.cat([e0, up(d1, e0)], 1), 6)
    out = (d0 * p[at:at + 16].reshape(1, 16, 1, 1)).sum(1).reshape(-1) + p[at + 16]
    loss = ((out - torch.from_numpy(target).double().to(dev)) ** 2).sum() / (N * N)
    (g,) = torch.autograd.grad(loss, p)
    #  without activation the network has no biases: they stay 0 and take no gradient
    g = g.clone()
    at = 0
    for ci, co, _ in CONVS:
        at += 9 * ci * co
        g[at:at + co] = 0.0
        at += co
    g[at + 16] = 0.0
    return float(loss), g.cpu().numpy()


def exact(case, seed):
    kind = case["kind"]
    if kind == "solve":
        #  the film's first Newton system, solved directly
        return {"ret": None, "x": _exact_solve(prepare(case, seed))}
    if kind == "unet":
        N = case["N"] + 4
        params, feat, target = _unet_inputs(N, sum(9 * ci * co + co for ci, co, _ in CONVS) + 17, seed)
        loss, g = _exact_unet(N, params, feat, target)
        return {"loss": np.float64(loss), "grad": g}
    #  whole time steps: nonlinear iterations with no plain form short of the framework itself
    return None
