"""The work a user has this framework do, as cases that can be timed and whose outputs can be compared.

A case is one pass through the public entry points: a run of a drop-impact simulation from its initial state
(`Fluid2D`, `Batch`), one solve of a linear system of the step (`MgsMac`, `MgsMacNeumann`, `MgsFem`, `ViscoImpl`,
`TriSolve`), or one prediction or training step of the learned guess's network (`learned.UNet`). Sizes, physics and
options are those of the repository's configurations, tests and benchmark.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import vdropimpact_b200 as V
from vdropimpact_b200 import learned

# ------------------------------------------------------------------ cases


def listed():
    return [
        # One tridiagonal system of the gas layer over 2048 liquid cells, on host arrays: the smallest call.
        {"name": "tri_2049", "kind": "tri", "m": 2049},
        # The projection system on a coarse grid, as in parameter studies: launches and latency.
        {"name": "mac_64x32", "kind": "mac", "m": 64, "n": 32, "prec": "fp64"},
        # The single-projection workload: 64 Gaussian sources on 2048 x 1024 square cells.
        {"name": "mac_2048x1024", "kind": "mac", "m": 2048, "n": 1024, "prec": "fp64"},
        # A projection on a grid with odd factors in its sides.
        {"name": "mac_1000x500", "kind": "mac", "m": 1000, "n": 500, "prec": "fp64"},
        # The finite-element projection of a 1024 x 512 simulation, in the mixed precision.
        {"name": "fem_1025x513_mixed", "kind": "fem", "m": 1025, "n": 513, "prec": "mixed"},
        # One implicit viscous system at the coupling of the 100 cSt workload (about 0.4).
        {"name": "visc_1024x512", "kind": "visc", "m": 1024, "n": 512, "prec": "fp64", "vf": 0.4, "x_sym": True,
         "horizontal": True},
        # The paper's initial-deceleration case with the class's default options (eager launches, FP64, linear guess).
        {"name": "sim_256x128_eager", "kind": "sim", "m": 256, "n": 128, "steps": 8, "nu": 32.0, "big": False,
         "x_sym": True, "implicit": True, "prec": "fp64", "guess": "linear", "graph": False, "rtol": 1e-10},
        # A grid with odd factors in its sides, at the tolerance of the parity tests, replayed as a graph.
        {"name": "sim_200x100", "kind": "sim", "m": 200, "n": 100, "steps": 5, "nu": 5.0, "big": False,
         "x_sym": True, "implicit": True, "prec": "fp64", "guess": "linear", "graph": True, "rtol": 1e-12},
        # The benchmark's workload and headline options: 100 cSt liquid deposition, 2048 x 1024.
        {"name": "sim_2048x1024_mixed", "kind": "sim", "m": 2048, "n": 1024, "steps": 8, "nu": 100.0, "big": True,
         "x_sym": True, "implicit": True, "prec": "mixed", "guess": "quadratic", "graph": True, "rtol": 1e-10},
        # A viscosity and velocity sweep over uneven grids stepped as one batch.
        {"name": "batch_6", "kind": "batch", "sizes": "256,512,256,1024,512,256", "steps": 5, "prec": "mixed",
         "guess": "quadratic", "rtol": 1e-10},
        # The learned guess of the 2048 x 1024 workload, restricted by 4: one prediction.
        {"name": "unet_256x512", "kind": "unet", "H": 256, "W": 512, "batch": 1},
        # The benchmark's training step of that network.
        {"name": "unet_train_256x512_b8", "kind": "train", "H": 256, "W": 512, "batch": 8},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    """One more case of the ranges the listed ones stand for."""
    kind = rng.choice(["tri", "mac", "mac", "neumann", "fem", "fem", "visc", "visc", "sim", "sim", "sim", "sim",
                       "unet", "train"])
    if kind == "tri":
        return {"kind": "tri", "m": int(_log(rng, 40, 4095))}
    if kind in ("unet", "train"):
        H = 8 * int(_log(rng, 4, 32))
        W = 16 * int(_log(rng, 4, 32))
        b = rng.randint(1, 8)
        return {"kind": kind, "H": H, "W": W, "batch": b}
    if kind == "sim":
        any_size = rng.random() < 0.4
        if any_size:
            # sizes without enough factors of two take the tests' tight tolerance
            m = int(_log(rng, 64, 900))
            n = max(32, int(m * rng.uniform(0.35, 0.7)))
        else:
            q = rng.choice([32, 64])
            m = q * 2 ** rng.randint(1, 5)
            n = m // 2
        prec = "fp64" if any_size else rng.choice(["fp64", "mixed", "mixed", "hybrid"])
        return {"kind": "sim", "m": m, "n": n, "steps": rng.randint(3, 6), "nu": round(_log(rng, 1, 100), 3),
                "big": rng.random() < 0.5, "x_sym": rng.random() < 0.8, "implicit": rng.random() < 0.85,
                "prec": prec, "guess": rng.choice(["linear", "quadratic"]), "graph": rng.random() < 0.75,
                "rtol": 1e-12 if any_size else 1e-10}
    if rng.random() < 0.5:
        m = int(_log(rng, 48, 1500))
        n = max(24, int(m * rng.uniform(0.35, 0.9)))
    else:
        q = rng.choice([16, 24, 32])
        m = q * 2 ** rng.randint(1, 6)
        n = m // 2
    prec = rng.choice(["fp64", "fp64", "mixed", "hybrid"]) if m <= 1024 else "fp64"
    if kind == "fem":
        return {"kind": "fem", "m": m + 1, "n": n + 1, "prec": prec}
    if kind == "visc":
        return {"kind": "visc", "m": m, "n": n, "prec": prec, "vf": round(_log(rng, 0.02, 2.0), 4),
                "x_sym": rng.random() < 0.8, "horizontal": rng.random() < 0.5}
    return {"kind": kind, "m": m, "n": n, "prec": prec}


# ----------------------------------------------------------------- inputs


def _cfg(m, n, nu, big, x_sym, implicit, rng):
    """A .cfg of the sweep's kind: viscosity and impact velocity vary with the seed."""
    nu = nu * math.exp(rng.uniform(-0.15, 0.15))
    vel = rng.uniform(0.4, 0.5)
    lines = [f"grid_points {m} {n}", f"L_nd {45 if big else 30}", "h0_nd 15", f"t_end_nd {100 if big else 50}",
             "frames 250", "tmult 8e-3", f"nul_cSt {nu:.9g}", "rhol 997.96", "R 1.5e-3", f"V {vel:.9g}", "gamma 1.4",
             "sigma 72e-3", "mug 1.820775e-5", "Pamb 1e5", "gas_layer_model"]
    if x_sym:
        lines.append("x_sym")
    if implicit:
        lines.append("implicit_visc")
    return "\n".join(lines) + "\n"


def _source(case, seed):
    """The source of a linear system, (n, m) float64 on the host."""
    m, n, kind = case["m"], case["n"], case["kind"]
    if kind in ("mac", "neumann"):
        b = V.projection_source(m, n, seed).reshape(n, m)
        return b + 0.37 if kind == "neumann" else b
    if kind == "fem":
        # sources scaled by the cell's area over a bottom row that sets the gas pressure (a_cc times its value)
        h = 1.0 / (m - 1)
        b = V.projection_source(m, n, seed).reshape(n, m) * h * h
        x = np.arange(m) * h
        rng = np.random.default_rng(seed + 1)
        p = rng.uniform(0.5, 1.5) * np.exp(-(x - rng.uniform(0, 0.2)) ** 2 / 0.05)
        a_cc = np.full(m, 4.0 / 3.0)
        a_cc[0] = a_cc[-1] = 2.0 / 3.0
        b[0] = a_cc * p
        return b
    # a velocity field: smooth structures with a little grid-scale content
    rng = np.random.default_rng(seed + 2)
    return V.projection_source(m, n, seed).reshape(n, m) + 0.01 * rng.standard_normal((n, m))


def _tri(case, seed):
    """A diagonally dominant system, as the gas layer's Newton steps give."""
    m = case["m"]
    rng = np.random.default_rng(seed)
    a = -rng.uniform(0.5, 1.5, m)
    c = -rng.uniform(0.5, 1.5, m)
    b = np.abs(a) + np.abs(c) + rng.uniform(0.05, 0.5, m)
    a[0] = c[-1] = 0.0
    return a, b, c, rng.standard_normal(m)


# the U-Net's layers: input and output channels, source sampling (0 direct, 1 upsampled by two, 2 pooled 2 x 2),
# ReLU, index of the skip added before it, index of the source layer
_NET = [(16, 16, 0, 1, -1, -1), (16, 16, 0, 1, -1, 0), (16, 32, 2, 1, -1, 1), (32, 32, 0, 1, -1, 2),
        (32, 64, 2, 1, -1, 3), (64, 64, 0, 1, -1, 4), (64, 64, 2, 1, -1, 5), (64, 64, 0, 1, -1, 6),
        (64, 64, 1, 1, 5, 7), (64, 32, 0, 1, -1, 8), (32, 32, 1, 1, 3, 9), (32, 16, 0, 1, -1, 10),
        (16, 16, 1, 1, 1, 11), (16, 16, 0, 0, -1, 12)]
_LEVEL = [0, 0, 1, 1, 2, 2, 3, 3, 2, 2, 1, 1, 0, 0]
_LR = 3e-4


def _net_params(seed):
    """All parameters in get_params' order (per layer: weights [9][cout][cin], then biases)."""
    rng = np.random.default_rng(seed + 3)
    out = []
    for ci, co, *_ in _NET:
        out.append(rng.standard_normal(9 * co * ci) * math.sqrt(1.6 / (9 * ci)))
        out.append(rng.uniform(-0.05, 0.05, co))
    return np.concatenate(out).astype(np.float32)


def _net_images(case, seed):
    """RMS-normalised residual-like images and their targets, (B, H, W) float32."""
    B, H, W = case["batch"], case["H"], case["W"]
    g = torch.Generator().manual_seed(seed)
    x = torch.randn(B, H, W, generator=g)
    s = torch.nn.functional.avg_pool2d(x[:, None], 5, 1, 2)[:, 0]
    x = x + 4 * s
    x = x / x.square().mean().sqrt()
    t = torch.nn.functional.avg_pool2d(x[:, None], 9, 1, 4)[:, 0]
    return x, t / t.square().mean().sqrt()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "tri":
        return {"kind": kind, "solver": V.TriSolve(case["m"]), "system": _tri(case, seed)}
    if kind in ("unet", "train"):
        net = learned.UNet(case["H"], case["W"], batch=case["batch"], seed=1)
        net.set_params(_net_params(seed))
        x, t = _net_images(case, seed)
        return {"kind": kind, "net": net, "x": x.cuda(), "t": t.cuda()}
    if kind == "sim":
        rng = np.random.default_rng(seed)
        f = V.Fluid2D(_cfg(case["m"], case["n"], case["nu"], case["big"], case["x_sym"], case["implicit"], rng),
                      mg_rtol=case["rtol"], mg_precision=case["prec"], mg_guess=case["guess"], graph=case["graph"])
        return {"kind": kind, "sim": f, "dt": f.frame_dt(), "steps": case["steps"]}
    if kind == "batch":
        rng = np.random.default_rng(seed)
        cfgs = [_cfg(int(m), int(m) // 2, nu, nu >= 25, True, True, rng)
                for m, nu in zip(case["sizes"].split(","), (30.0, 10.0, 3.0, 60.0, 20.0, 90.0))]
        b = V.Batch(cfgs, mg_rtol=case["rtol"], mg_precision=case["prec"], mg_guess=case["guess"])
        return {"kind": kind, "batch": b, "dts": b.frame_dts(), "steps": case["steps"]}
    m, n = case["m"], case["n"]
    if kind == "fem":
        s = V.MgsFem(m, n, 1.0 / (m - 1), 1.0 / (m - 1))
    elif kind == "visc":
        s = V.ViscoImpl(m, n, case["x_sym"], case["horizontal"], case["vf"], case["vf"])
    else:
        s = (V.MgsMac if kind == "mac" else V.MgsMacNeumann)(m, n, 1.0 / m, 1.0 / m)
    s.b.copy_(torch.from_numpy(_source(case, seed).ravel()))
    return {"kind": kind, "solver": s, "prec": case["prec"]}


class _Device:
    """A device array of the simulation, for torch.as_tensor, whose tensor keeps this object and so the simulation."""

    def __init__(self, sim, ptr, n):
        self.sim = sim
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<f8", "data": (ptr, False), "version": 3}


def _fields(sim):
    """The state a frame shows: velocity, pressure, gas-layer height and gas pressure, as views of device memory."""
    return {name: torch.as_tensor(_Device(sim, *sim.device_field(k)), device="cuda")
            for name, k in (("u", 0), ("v", 1), ("p", 2), ("h", 3), ("pg", 4))}


def run(state):
    kind = state["kind"]
    if kind == "tri":
        s = state["solver"]
        a, b, c, d = state["system"]
        s.a[:], s.b[:], s.c[:] = a, b, c
        s.d = d
        return {"d": s.solve_lapack()}
    if kind == "unet":
        return {"y": state["net"].forward(state["x"])}
    if kind == "train":
        loss = state["net"].train_step(state["x"], state["t"], _LR)
        return {"loss": loss, "params": state["net"].get_params()}
    if kind == "sim":
        f = state["sim"]
        f.init_fields()
        f.step_forward(state["dt"], state["steps"])
        return _fields(f)
    if kind == "batch":
        b = state["batch"]
        b.init_fields()
        b.step_forward(state["dts"], state["steps"])
        return [_fields(f) for f in b.sims]
    s = state["solver"]
    if kind == "visc":
        s.z.copy_(s.b)      # the velocity itself is the starting iterate
    else:
        s.z.zero_()
    s.solve_v_cycle(precision=state["prec"])
    return {"z": s.z}


# ------------------------------------------------------------------- work


def work(case):
    kind = case["kind"]
    if kind == "tri":
        return {"bytes": 40.0 * case["m"], "flops": 8.0 * case["m"]}
    if kind in ("unet", "train"):
        px = [case["batch"] * (case["H"] >> lv) * (case["W"] >> lv) for lv in _LEVEL]
        fl = sum(18.0 * ci * co * p for (ci, co, *_), p in zip(_NET, px))
        # every layer's BF16 output is written and read once (twice in the backward pass), with its FP32 gradient
        act = sum(2.0 * co * p for (_, co, *_), p in zip(_NET, px))
        if kind == "unet":
            return {"bytes": 2 * act, "flops": fl}
        return {"bytes": 8 * act, "flops": 3 * fl}
    if kind == "sim":
        # u, v and p read and written by every step
        return {"bytes": 48.0 * case["m"] * case["n"] * case["steps"], "flops": 200.0 * case["m"] * case["n"] * case["steps"]}
    if kind == "batch":
        cells = sum(int(m) * (int(m) // 2) for m in case["sizes"].split(","))
        return {"bytes": 48.0 * cells * case["steps"], "flops": 200.0 * cells * case["steps"]}
    return {"bytes": 16.0 * case["m"] * case["n"], "flops": 20.0 * case["m"] * case["n"]}


# ------------------------------------------------------------------ exact


def _thomas(lo, di, up, d):
    """Tridiagonal solves along dim 0 of d (n, k), one system per column, coefficients (n, k)."""
    n = d.shape[0]
    cp, dp = torch.empty_like(d), torch.empty_like(d)
    cp[0] = up[0] / di[0]
    dp[0] = d[0] / di[0]
    for j in range(1, n):
        den = di[j] - lo[j] * cp[j - 1]
        cp[j] = up[j] / den
        dp[j] = (d[j] - lo[j] * dp[j - 1]) / den
    x = torch.empty_like(d)
    x[n - 1] = dp[n - 1]
    for j in range(n - 2, -1, -1):
        x[j] = dp[j] - cp[j] * x[j + 1]
    return x


def _rows(n, k, v):
    return torch.full((n, k), float(v), dtype=torch.float64)


def _exact_cells(case, b):
    """The MAC systems: cosines in x, one tridiagonal system in y per mode."""
    m, n = case["m"], case["n"]
    kx = ky = float(m) * m
    neumann = case["kind"] == "neumann"
    if neumann:
        b = b - b.mean()
    i = torch.arange(m, dtype=torch.float64)
    B = torch.cos(math.pi * (i[:, None] + 0.5) * i[None, :] / m)
    w = torch.full((m,), 2.0 / m, dtype=torch.float64)
    w[0] = 1.0 / m
    beta = (b @ B) * w
    lam = -4.0 * kx * torch.sin(0.5 * math.pi * i / m) ** 2
    di = _rows(n, m, -2.0 * ky) + lam
    di[0] += ky if neumann else -ky
    di[n - 1] += ky
    lo, up = _rows(n, m, ky), _rows(n, m, ky)
    if neumann:
        # the constant mode is determined up to a constant: its last value is set to zero
        di[n - 1, 0], lo[n - 1, 0], beta[n - 1, 0] = 1.0, 0.0, 0.0
    z = _thomas(lo, di, up, beta) @ B.T
    return z - z.mean() if neumann else z


def _exact_fem(case, b):
    """The bilinear finite-element system on square cells: cosines over the nodes in x."""
    m, n = case["m"], case["n"]
    i = torch.arange(m, dtype=torch.float64)
    B = torch.cos(math.pi * i[:, None] * i[None, :] / (m - 1))
    end = torch.ones(m, dtype=torch.float64)
    end[0] = end[-1] = 0.5
    # each row of the operator carries the end weights, so row j's source is W B beta
    beta = (b @ B) * (2.0 / (m - 1)) * end
    co = torch.cos(math.pi * i / (m - 1))
    # rows: 8/3 on the point, -1/3 on each of its eight neighbours; half of both at the top
    di = _rows(n, m, 8.0 / 3.0) - (2.0 / 3.0) * co
    off = (-1.0 / 3.0 - (2.0 / 3.0) * co).expand(n, m).clone()
    di[n - 1] *= 0.5
    z0 = b[0] / (end * (4.0 / 3.0))
    a0 = (z0 * end) @ B * (2.0 / (m - 1)) * end
    rhs = beta[1:].clone()
    rhs[0] -= off[1] * a0
    a = _thomas(off[1:], di[1:], off[1:], rhs)
    return torch.cat([z0[None], a @ B.T])


def _exact_visc(case, b):
    """The viscous system: an eigenbasis of the x operator, one tridiagonal system in y per mode."""
    m, n, k = case["m"], case["n"], case["vf"]
    d = torch.full((m,), 2 * k, dtype=torch.float64)
    if case["x_sym"]:
        d[0] = 3 * k if case["horizontal"] else k
    off = torch.full((m - 1,), -k, dtype=torch.float64)
    lam, Q = torch.linalg.eigh(torch.diag(d) + torch.diag(off, 1) + torch.diag(off, -1))
    di = _rows(n, m, 1 + 2 * k) + lam
    di[0] -= k
    return _thomas(_rows(n, m, -k), di, _rows(n, m, -k), b @ Q) @ Q.T


def _net_forward(case, params, x):
    """The network in float64; returns its output and the parameter leaves."""
    inp = torch.zeros(case["batch"], 16, case["H"], case["W"], dtype=torch.float64, device=x.device)
    inp[:, 0] = x
    acts, leaves, off = [], [], 0
    for k, (ci, co, mode, relu, skip, src) in enumerate(_NET):
        w = params[off:off + 9 * ci * co].clone().requires_grad_()
        b = params[off + 9 * ci * co:off + 9 * ci * co + co].clone().requires_grad_()
        off += 9 * ci * co + co
        leaves += [w, b]
        s = inp if src < 0 else acts[src]
        if mode == 1:
            s = s.repeat_interleave(2, dim=2).repeat_interleave(2, dim=3)
        elif mode == 2:
            s = torch.nn.functional.avg_pool2d(s, 2)
        y = torch.nn.functional.conv2d(s, w.reshape(3, 3, co, ci).permute(2, 3, 0, 1), b, padding=1)
        if skip >= 0:
            y = y + acts[skip]
        acts.append(torch.relu(y) if relu else y)
    return acts[-1][:, 0], leaves


def exact(case, seed):
    kind = case["kind"]
    if kind in ("sim", "batch"):
        return None
    if kind == "tri":
        a, b, c, d = (torch.from_numpy(v)[:, None] for v in _tri(case, seed))
        return {"d": _thomas(a, b, c, d)[:, 0]}
    if kind in ("unet", "train"):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        x, t = (v.double().to(dev) for v in _net_images(case, seed))
        p = torch.from_numpy(_net_params(seed)).double().to(dev)
        y, leaves = _net_forward(case, p, x)
        if kind == "unet":
            return {"y": y.detach()}
        loss = torch.mean((y - t) ** 2)
        g = torch.cat([q.reshape(-1) for q in torch.autograd.grad(loss, leaves)])
        # the first Adam step: the moments' bias corrections cancel their weights
        return {"loss": float(loss.detach()), "params": (p - _LR * g / (g.abs() + 1e-8)).cpu().numpy()}
    b = torch.from_numpy(_source(case, seed))
    z = (_exact_fem if kind == "fem" else _exact_visc if kind == "visc" else _exact_cells)(case, b)
    return {"z": z.reshape(-1)}
