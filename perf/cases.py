"""Workloads of the residual path, for timing and for checking its results.

Each case is a job as a program of this framework runs it: a context set up
once (blocks, faces, conditions, precision), then passes that advance the
state a number of steps and read it back into host arrays for output, in the
precision the path keeps it in (FP32 primitives in the mixed precision, FP64
in the plain one).  The closure's training step is a case of its own.

`listed()` holds the named cases, `draw(rng)` another one of the same ranges;
`prepare` sets a case up, `run` is one pass, `work` counts the bytes and
operations a pass cannot do without, and `exact` is the same pass in FP64
PyTorch, written from the equations on whole arrays.
"""
import ctypes
import math

import numpy as np
import torch

import combustioncodegpu_b200 as cc
from combustioncodegpu_b200 import cases, closure

R_U = 8314.462618
GAMMA, MW_AIR = 1.4, 28.9647
G = 2  # ghost layers
FOUR = [("H2", {"H": 2}), ("O2", {"O": 2}), ("H2O", {"H": 2, "O": 1}), ("N2", {"N": 2})]
BC_IN, BC_OUT, WALL_T, WALL_Q = 5, 6, 2, 3  # labels: inflow, outflow, isothermal and adiabatic wall


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


# ------------------------------------------------------------------ the cases

def _case(name, kind, ni, nj, nk, precision="mixed", scheme="rk3", steps=10, species=9, viscous=True, cfl=0.5,
          distort=0.0, closure=False, monitor=False):
    """ni, nj, nk: points per axis, or a text with one size per block along the axis."""
    return {"name": name, "kind": kind, "ni": ni, "nj": nj, "nk": nk, "precision": precision, "scheme": scheme,
            "steps": steps, "species": species, "viscous": viscous, "cfl": cfl, "distort": distort,
            "closure": closure, "monitor": monitor}


def listed():
    return [
        # a shock tube, the smallest job: launch latency, no species, inviscid
        _case("sod_tube_fp64", "tube", 256, 8, 8, "fp64", steps=50, species=0, viscous=False),
        # a small box stepped one step at a time with its residual watched
        _case("box32_mixed_monitored", "box", 32, 32, 32, steps=20, monitor=True),
        # a four-species mixture: a mechanism of another size than the 9-species H2/O2/N2 set
        _case("box64_mixed_4species", "box", 64, 64, 64, steps=10, species=4),
        # the plain FP64 path on a curvilinear grid of odd sizes
        _case("box_fp64_curvilinear", "box", 97, 85, 71, "fp64", steps=15, distort=0.2),
        # the headline workload: 128^3 periodic viscous 9-species box, mixed precision, SSP-RK3
        _case("box128_mixed", "box", 128, 128, 128, steps=40),
        # uneven blocks joined at interfaces: halo-heavy, extents that are no multiples of a tile
        _case("multiblock_mixed", "blocks", "23,41,64", "33,48,20", "57,28", steps=10),
        # a thin mixing layer: half of the points are ghosts
        _case("mixing_layer_mixed", "layer", 512, 256, 4, steps=20),
        # a steady duct with inflow, outflow, both wall types; the residual of every step watched
        _case("channel_steady_mixed", "channel", 113, 66, 33, scheme="steady", steps=30, monitor=True),
        # implicit steady steps
        _case("box96_lusgs_mixed", "box", 96, 96, 96, scheme="lusgs", steps=10, cfl=5.0),
        # the learned transport closure in place of the Wilke evaluation
        _case("box112_closure_mixed", "box", 112, 112, 112, steps=10, closure=True),
        # training that closure: eight optimiser steps, forward and backward
        {"name": "closure_training", "kind": "training", "batch": 4096, "steps": 8},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["box", "box", "box", "box", "tube", "blocks", "layer", "channel", "training"])
    if kind == "training":
        return {"kind": kind, "batch": _log_int(rng, 1024, 12000), "steps": rng.randint(3, 8)}
    c = _case("", kind, 0, 0, 0, precision=rng.choice(["mixed", "mixed", "fp64"]), species=rng.choice([9, 9, 4]))
    if kind == "tube":
        c.update(ni=_log_int(rng, 64, 1024), nj=rng.randint(6, 16), nk=rng.randint(6, 16), species=0, viscous=False)
    elif kind == "blocks":
        sizes = lambda n: ",".join(str(_log_int(rng, 14, 60)) for _ in range(n))  # noqa: E731
        c.update(ni=sizes(rng.randint(2, 3)), nj=sizes(2), nk=sizes(2))
    elif kind == "layer":
        c.update(ni=_log_int(rng, 64, 640), nj=_log_int(rng, 48, 320), nk=rng.randint(4, 6))
    elif kind == "channel":
        c.update(ni=_log_int(rng, 24, 128), nj=_log_int(rng, 16, 80), nk=_log_int(rng, 8, 40),
                 scheme=rng.choice(["steady", "rk3"]), monitor=rng.random() < 0.5)
    else:
        n = _log_int(rng, 16, 100)
        side = lambda: max(12, min(112, int(n * rng.uniform(0.7, 1.3))))  # noqa: E731
        c.update(ni=side(), nj=side(), nk=side(), scheme=rng.choice(["rk3", "rk3", "rk3", "steady", "lusgs"]),
                 distort=rng.choice([0.0, 0.0, 0.2]), species=rng.choice([9, 9, 9, 4, 0]),
                 monitor=rng.random() < 0.3)
        if c["scheme"] == "lusgs":
            c["cfl"] = rng.choice([2.0, 5.0])
        c["closure"] = (c["precision"] == "mixed" and c["species"] == 9 and c["scheme"] == "rk3"
                        and rng.random() < 0.25)
    c["steps"] = max(2, min(20, int(1.5e7 / _points(c)) + rng.randint(0, 3)))
    if c["scheme"] == "lusgs":
        c["steps"] = min(c["steps"], 8)
    del c["name"]
    return c


def _axes(case):
    return [[int(v) for v in str(case[k]).split(",")] for k in ("ni", "nj", "nk")]


def _dims(case):
    """The blocks' extents, i fastest (block a + na (b + nb c) at place a, b, c)."""
    ni, nj, nk = _axes(case)
    return [(a, b, c) for c in nk for b in nj for a in ni]


def _points(case):
    return sum(a * b * c for a, b, c in _dims(case))


def _ghosted(case):
    return sum((a + 2 * G) * (b + 2 * G) * (c + 2 * G) for a, b, c in _dims(case))


def work(case):
    if case["kind"] == "training":
        n_in, h, n_out = 20, closure.HIDDEN, 11
        weights = n_in * h + 2 * h * h + h * n_out
        params = weights + 3 * h + n_out
        # per step: the batch, the parameters and both moments in, parameters, moments and gradient out
        return {"bytes": float(case["steps"] * 4 * (case["batch"] * (n_in + n_out) + 7 * params)),
                "flops": float(case["steps"] * 6 * case["batch"] * weights)}
    ns = case["species"]
    bulk = 8 if case["precision"] == "fp64" else 4
    nv = 5 + ns
    # per point and stage: the conserved state in, at the step's start and out (FP64), T in and out,
    # geometry in; then the read-out of the primitives
    stage = 3 * 8 * nv + 2 * bulk + 10 * bulk
    stages = case["steps"] * (3 if case["scheme"] == "rk3" else 1)
    per_face = 40 * nv + (50 * ns if ns else 60) + (80 + 30 * ns if case["viscous"] else 0)
    point = 30 * nv + 60 * ns + (4 * ns * ns if case["viscous"] else 0)
    if case["closure"]:
        point += 2 * (20 * 64 + 2 * 64 * 64 + 64 * 11)
    if case["scheme"] == "lusgs":
        point += 120 * nv
        stage += 8 * 2 * nv
    pts = _points(case)
    return {"bytes": float(pts * stage * stages + _ghosted(case) * (6 + ns) * bulk),
            "flops": float(pts * stages * (3 * per_face + point))}


# ----------------------------------------------------------- inputs of a case

_SPECIES = {}


def _species(n):
    if n not in _SPECIES:
        _SPECIES[n] = (None if n == 0 else cases.synthetic_species() if n == 9 else cases.synthetic_species(FOUR))
    return _SPECIES[n]


def _modes(gen, shape_phase, n_modes=12, kmax=4):
    """A sum of Fourier modes of the phases X, Y, Z (broadcastable), scaled to [-1, 1]."""
    X, Y, Z = shape_phase
    f = 0.0
    for _ in range(n_modes):
        k = torch.randint(-kmax, kmax + 1, (3,), generator=gen).tolist()
        if k == [0, 0, 0]:
            k = [1, 0, 0]
        amp = 0.2 + 0.8 * torch.rand(1, generator=gen).item()
        phase = 2 * math.pi * torch.rand(1, generator=gen).item()
        f = f + amp * torch.cos(k[0] * X + k[1] * Y + k[2] * Z + phase)
    lo, hi = f.min(), f.max()
    return 2 * (f - lo) / (hi - lo).clamp_min(1e-300) - 1


def _phases(dims, periodic, dev):
    """Phase 2 pi i / (n - 1) of the ghosted box per axis, shaped to broadcast over [k, j, i]."""
    out = []
    for a, n in enumerate(dims):
        i = torch.arange(-G, n + G, dtype=torch.float64, device=dev)
        if periodic[a]:
            i = torch.remainder(i, n - 1)
        shape = [1, 1, 1]
        shape[2 - a] = n + 2 * G
        out.append((2 * math.pi / (n - 1) * i).reshape(shape))
    return out


def _mixture(case, gen, dims, periodic, dev):
    """Smooth fields of a frozen mixture: T in [300, 1500] K, p = 1 atm +- 5 %, Taylor-Green
    velocities of 10 m/s, positive mass fractions.  [6 + ns, k, j, i]."""
    X, Y, Z = ph = _phases(dims, periodic, dev)
    ns = case["species"]
    T = 300.0 + 600.0 * (_modes(gen, ph) + 1)
    p = 101325.0 * (1 + 0.05 * _modes(gen, ph))
    u = 10.0 * torch.sin(X) * torch.cos(Y) * torch.cos(Z)
    v = -10.0 * torch.cos(X) * torch.sin(Y) * torch.cos(Z)
    w = 4.0 * torch.sin(X) * torch.sin(Y) * torch.sin(Z)
    if ns == 0:
        return torch.stack([p * MW_AIR / (R_U * T), u, v, w, p, T])
    yk = torch.stack([torch.log1p(torch.exp(2.0 * _modes(gen, ph))) + 1e-3 for _ in range(ns)])
    yk = yk / yk.sum(0)
    mw = torch.tensor(_species(ns)["mw"], device=dev)[:, None, None, None]
    return torch.cat([torch.stack([p / (R_U * T * (yk / mw).sum(0)), u, v, w, p, T]), yk])


def _geometry(dims, h, distort, dev):
    """[10, k, j, i]: J and the metrics by central differences of the coordinates; uniform spacing h,
    or every coordinate moved by a periodic sinusoid of the others (distort cells)."""
    ax = [torch.arange(-G - 1, n + G + 1, dtype=torch.float64, device=dev) * h for n in dims]
    z, y, x = torch.meshgrid(ax[2], ax[1], ax[0], indexing="ij")
    if distort:
        wx, wy, wz = (2 * math.pi / (h * (n - 1)) for n in dims)
        x, y, z = (x + distort * h * torch.sin(wy * y) * torch.cos(wz * z),
                   y + distort * h * torch.sin(wz * z) * torch.cos(wx * x),
                   z + distort * h * torch.sin(wx * x) * torch.cos(wy * y))
    c = slice(1, -1)

    def d(a):  # derivatives of a coordinate along i, j, k
        return (0.5 * (a[c, c, 2:] - a[c, c, :-2]), 0.5 * (a[c, 2:, c] - a[c, :-2, c]),
                0.5 * (a[2:, c, c] - a[:-2, c, c]))

    (x1, x2, x3), (y1, y2, y3), (z1, z2, z3) = d(x), d(y), d(z)
    m = [y2 * z3 - y3 * z2, x3 * z2 - x2 * z3, x2 * y3 - x3 * y2, y3 * z1 - y1 * z3, x1 * z3 - x3 * z1,
         x3 * y1 - x1 * y3, y1 * z2 - y2 * z1, x2 * z1 - x1 * z2, x1 * y2 - x2 * y1]
    jac = x1 * m[0] + x2 * m[3] + x3 * m[6]
    return torch.stack([jac] + [v / jac for v in m])


def _inputs(case, seed, dev):
    """Blocks as dicts: dims, geo [10, k, j, i], prim [6 + ns, k, j, i] on the device, and the faces:
    ("inner", face, target block) or ("bc", face, label)."""
    gen = torch.Generator().manual_seed(int(seed))
    dims, kind = _dims(case), case["kind"]
    ring = [("inner", f, 0) for f in ("i-", "i+", "j-", "j+", "k-", "k+")]
    if kind == "blocks":
        ni, nj, nk = sizes = _axes(case)
        whole = tuple(sum(n - 1 for n in s) + 1 for s in sizes)
        prim = _mixture(case, gen, whole, (True,) * 3, dev)
        blocks = []
        for b, d in enumerate(dims):
            at = (b % len(ni), b // len(ni) % len(nj), b // (len(ni) * len(nj)))
            o = [sum(n - 1 for n in s[:a]) for s, a in zip(sizes, at)]
            faces = []
            for ax in range(3):
                for side, step in (("-", -1), ("+", 1)):
                    t = list(at)
                    t[ax] = (t[ax] + step) % len(sizes[ax])
                    faces.append(("inner", "ijk"[ax] + side, t[0] + len(ni) * (t[1] + len(nj) * t[2])))
            cut = prim[:, o[2]:o[2] + d[2] + 4, o[1]:o[1] + d[1] + 4, o[0]:o[0] + d[0] + 4].clone()
            blocks.append({"dims": d, "geo": _geometry(d, 2e-3 / 127, 0.0, dev), "prim": cut, "faces": faces})
        return blocks
    d = dims[0]
    shape = tuple(n + 2 * G for n in reversed(d))
    if kind == "box":
        prim, faces, h = _mixture(case, gen, d, (True,) * 3, dev), ring, 2e-3 / (d[0] - 1)
    elif kind == "tube":
        # the shock tube's two states, with the membrane and the driver pressure drawn from the seed
        where, p_l = 0.4 + 0.2 * torch.rand(1, generator=gen).item(), 1e5 * (1 + torch.rand(1, generator=gen).item())
        x = torch.arange(-G, d[0] + G, dtype=torch.float64, device=dev) / (d[0] - 1)
        left = (x < where).expand(shape)
        rho = torch.where(left, 1.0, 0.125).double()
        p = torch.where(left, p_l, 1e4).double()
        o = torch.zeros_like(rho)
        prim, h = torch.stack([rho, o, o, o, p, p * MW_AIR / (rho * R_U)]), 1.0 / (d[0] - 1)
        faces = [("bc", "i-", BC_OUT), ("bc", "i+", BC_OUT)] + ring[2:]
    elif kind == "layer":
        # fuel stream (H2 in N2, 300 K, 50 m/s) over air (600 K, 10 m/s), 1 % velocity noise
        sp = _species(case["species"])
        names, mw = sp["names"], torch.tensor(sp["mw"], device=dev)[:, None, None, None]
        h = 4e-3 / 1023
        y = (torch.arange(-G, d[1] + G, dtype=torch.float64, device=dev) * h).reshape(1, -1, 1)
        s = (0.5 * (1 + torch.tanh((y - 0.5 * h * (d[1] - 1)) / (0.05 * h * d[1])))).expand(shape)
        mass = {}
        for stream, x in (("fuel", {"H2": 0.3, "N2": 0.7}), ("air", {"O2": 0.21, "N2": 0.79})):
            w = torch.tensor([x.get(n, 0.0) for n in names], dtype=torch.float64, device=dev)[:, None, None, None] * mw
            mass[stream] = w / w.sum()
        yk = mass["air"] * (1 - s) + mass["fuel"] * s
        noise = (0.4 * (2 * torch.rand((2,) + shape, generator=gen, dtype=torch.float64) - 1)).to(dev)
        T, p = 600.0 - 300.0 * s, torch.full(shape, 101325.0, dtype=torch.float64, device=dev)
        prim = torch.cat([torch.stack([p / (R_U * T * (yk / mw).sum(0)), 10 + 40 * s + noise[0], noise[1],
                                       torch.zeros_like(p), p, T]), yk])
        faces = ring[:2] + [("bc", "j-", BC_OUT), ("bc", "j+", BC_OUT)] + ring[4:]
    else:  # channel
        prim, h = _mixture(case, gen, d, (False, False, True), dev), 2e-3 / (d[0] - 1)
        faces = [("bc", "i-", BC_IN), ("bc", "i+", BC_OUT), ("bc", "j-", WALL_T), ("bc", "j+", WALL_Q)] + ring[4:]
    return [{"dims": d, "geo": _geometry(d, h, case["distort"], dev), "prim": prim, "faces": faces}]


def _conditions(case):
    """The boundary conditions of a case by label; the inflow is an equal-mass mixture at 600 K, 20 m/s."""
    if case["kind"] in ("tube", "layer"):
        return {BC_OUT: {"kind": 6}}
    if case["kind"] != "channel":
        return {}
    sp = _species(case["species"])
    y = np.full(case["species"], 1.0 / case["species"])
    return {BC_IN: {"kind": 5, "density": 101325.0 / (R_U * 600.0 * (y / sp["mw"]).sum()), "u": 20.0, "v": 0.0,
                    "w": 0.0, "pressure": 101325.0, "temperature": 600.0, "yk": y},
            BC_OUT: {"kind": 6},
            WALL_T: {"kind": 2, "thermal_type": 0, "t_wall": 500.0},
            WALL_Q: {"kind": 2, "thermal_type": 1, "t_wall": 300.0}}


def _training_inputs(case, seed, dev):
    """Initial weights of the closure network, and per step a batch of its features [batch, 20] and
    normalised log transport properties [batch, 11]."""
    gen = torch.Generator().manual_seed(int(seed))
    sp, n, k = _species(9), case["batch"], case["steps"]
    h, n_in, n_out = closure.HIDDEN, 20, 11
    flat = []
    for a, b in ((n_in, h), (h, h), (h, h), (h, n_out)):
        flat += [(torch.randn(b, a, generator=gen) / math.sqrt(a)).reshape(-1), 0.1 * torch.randn(b, generator=gen)]
    T = 300.0 + 2200.0 * torch.rand(n * k, generator=gen, dtype=torch.float64).to(dev)
    X = -torch.log(torch.rand((9, n * k), generator=gen, dtype=torch.float64).clamp_min(1e-12)).to(dev)
    X = X / X.sum(0)
    mw = torch.tensor(sp["mw"], device=dev)[:, None]
    Y = X * mw / (X * mw).sum(0)
    solver = _Exact({"species": 9, "closure": False, "precision": "fp64"}, dev)
    mu, lam, rd = solver.transport(T, Y)
    y = torch.log(torch.cat([mu[None], lam[None], rd]))
    mean, scale = y.mean(1, keepdim=True), y.std(1, keepdim=True)
    feat = _features(T, X).float().T.reshape(k, n, n_in).contiguous()
    return (torch.cat(flat).to(dev), feat, ((y - mean) / scale).float().T.reshape(k, n, n_out).contiguous(),
            scale.reshape(-1).float())


def _bf16(x):
    return x.to(torch.bfloat16).to(x.dtype)


def _features(T, X):
    """Network inputs [20, n]: t and the mole fractions as BF16 (high, low) pairs."""
    t = (T - closure.T_CENTER) / closure.T_SCALE
    t_hi, x_hi = _bf16(t), _bf16(X)
    return torch.cat([t_hi[None], _bf16(t - t_hi)[None], x_hi, _bf16(X - x_hi)])


# ------------------------------------------------------- set-up and one pass

LR, BETA1, BETA2, EPS, STEP0 = 1e-3, 0.9, 0.999, 1e-8, 1000


def _prepare_training(case, seed):
    lib = cc.load_library()
    params, x, y, scale = _training_inputs(case, seed, "cuda")
    n = params.numel()
    # in mid-training: the second moments are settled
    return {"case": case, "lib": lib, "n": n, "params": params, "x": x, "y": y, "scale": scale,
            "grad": torch.zeros_like(params), "m": torch.zeros_like(params), "v": torch.full_like(params, 1e-4),
            "loss": torch.zeros(1, device="cuda"), "step": STEP0,
            "work": torch.empty(lib.cc_mlp_workspace_bytes(20, closure.HIDDEN, 11, case["batch"]), dtype=torch.uint8,
                                device="cuda")}


def prepare(case, seed):
    if case["kind"] == "training":
        return _prepare_training(case, seed)
    sp = _species(case["species"])
    blocks = []
    host = lambda a: a.reshape(a.shape[0], -1).cpu().numpy()  # noqa: E731
    dims = _dims(case)
    for b in _inputs(case, seed, _device()):
        geo, prim = host(b["geo"]), host(b["prim"])
        bnd, inner = [], []
        for what, face, to in b["faces"]:
            if what == "bc":
                bnd.append(cases.boundary_raw(b["dims"], face, to))
            else:
                other = face[0] + ("+" if face[1] == "-" else "-")
                inner.append(cases.inner_face_raw(b["dims"], face, dims[to], other, to))
        blocks.append({"dims": b["dims"], "jac": geo[0], "metric": geo[1:], "bv": prim[:6], "yk": prim[6:],
                       "boundaries": bnd, "inner_faces": inner})
    bcs = [dict(v, label=k) for k, v in _conditions(case).items()]
    d = cc.Driver.from_case({"params": cases.default_params(sp, viscous=case["viscous"], cfl=case["cfl"]),
                             "blocks": blocks, "bcs": bcs}, case["precision"])
    if case["closure"]:
        d.set_closure(closure.load()[0])
        d.use_closure(True)
    d.initialize_computation()
    # host side of the read-out: per block pinned FP64 buffers, and the fields of all blocks in the
    # precision of the output
    ns = case["species"]
    ng = [b["bv"].shape[1] for b in blocks]
    pin = lambda n: torch.empty((n[0], n[1]), dtype=torch.float64, pin_memory=True)  # noqa: E731
    bv, yk = [pin((6, n)) for n in ng], [pin((ns, n)) for n in ng]
    rows = {"rho": 1, "velocity": 3, "p": 1, "T": 1, "Y": ns}
    if case["precision"] == "fp64" and len(ng) == 1:  # the buffers as they are
        out = {"rho": bv[0][0:1], "velocity": bv[0][1:4], "p": bv[0][4:5], "T": bv[0][5:6], "Y": yk[0]}
    else:
        kind = torch.float64 if case["precision"] == "fp64" else torch.float32
        out = {k: torch.empty((r, sum(ng)), dtype=kind) for k, r in rows.items()}
    if ns == 0:
        del out["Y"]
    return {"case": case, "driver": d, "ng": ng, "bv": bv, "yk": yk, "out": out}


def _ptr(t):
    return ctypes.cast(t.data_ptr(), cc._dp) if t.numel() else None


def _run_training(s):
    c, lib = s["case"], s["lib"]
    vp = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    for k in range(c["steps"]):
        s["step"] += 1
        cc._check(lib.cc_mlp_grad(20, closure.HIDDEN, 11, c["batch"], vp(s["params"]), vp(s["x"][k]), vp(s["y"][k]),
                                  vp(s["scale"]), vp(s["grad"]), vp(s["loss"]), vp(s["work"]), stream))
        cc._check(lib.cc_mlp_adam(s["n"], vp(s["params"]), vp(s["grad"]), vp(s["m"]), vp(s["v"]), LR, BETA1, BETA2,
                                  EPS, s["step"], stream))
    return {"loss": s["loss"], "grad": s["grad"], "params": s["params"]}


def run(state):
    c = state["case"]
    if c["kind"] == "training":
        return _run_training(state)
    d, out = state["driver"], dict(state["out"])
    if c["monitor"]:
        for _ in range(c["steps"]):
            d.simulate(1, c["scheme"], residual=True)
        out["residual"] = torch.from_numpy(d.residual()).to(state["out"]["rho"].dtype)
    else:
        d.simulate(c["steps"], c["scheme"])
    at = 0
    for b, (n, bv, yk) in enumerate(zip(state["ng"], state["bv"], state["yk"])):
        cc._check(d.lib.cc_get_state(d.ctx, b, _ptr(bv), _ptr(yk), None, 0))
        if out["rho"].data_ptr() != bv.data_ptr():
            at1 = at + n
            for key, src in (("rho", bv[0:1]), ("velocity", bv[1:4]), ("p", bv[4:5]), ("T", bv[5:6]), ("Y", yk)):
                if key in out:
                    out[key][:, at:at1].copy_(src)
            at = at1
    return out


# ------------------------------------------------------- the same in 64 bits

class _Exact:
    """The path on whole arrays in FP64: AUSM+ with MUSCL (kappa = 1/3, minmod), central viscous fluxes,
    NASA-7 thermodynamics, Wilke and constant-Schmidt transport, SSP-RK3, explicit and LU-SGS steps.
    Arrays are [field, k, j, i] over the ghosted box; prim = rho, u, v, w, p, T, Y."""

    def __init__(self, case, dev):
        self.case, self.dev, self.ns = case, dev, case["species"]
        self.renorm = self.ns > 0 and case["precision"] != "fp64"
        self.net = None
        if self.ns:
            sp = _species(self.ns)
            t = lambda k: torch.tensor(np.asarray(sp[k]), dtype=torch.float64, device=dev)  # noqa: E731
            self.mw, self.t_low, self.t_mid = t("mw"), t("t_low"), t("t_mid")
            self.low, self.high = t("low_temp_coeff"), t("high_temp_coeff")
            self.lj, self.vis = t("LJ_potent_inv"), t("vis_coeff")
            self.wj, self.sw = t("WjDivWi_to_One4th"), t("sqrt_WiDivWjPl1Mul8")
        if case["closure"]:
            w, _ = closure.load()
            self.net = {k: torch.tensor(np.asarray(v), device=dev) for k, v in w.items()}

    def h_cp(self, l, T):
        """Enthalpy and cp of species l per unit mass; h continues linearly below t_low."""
        te = T.clamp_min(self.t_low[l].item())
        low = (T < self.t_mid[l])[None]
        a = torch.where(low, self.low[l].reshape((-1,) + (1,) * T.dim()), self.high[l].reshape((-1,) + (1,) * T.dim()))
        cp = a[0] + te * (a[1] + te * (a[2] + te * (a[3] + te * a[4])))
        h = a[5] + te * (a[0] + te * (a[1] / 2 + te * (a[2] / 3 + te * (a[3] / 4 + te * a[4] / 5))))
        r = R_U / self.mw[l]
        return (h + cp * (T - te)) * r, cp * r

    def mixture(self, T, Y):
        """h, cp and R = R_u / W of the mixture."""
        h = cp = gas = 0.0
        for l in range(self.ns):
            hl, cl = self.h_cp(l, T)
            h, cp, gas = h + Y[l] * hl, cp + Y[l] * cl, gas + Y[l] * (R_U / self.mw[l])
        return h, cp, gas

    def transport(self, T, Y):
        """mu, lambda, rho D_k of the mixture."""
        ns, mw = self.ns, self.mw
        x = torch.stack([Y[l] / mw[l] for l in range(ns)])
        x = x / x.sum(0)
        mu_k = []
        for l in range(ns):
            t = T * self.lj[l]
            mu_k.append(self.vis[l] * torch.sqrt(T) / (1.147 * t ** -0.145 + (t + 0.5) ** -2))
        root = [torch.sqrt(v) for v in mu_k]
        mu = lam = 0.0
        for a in range(ns):
            s = x[a]
            for b in range(ns):
                if a != b:
                    s = s + (1 + root[a] / root[b] * self.wj[a, b]) ** 2 * self.sw[a, b] * x[b]
            lam_a = mu_k[a] * (self.h_cp(a, T)[1] + 1.25 * R_U / mw[a])
            mu = mu + mu_k[a] * x[a] / s
            lam = lam + lam_a * x[a] / (1.065 * s - 0.065 * x[a])
        rd = torch.stack([torch.where((x[l] - 1).abs() < 1e-3, mu, (1 - Y[l]) * mu / (1 - x[l])) / 0.9
                          for l in range(ns)])
        if self.net is not None:
            n = self.net
            a = _features(T.reshape(-1), x.reshape(ns, -1)).T
            for i in range(1, 5):
                a = a @ _bf16(n["w%d" % i].float()).double().T + n["b%d" % i].double()
                a = a * torch.sigmoid(a) if i < 4 else a
            o = torch.exp(a * n["out_scale"].double() + n["out_mean"].double()).T.reshape((2 + ns,) + T.shape)
            inside = (T >= n["t_min"]) & (T <= n["t_max"]) & (x.amax(0) < 0.998)
            mu, lam, rd = torch.where(inside, o[0], mu), torch.where(inside, o[1], lam), torch.where(inside, o[2:], rd)
        return mu, lam, rd

    def properties(self, V):
        """[4 + ns]: mu, lambda, gamma, c, rho D_k."""
        T = V[5]
        if self.ns == 0:
            c2 = GAMMA * R_U / MW_AIR
            mu = 1.716e-5 * (T / 273) ** 1.5 * 384 / (T + 111)
            return torch.stack([mu, mu * c2 / (GAMMA - 1) / 0.72, torch.full_like(T, GAMMA), torch.sqrt(c2 * T)])
        _, cp, gas = self.mixture(T, V[6:])
        gam = cp / (cp - gas)
        mu, lam, rd = self.transport(T, V[6:])
        return torch.cat([torch.stack([mu, lam, gam, torch.sqrt(gam * gas * T)]), rd])

    def energy(self, V):
        kin = 0.5 * V[0] * (V[1] ** 2 + V[2] ** 2 + V[3] ** 2)
        if self.ns == 0:
            return kin + V[4] / (GAMMA - 1)
        return kin + V[0] * self.mixture(V[5], V[6:])[0] - V[4]

    def conserved(self, V):
        return torch.cat([V[0:1], V[0] * V[1:4], self.energy(V)[None], V[0] * V[6:]])

    def primitives(self, Q, t):
        """Primitives of Q; the temperature by Newton from t until a step is below 1e-3."""
        rho, vel = Q[0], Q[1:4] / Q[0]
        kin = 0.5 * (vel ** 2).sum(0)
        if self.ns == 0:
            p = (GAMMA - 1) * (Q[4] - rho * kin)
            return torch.cat([rho[None], vel, torch.stack([p, p * MW_AIR / (rho * R_U)])])
        Y = Q[5:] / rho
        if self.renorm:
            Y = Y / Y.sum(0)
        e = Q[4] / rho - kin
        t, on = t.clone(), torch.ones_like(t, dtype=torch.bool)
        for _ in range(50):
            h, cp, gas = self.mixture(t, Y)
            t1 = t - (h - gas * t - e) / (cp - gas)
            err = (1 - t1 / t).abs()
            t = torch.where(on, t1, t)
            on = on & (err > 1e-3)
            if not bool(on.any()):
                break
        return torch.cat([rho[None], vel, torch.stack([rho * t * gas, t]), Y])

    def face_flux(self, d, V, prop, geo, dims):
        """Inviscid minus viscous flux of the faces between points -1..m-1 and their neighbours along d."""
        unit = [0, 0, 0]
        unit[d] = 1

        def at(a, off=(0, 0, 0)):  # the faces' first points, moved by off (i, j, k)
            s = [slice(G - unit[x] + off[x], G + dims[x] + off[x]) for x in range(3)]
            return a[..., s[2], s[1], s[0]]

        step = lambda n: tuple(n * x for x in unit)  # noqa: E731
        pts = [torch.cat([at(V, step(n))[:5], at(V, step(n))[6:]]) for n in (-1, 0, 1, 2)]
        d0, d1, d2 = (b - a for a, b in zip(pts, pts[1:]))
        mm = lambda a, b: torch.where(a * b > 0, torch.where(a.abs() < b.abs(), a, b), torch.zeros_like(a))  # noqa: E731
        L, R = pts[1] + 0.5 * mm(d0, d1), pts[2] - 0.5 * mm(d1, d2)
        J0, J1 = at(geo)[0], at(geo, step(1))[0]
        m0, m1 = at(geo)[1:].unflatten(0, (3, 3)), at(geo, step(1))[1:].unflatten(0, (3, 3))
        k = 0.5 * (J0 * m0[d] + J1 * m1[d])
        gk = torch.sqrt((k ** 2).sum(0))

        def thermo(S):  # total enthalpy per mass, gamma p / rho
            kin = 0.5 * (S[1] ** 2 + S[2] ** 2 + S[3] ** 2)
            if self.ns == 0:
                return kin + GAMMA / (GAMMA - 1) * S[4] / S[0], GAMMA * S[4] / S[0]
            gas = sum(S[5 + l] * (R_U / self.mw[l]) for l in range(self.ns))
            h, cp, _ = self.mixture(S[4] / (S[0] * gas), S[5:])
            return kin + h, cp / (cp - gas) * S[4] / S[0]

        (Hl, c2l), (Hr, c2r) = thermo(L), thermo(R)
        ul, ur = (k * L[1:4]).sum(0) / gk, (k * R[1:4]).sum(0) / gk
        c = 0.5 * (torch.sqrt(c2l) + torch.sqrt(c2r))
        Ml, Mr = ul / c, ur / c
        bl, br = (Ml ** 2 - 1) ** 2, (Mr ** 2 - 1) ** 2
        sub = lambda M, a, b: torch.where(M.abs() > 1, a, b)  # noqa: E731
        mp = sub(Ml, Ml.clamp_min(0), (Ml + 1) ** 2 / 4 + bl / 8)
        mn = sub(Mr, Mr.clamp_max(0), -((Mr - 1) ** 2) / 4 - br / 8)
        pp = sub(Ml, (Ml > 0).double(), (Ml + 1) ** 2 / 4 * (2 - Ml) + 3 / 16 * Ml * bl)
        pn = sub(Mr, (Mr < 0).double(), (Mr - 1) ** 2 / 4 * (2 + Mr) - 3 / 16 * Mr * br)
        half = mp + mn
        flux = c * (L[0] * half.clamp_min(0) + R[0] * half.clamp_max(0))
        up = flux >= 0
        S = torch.where(up, L, R)
        p = pp * L[4] + pn * R[4]
        mass = flux * gk
        F = torch.cat([mass[None], mass * S[1:4] + p * k, (mass * torch.where(up, Hl, Hr))[None], mass * S[5:]])
        if not self.case["viscous"]:
            return F
        met = 0.5 * (m0 + m1)

        def grad(a):  # physical gradient [3] of the field(s) a
            out = 0.0
            for x in range(3):
                if x == d:
                    dd = at(a, step(1)) - at(a)
                else:
                    e = [int(x == y) for y in range(3)]
                    e1 = [u + v for u, v in zip(unit, e)]
                    e2 = [u - v for u, v in zip(unit, e)]
                    dd = 0.25 * (at(a, e) - at(a, [-v for v in e]) + at(a, e1) - at(a, e2))
                out = out + dd[..., None, :, :, :] * met[x]
            return out

        mean = lambda a: 0.5 * (at(a) + at(a, step(1)))  # noqa: E731
        gv = grad(V[1:4])
        mu = mean(prop[0])
        div = gv[0][0] + gv[1][1] + gv[2][2]
        f = []
        for a in range(3):
            tau = [mu * (gv[a][b] + gv[b][a] - (2 / 3 * div if a == b else 0)) for b in range(3)]
            f.append(sum(k[b] * tau[b] for b in range(3)))
        e = sum(mean(V[1 + a]) * f[a] for a in range(3)) + mean(prop[1]) * (k * grad(V[5])).sum(0)
        if self.ns:
            tm, flux_y = mean(V[5]), []
            for l in range(self.ns):
                flux_y.append(mean(prop[4 + l]) * (k * grad(V[6 + l])).sum(0))
                e = e + flux_y[l] * self.h_cp(l, tm)[0]
            total = sum(flux_y)
            for l in range(self.ns):
                F[5 + l] -= flux_y[l] - mean(V[6 + l]) * total
        F[1:4] -= torch.stack(f)
        F[4] -= e
        return F

    def residual(self, b):
        """dq of the interior."""
        out = 0.0
        for d in range(3):
            F = self.face_flux(d, b["V"], b["prop"], b["geo"], b["dims"])
            n = F.shape[3 - d]
            out = out - (F.narrow(3 - d, 1, n - 1) - F.narrow(3 - d, 0, n - 1))
        return out

    @staticmethod
    def core(a):
        return a[..., G:-G, G:-G, G:-G]

    def radii(self, b):
        """Per direction |u . grad xi|, |grad xi| of the interior, and max(gamma, 4/3) mu / (rho Pr)."""
        V, prop, m = self.core(b["V"]), self.core(b["prop"]), self.core(b["geo"])[1:].unflatten(0, (3, 3))
        g = torch.sqrt((m ** 2).sum(1))
        u = (m * V[1:4]).sum(1).abs()
        return u, g, prop[3], prop[2].clamp_min(4 / 3) * prop[0] / V[0] / 0.72

    def local_dt(self, b):
        u, g, c, nu = self.radii(b)
        return self.case["cfl"] / ((u + c * g).sum(0) + nu * (g ** 2).sum(0))

    def advance(self, b, Q):
        """The interior's new conserved state and its primitives."""
        V = self.primitives(Q, self.core(b["V"])[5])
        self.core(b["Q"])[:] = Q
        self.core(b["V"])[:] = V
        b["speed"] = torch.sqrt((V[1:4] ** 2).sum(0))

    def exchange(self, blocks, conditions):
        """Ghost points: outflow, inflow, walls, then the interfaces in block order."""
        def layer(a, ax, n, pos):  # the layer at point pos along ax of an array whose extent there is n
            return a.select(3 - ax, G + pos)

        for kind in (6, 5, 2):
            for label, bc in conditions.items():
                if bc["kind"] != kind:
                    continue
                for b in blocks:
                    for what, face, to in b["faces"]:
                        if what == "bc" and to == label:
                            self.condition(b, face, bc, layer)
        for b in blocks:
            for what, face, to in b["faces"]:
                if what != "inner":
                    continue
                ax, t = "ijk".index(face[0]), blocks[to]
                n, nt = b["dims"][ax], t["dims"][ax]
                here = (lambda g: -g) if face[1] == "-" else (lambda g: n - 1 + g)  # noqa: E731
                there = (lambda g: nt - 1 - g) if face[1] == "-" else (lambda g: g)  # noqa: E731
                for a in ("V", "Q"):
                    src = [layer(t[a], ax, nt, there(g)).clone() for g in range(G + 1)]
                    mid = 0.5 * (layer(b[a], ax, n, here(0)) + src[0])
                    layer(b[a], ax, n, here(0))[:] = mid
                    layer(t[a], ax, nt, there(0))[:] = mid
                    for g in range(1, G + 1):
                        layer(b[a], ax, n, here(g))[:] = src[g]

    def condition(self, b, face, bc, layer):
        ax = "ijk".index(face[0])
        n = b["dims"][ax]
        pos = (lambda g: -g) if face[1] == "-" else (lambda g: n - 1 + g)  # noqa: E731
        if bc["kind"] == 6:
            for a in ("V", "Q"):
                for g in range(1, G + 1):
                    layer(b[a], ax, n, pos(g))[:] = layer(b[a], ax, n, pos(0))
        elif bc["kind"] == 5:
            v = torch.tensor([bc["density"], bc["u"], bc["v"], bc["w"], bc["pressure"], bc["temperature"]]
                             + list(bc["yk"]), dtype=torch.float64, device=self.dev)
            q = self.conserved(v.reshape(-1, 1))
            for g in range(1, G + 1):
                layer(b["V"], ax, n, pos(g))[:] = v[:, None, None]
                layer(b["Q"], ax, n, pos(g))[:] = q[:, :, None]
        else:
            cut = (slice(None), slice(G, -G), slice(G, -G))  # walls leave out the tangential ghosts
            at = lambda a, g: layer(b[a], ax, n, pos(g))[cut]  # noqa: E731
            inner = [at("V", -g).clone() for g in range(G + 1)]
            tw = inner[1][5].clone() if bc["thermal_type"] == 1 else torch.full_like(inner[1][5], bc["t_wall"])
            gas = lambda v: sum(v[6 + l] * (R_U / self.mw[l]) for l in range(self.ns))  # noqa: E731
            for g in range(G + 1):
                v = inner[max(g, 1)].clone()
                if g == 0:
                    v[1:4], v[5] = 0.0, tw
                else:
                    v[1:4] = -v[1:4]
                    if bc["thermal_type"] == 0:
                        tg = 2 * tw - v[5]
                        v[5] = torch.where(tg <= 0.1 * tw, tw, tg)
                v[0] = v[4] / (v[5] * gas(v))
                at("V", g)[:] = v
                at("Q", g)[:] = self.conserved(v)
            speed = b.get("speed")
            if speed is not None:
                speed.select(2 - ax, 0 if face[1] == "-" else n - 1)[:] = 0.0

    def settle(self, blocks, conditions):
        self.exchange(blocks, conditions)
        for b in blocks:
            b["prop"] = self.properties(b["V"])

    def lusgs(self, b, dt):
        """dQ of one LU-SGS step, hyperplane by hyperplane."""
        dims, nv = b["dims"], 5 + self.ns
        V, Q, geo = (self.core(b[a]).reshape(b[a].shape[0], -1) for a in ("V", "Q", "geo"))
        u, g, c, nu = (a.reshape(a.shape[:-3] + (-1,)) for a in self.radii(b))
        J, gam = geo[0], self.core(b["prop"])[2].reshape(-1)
        r = J * (u + c * g + (2 * nu * g ** 2 if self.case["viscous"] else 0))
        inv_d = 1 / (J / dt.reshape(-1) + r.sum(0))
        k = J * geo[1:].unflatten(0, (3, 3))
        psi = [gam * (R_U / self.mw[l]) * V[5] - (gam - 1) * self.h_cp(l, V[5])[0] for l in range(self.ns)]
        X = self.residual(b).reshape(nv, -1)
        # everything a point's flux Jacobian needs, a row per point
        rows = torch.cat([Q, V[4:5], gam[None], k.reshape(9, -1), r] + [torch.stack(psi)] * bool(psi)).T.contiguous()
        idx = torch.arange(J.numel(), device=self.dev)
        ijk = [idx % dims[0], idx // dims[0] % dims[1], idx // (dims[0] * dims[1])]
        stride = (1, dims[0], dims[0] * dims[1])
        order = torch.argsort(ijk[0] + ijk[1] + ijk[2], stable=True)
        planes = torch.split(order, torch.bincount(ijk[0] + ijk[1] + ijk[2]).tolist())
        X = X.T.contiguous()

        def term(q, d, sign):  # (A_d X + sign r_d X) / 2 at the points q
            w, x = rows[q].T, X[q].T
            vel, p, ga, kd, rad = w[1:4] / w[0], w[nv], w[nv + 1], w[nv + 2 + 3 * d:nv + 5 + 3 * d], w[nv + 11 + d]
            U, dm = (kd * vel).sum(0), (kd * x[1:4]).sum(0)
            dU = (dm - U * x[0]) / w[0]
            dp = (ga - 1) * (x[4] - (vel * x[1:4]).sum(0) + 0.5 * (vel ** 2).sum(0) * x[0])
            if self.ns:
                dp = dp + (w[nv + 14:] * x[5:]).sum(0)
            f = x * U + w[:nv] * dU
            f[0] = dm
            f[1:4] += kd * dp
            f[4] += dp * U + p * dU
            return 0.5 * (f + sign * rad * x)

        for way, todo in ((-1, planes), (1, reversed(planes))):
            for q in todo:
                acc = X[q].T.clone() if way < 0 else 0.0
                for d in range(3):
                    ok = (ijk[d][q] > 0) if way < 0 else (ijk[d][q] + 1 < dims[d])
                    n = torch.where(ok, q + way * stride[d], q)
                    acc = acc + torch.where(ok, term(n, d, -way), 0.0)
                X[q] = (acc * inv_d[q]).T if way < 0 else X[q] - (acc * inv_d[q]).T
        return X.T.reshape((nv,) + tuple(reversed(dims)))

    def run(self, blocks, conditions):
        """The case's steps from the primitives in blocks; returns the last step's residual norms."""
        case, norms = self.case, None
        for b in blocks:
            b["V"] = b["prim"].clone()
            b["Q"] = self.conserved(b["V"])
            b["speed"] = torch.sqrt((self.core(b["V"])[1:4] ** 2).sum(0))
        self.settle(blocks, conditions)
        watched = lambda b: torch.stack([self.core(b["V"])[0], b["speed"], self.core(b["V"])[4],  # noqa: E731
                                         self.core(b["V"])[5]])
        for _ in range(case["steps"]):
            last = [watched(b).clone() for b in blocks]
            if case["scheme"] == "rk3":
                dt = min(self.local_dt(b).min() for b in blocks)
                start = [self.core(b["Q"]).clone() for b in blocks]
                for a, w in ((0.0, 1.0), (0.75, 0.25), (1 / 3, 2 / 3)):
                    new = [a * q0 + w * (self.core(b["Q"]) + self.residual(b) * dt / self.core(b["geo"])[0])
                           for q0, b in zip(start, blocks)]
                    for b, q in zip(blocks, new):
                        self.advance(b, q)
                    self.settle(blocks, conditions)
            else:
                new = []
                for b in blocks:
                    dt = self.local_dt(b)
                    dq = (self.lusgs(b, dt) if case["scheme"] == "lusgs"
                          else self.residual(b) * dt / self.core(b["geo"])[0])
                    new.append(self.core(b["Q"]) + dq)
                for b, q in zip(blocks, new):
                    self.advance(b, q)
                self.settle(blocks, conditions)
            sums = sum(((watched(b) - l) ** 2).sum((1, 2, 3)) for b, l in zip(blocks, last))
            norms = torch.sqrt(sums / sum(l[0].numel() for l in last))
        return norms


def _exact_training(case, seed, dev):
    params, x, y, scale = _training_inputs(case, seed, dev)
    p, scale = params.double(), scale.double()
    m, v = torch.zeros_like(p), torch.full_like(p, 1e-4)
    h = closure.HIDDEN
    shapes = [(h, 20), (h, h), (h, h), (11, h)]
    for k in range(case["steps"]):
        W, b, o = [], [], 0
        for s in shapes:  # the forward and backward passes see the FP32 parameters, weights rounded to BF16
            W.append(_bf16(p[o:o + s[0] * s[1]].float()).double().reshape(s))
            b.append(p[o + s[0] * s[1]:o + s[0] * s[1] + s[0]])
            o += s[0] * s[1] + s[0]
        a, z = [x[k].double()], []
        for i in range(4):
            z.append(a[i] @ W[i].T + b[i])
            a.append(z[i] * torch.sigmoid(z[i]))
        err = (z[3] - y[k].double()) * scale
        loss = (err ** 2).mean()
        g, grad = 2 * err * scale / err.numel(), []
        for i in range(3, -1, -1):
            grad = [(g.T @ a[i]).reshape(-1), g.sum(0)] + grad
            if i:
                s = torch.sigmoid(z[i - 1])
                g = (g @ W[i]) * (s * (1 + z[i - 1] * (1 - s)))
        grad = torch.cat(grad)
        n = STEP0 + 1 + k
        m, v = BETA1 * m + (1 - BETA1) * grad, BETA2 * v + (1 - BETA2) * grad ** 2
        p = p - LR * (m / (1 - BETA1 ** n)) / (torch.sqrt(v / (1 - BETA2 ** n)) + EPS)
    return {"loss": loss.reshape(1), "grad": grad, "params": p}


def exact(case, seed):
    dev = _device()
    if case["kind"] == "training":
        return _exact_training(case, seed, dev)
    solver = _Exact(case, dev)
    blocks = _inputs(case, seed, dev)
    norms = solver.run(blocks, _conditions(case))
    rows = {"rho": slice(0, 1), "velocity": slice(1, 4), "p": slice(4, 5), "T": slice(5, 6), "Y": slice(6, None)}
    out = {k: torch.cat([b["V"][s].reshape(b["V"][s].shape[0], -1) for b in blocks], 1).cpu() for k, s in rows.items()
           if not (k == "Y" and case["species"] == 0)}
    if case["monitor"]:
        out["residual"] = norms.cpu()
    return out
