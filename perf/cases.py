"""Workloads the framework is timed on: what its users have it do, through the
public entry points of ``saras_gb300``.

Six kinds of pass:

* ``dropin``   time steps of the default mode (the reference algorithm) from a
               given state: fields uploaded, advanced, downloaded;
* ``target``   the same with the plain FP64 multigrid to a residual target;
* ``mixed``    a running simulation with the mixed-precision multigrid and the
               extrapolated guess: the next steps of it, then the fields;
* ``operators``  the field operators one by one, as a program with its own time
               stepping calls them;
* ``cn``       one Crank-Nicolson Jacobi solve on device arrays of the caller;
* ``unet``     one forward and backward pass of the warm-start network.

Sizes are grid indices: an axis of index n has 2^n + 1 vertex points.
"""
import ctypes
import math

import numpy as np
import torch

import saras_gb300 as S
from saras_gb300 import _abi as F

V3 = (F.FIELD_VX, F.FIELD_VY, F.FIELD_VZ)
NSE = (F.FIELD_NSE_X, F.FIELD_NSE_Y, F.FIELD_NSE_Z)
GRAD = (F.FIELD_GRAD_X, F.FIELD_GRAD_Y, F.FIELD_GRAD_Z)


def listed():
    return [
        # the lid-driven cavity every user starts with: the drop-in's damped-Jacobi V(3,3) at 33^3, thousands of small launches
        {"name": "ldc33_dropin", "kind": "dropin", "flow": "ldc", "ix": 5, "iy": 5, "iz": 5, "depth": 3, "gs": 0, "stretch": 0, "steps": 1},
        # the input file the reference ships: Taylor-Green 65^3, Gauss-Seidel V(4,4), at most 5 cycles a step
        {"name": "tgv65_gs_dropin", "kind": "dropin", "flow": "tgv", "ix": 6, "iy": 6, "iz": 6, "depth": 3, "gs": 1, "stretch": 0, "steps": 2},
        # the drop-in at a production size: Taylor-Green 129^3, as many cycles as the reference's stopping rule takes
        {"name": "tgv129_dropin", "kind": "dropin", "flow": "tgv", "ix": 7, "iy": 7, "iz": 7, "depth": 5, "gs": 0, "stretch": 0, "steps": 1},
        # convection in the drop-in, an anisotropic point count, the temperature equation in every step
        {"name": "rbc65_dropin", "kind": "dropin", "flow": "rbc", "ix": 6, "iy": 6, "iz": 5, "depth": 3, "gs": 0, "stretch": 0, "steps": 1},
        # the 2D validation run (65 x 65 cavity, Gauss-Seidel V(2,2), CFL time step): a few of its 50000 steps
        {"name": "cavity2d_65", "kind": "dropin", "flow": "cav2d", "ix": 6, "iy": 0, "iz": 6, "depth": 4, "gs": 1, "stretch": 0, "steps": 5},
        # the mixed-precision step on a small grid, where launches and round trips count
        {"name": "tgv65_mixed", "kind": "mixed", "flow": "tgv", "ix": 6, "iy": 6, "iz": 6, "depth": 4, "steps": 8},
        # the benchmark's size and settings
        {"name": "tgv257_mixed", "kind": "mixed", "flow": "tgv", "ix": 8, "iy": 8, "iz": 8, "depth": 6, "steps": 4},
        # the benchmark's other arm: FP64 V-cycles to the same residual
        {"name": "tgv257_plain", "kind": "target", "flow": "tgv", "ix": 8, "iy": 8, "iz": 8, "depth": 6, "steps": 3},
        # the convection study: 257 x 257 x 129, walls along z, buoyancy and temperature
        {"name": "rbc257_mixed", "kind": "mixed", "flow": "rbc", "ix": 8, "iy": 8, "iz": 7, "depth": 6, "steps": 4},
        # the operators of the reference's field classes, called one by one
        {"name": "operators129", "kind": "operators", "flow": "tgv", "ix": 7, "iy": 7, "iz": 7},
        # the smallest call: one allocation-free Jacobi solve on the caller's device arrays
        {"name": "cn33", "kind": "cn", "flow": "ldc", "ix": 5, "iy": 5, "iz": 5, "comp": 0, "fast": 0},
        # training of the warm start: one pass of the network on its 65^3 grid, output, loss and gradients
        {"name": "unet65_train", "kind": "unet", "flow": "tgv", "ix": 7, "iy": 7, "iz": 7, "depth": 5},
    ]


def _near(rng, i, lo, hi):
    return min(hi, max(lo, i + rng.choice((-1, 0, 0, 0, 1))))


def draw(rng):
    """One more case: each kind over its range of grid indices (the logarithm of
    the size), the axes not all alike, the drop-in's options as the parameters
    files use them."""
    kind = rng.choice(("dropin", "dropin", "dropin", "target", "mixed", "mixed", "operators", "cn", "unet"))
    if kind == "dropin":
        flow = rng.choice(("ldc", "tgv", "rbc", "cav2d"))
        if flow == "cav2d":
            i = rng.randint(4, 7)
            j = _near(rng, i, 4, 7)
            return {"kind": kind, "flow": flow, "ix": i, "iy": 0, "iz": j, "depth": min(i, j) - rng.randint(1, 2), "gs": 1,
                    "stretch": rng.choice((0, 0, 1)), "steps": rng.randint(3, 6)}
        i = rng.randint(4, 6)
        ix, iy, iz = i, _near(rng, i, 4, 6), _near(rng, i, 4, 6)
        gs = rng.choice((0, 0, 1))
        stretch = rng.choice((0, 0, 0, 1)) if flow != "tgv" else 0
        if flow == "rbc":                    # the 2:2:1 box
            iz = max(4, i - 1)
            if stretch:
                iy = ix
        if flow == "tgv" and not gs:         # the cube (Jacobi cycles want equal spacings on a periodic box)
            iy = iz = ix
        return {"kind": kind, "flow": flow, "ix": ix, "iy": iy, "iz": iz, "depth": min(ix, iy, iz) - rng.randint(1, 2),
                "gs": gs, "stretch": stretch, "steps": 1, "cycles": rng.randint(10, 40)}
    if kind in ("mixed", "target"):
        flow = rng.choice(("tgv", "rbc")) if kind == "mixed" else "tgv"
        i = rng.randint(5, 8)
        iz = i - 1 if flow == "rbc" else i
        return {"kind": kind, "flow": flow, "ix": i, "iy": i, "iz": iz, "depth": iz - rng.randint(1, 2), "steps": rng.randint(2, 3) if i > 7 else rng.randint(3, 8)}
    if kind == "operators":
        i = rng.randint(4, 7)
        return {"kind": kind, "flow": "tgv", "ix": i, "iy": _near(rng, i, 4, 7), "iz": _near(rng, i, 4, 7)}
    if kind == "cn":
        i = rng.randint(4, 7)
        flow = rng.choice(("ldc", "tgv", "rbc"))
        return {"kind": kind, "flow": flow, "ix": i, "iy": _near(rng, i, 4, 7), "iz": _near(rng, i, 4, 7),
                "comp": rng.randint(0, 3 if flow == "rbc" else 2), "fast": rng.choice((0, 1, 2))}
    i = rng.randint(5, 7)
    return {"kind": kind, "flow": "tgv", "ix": i, "iy": _near(rng, i, 5, 7), "iz": _near(rng, i, 5, 7), "depth": rng.randint(3, 4)}


# ---------------------------------------------------------------- parameters and initial states
def _params(case):
    p = F.default_params()
    p.xInd, p.yInd, p.zInd = case["ix"], case["iy"], case["iz"]
    p.vcDepth = case.get("depth") or max(1, min(case["ix"], case["iy"], case["iz"]) - 2)
    p.cnTolerance = p.mgTolerance = 1.0e-8
    p.preSmooth = p.postSmooth = 3
    p.gsSmooth, p.vcCount, p.resType = 0, 200, 1
    flow = case["flow"]
    if flow == "tgv":
        p.probType, p.icType = 2, 1
        p.xPer = p.yPer = p.zPer = 1
        p.Lx = p.Ly = p.Lz = 2.0 * math.pi
        p.Re, p.tStp = 1600.0, 5.0e-4
    elif flow == "ldc":
        p.probType, p.icType = 1, 0
        p.xPer = p.yPer = p.zPer = 0
        p.Lx = p.Ly = p.Lz = 1.0
        p.Re, p.tStp = 1000.0, 1.0e-3
    elif flow == "rbc":
        p.probType, p.icType = 5, 0
        p.xPer = p.yPer = 1
        p.zPer = 0
        p.Lx, p.Ly, p.Lz = 2.0, 2.0, 1.0
        p.Ra, p.Pr, p.rbcType, p.forceType = 1.0e7, 1.0, 2, 3
        p.Re, p.tStp = 1.0, 5.0e-4
    else:                                    # the 2D cavity in x-z
        p.probType, p.icType = 1, 0
        p.xPer = p.yPer = p.zPer = 0
        p.Lx = p.Ly = p.Lz = 1.0
        p.Re, p.tStp, p.tMax = 1000.0, 1.0e-3, 50.0
        p.useCFL, p.courantNumber = 1, 0.1
        p.cnTolerance = p.mgTolerance = 1.0e-6
        p.preSmooth = p.postSmooth = 2
        p.vcCount = 7
    if case.get("gs"):
        p.gsSmooth = 1
        if flow != "cav2d":                  # the shipped input file
            p.cnTolerance = p.mgTolerance = 1.0e-6
            p.preSmooth = p.postSmooth = 4
            p.vcCount = 5
            if flow == "tgv":
                p.Lx = p.Ly = p.Lz = 1.0
                p.Re, p.tStp = 1000.0, 1.0e-3
    if case.get("cycles") and not case["gs"]:  # a cap on the V-cycles, as the shipped file sets one
        p.vcCount = case["cycles"]
    if case.get("stretch"):                  # Mesh Type 'D' along the wall-normal axis
        p.zGrid, p.betaZ = 2, 1.2
    if case["kind"] in ("mixed", "target"):
        p.mgMode = F.MG_MIXED if case["kind"] == "mixed" else F.MG_PLAIN_TARGET
        p.mgTarget, p.mgMaxCycles, p.mixedCycles = 1.0e-8, 100, 0
        p.smoother = F.SMOOTHER_CHEBYSHEV
        p.jacobiWeight = 6.0 / 7.0
        p.fastKernels = 2
        p.coarseCycles = 3 if case["kind"] == "target" else 1
        p.preSmooth = p.postSmooth = 2 if case["kind"] == "target" else 3
    if case["kind"] == "cn":
        p.fastKernels = case["fast"]
    return p


def _waves(p, axis_field, rng, walls):
    """Smooth seeded values on the padded points of velocity component `axis_field`:
    waves that vary along the other two axes only on periodic axes (so the field has
    no divergence of its own), and vanish on walls."""
    co = S.grid_coords(p)
    x = [co[d][1 if d == axis_field else 0] for d in range(3)]
    L = (p.Lx, p.Ly, p.Lz)
    out = np.zeros([len(v) for v in x])
    for d in range(3):
        if (p.xPer, p.yPer, p.zPer)[d] and d == axis_field:
            continue
        a, ph, n = 0.1 + 0.2 * rng.random(), 2 * math.pi * rng.random(), rng.integers(1, 3)
        w = a * np.sin(2 * math.pi * n * x[d] / L[d] + ph)
        out += w.reshape([-1 if q == d else 1 for q in range(3)])
    for d in range(3):
        if walls[d]:
            out *= np.sin(math.pi * x[d] / L[d]).reshape([-1 if q == d else 1 for q in range(3)])
    return out


def _initial(p, flow, seed):
    """{field: padded array}: the flow's initial condition with seeded waves added."""
    rng = np.random.default_rng(seed)
    walls = [not p.xPer, not p.yPer and p.yInd, not p.zPer]
    q = {}
    if flow == "tgv":
        Vx, Vy = S.taylor_green_velocity(p)
        q[F.FIELD_VX] = Vx + _waves(p, 0, rng, walls)
        q[F.FIELD_VY] = Vy + _waves(p, 1, rng, walls)
        q[F.FIELD_VZ] = _waves(p, 2, rng, walls)
        q[F.FIELD_P] = S.taylor_green_pressure(p)
    else:
        amp = 0.3 if flow == "rbc" else 0.5
        for d in range(3):
            if p.yInd or d != 1:
                q[F.FIELD_VX + d] = amp * _waves(p, d, rng, walls)
    if flow == "rbc":
        q[F.FIELD_T] = S.rbc_temperature(p, seed=int(seed) & 0xFFFF, amplitude=1.0e-2)
    return q


def _pinned(g, fields):
    return [torch.empty(g.dims(f), dtype=torch.float64, pin_memory=torch.cuda.is_available()) for f in fields]


def _ptrs(bufs):
    return [b.data_ptr() for b in bufs]


def _start(p, flow, seed):
    """A solver in the flow's initial state, boundaries filled."""
    g = S.Solver(p)
    g.set(F.FIELD_P, np.ones(g.dims(F.FIELD_P)))
    for f, a in _initial(p, flow, seed).items():
        g.set(f, np.broadcast_to(a, g.dims(f)))
    for f in V3 + ((F.FIELD_T,) if flow == "rbc" else ()):
        g.apply_bc(f)
    return g


def prepare(case, seed):
    kind, flow = case["kind"], case["flow"]
    p = _params(case)
    if kind == "unet":
        g = S.Solver(p)
        n, dims = g.unet_shape()
        rng = np.random.default_rng(seed)
        w, off = np.empty(n, dtype=np.float32), 0
        for cin, co in _LAYERS:
            m = 27 * cin * co
            w[off:off + m] = rng.uniform(-1, 1, m) * math.sqrt(6.0 / (27 * cin))
            w[off + m:off + m + co] = rng.uniform(-0.1, 0.1, co)
            off += m + co
        return {"kind": kind, "g": g, "feat": rng.standard_normal(dims + (3,)).astype(np.float32),
                "target": rng.standard_normal(dims).astype(np.float32), "params": w}
    if kind == "cn":
        v, rhs = _cn_inputs(case, p, seed)
        return {"kind": kind, "p": p, "comp": case["comp"], "v0": v, "v": v.clone(), "rhs": rhs, "lib": F.load()}
    if kind == "operators":
        p.mgMode = F.MG_REFERENCE
        g = _start(p, flow, seed)
        out = NSE + GRAD + (F.FIELD_MGRHS,)
        return {"kind": kind, "g": g, "fields": out, "out": _pinned(g, out), "nu": 1.0 / p.Re}
    g = _start(p, flow, seed)
    fields = V3 + (F.FIELD_P,) + ((F.FIELD_T,) if flow == "rbc" else ())
    if flow == "cav2d":
        fields = (F.FIELD_VX, F.FIELD_VZ, F.FIELD_P)
    s = {"kind": kind, "g": g, "fields": fields, "out": _pinned(g, fields), "steps": case["steps"], "cfl": p.useCFL, "dt": p.tStp}
    if kind == "mixed":                      # a simulation under way: its start-up steps, the history of the guess filled
        for _ in range(3):
            _step(g)
        g.set_guess_mode(F.GUESS_EXTRAPOLATE)
        for _ in range(5 if flow == "tgv" else 40):
            _step(g)
        return s
    for _ in range(5 if kind == "target" else 2 if max(case["ix"], case["iz"]) < 7 else 1):
        _step(g)
    s["state"] = fields + (F.FIELD_PP,)
    s["in"] = _pinned(g, s["state"])
    g.download_fields_ptr(s["state"], _ptrs(s["in"]))
    return s


def _step(g):
    status, st = g.time_advance()
    if status != 0:
        raise RuntimeError("time_advance: status %d" % status)
    return st


def run(state):
    kind = state["kind"]
    if kind == "unet":
        out, loss, grad = state["g"].unet_grad_check(state["feat"], state["target"], state["params"])
        return {"out": out, "loss": loss, "grad": grad}
    if kind == "cn":
        state["v"].copy_(state["v0"])
        it, err = ctypes.c_int(), ctypes.c_double()
        s = state["lib"].saras_cn_solve_noalloc(ctypes.byref(state["p"]), state["comp"], ctypes.c_void_p(state["v"].data_ptr()),
                                                ctypes.c_void_p(state["rhs"].data_ptr()), None, ctypes.byref(it), ctypes.byref(err))
        if s != 0:
            raise RuntimeError("saras_cn_solve_noalloc: status %d" % s)
        return {"v": state["v"], "iterations": it.value}
    g = state["g"]
    if kind == "operators":
        for f in NSE:
            g.axpby(f, 0.0, -1, 0.0)
        g.vfield_compute_diff()
        for f in NSE:
            g.axpby(f, state["nu"], -1, 0.0)
        g.vfield_compute_nlin()
        g.sfield_gradient(F.FIELD_P)
        g.vfield_divergence()
        g.download_fields_ptr(state["fields"], _ptrs(state["out"]))
        return state["out"]
    counts = []
    if "in" in state:
        g.upload_fields_ptr(state["state"], _ptrs(state["in"]))
        if state["cfl"]:
            g.set_dt(state["dt"])
    for _ in range(state["steps"]):
        st = _step(g)
        if state["cfl"]:                     # solvePDE's time step
            g.set_dt(min(g.compute_tstp(), state["dt"]))
        if kind == "dropin":                 # the drop-in takes the reference's iteration counts
            counts += list(st.cn_iters) + [st.vcycles]
    g.download_fields_ptr(state["fields"], _ptrs(state["out"]))
    return {"fields": state["out"], "counts": np.array(counts, dtype=np.int64)} if counts else state["out"]


def work(case):
    n = [2 ** case["ix"] + 1, 2 ** case["iy"] + 1 if case["iy"] else 1, 2 ** case["iz"] + 1]
    pts = float(n[0] * n[1] * n[2])
    kind = case["kind"]
    if kind == "cn":                         # the iterate and the right-hand side in, the solution out; two sweeps of 13 operations
        return {"bytes": 24.0 * pts, "flops": 26.0 * pts}
    if kind == "operators":                  # four fields in, seven out
        return {"bytes": 88.0 * pts, "flops": 170.0 * pts}
    if kind == "unet":                       # 3 x the forward convolutions; features, target and parameters in, output and gradients out
        m = [2 ** max(1, case[q] - 1) + 1 for q in ("ix", "iy", "iz")]
        v = [float(np.prod([(q - 1) // 2 ** k + 1 for q in m])) for k in range(3)]
        lvl = (0, 0, 1, 1, 2, 2, 1, 1, 0, 0, 0)
        fwd = sum(54.0 * cin * co * v[k] for (cin, co), k in zip(_LAYERS, lvl))
        npar = sum(27 * cin * co + co for cin, co in _LAYERS)
        return {"bytes": 4.0 * (5 * v[0] + 2 * npar), "flops": 3.0 * fwd}
    fields = 7 if case["flow"] == "rbc" else 4 if case["flow"] == "cav2d" else 5
    # a step reads and writes its fields once; right-hand sides, projection and one V-cycle are the arithmetic at least
    return {"bytes": 16.0 * fields * pts * case["steps"], "flops": 400.0 * pts * case["steps"]}


# ---------------------------------------------------------------- the Jacobi solve on the caller's arrays
_STAG = ((0, 1, 1), (1, 0, 1), (1, 1, 0), (1, 1, 1))


def _cn_shape(p, comp):
    return [2 ** i + _STAG[comp][d] for d, i in enumerate((p.xInd, p.yInd, p.zInd))]


def _cn_inputs(case, p, seed):
    """An iterate and a right-hand side near it, as a time step forms them."""
    n = _cn_shape(p, case["comp"])
    gen = torch.Generator(device="cpu").manual_seed(int(seed))
    x = [torch.linspace(0, 1, m + 2, dtype=torch.float64) for m in n]
    v = torch.zeros([m + 2 for m in n], dtype=torch.float64)
    for d in range(3):
        a, ph = torch.rand(2, generator=gen, dtype=torch.float64)
        v += (a * torch.sin(2 * math.pi * (x[d] + ph))).reshape([-1 if q == d else 1 for q in range(3)])
    r = v + 1.0e-3 * torch.randn(v.shape, generator=gen, dtype=torch.float64)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    return v.to(dev), r.to(dev)


def _cn_boundary(p, comp, n, v):
    """Periodic copies, edges and walls of component `comp` on the padded array v."""
    per = (p.xPer, p.yPer, p.zPer)
    st = _STAG[comp]
    lo = [1 if st[d] else 0 for d in range(3)]
    hi = [n[d] - 1 - (1 if st[d] else 0) for d in range(3)]
    core = [slice(1, n[d] + 1) for d in range(3)]

    def copy(to, src):
        v[tuple(to)] = v[tuple(src)].clone()

    for d in (0, 1):
        if per[d]:
            for ghost, image in ((-1, hi[d]), (n[d], lo[d])):
                t, s = list(core), list(core)
                t[d], s[d] = ghost + 1, image + 1
                copy(t, s)
    for gx, ix in ((-1, hi[0]), (n[0], lo[0])):
        for gy, iy in ((-1, hi[1]), (n[1], lo[1])):
            copy([gx + 1, gy + 1, core[2]], [ix + 1, iy + 1, core[2]])
    blo = [1 if st[d] and not per[d] else 0 for d in range(3)]
    bhi = [n[d] - 1 - (1 if st[d] and not per[d] else 0) for d in range(3)]
    full = [slice(None)] * 3
    for wall in (0, 1, 2, 3, 5, 4):
        d, even = wall // 2, wall % 2 == 0
        w = blo[d] - 1 if even else bhi[d] + 1
        t, s = list(full), list(full)
        t[d] = w + 1
        if per[d]:
            if d == 2:                       # x and y are the periodic copies above
                src = (bhi[2] - 1 if even else blo[2] + 1) if st[2] else (bhi[2] if even else blo[2])
                s[2] = src + 1
                copy(t, s)
            continue
        s[d] = w + 1 + (1 if even else -1)
        if comp == 3:
            if d == 2:
                v[tuple(t)] = 1.0 if even else 0.0
            else:
                copy(t, s)
        elif st[d]:
            v[tuple(t)] = 1.0 if p.probType == 1 and comp == 0 and wall == 5 else 0.0
        else:
            v[tuple(t)] = -v[tuple(s)]


def _cn_exact(case, seed):
    p = _params(case)
    comp = case["comp"]
    n = _cn_shape(p, comp)
    v, rhs = _cn_inputs(case, p, seed)
    nu = 1.0 / p.Re if case["flow"] != "rbc" else math.sqrt(p.Pr / p.Ra) if comp < 3 else 1.0 / math.sqrt(p.Pr * p.Ra)
    per, st = (p.xPer, p.yPer, p.zPer), _STAG[comp]
    c = [0.5 * p.tStp * nu * (2.0 ** i / L) ** 2 for i, L in zip((p.xInd, p.yInd, p.zInd), (p.Lx, p.Ly, p.Lz))]
    b = [slice(1 + (1 if st[d] and not per[d] else 0), n[d] + 1 - (1 if st[d] and not per[d] else 0)) for d in range(3)]

    def off(d, s):
        q = list(b)
        q[d] = slice(b[d].start + s, b[d].stop + s)
        return tuple(q)
    b = tuple(b)
    for _ in range(400):
        a = rhs[b].clone()
        for d in range(3):
            a += c[d] * (v[off(d, 1)] + v[off(d, -1)])
        a /= 1.0 + 2.0 * sum(c)
        w = torch.zeros_like(v)
        w[b] = a
        _cn_boundary(p, comp, n, w)
        done = bool((w - v).abs().max() < 1.0e-15)
        v = w
        if done:
            break
    return {"v": v, "iterations": None}


# ---------------------------------------------------------------- the operators in plain torch
def _ops_exact(case, seed):
    p = _params(case)
    g = _start(p, case["flow"], seed)        # the inputs a program has in hand: its fields with their boundaries filled
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    v = [torch.from_numpy(g.get(f)).to(dev) for f in V3]
    pr = torch.from_numpy(g.get(F.FIELD_P)).to(dev)
    g.close()
    ih = [2.0 ** i / L for i, L in zip((p.xInd, p.yInd, p.zInd), (p.Lx, p.Ly, p.Lz))]
    half = 0.5 if p.iScheme == 1 else 1.0

    def sh(a, o):                            # a at the core points displaced by o
        return a[tuple(slice(1 + o[d], a.shape[d] - 1 + o[d]) for d in range(3))]

    def at(a, o, n):                         # the same on the first n points of each axis
        return a[tuple(slice(1 + o[d], 1 + o[d] + n[d]) for d in range(3))]
    e = ((1, 0, 0), (0, 1, 0), (0, 0, 1))
    neg = tuple(tuple(-q for q in r) for r in e)
    nse, grad = [], []
    for q in range(3):
        f = v[q]
        n = [m - 2 for m in f.shape]
        h = sum(half * ih[d] ** 2 * (sh(f, e[d]) - 2.0 * sh(f, (0, 0, 0)) + sh(f, neg[d])) for d in range(3)) / p.Re
        for d in range(3):
            if d == q:
                u = sh(f, (0, 0, 0))
            else:                            # component d averaged to the points of component q
                u = 0.25 * sum(at(v[d], [a * e[q][x] - b * e[d][x] for x in range(3)], n) for a in (0, 1) for b in (0, 1))
            h = h - u * 0.5 * ih[d] * (sh(f, e[d]) - sh(f, neg[d]))
        whole = torch.zeros_like(f)
        whole[1:-1, 1:-1, 1:-1] = h
        nse.append(whole)
        whole = torch.zeros_like(f)
        whole[1:-1, 1:-1, 1:-1] = ih[q] * (at(pr, e[q], n) - at(pr, (0, 0, 0), n))
        grad.append(whole)
    div = torch.zeros_like(pr)
    full = [m - 2 for m in pr.shape]
    d = sum(ih[q] * (v[q][tuple(slice(1, 1 + full[x]) for x in range(3))] - v[q][tuple(slice(1 - e[q][x], 1 - e[q][x] + full[x]) for x in range(3))])
            for q in range(3))
    div[1:-1, 1:-1, 1:-1] = d
    return nse + grad + [div]


# ---------------------------------------------------------------- the network in plain torch
_LAYERS = ((16, 16), (16, 16), (16, 32), (32, 32), (32, 64), (64, 64), (96, 32), (32, 32), (48, 16), (16, 16), (16, 16))


def _unet_exact(case, seed):
    s = prepare(case, seed)
    s["g"].close()
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    f64 = torch.float64
    bf = lambda a: torch.from_numpy(a).to(torch.bfloat16).to(f64).to(dev)  # noqa: E731  (the tensor cores' operands)
    conv3d = torch.nn.functional.conv3d
    ws, off = [], 0
    for cin, co in _LAYERS:
        m = 27 * cin * co
        w = bf(s["params"][off:off + m]).reshape(co, 3, 3, 3, cin).permute(0, 4, 1, 2, 3).contiguous().requires_grad_(True)
        b = torch.from_numpy(s["params"][off + m:off + m + co]).to(f64).to(dev).requires_grad_(True)
        ws.append((w, b))
        off += m + co

    def conv(q, x):
        y = conv3d(x, ws[q][0], ws[q][1], padding=1)
        return torch.relu(y) if q < len(_LAYERS) - 1 else y

    def down(x):
        k1 = torch.tensor([0.25, 0.5, 0.25], dtype=f64, device=dev)
        k = (k1[:, None, None] * k1[None, :, None] * k1[None, None, :]).expand(x.shape[1], 1, 3, 3, 3)
        return conv3d(x, k, stride=2, padding=1, groups=x.shape[1])

    def up(x, shape):
        for d in range(3):
            i = torch.arange(shape[d], device=dev)
            a = i // 2
            x = 0.5 * (x.index_select(2 + d, a) + x.index_select(2 + d, torch.clamp(a + i % 2, max=x.shape[2 + d] - 1)))
        return x

    x0 = torch.zeros((1, 16) + s["target"].shape, dtype=f64, device=dev)
    x0[0, :3] = bf(s["feat"]).permute(3, 0, 1, 2)
    e1 = conv(1, conv(0, x0))
    e2 = conv(3, conv(2, down(e1)))
    e3 = conv(5, conv(4, down(e2)))
    f2 = conv(7, conv(6, torch.cat([up(e3, e2.shape[2:]), e2], 1)))
    f1 = conv(9, conv(8, torch.cat([up(f2, e1.shape[2:]), e1], 1)))
    y = conv(10, f1)[0, 0]
    loss = 0.5 * torch.mean((y - torch.from_numpy(s["target"]).to(f64).to(dev)) ** 2)
    loss.backward()
    grad = torch.cat([torch.cat([w.grad.permute(0, 2, 3, 4, 1).reshape(-1), b.grad]) for w, b in ws])
    return {"out": y.detach(), "loss": float(loss.item()), "grad": grad}


def exact(case, seed):
    """64-bit values of the operators, the Jacobi solve and the network.  A time
    step's outputs are where its stopping rules leave the iterations: no value
    but the algorithm's own."""
    if case["kind"] == "operators":
        return _ops_exact(case, seed)
    if case["kind"] == "cn":
        return _cn_exact(case, seed)
    if case["kind"] == "unet":
        return _unet_exact(case, seed)
    return None
