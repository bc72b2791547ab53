"""Timed cases of the framework's main path: advancing grids that live on the GPU.

A case is one grid (or one batch of grids) of the kind a DRAGON user steps:
the Sod tube, the shear layer, the Orszag-Tang vortex, the 3D blast and the
batch of uneven small grids, at the sizes of the tests, the benchmark and the
examples, plus ragged ones. A pass advances it through the public Python API,
as a stepping loop does, and returns the state it ends in. The state evolves
from pass to pass, as it does in a run.

exact() restates the scheme in plain torch, FP64, from the formulas (whole
padded arrays, shifts and masks; no code of the framework).
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

import dragon_b200 as dg
from dragon_b200 import _lib
from dragon_b200.batch import Batch
from dragon_b200.boundary import Outflow, Periodic, Reflective

RIEMANN = {"hllc": dg.RIEMANN_HLLC, "hlle": dg.RIEMANN_HLLE, "hll": dg.RIEMANN_HLL, "roe": dg.RIEMANN_ROE,
           "exact": dg.RIEMANN_EXACT, "hlld": dg.RIEMANN_HLLD}
LIMITER = {"minmod": dg.LIMITER_MINMOD, "mc": dg.LIMITER_MC, "vanleer": dg.LIMITER_VANLEER,
           "superbee": dg.LIMITER_SUPERBEE}
BOUNDARY = {"periodic": Periodic, "outflow": Outflow, "walls": lambda: Reflective("X") + Periodic("YZ")}


def _case(name, kind, nx, ny=0, nz=0, mhd=False, mixed=False, solver="hllc", limiter="vanleer", boundary="periodic",
          how="steps", steps=4):
    c = {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "mhd": mhd, "mixed": mixed, "solver": solver, "limiter": limiter,
         "boundary": boundary, "how": how, "steps": steps}
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest grid a user steps: the README's Sod tube to an output time (latency and launches count)
        _case("sod tube 512", "tube", 512, limiter="mc", boundary="outflow", how="interval", steps=40),
        # a long MHD tube (Dai-Woodward and Brio-Wu type states), one-dimensional throughput, ragged length
        _case("mhd tube 200003", "tube", 200003, mhd=True, solver="hlld", limiter="mc", boundary="outflow", steps=10),
        # a small 2D grid in the examples' main loop (boundary, dt = cfl_time(), advance(dt)): the user looks at every step
        _case("shear layer 96 loop", "shear", 96, 96, how="loop", steps=10),
        # the headline configuration of the benchmark
        _case("shear layer 1024", "shear", 1024, 1024),
        # the same in mixed precision
        _case("shear layer 1024 mixed", "shear", 1024, 1024, mixed=True, steps=8),
        # a ragged 2D grid between walls with another solver and limiter
        _case("walls 777x1301 roe", "shear", 777, 1301, solver="roe", limiter="mc", boundary="walls"),
        # 2D MHD: Orszag-Tang at the size the accuracy tests use
        _case("vortex 384", "vortex", 384, 384, mhd=True, solver="hlld", limiter="mc"),
        # 2D MHD at the benchmark's size in mixed precision
        _case("vortex 1024 mixed", "vortex", 1024, 1024, mhd=True, mixed=True, solver="hlld", limiter="mc"),
        # 3D blast, approximate solver
        _case("blast 128", "blast", 128, 128, 128, limiter="mc", boundary="outflow", steps=3),
        # 3D blast with the exact solver (the reference's default comparison), ragged box
        _case("blast 110x87x93 exact", "blast", 110, 87, 93, solver="exact", limiter="mc", boundary="outflow", steps=2),
        # 3D MHD blast
        _case("blast mhd 96", "blast", 96, 96, 96, mhd=True, solver="hlld", limiter="mc", boundary="outflow", steps=2),
        # many uneven small grids together: 1D tubes and 2D MHD blasts, the batched step
        _case("batch 40+8", "batch", 4096, 160, mhd=True, solver="hlld", limiter="mc", steps=8),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["tube", "tube", "shear", "shear", "shear", "vortex", "vortex", "blast", "blast", "batch"])
    mhd = kind in ("vortex", "batch") or (kind in ("tube", "blast") and rng.random() < 0.4)
    mixed = rng.random() < 0.25
    solver = rng.choice(["hlld", "hlld", "hlle"]) if mhd else rng.choice(["hllc", "hllc", "roe", "hlle", "exact"])
    if mixed and solver in ("roe", "exact"):
        solver = "hllc"
    limiter = rng.choice(["mc", "vanleer", "minmod"])
    if kind == "tube":
        how = rng.choice(["interval", "steps", "loop"])
        return _case(None, kind, _log(rng, 64, 500000), mhd=mhd, mixed=mixed, solver=solver, limiter=limiter,
                     boundary="outflow", how=how, steps=rng.randint(5, 40) if how == "interval" else rng.randint(4, 12))
    if kind == "shear":
        return _case(None, kind, _log(rng, 24, 1100), _log(rng, 24, 1100), mixed=mixed, solver=solver, limiter=limiter,
                     boundary=rng.choice(["periodic", "walls"]), how=rng.choice(["steps", "steps", "loop"]),
                     steps=rng.randint(2, 5))
    if kind == "vortex":
        return _case(None, kind, _log(rng, 32, 800), _log(rng, 32, 800), mhd=True, mixed=mixed, solver=solver,
                     limiter=limiter, steps=rng.randint(2, 4))
    if kind == "blast":
        n = [_log(rng, 20, 112) for _ in range(3)]
        return _case(None, kind, *n, mhd=mhd, mixed=mixed, solver=solver, limiter=limiter, boundary="outflow",
                     steps=rng.randint(1, 2))
    return _case(None, kind, _log(rng, 256, 4096), _log(rng, 48, 192), mhd=True, mixed=mixed, solver="hlld",
                 limiter="mc", steps=rng.randint(4, 8))


# ---- initial states: interior arrays, fields last --------------------------------------------------------------


def _centres(n, lo=0.0, hi=1.0):
    return lo + (np.arange(n) + 0.5) * ((hi - lo) / n)


def _tube(rng, n, mhd):
    w = np.zeros((n, 8 if mhd else 5))
    left = np.arange(n) < n // 2
    w[:, 0] = np.where(left, 1.0 + 0.2 * rng.random(), 0.125 + 0.02 * rng.random())
    w[:, 1] = np.where(left, 1.0 + 0.2 * rng.random(), 0.1 + 0.02 * rng.random())
    w[:, 2] = 0.1 * rng.random()
    if mhd:
        w[:, 5] = 0.75 * math.sqrt(4 * math.pi)
        w[:, 6] = np.where(left, 1.0, -1.0) * math.sqrt(4 * math.pi) * (0.8 + 0.2 * rng.random())
        w[:, 7] = 0.1 * rng.random()
    return w, None, (1.0 / n,)


def _shear(rng, nx, ny):
    w = np.zeros((nx, ny, 5))
    inner = np.abs(_centres(ny) - 0.5) < 0.25
    w[..., 0] = np.where(inner, 2.0, 1.0)
    w[..., 1] = 2.5
    w[..., 2] = np.where(inner, 0.5, -0.5)
    w[..., 3] = rng.uniform(-0.01, 0.01, (nx, ny))
    return w, None, (1.0 / nx, 1.0 / ny)


def _vortex(rng, nx, ny):
    b0, tau = 1.0 / math.sqrt(4 * math.pi), 2 * math.pi
    w, B = np.zeros((nx, ny, 8)), np.zeros((nx + 1, ny + 1, 3))
    x, y = _centres(nx), _centres(ny)
    w[..., 0] = 25 / (36 * math.pi)
    w[..., 1] = 5 / (12 * math.pi)
    w[..., 2] = -np.sin(tau * y)[None, :]
    w[..., 3] = np.sin(tau * x)[:, None]
    w[..., 2:4] += rng.uniform(-1e-3, 1e-3, (nx, ny, 2))
    B[:, :ny, 0] = -b0 * np.sin(tau * y)[None, :]
    B[:nx, :, 1] = b0 * np.sin(2 * tau * x)[:, None]
    B[..., 2] = 0.01
    return w, B, (1.0 / nx, 1.0 / ny)


def _blast(rng, n, mhd, p_in=10.0, radius=0.15):
    d = tuple(1.0 / k for k in n)
    c = rng.uniform(-0.05, 0.05, len(n))
    r2 = sum(np.square(q) for q in np.meshgrid(*[_centres(k, -0.5, 0.5) - s for k, s in zip(n, c)], indexing="ij"))
    w = np.zeros(n + (8 if mhd else 5,))
    w[..., 0] = 1.0
    w[..., 1] = np.where(r2 < radius * radius, p_in * (0.8 + 0.4 * rng.random()), 0.1)
    B = None
    if mhd:
        B = np.zeros(tuple(k + 1 for k in n) + (3,))
        B[...] = np.array([0.5, 0.3, 0.2]) * (0.9 + 0.2 * rng.random())
    return w, B, d


def _members(case, seed):
    """The 1D tubes and 2D MHD blasts of a batch: their states from the seed, their sizes from the case."""
    rng, size = np.random.default_rng(seed), np.random.default_rng(9)
    out = []
    for k in range(40):
        n = int(round(math.exp(size.uniform(math.log(64), math.log(case["nx"] + 1)))))
        out.append((_tube(rng, n, False), False, "outflow"))
    for k in range(8):
        n = int(size.choice([case["ny"], 2 * case["ny"] // 3, case["ny"] // 2]))
        out.append((_blast(rng, (n, n), True, p_in=5.0, radius=0.1), True, "periodic"))
    return out


def _initial(case, seed):
    rng = np.random.default_rng(seed)
    if case["kind"] == "tube":
        return _tube(rng, case["nx"], case["mhd"])
    if case["kind"] == "shear":
        return _shear(rng, case["nx"], case["ny"])
    if case["kind"] == "vortex":
        return _vortex(rng, case["nx"], case["ny"])
    return _blast(rng, (case["nx"], case["ny"], case["nz"]), case["mhd"])


# ---- a grid on the GPU and views of its state -------------------------------------------------------------------


class _Planes:
    """The field planes of a grid's device state, for torch (no copy); the tensor keeps the grid alive."""

    def __init__(self, grid, ptr, shape, strides):
        self.grid = grid
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<f8", "data": (ptr, False), "strides": strides,
                                         "version": 2}


def _grid(case, w, B, d, mhd, boundary):
    cls = (dg.Grid1D, dg.Grid2D, dg.Grid3D)[len(d) - 1]
    solver = case["solver"] if mhd == case["mhd"] else "hllc"
    cfg = dg.Config(mhd=mhd, riemann=RIEMANN[solver], limiter=LIMITER[case["limiter"]],
                    precision=dg.PREC_MIXED if case["mixed"] else dg.PREC_FP64)
    G = cls(*w.shape[:-1], *d, ghosts=3 if mhd else 2, config=cfg)
    G.boundary = BOUNDARY[boundary]()
    g = G.ghosts
    G.w[tuple(slice(g, g + n) for n in G.n)] = w
    if B is not None:
        G.B[tuple(slice(g, g + n + 1) for n in G.n)] = B
        G.initialize_B_fields()
    G.upload() if B is None else None
    return G


def _state_view(G, seen):
    """The interior of the current state, (field, i[, j[, k]]): a view of the device planes."""
    p, plane, pitch = ctypes.c_void_p(), ctypes.c_longlong(), ctypes.c_longlong()
    _lib.check(G._lib.dragon_gpu_device_state(G._h, ctypes.byref(p), ctypes.byref(plane), ctypes.byref(pitch)))
    at = p.value
    if at not in seen:
        g, n = G.ghosts, G.n
        strides = {1: (8,), 2: (8 * pitch.value, 8), 3: (8 * pitch.value * (n[1] + 2 * g if G.dim == 3 else 0),
                                                         8 * pitch.value, 8)}[G.dim]
        first = at + g * sum(strides)
        planes = _Planes(G, first, (G.nfields, *n), (8 * plane.value, *strides))
        seen[at] = torch.as_tensor(planes, device="cuda")
    return seen[at]


def _face_buffer(G):
    """A device buffer for the face-centred B of the interior faces and its views per component."""
    count = ctypes.c_longlong()
    _lib.check(G._lib.dragon_gpu_halo_size(G._h, 0, G.n[0] + 1, 1, 0, ctypes.byref(count)))
    return torch.empty(count.value, dtype=torch.float64, device="cuda")


def prepare(case, seed):
    if case["kind"] == "batch":
        grids = [_grid(case, *state, mhd, bc) for state, mhd, bc in _members(case, seed)]
        return {"case": case, "grids": grids, "batch": Batch(grids), "seen": {}}
    w, B, d = _initial(case, seed)
    G = _grid(case, w, B, d, case["mhd"], case["boundary"])
    s = {"case": case, "grid": G, "seen": {}, "faces": None if B is None else _face_buffer(G)}
    if case["how"] == "interval":
        s["interval"] = 0.1 * case["steps"] / case["nx"]
    return s


def run(state):
    case = state["case"]
    if case["kind"] == "batch":
        state["batch"].advance_steps(case["steps"])
        return {"w": [_state_view(G, state["seen"]) for G in state["grids"]]}
    G = state["grid"]
    t = 0.0
    if case["how"] == "interval":
        t = G.advance(state["interval"]).time_advanced
    elif case["how"] == "loop":
        for _ in range(case["steps"]):
            G.apply_boundary()
            t += G.advance(G.cfl_time()).time_advanced
    else:
        t = G.advance_steps(case["steps"]).time_advanced
    out = {"w": _state_view(G, state["seen"]), "t": t}
    if state["faces"] is not None:
        buf = state["faces"]
        _lib.check(G._lib.dragon_gpu_halo_pack(G._h, 0, 0, G.n[0] + 1, 1, 0, ctypes.cast(buf.data_ptr(), _lib.c_double_p), 1))
        out["B"] = buf
    return out


# floating-point operations of one cell update (every division and square root one operation, no halo)
_FLOPS = {(1, False): 350, (1, True): 800, (2, False): 1400, (2, True): 3400, (3, False): 4200, (3, True): 6500}


def work(case):
    if case["kind"] == "batch":
        n1 = 40 * (case["nx"] - 64) / math.log((case["nx"] + 1) / 64)
        n2 = 8 * case["ny"] ** 2 * (1 + 4 / 9 + 1 / 4) / 3
        return {"bytes": n1 * 80 + n2 * 176, "flops": case["steps"] * (n1 * _FLOPS[1, False] + n2 * _FLOPS[2, True])}
    n = [k for k in (case["nx"], case["ny"], case["nz"]) if k]
    cells = math.prod(n)
    fields = (8 + (3 if len(n) > 1 else 0)) if case["mhd"] else 5
    return {"bytes": 16.0 * cells * fields, "flops": float(case["steps"]) * cells * _FLOPS[len(n), case["mhd"]]}


# ---- the scheme in plain torch, FP64 ----------------------------------------------------------------------------
# States are (field, i[, j[, k]]) over the padded grid; _at(a, ax, k)[i] = a[i + k] along axis ax. The outermost
# layers of the shifted arrays are meaningless and never reach the interior.

GAMMA = 5.0 / 3.0
GM1, GP1 = GAMMA - 1.0, GAMMA + 1.0
Q4, Q8 = 0.25 / math.pi, 0.125 / math.pi


def _at(a, ax, k):
    return torch.roll(a, -k, ax + 1) if a.dim() > 1 else a


def _sh(a, ax, k):
    """_at for an array without a field axis."""
    return torch.roll(a, -k, ax)


def _swap(a, ax):
    """The frame in which axis ax is x."""
    if ax == 0:
        return a
    i = list(range(a.shape[0]))
    i[2], i[2 + ax] = i[2 + ax], i[2]
    if len(i) == 8:
        i[5], i[5 + ax] = i[5 + ax], i[5]
    return a[i]


def _dot(a, b):
    return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]


def _cons(w):
    u = w.clone()
    u[2:5] = w[2:5] * w[0]
    u[1] = w[1] / GM1 + 0.5 * w[0] * _dot(w[2:5], w[2:5])
    if w.shape[0] == 8:
        u[1] += _dot(w[5:8], w[5:8]) * Q8
    return u


def _prim(u):
    w = u.clone()
    w[2:5] = u[2:5] / u[0]
    e = u[1] - _dot(u[2:5], u[2:5]) / (2 * u[0])
    if u.shape[0] == 8:
        e = e - _dot(u[5:8], u[5:8]) * Q8
    w[1] = GM1 * e
    return w


def _xflux(w):
    """Flux along x of a primitive state."""
    u = _cons(w)
    f = u * w[2]
    f[2] += w[1]
    f[1] += w[1] * w[2]
    if w.shape[0] == 8:
        pm, t = _dot(w[5:8], w[5:8]) * Q8, w[5:8] * w[5] * Q4
        f[2] += pm
        f[1] += pm * w[2] - _dot(w[2:5], t)
        f[2:5] -= t
        f[5:8] = w[5:8] * w[2] - w[2:5] * w[5]
        f[5] = 0
    return f


def _sound(w):
    return torch.sqrt(GAMMA * w[1] / w[0])


def _fast(w, bn):
    c2, a2 = GAMMA * w[1] / w[0], _dot(w[5:8], w[5:8]) / w[0] * Q4
    s = c2 + a2
    return torch.sqrt(0.5 * s + torch.sqrt(torch.clamp(0.25 * s * s - bn * bn / w[0] * Q4 * c2, min=0)))


def _minmod(a, b):
    return torch.where(a * b <= 0, torch.zeros_like(a), torch.where(a.abs() < b.abs(), a, b))


def _limit(name, a, b):
    zero = torch.zeros_like(a)
    if name == "minmod":
        return _minmod(a, b)
    if name == "vanleer":
        same = a * b > 0
        return torch.where(same, 2 * a * b / torch.where(same, a + b, zero + 1), zero)
    c = (a + b).abs()
    mc = torch.where((c < 4 * a.abs()) & (c < 4 * b.abs()), torch.sign(a) * c / 2, 2 * _minmod(a, b))
    return torch.where(a * b <= 0, zero, mc)


def _physical(w):
    return torch.isfinite(w).all(0) & (w[0] > 0) & (w[1] > 0)


def _muscl(limiter, wl, wc, wr, r, dB):
    """Half-step states at the low and the high face of each cell, x frame (r = dt / dx)."""
    dw = _limit(limiter, wc - wl, wr - wc)
    lo, hi = wc - 0.5 * dw, wc + 0.5 * dw
    corr = (_xflux(hi) - _xflux(lo)) * (0.5 * r)
    if wc.shape[0] == 8:
        a = (hi[5] - lo[5]) * r
        for q in (3, 4):
            s = 0.5 * wc[q] * _minmod(dB[0], -dB[q - 2]) - 0.5 * (0.5 * (lo[q] + hi[q])) * a
            corr[q + 3] -= s
            corr[1] -= Q4 * wc[q + 3] * s
    lo, hi = _prim(_cons(lo) - corr), _prim(_cons(hi) - corr)
    ok = _physical(lo) & _physical(hi)
    return torch.where(ok, lo, wc), torch.where(ok, hi, wc)


def _roe_mean(L, R):
    l, r = torch.sqrt(L[0]), torch.sqrt(R[0])
    l, r = l / (l + r), r / (l + r)
    v = L[2:5] * l + R[2:5] * r
    h = l * (_cons(L)[1] + L[1]) / L[0] + r * (_cons(R)[1] + R[1]) / R[0]
    return l, r, v, h, torch.sqrt(GM1 * (h - _dot(v, v) / 2))


def _hll_of(L, R, sl, sr):
    fl, fr = _xflux(L), _xflux(R)
    mid = (fl * sr - fr * sl + (_cons(R) - _cons(L)) * (sl * sr)) / (sr - sl)
    return torch.where(sl >= 0, fl, torch.where(sr <= 0, fr, mid))


def _hlle(L, R):
    if L.shape[0] == 8:
        aL, aR = _fast(L, L[5]), _fast(R, R[5])
    else:
        aL, aR = _sound(L), _sound(R)
    l, r = torch.sqrt(L[0]), torch.sqrt(R[0])
    s = l + r
    v = (R[2] - L[2]) / s
    d = torch.sqrt((l / s) * aL * aL + (r / s) * aR * aR + 0.5 * l * r * v * v)
    u = (l / s) * L[2] + (r / s) * R[2]
    return _hll_of(L, R, torch.minimum(L[2] - aL, u - d), torch.maximum(R[2] + aR, u + d))


def _hllc(L, R):
    _, _, v, _, a = _roe_mean(L, R)
    sl, sr = torch.minimum(L[2] - _sound(L), v[0] - a), torch.maximum(R[2] + _sound(R), v[0] + a)
    sc = ((R[1] + R[0] * R[2] * (R[2] - sr)) - (L[1] + L[0] * L[2] * (L[2] - sl))) / (
        R[0] * (R[2] - sr) - L[0] * (L[2] - sl))
    left = sc > 0
    X, sx = torch.where(left, L, R), torch.where(left, sl, sr)
    ux = _cons(X)
    u = ux * ((sx - X[2]) / (sx - sc))
    u[2] = u[0] * sc
    u[1] += u[0] * (sc - X[2]) * (sc + X[1] / (X[0] * (sx - X[2])))
    mid = _xflux(X) + (u - ux) * sx
    return torch.where(sl >= 0, _xflux(L), torch.where(sr <= 0, _xflux(R), mid))


def _roe(L, R):
    _, _, v, h, a = _roe_mean(L, R)
    rho, zero, one = torch.sqrt(L[0] * R[0]), torch.zeros_like(a), torch.ones_like(a)
    v2 = _dot(v, v)
    lam = [v[0] - a, v[0], v[0], v[0], v[0] + a]
    K = [torch.stack([one, h - v[0] * a, v[0] - a, v[1], v[2]]), torch.stack([one, v2 / 2, v[0], v[1], v[2]]),
         torch.stack([zero, v[1], zero, one, zero]), torch.stack([zero, v[2], zero, zero, one]),
         torch.stack([one, h + v[0] * a, v[0] + a, v[1], v[2]])]
    dp, du = R[1] - L[1], R[2] - L[2]
    al = [(dp - rho * a * du) / (2 * a * a), (R[0] - L[0]) - dp / (a * a), rho * (R[3] - L[3]), rho * (R[4] - L[4]),
          (dp + rho * a * du) / (2 * a * a)]
    fl, fr = _xflux(L), _xflux(R)
    out = (fl + fr - sum(k * (c * s.abs()) for k, c, s in zip(K, al, lam))) / 2
    ul, ur = _prim(_cons(L) + K[0] * al[0]), _prim(_cons(R) - K[4] * al[4])
    l0, l1 = L[2] - _sound(L), ul[2] - _sound(ul)
    r0, r1 = R[2] + _sound(R), ur[2] + _sound(ur)
    out = torch.where((r0 > 0) & (r1 < 0), fr - K[4] * (r0 * (lam[4] - r1) / (r0 - r1) * al[4]), out)
    return torch.where((l0 < 0) & (l1 > 0), fl + K[0] * (l0 * (lam[0] - l1) / (l0 - l1) * al[0]), out)


def _exact_f(p, w):
    a, b = 2 / GP1 / w[0], GM1 / GP1 * w[1]
    return torch.where(p > w[1], (p - w[1]) * torch.sqrt(a / (b + p)),
                       2 / GM1 * _sound(w) * ((p / w[1]) ** (GM1 / (2 * GAMMA)) - 1))


def _exact_df(p, w):
    a, b = 2 / GP1 / w[0], GM1 / GP1 * w[1]
    return torch.where(p > w[1], torch.sqrt(a / (p + b)) * (1 - (p - w[1]) / (2 * (b + p))),
                       (p / w[1]) ** (-GP1 / (2 * GAMMA)) / (w[0] * _sound(w)))


def _exact_rho(p, w):
    k = GM1 / GP1
    return torch.where(p > w[1], w[0] * (p + k * w[1]) / (k * p + w[1]), w[0] * (p / w[1]) ** (1 / GAMMA))


def _exact(L, R):
    aL, aR = _sound(L), _sound(R)
    low = torch.minimum(L[1], R[1])
    two = _exact_f(low, L) + _exact_f(low, R) + R[2] - L[2] >= 0
    q = (L[1] / R[1]) ** (GM1 / (2 * GAMMA)) * aR / aL
    v2 = (q * L[2] + R[2] + 2 / GM1 * (q * aL - aR)) / (q + 1)
    p2 = L[1] * (1 - GM1 / 2 * (v2 - L[2]) / aL) ** (2 * GAMMA / GM1)
    p, live = (L[1] + R[1]) / 2, ~two
    for _ in range(6):
        d = (_exact_f(p, L) + _exact_f(p, R) + R[2] - L[2]) / (_exact_df(p, L) + _exact_df(p, R))
        d = torch.where(live, torch.minimum(d, 0.8 * p), torch.zeros_like(d))
        p = p - d
        live = live & ((d / (p + d / 2)).abs() > 1e-12)
    v = torch.where(two, v2, (L[2] + R[2] + _exact_f(p, R) - _exact_f(p, L)) / 2)
    p = torch.where(two, p2, p)
    rl = torch.where(two, L[0] * (p / L[1]) ** (1 / GAMMA), _exact_rho(p, L))
    rr = torch.where(two, R[0] * (p / R[1]) ** (1 / GAMMA), _exact_rho(p, R))
    sL, sR = torch.stack([rl, p, v, L[3], L[4]]), torch.stack([rr, p, v, R[3], R[4]])
    # the state on x / t = 0: the side the contact leaves behind, mirrored so that it is the right one
    left = v > 0
    sign = torch.where(left, -1.0, 1.0).to(v)
    W, S = torch.where(left, L, R), torch.where(left, sL, sR)
    wv, sv, a = W[2] * sign, v * sign, _sound(W)
    shock = S[1] > W[1]
    speed = torch.sqrt(GP1 / (2 * GAMMA) * S[1] / W[1] + GM1 / (2 * GAMMA)) * a
    tail = a * (S[1] / W[1]) ** (GM1 / (2 * GAMMA))
    outer = torch.where(shock, -wv > speed, -wv > a)
    fan = ~shock & ~outer & ((-sv > a) | (-sv > tail))
    f = 2 / GP1 - GM1 / GP1 * wv / a
    fw = torch.stack([W[0] * f.abs() ** (2 / GM1), W[1] * f.abs() ** (2 * GAMMA / GM1),
                      sign * (2 / GP1 * (wv * GM1 / 2 - a)), W[3], W[4]])
    w = torch.where(outer, W, torch.where(fan, fw, S))
    l, r = torch.sqrt(rl), torch.sqrt(rr)
    contact = _prim((_cons(sL) * l + _cons(sR) * r) / (l + r))
    return _xflux(torch.where(v.abs() < 1e-12, contact, w))


def _hlld(L, R):
    L, R = L.clone(), R.clone()
    L[5] = R[5] = bx = (L[5] + R[5]) / 2
    cl, cr = _fast(L, bx), _fast(R, bx)
    sl, sr = torch.minimum(L[2] - cl, R[2] - cr), torch.maximum(L[2] + cl, R[2] + cr)
    cut = torch.clamp(_dot(L[5:8], L[5:8]) + _dot(R[5:8], R[5:8]), min=1e-100)
    plain = bx * bx < 1e-12 * cut
    pl, pr = L[1] + _dot(L[5:8], L[5:8]) * Q8, R[1] + _dot(R[5:8], R[5:8]) * Q8
    xl, xr = L[0] * (sl - L[2]), R[0] * (sr - R[2])
    sm = ((xr * R[2] - xl * L[2]) - (pr - pl)) / (xr - xl)
    pt = (xr * pl - xl * pr + xl * xr * (R[2] - L[2])) / (xr - xl)
    b2, root = bx * bx * Q4, math.sqrt(4 * math.pi)

    def star(K, x, sk, pk):
        u = torch.zeros_like(K)
        u[0] = x / (sk - sm)
        den = x * (sk - sm) - b2
        flat = den.abs() < 1e-12
        den = torch.where(flat, torch.ones_like(den), den)
        bs = torch.where(flat, K[5:8], K[5:8] * (x * (sk - K[2]) - b2) / den)
        vs = torch.where(flat, K[2:5], K[2:5] - K[5:8] * bx * (sm - K[2]) / den * Q4)
        bs = torch.where(plain, K[5:8] * (sk - K[2]) / (sk - sm), bs)
        vs = torch.where(plain, K[2:5], vs)
        bs[0] = torch.where(plain, torch.zeros_like(bx), bx)
        vs[0] = sm
        u[2:5], u[5:8] = vs * u[0], bs
        work_ = bx * (_dot(K[2:5], K[5:8]) - _dot(vs, bs)) * Q4
        e = _cons(K)[1] * (sk - K[2]) + pt * sm - pk * K[2] + torch.where(plain, torch.zeros_like(bx), work_)
        u[1] = e / (sk - sm)
        f = _xflux(K) + (u - _cons(K)) * sk
        f[5] = 0
        return u, torch.cat([vs, bs]), f

    ul, wl, fl = star(L, xl, sl, pl)
    ur, wr, fr = star(R, xr, sr, pr)
    ql, qr = torch.sqrt(ul[0].abs()), torch.sqrt(ur[0].abs())
    q = ql + qr
    ssl, ssr = sm - bx.abs() / (root * ql), sm + bx.abs() / (root * qr)
    sg = torch.sign(bx) * root
    v = wl[0:3] * (ql / q) + wr[0:3] * (qr / q) + (ur[5:8] - ul[5:8]) * sg * Q4 / q
    b = ur[5:8] * (ql / q) + ul[5:8] * (qr / q) + (wr[0:3] - wl[0:3]) * sg * ql * qr / q
    v[0], b[0] = sm, bx
    pos = sm >= 0
    us, ws, fs = torch.where(pos, ul, ur), torch.where(pos, wl, wr), torch.where(pos, fl, fr)
    uu = us.clone()
    uu[2:5], uu[5:8] = v * us[0], b
    de = sg * (_dot(ws[0:3], ws[3:6]) - _dot(v, b)) * Q4 * torch.sqrt(us[0].abs())
    uu[1] = torch.where(pos, ul[1] - de, ur[1] + de)
    mid = fs + (uu - us) * torch.where(pos, ssl, ssr)
    mid = torch.where(ssl >= 0, fl, torch.where(ssr <= 0, fr, mid))
    both = (fl * ql + fr * qr) / q
    flat = torch.where(sm > 0, fl, torch.where(sm < 0, fr, both))
    mid = torch.where(plain, flat, mid)
    return torch.where(sl >= 0, _xflux(L), torch.where(sr <= 0, _xflux(R), mid))


def _face(case, low, high, ax):
    """Flux through the low face of every cell from the states on its two sides."""
    L, R = _swap(_at(low, ax, -1), ax), _swap(high, ax)
    if L.shape[0] == 8:
        if case["solver"] == "hlld":
            f = _hlld(L, R)
        else:
            L, R = L.clone(), R.clone()
            L[5] = R[5] = (L[5] + R[5]) / 2
            f = _hlle(L, R)
            f[5] = 0
    else:
        f = {"hllc": _hllc, "hlle": _hlle, "roe": _roe, "exact": _exact, "hlld": _hllc}[case["solver"]](L, R)
    return _swap(f, ax)


def _fill(w, g, n, boundary, faces=False):
    """Ghost layers, axis after axis over the padded extents (w: the last len(n) axes; faces: n + 1 points)."""
    first = w.dim() - len(n)
    for ax, na in enumerate(n):
        kind = "periodic" if boundary == "walls" and ax else boundary
        v = w.movedim(first + ax, 0)
        for k in range(1, g + 1) if kind == "periodic" or not faces else ():
            if kind == "periodic":
                v[g - k] = v[g + na - k]
                v[g + na - 1 + k] = v[g + k - 1]
            elif kind == "outflow":
                v[g - k], v[g + na - 1 + k] = v[g], v[g + na - 1]
            else:
                v[g - k], v[g + na - 1 + k] = v[g + k - 1], v[g + na - k]
                w.movedim(first + ax, 0)[g - k, 2 + ax] *= -1
                w.movedim(first + ax, 0)[g + na - 1 + k, 2 + ax] *= -1
        if faces and kind == "periodic":
            v[g + na + g] = v[g + g]
        elif faces:
            for c in range(3):
                b = w[c].movedim(ax, 0)
                if c == ax:
                    for k in range(1, g + 1):
                        b[g - k] = 2 * b[g - k + 1] - b[g - k + 2]
                        b[g + na + k] = 2 * b[g + na + k - 1] - b[g + na + k - 2]
                else:
                    for k in range(0, g + 1):
                        b[g + na + k] = b[g + na - 1]
                        b[g - k] = b[g]


def _transverse(w, f, ax, weight):
    return _prim(_cons(w) - (_at(f, ax, 1) - f) * weight)


def _hydro_step(case, w, r):
    """One unsplit step on filled ghosts: r[ax] = dt / d[ax]."""
    D = len(r)
    half = []
    for ax in range(D):
        lo, hi = _muscl(case["limiter"], _swap(_at(w, ax, -1), ax), _swap(w, ax), _swap(_at(w, ax, 1), ax), r[ax], None)
        half.append((_swap(lo, ax), _swap(hi, ax)))
    if D == 2:
        pre = [_face(case, half[ax][1], half[ax][0], ax) for ax in range(2)]
        half = [tuple(_transverse(s, pre[1 - ax], 1 - ax, 0.5 * r[1 - ax]) for s in half[ax]) for ax in range(2)]
    elif D == 3:
        pre = [_face(case, half[ax][1], half[ax][0], ax) for ax in range(3)]
        corner = {}
        for ax in range(3):
            for t in range(3):
                if t != ax:
                    lo, hi = (_transverse(s, pre[t], t, r[t] / 3) for s in half[ax])
                    corner[ax, t] = _face(case, hi, lo, ax)
        new = []
        for ax in range(3):
            t, s = [q for q in range(3) if q != ax]
            new.append(tuple(_transverse(_transverse(h, corner[t, s], t, 0.5 * r[t]), corner[s, t], s, 0.5 * r[s])
                             for h in half[ax]))
        half = new
    u = _cons(w)
    for ax in range(D):
        f = _face(case, half[ax][1], half[ax][0], ax)
        u = u + (f - _at(f, ax, 1)) * r[ax]
    return _prim(u)


def _edge_e(f, ref, D):
    """Edge electric field from the face fluxes f[ax] (field planes: B at 5..7), upwinded against the cells' ref."""

    def up(m, em, ep, rm, rp):
        mid = 0.125 * (em + ep - rm - rp)
        return torch.where(m > 1e-18, 0.25 * (em - rm), torch.where(m < -1e-18, 0.25 * (ep - rp), mid))

    E = [None] * 3
    for c in range(3):
        a, b = (c + 1) % 3, (c + 2) % 3
        if D == 2 and c < 2:
            # no z faces: the single in-plane flux gives the component
            o = 1 - c
            s = -1.0 if c == 0 else 1.0
            E[c] = s * f[o][7] + 0.25 * (2 * s * f[o][7] - ref[c] - _sh(ref[c], o, -1))
            continue
        # faces along a carry -flux of b, faces along b carry +flux of a
        ea, eb = -f[a][5 + b], f[b][5 + a]
        e = 0.25 * (_sh(eb, a, -1) + _sh(ea, b, -1) + eb + ea)
        for q, o, eq in ((a, b, eb), (b, a, ea)):
            for k in (0, -1):
                m = _sh(f[q][0], o, k)
                e = e + up(m, _sh(eq, q, -1), eq, _sh(_sh(ref[c], q, -1), o, k), _sh(ref[c], o, k))
        E[c] = e
    return E


def _faraday(B, E, h):
    D = len(h)

    def d(a, ax):
        return (_sh(a, ax, 1) - a) * h[ax] if ax < D else torch.zeros_like(a)

    return torch.stack([B[c] - (d(E[(c + 2) % 3], (c + 1) % 3) - d(E[(c + 1) % 3], (c + 2) % 3)) for c in range(3)])


def _body(w, B, D):
    """Cells with the face field averaged into them; the thermal energy is kept where the field dominates."""
    b = torch.stack([0.5 * (B[c] + _sh(B[c], c, 1)) if c < D else B[c] for c in range(3)])
    b2 = _dot(w[5:8], w[5:8])
    keep = (b2 != 0) & (8 * math.pi * w[1] / b2 <= 0.1)
    u = _cons(w)
    u[5:8] = b
    out = _prim(u)
    out[1] = torch.where(keep, w[1], out[1])
    return out


def _cell_e(w):
    v, b = w[2:5], w[5:8]
    return [b[1] * v[2] - b[2] * v[1], b[2] * v[0] - b[0] * v[2], b[0] * v[1] - b[1] * v[0]]


def _mhd_step(case, w, B, r):
    """One unsplit CTU + CT step in 2D or 3D; B has the face fields on the cells' padded extents (low faces)."""
    D = len(r)
    h = [0.5 * q for q in r]
    dB = [(_sh(B[c], c, 1) - B[c]) * r[c] if c < D else torch.zeros_like(B[0]) for c in range(3)]
    half = []
    for ax in range(D):
        order = [0, 1, 2]
        order[0], order[ax] = ax, 0
        lo, hi = _muscl(case["limiter"], _swap(_at(w, ax, -1), ax), _swap(w, ax), _swap(_at(w, ax, 1), ax), r[ax],
                        [dB[q] for q in order])
        lo, hi = _swap(lo, ax).clone(), _swap(hi, ax).clone()
        lo[5 + ax], hi[5 + ax] = B[ax], _sh(B[ax], ax, 1)
        half.append((lo, hi))
    f = [_face(case, half[ax][1], half[ax][0], ax) for ax in range(D)]
    E = _edge_e(f, _cell_e(w), D)
    Bh = _faraday(B, E, h)
    diff = [(f[ax] - _at(f[ax], ax, 1)) * r[ax] for ax in range(D)]
    wh = _body(_prim(_cons(w) + 0.5 * sum(diff)), Bh, D)
    for ax in range(D):
        corr = 0.5 * sum(diff[t] for t in range(D) if t != ax)
        corr[5:8] = 0
        for c in range(3):
            if c == ax:
                continue
            o = 3 - ax - c  # the field component c of the states along ax feels E[ax], differenced along o
            lim = _minmod(-dB[o], dB[ax]) if o < D else torch.zeros_like(B[0])
            corr[1] += Q8 * w[5 + c] * w[2 + c] * lim
            if o < D:
                e = _sh(E[ax], o, 1) - E[ax]
                e = 0.25 * (e + _sh(e, c, 1)) if c < D else 0.5 * e
                s = 1.0 if (c - ax) % 3 == 2 else -1.0
                corr[5 + c] += s * r[o] * e + 0.5 * w[2 + c] * lim
        new = []
        for k, s in enumerate(half[ax]):
            u = _cons(s) + corr
            u[5 + ax] = _sh(Bh[ax], ax, k)
            new.append(_prim(u))
        half[ax] = tuple(new)
    f = [_face(case, half[ax][1], half[ax][0], ax) for ax in range(D)]
    E = _edge_e(f, _cell_e(wh), D)
    Bn = _faraday(B, E, r)
    u = _cons(w) + sum((f[ax] - _at(f[ax], ax, 1)) * r[ax] for ax in range(D))
    return _body(_prim(u), Bn, D), Bn


def _advance(case, w0, B0, d, mhd, boundary, steps, interval, device):
    """The interior state (fields first) after `steps` CFL steps, or after `interval`; face B; the time advanced."""
    n, g, D = w0.shape[:-1], 4, len(d)
    inner = tuple(slice(g, g + k) for k in n)
    w = torch.zeros((w0.shape[-1],) + tuple(k + 2 * g for k in n), dtype=torch.float64, device=device)
    w[(slice(None),) + inner] = torch.from_numpy(np.ascontiguousarray(np.moveaxis(w0, -1, 0))).to(device)
    B = None
    if B0 is not None:
        B = torch.zeros((3,) + tuple(k + 1 + 2 * g for k in n), dtype=torch.float64, device=device)
        B[(slice(None),) + tuple(slice(g, g + k + 1) for k in n)] = torch.from_numpy(
            np.ascontiguousarray(np.moveaxis(B0, -1, 0))).to(device)
        _fill(w, g, n, boundary)
        _fill(B, g, n, boundary, faces=True)
        low = (slice(None),) + tuple(slice(0, k + 2 * g) for k in n)
        for c in range(3):
            b = B[c]
            if c < D:
                b = 0.5 * (b.narrow(c, 0, n[c] + 2 * g) + b.narrow(c, 1, n[c] + 2 * g))
            w[5 + c] = b[low[1:]]
    t = 0.0
    k = 0
    while (k < steps) if interval is None else (interval - t > 1e-14):
        _fill(w, g, n, boundary)
        x = w[(slice(None),) + inner]
        if mhd:
            b2 = x[5:8] * x[5:8]
            a = _fast(x, torch.sqrt(b2.min(0).values))
        else:
            a = _sound(x)
        speed = sum((x[2 + ax].abs() + a) / d[ax] for ax in range(D))
        dt = 0.3 / float(speed.max())
        if interval is not None:
            dt = min(dt, interval - t)
        r = [dt / q for q in d]
        if B is None:
            if mhd:
                lo, hi = _muscl(case["limiter"], _at(w, 0, -1), w, _at(w, 0, 1), r[0], [torch.zeros_like(w[0])] * 3)
                f = _face(case, hi, lo, 0)
                w = _prim(_cons(w) + (f - _at(f, 0, 1)) * r[0])
            else:
                w = _hydro_step(case, w, r)
        else:
            _fill(B, g, n, boundary, faces=True)
            cells = tuple(slice(0, q + 2 * g) for q in n)
            w, Bn = _mhd_step(case, w, B[(slice(None),) + cells].clone(), r)
            for c in range(3):
                up = tuple(slice(g, g + q + (1 if (ax == c and c < D) else 0)) for ax, q in enumerate(n))
                B[c][up] = Bn[c][up]
        t += dt
        k += 1
    faces = None if B is None else (B, g, n)
    return w[(slice(None),) + inner], faces, t


def _packed_faces(B, g, n):
    """Component, layer along x, transverse cells and one more point: the order of the packed faces."""
    return B[(slice(None),) + tuple(slice(g, g + k + 1) for k in n)].reshape(-1)


def exact(case, seed):
    device = "cuda" if torch.cuda.is_available() else "cpu"
    if case["kind"] == "batch":
        out = []
        for (w, B, d), mhd, bc in _members(case, seed):
            c = case if mhd else dict(case, solver="hllc")
            out.append(_advance(c, w, B, d, mhd, bc, case["steps"], None, device)[0])
        return {"w": out}
    w, B, d = _initial(case, seed)
    interval = 0.1 * case["steps"] / case["nx"] if case["how"] == "interval" else None
    w, faces, t = _advance(case, w, B, d, case["mhd"], case["boundary"], case["steps"], interval, device)
    out = {"w": w, "t": t}
    if faces is not None:
        # the highest layer of a component that no cell updates is a ghost: as the last fill left it
        out["B"] = _packed_faces(*faces)
    return out
