"""The forms of the branch-free routines that test_gpu_fast64.py does not call:
small numerators divided on the spot (the 3D hydro step), one and three axes,
the exact solver's counters, and states in other units. Bit for bit against the
plain operators but for the exact solver, whose Newton derivative takes one
power where the plain form takes two."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

from test_gpu_fast64 import D, N, division_boundaries, neighbour, p, same_bits, states

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))
EXACT, HLL, HLLC, HLLD, HLLE, ROE = 0, 1, 2, 3, 4, 6
# density, velocity and cell width of a problem, in cgs
UNITS = {
    "order one": (1.0, 1.0, 0.01),
    "interstellar gas": (2e-24, 1e6, 3e18),
    "cluster gas at 1e8 K": (1e-26, 1.5e8, 3e21),
    "cosmological": (1e-30, 3e7, 3e24),
    "stellar interior": (150.0, 6e7, 1e8),
    "white dwarf": (1e7, 5e8, 1e5),
}
MHD_UNITS = {"order one": (1.0, 1.0, 0.01), "interstellar gas": (2e-24, 1e5, 3e18), "photosphere": (3e-7, 8e5, 1e7),
             "stellar interior": (150.0, 6e7, 1e8), "neutron star crust": (1e11, 3e9, 1e4)}


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    so = str(tmp_path_factory.mktemp("forms") / "libforms.so")
    subprocess.run([nvcc, "-std=c++17", "-O3", "-gencode", "arch=compute_100a,code=sm_100a", "--fmad=false", "-shared",
                    "-Xcompiler", "-fPIC", os.path.join(HERE, "devcheck", "fast64_forms.cu"), "-o", so], check=True)
    L = ctypes.CDLL(so)
    i, n, d = ctypes.c_int, ctypes.c_longlong, ctypes.c_double
    L.forms_arith.argtypes = [i, n, D, D, D, ctypes.POINTER(i)]
    L.forms_face.argtypes = [i, i, n, D, D, d, D]
    L.forms_mhd_face.argtypes = [i, n, D, D, d, D]
    L.forms_muscl.argtypes = [i, i, n, D, D, D, d, D]
    L.forms_cell.argtypes = [i, i, i, n, D, D, D]
    L.forms_flags.argtypes = [i, i, i, n, D, D, D, d, d, ctypes.POINTER(i)]
    return L


def in_units(w, rho, v):
    """States of order one with their density, velocity (and field) units changed."""
    s = np.ones(w.shape[1])
    s[:5] = rho, rho * v * v, v, v, v
    s[5:] = np.sqrt(rho) * v
    with np.errstate(over="ignore", under="ignore", invalid="ignore"):
        return np.ascontiguousarray(w * s)


def calm(rng, n, mhd):
    """Ordinary subsonic states and neighbours a few per cent away."""
    w = np.empty((n, 8 if mhd else 5))
    w[:, :2] = rng.uniform(0.7, 1.4, (n, 2))
    w[:, 2:5] = rng.uniform(-0.4, 0.4, (n, 3))
    w[:, 5:] = rng.uniform(-1, 1, (n, w.shape[1] - 5))
    near = lambda: np.ascontiguousarray(w * (1 + rng.uniform(-0.03, 0.03, w.shape)) + 1e-3 * rng.uniform(-1, 1, w.shape))
    return near(), w, near()


@pytest.mark.parametrize("units", ["order one", "cluster gas at 1e8 K", "white dwarf"])
@pytest.mark.parametrize("solver", [HLL, HLLC, HLLE, ROE])
@pytest.mark.parametrize("local", [0, 1])
def test_faces(lib, local, solver, units):
    rng = np.random.default_rng(31 + solver)
    w = states(rng, N, False)
    rho, v, _ = UNITS[units]
    L, R = in_units(w, rho, v), in_units(neighbour(rng, w), rho, v)
    out = np.zeros((2, N, 14))
    assert lib.forms_face(solver, local, N, p(L), p(R), 0.2 / v, p(out)) == 0
    # an unphysical face (no flux found) has no flux to compare
    ok = same_bits(out[0], out[1]) | ((out[0, :, 8:9] == 0) & (out[1, :, 8:9] == 0))
    assert ok.all(), (L[~ok.all(1)][:3], R[~ok.all(1)][:3], out[:, ~ok.all(1)][:, :3])


@pytest.mark.parametrize("local", [0, 1])
def test_exact_solver_counters(lib, local):
    """Counters as the plain solve's: a differing count needs a change within
    rounding (1e-16 / 1e-12 of it) of the tolerance, fewer than one solve in
    1000. Fluxes of solves that the cap did not end: the last step left less
    than the tolerance squared, so rounding of a few operations, 1e-13."""
    rng = np.random.default_rng(2)
    L = states(rng, 4 * N, False)
    R = neighbour(rng, L)
    good = np.isfinite(L).all(1) & np.isfinite(R).all(1) & (L[:, :2] > 1e-3).all(1) & (R[:, :2] > 1e-3).all(1)
    good &= (np.abs(L[:, 2:]) < 10).all(1) & (np.abs(R[:, 2:]) < 10).all(1)
    L, R = np.ascontiguousarray(L[good]), np.ascontiguousarray(R[good])
    n = len(L)
    out = np.zeros((2, n, 14))
    assert lib.forms_face(EXACT, local, n, p(L), p(R), 0.05, p(out)) == 0
    same = (out[0, :, 8:] == out[1, :, 8:]).all(1)
    assert (~same).sum() <= n // 1000, (~same).sum()
    assert (out[0, :, 11:13] == out[1, :, 11:13]).all()
    done = same & (out[1, :, 8] == 1) & (out[1, :, 13] == 0)
    scale = np.abs(out[1, done, :8]).max(1, keepdims=True)
    assert (np.abs(out[0, done, :8] - out[1, done, :8]) / scale).max() < 1e-13


@pytest.mark.parametrize("units", list(MHD_UNITS))
@pytest.mark.parametrize("solver", [HLLD, HLLE])
def test_mhd_faces(lib, solver, units):
    rng = np.random.default_rng(41 + solver)
    w = states(rng, N, True)
    rho, v, _ = MHD_UNITS[units]
    L, R = in_units(w, rho, v), in_units(neighbour(rng, w), rho, v)
    out = np.zeros((2, N, 14))
    assert lib.forms_mhd_face(solver, N, p(L), p(R), 0.2 / v, p(out)) == 0
    ok = same_bits(out[0], out[1]).all(1)
    assert ok.all(), (L[~ok][:3], R[~ok][:3], out[:, ~ok][:, :3])


@pytest.mark.parametrize("units", ["order one", "cluster gas at 1e8 K"])
@pytest.mark.parametrize("limiter", range(5))
@pytest.mark.parametrize("local", [0, 1])
def test_half_states(lib, local, limiter, units):
    rng = np.random.default_rng(23 + limiter)
    w = states(rng, N, False)
    rho, v, _ = UNITS[units]
    L, C, R = (in_units(a, rho, v) for a in (neighbour(rng, w), w, neighbour(rng, w)))
    out = np.zeros((2, N, 17))
    assert lib.forms_muscl(local, limiter, N, p(L), p(C), p(R), 0.2 / v, p(out)) == 0
    ok = same_bits(out[0], out[1]).all(1)
    assert ok.all(), (L[~ok][:2], C[~ok][:2], R[~ok][:2], out[:, ~ok][:, :2])


@pytest.mark.parametrize("mhd,nd", [(0, 1), (0, 3), (1, 1), (1, 3)])
@pytest.mark.parametrize("cfl", [0, 1, 3])
def test_cells(lib, mhd, nd, cfl):
    rng = np.random.default_rng(5)
    W = states(rng, N, bool(mhd))
    with np.errstate(over="ignore", invalid="ignore"):
        dU = np.ascontiguousarray(states(rng, N, bool(mhd)) * rng.choice([0.0, 1e-3, 0.1, 1e-20], (N, 1)))
    out = np.zeros((2, N, 18))
    assert lib.forms_cell(mhd, nd, cfl, N, p(W), p(dU), p(out)) == 0
    ok = same_bits(out[0], out[1]).all(1)
    assert ok.all(), (W[~ok][:2], dU[~ok][:2], out[:, ~ok][:, :2])


@pytest.mark.parametrize("mhd,solver,limiter,units",
                         [(0, s, k, u) for s in (EXACT, HLL, HLLC, HLLE, ROE) for k, u in ((2, n) for n in UNITS)] +
                         [(0, HLLC, 4, u) for u in UNITS] + [(1, s, 2, u) for s in (HLLD, HLLE) for u in MHD_UNITS])
def test_ordinary_states_raise_no_flag_in_other_units(lib, mhd, solver, limiter, units):
    """A raised flag repeats the work with the plain operators, up to three times."""
    rho, v, dx = (MHD_UNITS if mhd else UNITS)[units]
    L, C, R = (in_units(a, rho, v) for a in calm(np.random.default_rng(9), N, bool(mhd)))
    out = np.zeros(N, dtype=np.int32)
    assert lib.forms_flags(mhd, solver, limiter, N, p(L), p(C), p(R), 0.2 / v, dx,
                           out.ctypes.data_as(ctypes.POINTER(ctypes.c_int))) == 0
    assert (out & 6 == 0).all() and (out & 1).mean() < 1e-3, np.bincount(out & 7)


@pytest.mark.parametrize("op,top,floor", [(0, 400, -970), (1, 102, -1022), (2, 120, -1020), (3, 400, -950)])
def test_large_divisors(lib, op, top, floor):
    """Operands near rounding boundaries and random ones, up to the largest
    divisor and down to the smallest quotient: the plain quotient or a flag, and
    no flag inside the range."""
    rng = np.random.default_rng(17)
    lowest = -920 if op < 2 else -900  # of a numerator
    pairs = np.array(division_boundaries(), dtype=np.float64) * 2.0 ** -52
    a, b = [], []
    for eb in [48, 51, 75, 100, top - 1]:
        for eq in (-60, 0, 200, floor + 2, floor + 40):
            if lowest + 1 <= eb + eq < 820:
                a.append(np.ldexp(pairs[:, 0], eb + eq))
                b.append(np.ldexp(pairs[:, 1], eb))
    n = 300000
    eb = rng.integers(40, top, n)
    ea = np.maximum(eb + rng.integers(floor + 2, floor + 300, n), lowest + 1)
    a, b = np.concatenate(a + [np.ldexp(rng.uniform(1, 2, n), ea)]), np.concatenate(b + [np.ldexp(rng.uniform(1, 2, n), eb)])
    if op < 2:
        a *= rng.choice([-1, 1], a.size)
    inside = a.size
    ea = rng.integers(-1060, -600, n)  # across the floors
    a, b = np.concatenate([a, np.ldexp(rng.uniform(1, 2, n), ea)]), np.concatenate([b, np.ldexp(rng.uniform(1, 2, n), eb)])
    out, flag = np.zeros((2, a.size)), np.zeros(a.size, dtype=np.int32)
    assert lib.forms_arith(op, a.size, p(a), p(b), p(out), flag.ctypes.data_as(ctypes.POINTER(ctypes.c_int))) == 0
    assert not flag[:inside].any()
    assert (same_bits(out[0], out[1]) | (flag == 1)).all()
    assert flag[inside:].any()
