"""The branch-free FP64 divisions, square roots, reconstruction, solvers and
updates of the step kernels (csrc/fast64.cuh, solve64.cuh, update64.cuh) give
the plain operators' results bit for bit: on operands near every rounding
boundary that the proofs leave to a check, on random ones, and on states of
every kind the kernels can meet (ordinary, uniform, at rest, tiny, huge,
unphysical, infinite, NaN), where the fast form has to notice what it cannot
do. The tolerance is zero."""
import ctypes
import math
import os
import shutil
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))
D = ctypes.POINTER(ctypes.c_double)


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    so = str(tmp_path_factory.mktemp("fast64") / "libfast64.so")
    subprocess.run([nvcc, "-std=c++17", "-O3", "-gencode", "arch=compute_100a,code=sm_100a", "--fmad=false", "-shared",
                    "-Xcompiler", "-fPIC", os.path.join(HERE, "devcheck", "fast64_check.cu"), "-o", so], check=True)
    L = ctypes.CDLL(so)
    L.f64_arith.argtypes = [ctypes.c_int, ctypes.c_longlong, D, D, D, ctypes.POINTER(ctypes.c_int)]
    L.f64_face.argtypes = [ctypes.c_int, ctypes.c_int, ctypes.c_longlong, D, D, ctypes.c_double, D]
    L.f64_muscl.argtypes = [ctypes.c_int, ctypes.c_int, ctypes.c_longlong, D, D, D, ctypes.c_double, D]
    L.f64_cell.argtypes = [ctypes.c_int, ctypes.c_int, ctypes.c_longlong, D, D, D]
    return L


def p(a):
    return a.ctypes.data_as(D)


def same_bits(x, y):
    """Equal bits, any NaN standing for any other."""
    return (x.view(np.int64) == y.view(np.int64)) | (np.isnan(x) & np.isnan(y))


def division_boundaries():
    """(a, b) significands: b among the last 64 below 2 and every a whose
    quotient a / b lies within 8 units of 2^-53 / b of a rounding boundary."""
    out = []
    for j in range(1, 65):
        b = 2 ** 53 - j
        for s in (53, 54):
            for k in range(-8, 9):
                g = math.gcd(2 ** s, b)
                if k % g:
                    continue
                a = (k // g * pow((2 ** s // g) % (b // g), -1, b // g)) % (b // g)
                while a < 2 ** 53:
                    m, r = divmod(a * 2 ** s - k, b)
                    if a >= 2 ** 52 and r == 0 and m % 2 == 1 and 2 ** 53 <= m < 2 ** 54:
                        out.append((a, b))
                    a += b // g
    return sorted(set(out))


def root_boundaries(limit=130):
    """Radicands in [1, 4) with a 2^106 - M^2 = d, M odd with 54 bits, |d| < limit."""
    out = set()
    for d in range(-limit + 1, limit):
        if d % 8 != 7:
            continue
        for k, scale in ((54, 1.0), (55, 2.0)):
            roots = {x for x in (1, 3, 5, 7) if (x * x + d) % 8 == 0}
            for m in range(4, k + 1):
                roots = {y % 2 ** m for x in roots for y in (x, x + 2 ** (m - 1)) if (y * y + d) % 2 ** m == 0}
            for x in roots:
                for m in range(x, 2 ** 54, 2 ** k):
                    a, r = divmod(m * m + d, 2 ** k)
                    if m >= 2 ** 53 and r == 0 and 2 ** 52 <= a < 2 ** 53:
                        out.add(math.ldexp(float(a), -52) * scale)
    return sorted(out)


def test_division_and_root_bits(lib):
    rng = np.random.default_rng(3)
    pairs = division_boundaries()
    assert len(pairs) > 200 and (2 ** 52, 2 ** 53 - 1) in pairs
    a = [np.ldexp(float(x), -52 + e) for x, _ in pairs for e in (-800, -60, 0, 300)]
    b = [np.ldexp(float(y), -52 + e) for _, y in pairs for e in (-100, -7, 0, 30)]
    n = 400000
    ra = rng.uniform(1, 2, n) * np.exp2(rng.integers(-915, 845, n)) * rng.choice([-1, 1], n)
    rb = rng.uniform(1, 2, n) * np.exp2(rng.integers(-119, 49, n)) * rng.choice([-1, 1], n)
    ra[::50] = 0.0
    ra[1::50] = -0.0
    rb[2::50] = np.nextafter(np.exp2(rng.integers(-100, 40, len(rb[2::50]))), 0)
    ra[3::50] = rb[3::50]
    a, b = np.concatenate([a, ra]), np.concatenate([b, rb])
    out, flag = np.zeros((2, a.size)), np.zeros(a.size, dtype=np.int32)
    for op in (0, 1):
        assert lib.f64_arith(op, a.size, p(a), p(b), p(out), flag.ctypes.data_as(ctypes.POINTER(ctypes.c_int))) == 0
        assert not flag.any()
        assert same_bits(out[0], out[1]).all(), op
    hard = root_boundaries()
    assert len(hard) > 40
    x = np.concatenate([[np.ldexp(v, e) for v in hard for e in range(-800, 801, 50)],
                        rng.uniform(1, 4, n) * np.exp2(rng.integers(-300, 300, n) * 2), np.linspace(0.9, 1.1, 1001)])
    out, flag = np.zeros((2, x.size)), np.zeros(x.size, dtype=np.int32)
    for op in (2, 3, 4, 5, 6):
        y = np.abs(x[np.abs(np.log2(x)) < 840]) if op > 3 else x
        o, f = np.zeros((2, y.size)), np.zeros(y.size, dtype=np.int32)
        assert lib.f64_arith(op, y.size, p(y), p(y), p(o), f.ctypes.data_as(ctypes.POINTER(ctypes.c_int))) == 0
        assert not f.any()
        assert same_bits(o[0], o[1]).all(), op


def test_out_of_range_raises_the_flag(lib):
    big, small = np.exp2(900.0), np.exp2(-1000.0)
    a = np.array([1.0, big, small, np.nan, np.inf, -np.inf, 1.0, 1.0, 1.0, 5e-324])
    b = np.array([0.0, 1.0, 1.0, 1.0, 1.0, 1.0, np.nan, np.inf, 5e-324, 1.0])
    out, flag = np.zeros((2, a.size)), np.zeros(a.size, dtype=np.int32)
    for op in (0, 1):
        assert lib.f64_arith(op, a.size, p(a), p(b), p(out), flag.ctypes.data_as(ctypes.POINTER(ctypes.c_int))) == 0
        assert flag.all()
    x = np.array([-1.0, np.nan, np.inf, small * small, -0.0])
    out, flag = np.zeros((2, x.size)), np.zeros(x.size, dtype=np.int32)
    assert lib.f64_arith(2, x.size, p(x), p(x), p(out), flag.ctypes.data_as(ctypes.POINTER(ctypes.c_int))) == 0
    assert flag.all()


def states(rng, n, mhd):
    """n states: every kind in turn."""
    nf = 8 if mhd else 5
    w = np.zeros((n, nf))
    w[:, 0] = 10 ** rng.uniform(-2, 1, n)
    w[:, 1] = 10 ** rng.uniform(-2, 2, n)
    w[:, 2:5] = rng.uniform(-2, 2, (n, 3)) * rng.choice([0.0, 0.1, 1.0, 4.0], (n, 1))
    if mhd:
        w[:, 5:] = rng.uniform(-1, 1, (n, 3)) * rng.choice([0.0, 0.05, 1.0, 5.0], (n, 1))
        w[::7, 5] = 0.0
    kind = rng.integers(0, 12, n)
    for k, s in ((1, 1e-160), (2, 1e-280), (3, 3e-310), (4, 1e-70)):
        w[kind == k, 2:5] *= s
        if mhd:
            w[kind == k, 6:] *= rng.choice([1.0, s], ((kind == k).sum(), 1))
    one = kind == 5
    w[one, :2] = np.nextafter(1.0, rng.choice([0.0, 1.0, 2.0], (one.sum(), 2)))
    w[kind == 6, :2] *= 1e-40
    w[kind == 7, 1] *= -0.1
    odd = kind == 8
    w[odd, rng.integers(0, nf, odd.sum())] = rng.choice([np.nan, np.inf, -np.inf, 1e300, -1e-300, 0.0], odd.sum())
    w[kind == 9, 2:5] *= 1e3
    return w


def neighbour(rng, w):
    """A state beside w: the same, a small step away, one part in 1e12 away, or another."""
    n = len(w)
    c = rng.integers(0, 4, (n, 1))
    step = np.where(c == 1, 0.05, np.where(c == 2, 1e-12, 0.0))
    with np.errstate(over="ignore", invalid="ignore"):
        v = w * (1 + step * rng.uniform(-1, 1, w.shape))
    return np.ascontiguousarray(np.where(c == 3, states(rng, n, w.shape[1] == 8), v))


N = 60000


@pytest.mark.parametrize("mhd,solver", [(0, 1), (0, 2), (0, 4), (0, 6), (1, 3), (1, 4)])
def test_faces_bits(lib, mhd, solver):
    rng = np.random.default_rng(11 + solver)
    L = states(rng, N, bool(mhd))
    R = neighbour(rng, L)
    for dt_dx in (0.05, 0.4):
        out = np.zeros((2, N, 10))
        assert lib.f64_face(mhd, solver, N, p(L), p(R), dt_dx, p(out)) == 0
        # an unphysical hydro face (no flux found) has no flux to compare
        ok = same_bits(out[0], out[1]) | ((out[0, :, 8:9] == 0) & (out[1, :, 8:9] == 0))
        assert ok.all(), (L[~ok.all(1)][:3], R[~ok.all(1)][:3], out[:, ~ok.all(1)][:, :3])


def test_exact_solver_faces(lib):
    """The exact solver's Newton derivative takes one power where the plain form
    takes two, so its star pressure may differ in the last places: a flux to
    1e-13 of its largest component (the solve stops at a relative change of
    1e-12, after which the quadratic convergence leaves rounding error), and the
    same fallback decisions, on pairs of physical states a step apart."""
    rng = np.random.default_rng(2)
    L = states(rng, N, False)
    R = neighbour(rng, L)
    good = np.isfinite(L).all(1) & np.isfinite(R).all(1) & (L[:, :2] > 1e-3).all(1) & (R[:, :2] > 1e-3).all(1)
    good &= (np.abs(L[:, 2:]) < 10).all(1) & (np.abs(R[:, 2:]) < 10).all(1)
    L, R = np.ascontiguousarray(L[good]), np.ascontiguousarray(R[good])
    n = len(L)
    assert n > N // 3
    out = np.zeros((2, n, 10))
    assert lib.f64_face(0, 0, n, p(L), p(R), 0.05, p(out)) == 0
    done = (out[0, :, 8] == 1) & (out[1, :, 8] == 1)
    assert (out[0, :, 8:] == out[1, :, 8:]).all()
    scale = np.abs(out[1, done, :8]).max(1, keepdims=True)
    # six iterations cap the reference's Newton: a solve the cap ended is as far on either side
    err = np.abs(out[0, done, :8] - out[1, done, :8]) / scale
    assert np.quantile(err.max(1), 0.99) < 1e-13
    assert err.max() < 1e-9


@pytest.mark.parametrize("mhd", [0, 1])
@pytest.mark.parametrize("limiter", range(5))
def test_half_states_bits(lib, mhd, limiter):
    rng = np.random.default_rng(23 + limiter)
    C = states(rng, N, bool(mhd))
    L, R = neighbour(rng, C), neighbour(rng, C)
    out = np.zeros((2, N, 17))
    assert lib.f64_muscl(mhd, limiter, N, p(L), p(C), p(R), 0.2, p(out)) == 0
    ok = same_bits(out[0], out[1]).all(1)
    assert ok.all(), (L[~ok][:2], C[~ok][:2], R[~ok][:2], out[:, ~ok][:, :2])


@pytest.mark.parametrize("mhd", [0, 1])
@pytest.mark.parametrize("cfl", [0, 1, 2])
def test_cells_bits(lib, mhd, cfl):
    rng = np.random.default_rng(5)
    W = states(rng, N, bool(mhd))
    with np.errstate(over="ignore", invalid="ignore"):
        dU = np.ascontiguousarray(states(rng, N, bool(mhd)) * rng.choice([0.0, 1e-3, 0.1, 1e-20], (N, 1)))
    out = np.zeros((2, N, 18))
    assert lib.f64_cell(mhd, cfl, N, p(W), p(dU), p(out)) == 0
    ok = same_bits(out[0], out[1]).all(1)
    assert ok.all(), (W[~ok][:2], dU[~ok][:2], out[:, ~ok][:, :2])
