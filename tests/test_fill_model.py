"""The one-pass ghost fill on the CPU (tests/hostcheck/fill_check.cu runs the
device's own functions): for every boundary list it accepts, the values it
works out equal the passes' bit for bit whether it reads the arrays as they
were or as its own writes leave them, in either order. A launch whose threads
read what others write would differ. Lists of one and two entries of every
type and set of faces in 2D, sampled longer ones and 3D ones."""
import ctypes
import itertools
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
OUTFLOW, GATED, FIXED, REFLECTIVE, PERIODIC, IGNORE = range(6)
I = ctypes.POINTER(ctypes.c_int)


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    so = str(tmp_path_factory.mktemp("fill") / "libfill.so")
    subprocess.run([nvcc, "-std=c++17", "-O2", "-gencode", "arch=compute_100a,code=sm_100a", "-shared", "-Xcompiler",
                    "-fPIC,-ffp-contract=off", os.path.join(HERE, "hostcheck", "fill_check.cu"), "-o", so], check=True)
    f = ctypes.CDLL(so).fill_check
    f.argtypes = [ctypes.c_int, I, ctypes.c_int, ctypes.c_int, ctypes.c_int, I, I, ctypes.c_uint]

    def run(n, g, mhd, entries):
        arr = lambda v: (ctypes.c_int * len(v))(*v)
        return f(len(n), arr(list(n) + [1] * (3 - len(n))), g, int(mhd), len(entries), arr([t for t, _ in entries]),
                 arr([s for _, s in entries]), 7)
    return run


def entries(dim):
    return [(t, s) for t in range(6) for s in range(1, 4 ** dim)]


def sampled(dim, length, count, seed):
    rng = np.random.default_rng(seed)
    e = entries(dim)
    return [[e[i] for i in rng.integers(0, len(e), length)] for _ in range(count)]


@pytest.mark.parametrize("mhd", [False, True])
def test_every_pair_of_entries_2d(check, mhd):
    g = 3 if mhd else 2
    taken = 0
    for pair in itertools.chain(([e] for e in entries(2)), itertools.product(entries(2), repeat=2)):
        got = check((g + 1, g + 2), g, mhd, pair)
        assert got <= 0, (pair, got)
        taken += got == 0
    assert taken > 1000


@pytest.mark.parametrize("mhd", [False, True])
@pytest.mark.parametrize("n,length,count", [((4, 6), 4, 3000), ((4, 4, 5), 2, 400), ((5, 4, 4), 4, 200)])
def test_sampled_lists(check, n, length, count, mhd):
    for k, es in enumerate(sampled(len(n), length, count, 5)):
        got = check(n, 3 if mhd else 2, mhd, es)
        assert got <= 0, (es, got)


def test_lists_in_use_take_the_one_pass(check):
    full = 15
    for mhd in (False, True):
        g = 3 if mhd else 2
        for es in ([(OUTFLOW, full)], [(PERIODIC, full)], [(OUTFLOW, 3), (PERIODIC, 12)], [(GATED, 3), (OUTFLOW, 12)]):
            assert check((8, 9), g, mhd, es) == 0, es
