"""The one-CTA eigensolver's device code run on the CPU (tests/cpp/cta_emulator.h), on matrices whose
small numbers leave the range in which squares can be formed: tridiagonal matrices with degenerate
pairs that are coupled by next to nothing, parts that are tiny beside the rest, matrices of low rank, blocks of denormal norm; and what it does with numbers that are
not finite."""
import ctypes
import os
import re
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "nrgljubljana_b200", "csrc")
PTR = ctypes.POINTER(ctypes.c_double)


def _replace(text, pattern, new):
    out, count = re.subn(pattern, lambda m: new, text, flags=re.S)
    assert count == 1, (count, pattern)
    return out


@pytest.fixture(scope="module")
def solver(tmp_path_factory):
    tmp = tmp_path_factory.mktemp("small_solver")
    read = lambda f: open(os.path.join(CSRC, f)).read()  # noqa: E731
    common = _replace(read("common.cuh"), r"NRG_DEV void dmma884\(.*?\n}\n",
                      "NRG_DEV void dmma884(double& d0, double& d1, double a, double b) { emu_dmma884(d0, d1, a, b); }\n")
    common = _replace(common, r"// FP64 tensor-core MMA: D\(16x8\).*\Z", "}\n")
    small = _replace(read("eig_small.cu"), r'#include "kernels.h"\n', "")
    small = _replace(small, r"extern __shared__ __align__\(16\) double sm\[\];", "double* sm = emu_smem();")
    small = _replace(small, r"template <int R, int T, int CTAS>\s+cudaError_t launch.*\Z", "}\n}\n")
    for name, text in (("cuda_runtime.h", '#include "cta_emulator.h"\n'), ("common.cuh", common),
                       ("eig_small.cuh", read("eig_small.cuh")), ("eig_small.cu", small)):
        (tmp / name).write_text(text)
    lib = tmp / "small_solver.so"
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-march=native", "-U_FORTIFY_SOURCE", "-fPIC", "-shared", "-w", "-I", str(tmp),
                        "-I", os.path.join(HERE, "cpp"), os.path.join(HERE, "cpp", "small_solver_cpu.cpp"), "-o", str(lib)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return ctypes.CDLL(str(lib))


def solve(lib, h, threads=256):
    """Status, eigenvalues and eigenvector rows of the symmetric matrix with h's upper triangle; by 64 threads up
    to order 16."""
    H = np.ascontiguousarray(np.triu(h) + np.triu(h, 1).T)
    n = len(H)
    w, v = np.full(n, np.nan), np.full((n, n), np.nan)
    st = lib.solve(n, threads, *(x.ctypes.data_as(PTR) for x in (H, w, v)), ctypes.c_double(np.nan))
    return st, w, v


def check(lib, h, unit=1.0):
    for threads in (64, 256) if len(h) <= 16 else (256,):
        w = check_with(lib, h, unit, threads)
    return w


def check_with(lib, h, unit, threads):
    """`unit`: a power of two that brings the matrix to order one. Tolerances: 2 n roundings of relative size
    2^-53 per entry of a vector, in norm."""
    st, w, v = solve(lib, h, threads)
    n = len(w)
    assert st == 0 and np.isfinite(w).all() and np.isfinite(v).all()
    H = (np.triu(h) + np.triu(h, 1).T) * unit
    w = w * unit
    ref = np.linalg.eigvalsh(H)
    nrm, tol = np.abs(ref).max(), 4 * n * 2.0 ** -52
    assert (np.diff(w) >= 0).all() and np.abs(w - ref).max() <= tol * nrm
    assert np.abs(v @ v.T - np.eye(n)).max() <= tol
    assert np.abs(v @ H - w[:, None] * v).max() <= tol * nrm
    return w


@pytest.mark.parametrize("n", [3, 9, 40, 96])
@pytest.mark.parametrize("t", [1e-150, 1e-160, 1e-163, 1e-200, 1e-300, 5e-324])
def test_degenerate_pair(solver, n, t):
    """Two states of energy zero, coupled by t: the pair's eigenvalues are -t and t."""
    h = np.diag(np.r_[1.0 / np.arange(1, n - 1), 0.0, 0.0])
    h[-2, -1] = t
    w = check(solver, h)
    assert abs(w[0] + t) <= 1e-15 * t and abs(w[1] - t) <= 1e-15 * t


@pytest.mark.parametrize("norm", [2.0 ** -1000, 2.0 ** -1022, 2.0 ** -1060, 2.0 ** 1020])
def test_norms_without_room_for_the_scale(solver, norm):
    """Norms whose reciprocal, or the power of two that scales them, is out of range."""
    for h, threads in ((h, t) for t in (64, 256) for h in (np.array([[1.0, 0.5], [0.0, 1.0]]),
                                                           np.array([[0.0, 1.0], [0.0, 0.0]]))):
        st, w, v = solve(solver, h * norm, threads)
        ref = np.linalg.eigvalsh(np.triu(h) + np.triu(h, 1).T)
        assert st == 0 and np.abs(v @ v.T - np.eye(2)).max() <= 1e-15
        assert np.abs(w / norm - ref).max() <= 1e-15 + 2 * 5e-324 / norm


@pytest.mark.parametrize("n", [4, 9, 33, 64, 67, 96])
@pytest.mark.parametrize("x", [np.nan, np.inf])
def test_not_finite_is_flagged_and_indexes_nothing(solver, n, x):
    """Poles that are not finite (planted here; the kernels check their input) end in a status, and the
    order of the poles stays a permutation: rows are looked up by it."""
    for at in (0, n // 2, n - 1):
        d, e, z = np.arange(1.0, n + 1), np.full(n, 0.1), np.empty((n, n))
        d[at] = x
        st = solver.divide_and_conquer(n, *(a.ctypes.data_as(PTR) for a in (d, e, z)), ctypes.c_double(np.nan))
        assert 0 < st <= n and not np.isnan(d).any()


@pytest.mark.parametrize("n", [12, 20, 40, 96])
@pytest.mark.parametrize("x", [1e-100, 1e-155, 1e-163, 1e-250, 1e-300])
def test_tiny_tail(solver, n, x):
    """A tridiagonal matrix of order one whose last two thirds are x: the merges there have poles and couplings of
    size x. (The reduction leaves such tails of matrices of low rank.)"""
    d, e = np.full(n, x), np.full(n, x)
    d[: n // 3], e[: n // 3] = 1.0 + np.arange(n // 3), 0.5
    h = np.diag(d) + np.diag(e[:-1], 1)
    check(solver, h)


@pytest.mark.parametrize("t", [1e-100, 1e-135, 1e-150, 1e-157, 1e-160, 1e-162, 1e-170, 1e-250, 1e-300])
@pytest.mark.parametrize("n", [3, 17, 64, 96])
def test_tiny_column(solver, n, t):
    """The first row couples to the rest by numbers whose squares underflow, wholly or in part."""
    h = np.random.default_rng(n).standard_normal((n, n))
    h[0, 1:] *= t
    check(solver, h)


@pytest.mark.parametrize("c", [1.0, 0.3, 0.7, 1 / 3, np.pi])
def test_constant(solver, c):
    """Rank one: column after column the reduction leaves 1e-16 of the last."""
    for n in range(2, 97):
        check(solver, np.full((n, n), c))


@pytest.mark.parametrize("norm", [2.0 ** -500, 2.0 ** -400, 2.0 ** 450])
def test_graded_in_small_and_large_norms(solver, norm):
    """Rows of sizes 1 to 1e-150 of the norm, as far down as the doubles go."""
    for n in (5, 40, 96):
        rng = np.random.default_rng(n)
        s = 10.0 ** rng.uniform(-75.0, 0.0, n)
        check(solver, rng.standard_normal((n, n)) * np.outer(s, s) * norm, unit=1.0 / norm)


def test_diagonal(solver):
    for n in (1, 2, 16, 17, 64, 96):
        w = check(solver, np.diag(np.round(np.random.default_rng(n).standard_normal(n), 1)))
        assert len(w) == n


def test_every_order(solver):
    """All orders, and that all threads of the CTA come to the same barriers (nodes of a level differ in
    size: of order 67, eighths are of 8 and 9 rows)."""
    for n in range(1, 97):
        check(solver, np.random.default_rng(n).standard_normal((n, n)))
