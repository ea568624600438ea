"""The exchange between the CTAs of tridiag_dsm_kernel, run on the CPU (tests/cpp/cta_emulator.h) with one
CTA lagging behind the others as far as the exchange lets it: the reduction must not depend on
how fast a CTA is, also not on one that has no column left."""
import ctypes
import os
import re
import subprocess

import numpy as np
import pytest

from test_small_solver_cpu import CSRC, HERE, PTR, _replace


def _function(text, name):
    return re.search(r"(template <[^\n]*\n)?NRG_DEV [^\n]*\b" + name + r"\(.*?\n}\n", text, flags=re.S).group(0)


@pytest.fixture(scope="module")
def reduction(tmp_path_factory):
    tmp = tmp_path_factory.mktemp("cluster_exchange")
    read = lambda f: open(os.path.join(CSRC, f)).read()  # noqa: E731
    common = _replace(read("common.cuh"), r"NRG_DEV void dmma884\(.*?\n}\n",
                      "NRG_DEV void dmma884(double& d0, double& d1, double a, double b) { emu_dmma884(d0, d1, a, b); }\n")
    common = _replace(common, r"// FP64 tensor-core MMA: D\(16x8\).*\Z", "}\n")
    large = read("eig_large.cu")
    kernel = re.search(r"constexpr int kDsmThreads.*?(?=// -+ large blocks, few of them)", large, flags=re.S).group(0)
    for name, body in (("cluster_addr", "return (smem_addr & 0xffffff) | rank << 24;"),
                       ("st_async_pair", "double* p = static_cast<double*>(emu_pointer(addr)); p[0] = x; p[1] = y; "
                                         "emu_mbar_complete(bar, 16);"),
                       ("mbar_wait_cluster", "return emu_mbar_wait(bar, parity);")):
        head = _function(kernel, name).split("{")[0]
        kernel = kernel.replace(_function(kernel, name), head + "{ " + body + " }\n")
    kernel = _replace(kernel, r"namespace cg = cooperative_groups;\s+extern __shared__ __align__\(16\) double sm\[\];\s+"
                              r"__shared__ __align__\(8\) uint64_t bars\[2\];\s+__shared__ double sc\[4\];[^\n]*",
                      "const LargeBlock& B0 = *blocks; double* sm = emu_smem();\n"
                      "uint64_t* bars = reinterpret_cast<uint64_t*>(sm + dsm_smem_doubles(B0.n, C)); "
                      "double* sc = sm + dsm_smem_doubles(B0.n, C) + 2;")
    kernel = kernel.replace("cg::this_cluster().sync()", "emu_cluster_sync()")
    inc = "NRG_DEV unsigned smem_u32(const void* p) { return emu_address(p); }\n" \
          "NRG_DEV void mbar_init(uint64_t* b, unsigned) { emu_mbar_init(b); }\nNRG_DEV void fence_mbar_init() {}\n" \
          "NRG_DEV void mbar_expect_tx(uint64_t* b, unsigned bytes) { emu_mbar_expect(b, bytes); }\n" \
          + _function(large, "block_sum_mma") + _function(large, "colsum8_mma") + kernel
    for name, text in (("cuda_runtime.h", '#include "cta_emulator.h"\n'), ("common.cuh", common),
                       ("eig_small.cuh", read("eig_small.cuh")), ("dsm_kernel.inc", inc)):
        (tmp / name).write_text(text)
    lib = tmp / "cluster_exchange.so"
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-march=native", "-U_FORTIFY_SOURCE", "-fPIC", "-shared", "-w", "-I", str(tmp),
                        "-I", os.path.join(HERE, "cpp"), os.path.join(HERE, "cpp", "cluster_exchange_cpu.cpp"), "-o",
                        str(lib)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return ctypes.CDLL(str(lib))


def reduce(lib, h, C, slow):
    n = len(h)
    ld = (n + 31) // 32 * 32
    H, W1 = np.ascontiguousarray(h), np.zeros((n, ld))
    d, e, tau = np.zeros(n), np.zeros(n), np.zeros(n)
    p = lambda a: a.ctypes.data_as(PTR)  # noqa: E731
    st = lib.reduce(n, C, slow, p(H), p(W1), ld, p(d), p(e), p(tau))
    return st, d, e, tau, W1


@pytest.mark.parametrize("n,C", [(19, 2), (34, 16)])
@pytest.mark.parametrize("kind", ["diagonal", "tridiagonal", "two parts", "last rows", "every other column"])
def test_columns_that_are_reduced_already(reduction, n, C, kind):
    h = np.triu(np.random.default_rng(n).standard_normal((n, n)))
    i, j = np.indices((n, n))
    h[{"diagonal": i != j, "tridiagonal": j > i + 1, "two parts": (i < n // 2) & (j >= n // 2),
       "last rows": (i != j) & (i < n - 5), "every other column": (i % 2 == 0) & (j > i + 1)}[kind]] = 0.0
    st, d, e, tau, W1 = reduce(reduction, h, C, -1)
    H = np.triu(h) + np.triu(h, 1).T
    Q = np.eye(n)
    for k in range(n - 3, -1, -1):
        v = np.r_[np.zeros(k + 1), W1[k, k + 1:n]]
        Q -= tau[k] * np.outer(v, v @ Q)
    T = np.diag(d) + np.diag(e[:-1], 1) + np.diag(e[:-1], -1)
    assert st == 0 and np.abs(Q @ Q.T - np.eye(n)).max() <= 1e-14
    assert np.abs(Q @ T @ Q.T - H).max() <= 1e-14 * np.abs(H).max() * n


@pytest.mark.parametrize("n,C", [(19, 2), (21, 4), (21, 8), (21, 16), (34, 16)])
def test_any_cta_may_lag(reduction, n, C):
    h = np.triu(np.random.default_rng(n).standard_normal((n, n)))
    ref = reduce(reduction, h, C, -1)
    assert ref[0] == 0
    T = np.diag(ref[1]) + np.diag(ref[2][:-1], 1) + np.diag(ref[2][:-1], -1)
    w = np.linalg.eigvalsh(np.triu(h) + np.triu(h, 1).T)
    assert np.abs(np.linalg.eigvalsh(T) - w).max() <= 1e-13 * np.abs(w).max()
    for slow in {0, C // 2, C - 1, (n - 1) % C}:
        got = reduce(reduction, h, C, slow)
        assert got[0] == 0, slow
        assert all(np.array_equal(a, b) for a, b in zip(ref[1:], got[1:])), slow
