"""Eigenvectors of the tridiagonal by a twisted factorisation and one step of inverse iteration with its
factors (scc.cu: twisted_vector), compiled for the host with two threads a column, against the
orthogonality that two pivoted inverse iterations reach (CPU only)."""
import ctypes
import os
import re
import subprocess

import numpy as np
import pytest
from scipy.linalg import hessenberg

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gfn1-rs_b200", "csrc")
EPS = np.finfo(float).eps

SHIM = r"""
#include <algorithm>
#include <barrier>
#include <cmath>
#include <thread>
#define __device__
#define __forceinline__ inline
#define __restrict__
using std::fabs; using std::fma; using std::max; using std::min;
static thread_local std::barrier<>* t_bar;
static void __syncthreads() { t_bar->arrive_and_wait(); }
"""

MAIN = r"""
extern "C" void vectors(const double* d, const double* e, int n, int nv, const double* lam, double norm, double* work,
                        double* Z, double* scale) {
  for (int j = 0; j < nv; ++j) {
    std::barrier<> bar(2);
    double pa = 0, pb = 0, pc = 0;
    auto run = [&](bool top) {
      t_bar = &bar;
      const long long n2 = (long long)n * nv;
      const double s = twisted_vector<8>(d, e, n, lam[j], 2.220446049250313e-16 * norm, 64 * 2.220446049250313e-16 * norm,
                                         true, top, work + j, n2, Z + j, nv, &pa, &pb, &pc);
      if (top) scale[j] = s;
    };
    std::thread t([&] { run(false); });
    run(true);
    t.join();
  }
}
"""


@pytest.fixture(scope="module")
def vectors(tmp_path_factory):
    with open(os.path.join(CSRC, "scc.cu")) as fh:
        text = fh.read()
    at = text.index("template <int U>\n__device__ __forceinline__ double twisted_vector(")
    part = re.sub(r"#pragma unroll[^\n]*", "", text[at:text.index("\n}\n", at) + 3])
    tmp = tmp_path_factory.mktemp("twist")
    src, so = tmp / "twist.cpp", tmp / "twist.so"
    src.write_text(SHIM + part + MAIN)
    subprocess.run(["g++", "-std=c++20", "-O2", "-shared", "-fPIC", "-pthread", "-o", str(so), str(src)], check=True)
    lib = ctypes.CDLL(str(so))
    P = ctypes.POINTER(ctypes.c_double)
    lib.vectors.argtypes = [P, P, ctypes.c_int, ctypes.c_int, P, ctypes.c_double, P, P, P]

    def run(d, e, lam):
        n, nv = len(d), len(lam)
        Z, work, scale = np.zeros((n, nv)), np.zeros(5 * n * nv), np.zeros(nv)
        norm = np.abs(d).max() + 2 * (np.abs(e).max() if n > 1 else 0.0)
        ptr = lambda a: a.ctypes.data_as(P)  # noqa: E731
        e = np.append(e, 0.0)
        lib.vectors(ptr(d), ptr(e), n, nv, ptr(lam), norm, ptr(work), ptr(Z), ptr(scale))
        return Z * scale, scale, norm

    return run


def tridiagonal(n, gap, rng):
    """A reduced dense matrix with the spectrum of an occupied block: pairs of levels `gap` apart."""
    w = np.sort(rng.uniform(-1.0, 1.0, n // 2))
    w = np.sort(np.concatenate([w, w + gap, np.zeros(n % 2) + 1.1]))
    q, _ = np.linalg.qr(rng.normal(size=(n, n)))
    h = hessenberg((q * w) @ q.T)
    return np.diag(h).copy(), 0.5 * (np.diag(h, 1) + np.diag(h, -1))


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 8, 9, 33, 64, 128, 257])
def test_vectors_are_orthogonal(vectors, n):
    """Eigenvalues off by 3 eps |T|.  Two vectors of eigenvalues `gap` apart overlap by the square of
    (error of lam) / gap times the ratio of their entries in the twist row, and by the rounding of the
    factors, eps |T| / gap over many rows with random signs: eps |T| / gap + 1e3 (3 eps |T| / gap)^2 (one
    solve leaves the first power of the error, 3 eps |T| / gap and more)."""
    rng = np.random.default_rng(n)
    for gap in (1e-2, 1e-4):
        d, e = tridiagonal(n, gap, rng) if n > 1 else (np.array([0.3]), np.zeros(0))
        ref = np.linalg.eigvalsh(np.diag(d) + np.diag(e, 1) + np.diag(e, -1))
        norm = np.abs(d).max() + 2 * (np.abs(e).max() if n > 1 else 0.0)
        lam = ref + 3 * EPS * norm * rng.choice([-1.0, 1.0], n)
        far = np.diff(ref).min() if n > 1 else 1.0
        Z, scale, _ = vectors(d, e, lam)
        assert (scale > 0).all()
        T = np.diag(d) + np.diag(e, 1) + np.diag(e, -1)
        overlap = np.abs(Z.T @ Z - np.eye(n)).max()
        residual = np.abs(T @ Z - Z * ref).max()
        far = min(far, gap)
        assert overlap <= EPS * norm / far + 1e3 * (3 * EPS * norm / far) ** 2
        assert residual <= 16 * EPS * norm
