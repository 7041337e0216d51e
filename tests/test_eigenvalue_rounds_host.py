"""The shared-count eigenvalue search of the SCC kernels (scc.cu: sturm_poly, eigenvalues), compiled
for the host with one thread per CUDA thread, against LAPACK (CPU only)."""
import ctypes
import os
import re
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gfn1-rs_b200", "csrc")

SHIM = r"""
#include <algorithm>
#include <barrier>
#include <cfloat>
#include <cmath>
#include <cstring>
#include <thread>
#include <vector>
#define __device__
#define __forceinline__ inline
using std::fabs; using std::fma; using std::fmax; using std::fmin; using std::max; using std::min;
struct Idx { int x; };
static thread_local Idx threadIdx;
static std::barrier<>* g_bar;
static int g_or[3];
static thread_local int g_round;
static long long __double_as_longlong(double v) { long long r; std::memcpy(&r, &v, 8); return r; }
static double __longlong_as_double(long long v) { double r; std::memcpy(&r, &v, 8); return r; }
static int __double2hiint(double v) { return (int)(__double_as_longlong(v) >> 32); }
static double __hiloint2double(int h, int l) { return __longlong_as_double(((long long)h << 32) | (unsigned)l); }
static void __syncthreads() { g_bar->arrive_and_wait(); }
static bool __syncthreads_or(bool v) {  // three words in turn: the one after next is cleared meanwhile
  const int r = g_round++ % 3;
  if (v) __atomic_store_n(&g_or[r], 1, __ATOMIC_SEQ_CST);
  g_bar->arrive_and_wait();
  const bool any = __atomic_load_n(&g_or[r], __ATOMIC_SEQ_CST);
  __atomic_store_n(&g_or[(r + 2) % 3], 0, __ATOMIC_SEQ_CST);
  return any;
}
"""

MAIN = r"""
constexpr int NT = 64;
extern "C" void search(const double* d, const double* esq, int N, int nneed, int nwarm, double gl, double gu,
                       double pivmin, double atol, double* eps) {
  const int nall = nneed < N ? nneed + 1 : N;
  for (int base = 0; base < nall; base += NT) {
    std::barrier<> bar(NT);
    g_bar = &bar;
    g_or[0] = g_or[1] = g_or[2] = 0;
    std::vector<double> px(NT + 2), pc(NT);
    std::vector<std::thread> t;
    for (int i = 0; i < NT; ++i)
      t.emplace_back([&, i] {
        threadIdx.x = i;
        g_round = 0;
        eigenvalues<NT, true>(d, esq, N, nneed, nwarm, gl, gu, pivmin, atol, eps, px.data(), pc.data(), base);
      });
    for (auto& x : t) x.join();
  }
}
"""


@pytest.fixture(scope="module")
def search(tmp_path_factory):
    with open(os.path.join(CSRC, "scc.cu")) as fh:
        text = fh.read()
    part = text[text.index("__device__ __forceinline__ double pow2_inv_scale"):text.index("__device__ __forceinline__ double hash_unit")]
    at = re.search(r"template <int NT, bool Part = false>\n__device__ __forceinline__ void eigenvalues\(", text).start()
    part += text[at:text.index("\n}\n", at) + 3]
    part = re.sub(r"#pragma unroll[^\n]*", "", part)
    tmp = tmp_path_factory.mktemp("eig")
    src = tmp / "eig.cpp"
    src.write_text(SHIM + part + MAIN)
    so = tmp / "eig.so"
    subprocess.run(["g++", "-std=c++20", "-O2", "-ffp-contract=off", "-shared", "-fPIC", "-pthread", "-o", str(so), str(src)],
                   check=True)
    lib = ctypes.CDLL(str(so))
    P = ctypes.POINTER(ctypes.c_double)
    lib.search.argtypes = [P, P, ctypes.c_int, ctypes.c_int, ctypes.c_int] + [ctypes.c_double] * 4 + [P]

    def run(d, e, nneed, gl, gu):
        n = len(d)
        esq = np.append(e * e, 0.0)
        eps = np.zeros(n)
        norm = np.abs(d).max() + 2 * (np.abs(e).max() if n > 1 else 0.0)
        ptr = lambda a: a.ctypes.data_as(P)  # noqa: E731
        lib.search(ptr(d), ptr(esq), n, nneed, 0, gl, gu, np.finfo(float).tiny * max(1.0, esq.max()),
                   4 * np.finfo(float).eps * norm, ptr(eps))
        ref = np.linalg.eigvalsh(np.diag(d) + np.diag(e, 1) + np.diag(e, -1))
        return eps, ref, norm

    return run


@pytest.mark.parametrize("first", [False, True])
def test_search_in_parts(search, first):
    """150 eigenvalues in three parts, from no earlier iteration.  With `first` an even point of the first
    round falls on the first eigenvalue, whose thread is then done while the others go on."""
    rng = np.random.default_rng(3)
    n = 150
    d = np.sort(rng.uniform(20.0, 400.0, n))
    e = rng.uniform(-1.0, 1.0, n - 1)
    gl, gu = 0.0, 512.0
    if first:
        d[0], e[0] = gl + (gu - gl) * (0.5 / 64), 0.0
    eps, ref, norm = search(d, e, n, gl, gu)
    assert np.abs(eps - ref).max() <= 32 * np.finfo(float).eps * norm
