// Persistent SCC kernel: each CTA pulls molecules from a work queue (most
// expensive first) and runs the complete self-consistent-charge loop of
// gfn1-rs `run_scc_with_core` (src/electronic.rs:849-2054, plain charge-vector
// branch, ladder rung 0) on the device.  Three instantiations run side by side,
// each with the molecules whose matrix its CTA keeps on chip for the Householder
// reduction (kSccKinds in common.cuh): up to 64 AOs on 128-thread CTAs, four per
// SM; up to 128 on 256 threads, two per SM; up to 192 on 256 threads, one per SM
// (more CTAs per SM hide barriers and latencies better, but a reduction that
// fetches its matrix from L1 per column costs more: 128-thread CTAs, four per SM
// at every size, took 60.5 ms for the SCC of the 4096-molecule batch, these
// 42.4).  A batch with few small molecules runs them on 256 threads.  Shared
// memory holds the molecule's state, the index tables, the N-vectors and the
// scratch of the reduction and of the back-transformation; the matrices live in
// the CTA's global workspace slot.  The stages are functions of their own that
// read the molecule's state from shared memory, so that each has the whole
// register budget.
//
// Algorithmic choices that differ from the reference but give the same results
// up to FP64 rounding:
//  * orthogonaliser: Cholesky S = L L^T instead of Lowdin S^-1/2
//    (src/linalg.rs:193-217).  The density P = C f C^T is invariant to the choice.
//    H0' = L^-1 H0 L^-T is formed once per molecule, and each iteration only adds
//    the potential term  -1/2 (M + M^T),  M = L^-1 diag(v) L  (lower triangular),
//    because  L^-1 (S o V) L^-T = L^-1 diag(v) L + (L^-1 diag(v) L)^T  for
//    V_mu,nu = v_mu + v_nu (src/electronic.rs:3133-3158).
//  * eigensolver: Householder tridiagonalisation with the matrix on chip
//    (tridiag.cuh), Sturm counts shared by the CTA plus Laguerre steps,
//    warm-started from the previous iteration, for the eigenvalues the
//    occupations need, twisted factorisations (inverse iteration with modified
//    Gram-Schmidt inside eigenvalue clusters) for the occupied eigenvectors only,
//    and a compact-WY back-transformation with the orbitals in registers
//    (orbitals.cuh; replaces faer's self_adjoint_eigen, src/linalg.rs:153-191).
//  * electronic energy: tr(H0 P) = sum_i f_i eps_i + sum_mu v_mu (S P)_mu,mu,
//    which holds exactly for the F that was diagonalised, so P is only formed once
//    the SCC has converged (src/electronic.rs:3182-3188, :2173-2191).
//  * Mulliken populations (S P)_mu,mu = sum_i f_i (L z_i)_mu (L^-T z_i)_mu
//    (src/electronic.rs:3160-3180).
// Fermi smearing (bisection to the bracket fixed point, :3853-3921), the
// convergence test (:1881), Broyden mixing (:3203-3309, :3759-3806) and the final
// energy assembly (:1957-2053) follow the reference step by step.
#include <float.h>

#include "common.cuh"
#include "model.cuh"
#include "orbitals.cuh"
#include "tridiag.cuh"
#include "tridiag_cluster.cuh"
#include "tridiag_grid.cuh"

namespace gfn1 {

constexpr double kBoltzmann = 3.1668115634556e-6;  // src/constants.rs:26
constexpr int kVecSlots = 8;  // N-length vectors kept in shared memory

struct SccShared {
  double red[32];
  double scal[16];
  int iscal[16];
  double Ld[8][9];      // Cholesky: diagonal block and reciprocal pivots
  int first[2][16];     // occupations: each warp's first trial level that holds the electrons
};

// Per-stage clock accounting by thread 0 of the CTA (no-op without a buffer).
struct StageClock {
  unsigned long long* out;
  long long t0;
  __device__ explicit StageClock(unsigned long long* o) {
    out = o;
    t0 = clock64();
  }
  __device__ __forceinline__ void mark(int stage) {
    if (!out) return;
    __syncthreads();
    if (threadIdx.x == 0) {
      const long long t = clock64();
      atomicAdd(out + stage, (unsigned long long)(t - t0));
      t0 = t;
    } else {
      t0 = clock64();
    }
  }
};

// Layout of one CTA's global workspace slot (doubles).
struct CtaWs {
  double *L, *LiT, *Hp, *F, *Z, *Ct, *V, *iw, *popw;
  double *df, *u, *dots, *omega, *beta, *cvec, *qin, *qout, *vsh, *qlast, *dqlast, *qnext, *vout, *qat;
};
// Leading dimension of the matrices: whole 8 x 8 tiles.
__host__ __device__ inline int work_ld(int n) { return (n + 7) & ~7; }
// Reflectors of the register-resident reduction: rows padded to 32 columns, and
// room for zero rows up to a multiple of 16.
__host__ __device__ inline int refl_ld(int n) { return (n + 31) & ~31; }
__host__ __device__ inline long long refl_size(int n) { return (long long)(n + 16) * refl_ld(n); }
constexpr int kMaxSccWarps = 8;

// Slot sizes in doubles; every matrix starts on a 32-byte boundary.
__host__ __device__ inline long long cta_ws_size(int maxn, int maxnsh, int cap, int maxnat) {
  const long long n2 = (long long)work_ld(maxn) * work_ld(maxn);
  const long long t = 11 * n2 + refl_size(maxn) + (long long)kMaxSccWarps * work_ld(maxn) + 2LL * cap * maxnsh +
                      2LL * cap * cap + 2LL * cap + 8LL * maxnsh + maxnat + 64;
  return (t + 3) & ~3LL;
}
__device__ __forceinline__ CtaWs cta_ws(double* base, int maxn, int maxnsh, int cap) {
  CtaWs w;
  const long long n2 = (long long)work_ld(maxn) * work_ld(maxn);
  w.L = base;
  w.LiT = w.L + n2;
  w.Hp = w.LiT + n2;
  w.F = w.Hp + n2;
  w.Z = w.F + n2;
  w.Ct = w.Z + n2;
  w.iw = w.Ct + n2;  // 5 * n2
  w.V = w.iw + 5 * n2;
  w.popw = w.V + refl_size(maxn);
  w.df = w.popw + (long long)kMaxSccWarps * work_ld(maxn);
  w.u = w.df + (long long)cap * maxnsh;
  w.dots = w.u + (long long)cap * maxnsh;
  w.beta = w.dots + (long long)cap * cap;
  w.omega = w.beta + (long long)cap * cap;
  w.cvec = w.omega + cap;
  w.qin = w.cvec + cap;
  w.qout = w.qin + maxnsh;
  w.vsh = w.qout + maxnsh;
  w.qlast = w.vsh + maxnsh;
  w.dqlast = w.qlast + maxnsh;
  w.qnext = w.dqlast + maxnsh;
  w.vout = w.qnext + maxnsh;
  w.qat = w.vout + maxnsh;
  return w;
}

__host__ __device__ inline int scc_ints(int maxnsh, int maxn, int maxnat) {
  return 3 * maxnsh + maxn + maxnat + 1;
}
// Byte offset of the N-vectors in the SCC kernel's dynamic shared memory: after
// the CTA's state and the index tables.
struct SccCta;
__host__ __device__ constexpr size_t scc_cta_bytes();
__host__ __device__ inline size_t scc_vec_bytes(int maxnsh, int maxn, int maxnat) {
  return (scc_cta_bytes() + (size_t)4 * scc_ints(maxnsh, maxn, maxnat) + 15) & ~(size_t)15;
}
__host__ __device__ inline size_t scc_smem_fixed(int maxnsh, int maxn, int maxnat) {
  const size_t ib = scc_vec_bytes(maxnsh, maxn, maxnat);
  return ib + sizeof(double) * ((kVecSlots * (size_t)maxn + 1) & ~(size_t)1);
}

// Sturm count and characteristic polynomial at x for the symmetric tridiagonal
// (d, esq = e^2): returns #eigenvalues <= x and the values p, p', p'' of
// p_n(x) = det(T - x I) up to one common positive factor.  The recurrence
//   p_i = (d_i - x) p_{i-1} - e_{i-1}^2 p_{i-2}
// is LAPACK dlaebz's ratio recurrence q_i = p_i / p_{i-1} multiplied through by
// p_{i-1}, so the count (the number of negative q_i) is the same but the loop
// needs no division.  The pair (p_i, p_{i-1}) and its derivatives are rescaled
// by an exact power of two every 8 steps.  The pivot guard |q_i| < pivmin sets
// q_i = -2^-600 (LAPACK: -pivmin; the two differ only when e_i^2 < 2^-600 |d_i -
// x|, an exact split) and moves the pair to a scale where |p_i| is near 1.  The
// derivatives may overflow; they only steer the Laguerre step.
__device__ __forceinline__ double pow2_inv_scale(double m) {  // 2^-floor(log2 m), clamped to 2^+-1000
  const long long ex = ((__double_as_longlong(m) >> 52) & 0x7ff) - 1023;
  const long long sc = 1023 - (ex < -1000 ? -1000 : (ex > 1000 ? 1000 : ex));
  return __longlong_as_double(sc << 52);
}
struct SturmState {
  double p, pm, dp, dpm, ddp, ddpm;
  int c;
};
// One step with the pivot guard.
__device__ __forceinline__ void sturm_step(SturmState& s, double t, double e2, double pivmin) {
  constexpr double kGuardScale = 0x1p600;
  double pn = fma(t, s.p, -(e2 * s.pm));
  double dpn = fma(t, s.dp, fma(-e2, s.dpm, -s.p));
  double ddpn = fma(t, s.ddp, fma(-e2, s.ddpm, -2.0 * s.dp));
  if (fabs(pn) <= pivmin * fabs(s.p)) {
    const double sc = pow2_inv_scale(fabs(s.p)) * kGuardScale;
    pn = s.p * -pow2_inv_scale(fabs(s.p));
    s.p = pn * -kGuardScale;
    s.dp *= sc;
    dpn *= sc;
    s.ddp *= sc;
    ddpn *= sc;
  }
  s.c += (pn > 0.0) != (s.p > 0.0);
  s.pm = s.p;
  s.p = pn;
  s.dpm = s.dp;
  s.dp = dpn;
  s.ddpm = s.ddp;
  s.ddp = ddpn;
}
__device__ __forceinline__ int exp_bits(double x) { return __double2hiint(x) & 0x7ff00000; }
// G steps and a rescale.  The guard's test and branch after every step would
// take most of the time (96 cycles a step, where a multiply-add's latency is 8).
// The pair (p, pm) starts a group at a scale near 1 and the guard needs
// |pn| <= pivmin |p| ~ 2^-1022, so a group whose values all stay above 2^-700 has
// none; otherwise the group is done step by step.
template <int G>
__device__ __forceinline__ void sturm_group(SturmState& s, const double (&t)[8], const double (&e2)[8], double pivmin) {
  double a = s.p, b = s.pm, da = s.dp, db = s.dpm, va = s.ddp, vb = s.ddpm;
  int low = 0x7ff00000, c = 0;
#pragma unroll
  for (int i = 0; i < G; ++i) {
    const double q = fma(t[i], a, -(e2[i] * b));
    const double u = fma(t[i], da, fma(-e2[i], db, -a));
    const double v = fma(t[i], va, fma(-e2[i], vb, -2.0 * da));
    c += (unsigned)(__double2hiint(q) ^ __double2hiint(a)) >> 31;
    low = min(low, exp_bits(q));
    b = a;
    a = q;
    db = da;
    da = u;
    vb = va;
    va = v;
  }
  if (low >= (1023 - 700) << 20) {
    s.p = a;
    s.pm = b;
    s.dp = da;
    s.dpm = db;
    s.ddp = va;
    s.ddpm = vb;
    s.c += c;
  } else {
#pragma unroll 1
    for (int i = 0; i < G; ++i) {
      double ti = t[0], ei = e2[0];
#pragma unroll
      for (int j = 1; j < G; ++j)
        if (j == i) {
          ti = t[j];
          ei = e2[j];
        }
      sturm_step(s, ti, ei, pivmin);
    }
  }
  // exact power of two; (p, pm) is never zero
  const int ex = max(exp_bits(s.p), exp_bits(s.pm));
  const double sc = __hiloint2double(min(max(0x7fe00000 - ex, 23 << 20), 2023 << 20), 0);
  s.p *= sc;
  s.pm *= sc;
  s.dp *= sc;
  s.dpm *= sc;
  s.ddp *= sc;
  s.ddpm *= sc;
}
__device__ __forceinline__ int sturm_poly(const double* d, const double* esq, int n, double x, double pivmin,
                                          double& pout, double& dpout, double& ddpout) {
  SturmState s{d[0] - x, 1.0, -1.0, 0.0, 0.0, 0.0, 0};
  if (fabs(s.p) < pivmin) {
    constexpr double kGuardScale = 0x1p600;
    s.p = -1.0;
    s.pm = kGuardScale;
    s.dp = -kGuardScale;
  }
  s.c = s.p <= 0.0;
  double t[8], e2[8], tn[8], en[8];
  auto load = [&](int i, double (&tt)[8], double (&ee)[8]) {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int k = min(i + j, n - 1);
      tt[j] = d[k] - x;
      ee[j] = esq[max(k, 1) - 1];
    }
  };
  int i = 1;
  load(1, t, e2);
  for (; i + 7 < n; i += 8) {  // the next group's entries are fetched before this one's steps
    load(i + 8, tn, en);
    sturm_group<8>(s, t, e2, pivmin);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      t[j] = tn[j];
      e2[j] = en[j];
    }
  }
  if (i + 3 < n) {
    sturm_group<4>(s, t, e2, pivmin);
    i += 4;
    t[0] = t[4];
    t[1] = t[5];
    t[2] = t[6];
    e2[0] = e2[4];
    e2[1] = e2[5];
    e2[2] = e2[6];
  }
#pragma unroll 1
  for (; i < n; ++i) {  // at most three
    sturm_step(s, t[0], e2[0], pivmin);
    t[0] = t[1];
    e2[0] = e2[1];
    t[1] = t[2];
    e2[1] = e2[2];
  }
  pout = s.p;
  dpout = s.dp;
  ddpout = s.ddp;
  return s.c;
}

__device__ __forceinline__ double hash_unit(unsigned a, unsigned b) {
  unsigned h = a * 0x9E3779B1u ^ (b + 0x7F4A7C15u) * 0x85EBCA77u;
  h ^= h >> 15;
  h *= 0x2C1B3C6Du;
  h ^= h >> 12;
  h *= 0x297A2D39u;
  h ^= h >> 15;
  return (double)(h & 0xFFFFFF) / 16777216.0 - 0.5;
}

// Gaussian elimination with partial pivoting of the tridiagonal T - lam I.
// The five factor arrays of eigenvector column j are stored interleaved,
// w[(a * n + i) * ldw + j], so the threads of a warp access consecutive words;
// the pivots are kept as reciprocals, so the solves only multiply.
__device__ void tri_factor(const double* d, const double* e, int n, double lam, double tiny, double* w, int ldw) {
  double a = d[0] - lam;
  double c = n > 1 ? e[0] : 0.0;
  const long long s = (long long)n * ldw;
  for (int k = 0; k < n - 1; ++k) {
    const double b = e[k];
    const double an = d[k + 1] - lam;
    const double cn = (k + 1 < n - 1) ? e[k + 1] : 0.0;
    double* wk = w + (long long)k * ldw;
    if (fabs(a) >= fabs(b)) {
      double piv = a;
      if (fabs(piv) < tiny) piv = piv >= 0.0 ? tiny : -tiny;
      const double r = 1.0 / piv;
      wk[0] = r;
      wk[s] = c;
      wk[2 * s] = 0.0;
      wk[3 * s] = b * r;
      wk[4 * s] = 0.0;
      a = an - b * r * c;
      c = cn;
    } else {
      const double r = 1.0 / b;
      const double mult = a * r;
      wk[0] = r;
      wk[s] = an;
      wk[2 * s] = cn;
      wk[3 * s] = mult;
      wk[4 * s] = 1.0;
      a = c - mult * an;
      c = -mult * cn;
    }
  }
  if (fabs(a) < tiny) a = a >= 0.0 ? tiny : -tiny;
  w[(long long)(n - 1) * ldw] = 1.0 / a;
}

// Back substitution of tri_solve from the last forward-eliminated entry
// `cur`; returns |x|^2 of the solution.
__device__ double tri_back(const double* w, int n, int ldw, double* x, long long stride, double cur) {
  const long long s = (long long)n * ldw;
  double x2 = cur * w[(long long)(n - 1) * ldw];  // x[n-1]
  x[(n - 1) * stride] = x2;
  double nrm = x2 * x2;
  if (n == 1) return nrm;
  const double* w2 = w + (long long)(n - 2) * ldw;
  double x1 = (x[(n - 2) * stride] - w2[s] * x2) * w2[0];  // x[n-2]
  x[(n - 2) * stride] = x1;
  nrm += x1 * x1;
  int k = n - 3;
  for (; k >= 3; k -= 4) {
    double rh[4], u1[4], u2[4], rp[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const double* wk = w + (long long)(k - q) * ldw;
      rh[q] = x[(k - q) * stride];
      u1[q] = wk[s];
      u2[q] = wk[2 * s];
      rp[q] = wk[0];
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const double x0 = (rh[q] - u1[q] * x1 - u2[q] * x2) * rp[q];
      x[(k - q) * stride] = x0;
      nrm += x0 * x0;
      x2 = x1;
      x1 = x0;
    }
  }
  for (; k >= 0; --k) {
    const double* wk = w + (long long)k * ldw;
    const double x0 = (x[k * stride] - wk[s] * x1 - wk[2 * s] * x2) * wk[0];
    x[k * stride] = x0;
    nrm += x0 * x0;
    x2 = x1;
    x1 = x0;
  }
  return nrm;
}

// Solves (T - lam I) x = b in place with the factors of tri_factor.  The
// running entries are carried in registers and the loads of x and of the
// factors are issued four steps ahead of their use, so the serial recurrences
// do not wait on memory at every step.  Returns |x|^2 of the solution.
__device__ double tri_solve(const double* w, int n, int ldw, double* x, long long stride) {
  const long long s = (long long)n * ldw;
  double cur = x[0];
  int k = 0;
  for (; k + 4 <= n - 1; k += 4) {
    double fl[4], mu[4], xn[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const double* wk = w + (long long)(k + q) * ldw;
      fl[q] = wk[4 * s];
      mu[q] = wk[3 * s];
      xn[q] = x[(k + q + 1) * stride];
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      double xk = cur, xk1 = xn[q];
      if (fl[q] != 0.0) {
        xk = xn[q];
        xk1 = cur;
      }
      xk1 -= mu[q] * xk;
      x[(k + q) * stride] = xk;
      cur = xk1;
    }
  }
  for (; k < n - 1; ++k) {
    const double* wk = w + (long long)k * ldw;
    double xk = cur, xk1 = x[(k + 1) * stride];
    if (wk[4 * s] != 0.0) {
      const double t = xk;
      xk = xk1;
      xk1 = t;
    }
    xk1 -= wk[3 * s] * xk;
    x[k * stride] = xk;
    cur = xk1;
  }
  return tri_back(w, n, ldw, x, stride, cur);
}

// tri_factor for the shift lam together with the forward elimination of the
// right-hand side b_i = hash_unit(i, col) + 1e-3 (the start vector of inverse
// iteration), stored in x; returns the last eliminated entry, from which
// tri_back completes the first solve.
__device__ double tri_factor_rhs(const double* d, const double* e, int n, double lam, double tiny, double* w,
                                 int ldw, double* x, long long stride, unsigned col) {
  double a = d[0] - lam;
  double c = n > 1 ? e[0] : 0.0;
  const long long s = (long long)n * ldw;
  double cur = hash_unit(0, col) + 1e-3;
  for (int k = 0; k < n - 1; ++k) {
    const double b = e[k];
    const double an = d[k + 1] - lam;
    const double cn = (k + 1 < n - 1) ? e[k + 1] : 0.0;
    double* wk = w + (long long)k * ldw;
    double xk = cur, xk1 = hash_unit(k + 1, col) + 1e-3;
    if (fabs(a) >= fabs(b)) {
      double piv = a;
      if (fabs(piv) < tiny) piv = piv >= 0.0 ? tiny : -tiny;
      const double r = 1.0 / piv;
      wk[0] = r;
      wk[s] = c;
      wk[2 * s] = 0.0;
      wk[3 * s] = b * r;
      wk[4 * s] = 0.0;
      xk1 -= (b * r) * xk;
      a = an - b * r * c;
      c = cn;
    } else {
      const double r = 1.0 / b;
      const double mult = a * r;
      wk[0] = r;
      wk[s] = an;
      wk[2 * s] = cn;
      wk[3 * s] = mult;
      wk[4 * s] = 1.0;
      const double t = xk;
      xk = xk1;
      xk1 = t - mult * xk;
      a = c - mult * an;
      c = -mult * cn;
    }
    x[k * stride] = xk;
    cur = xk1;
  }
  if (fabs(a) < tiny) a = a >= 0.0 ? tiny : -tiny;
  w[(long long)(n - 1) * ldw] = 1.0 / a;
  return cur;
}

// ---------------------------------------------------------------- stages

// Eigenvalues k = 0..nneed-1 and N-1 of the tridiagonal, one thread each.
// Bisection on the Sturm count until the count at the iterate x says that
// eigenvalue k is the nearest one above (count k) or below (count k+1); from
// there Laguerre steps toward it.  For a polynomial with real roots the
// Laguerre step in a chosen direction lands between x and the adjacent root on
// that side, so the iterates approach eigenvalue k monotonically and converge
// cubically (Li & Zeng, "Laguerre's iteration in solving the symmetric
// tridiagonal eigenproblem - revisited", SIAM J. Sci. Comput. 15, 1994).
// Every evaluation also tightens the bisection bracket, and a step that leaves
// it falls back to bisection.
// Eigenvalue k of the tridiagonal (one thread).  x0: a first iterate inside
// (gl, gu), e.g. the eigenvalue of the previous SCC iteration (the search then
// usually starts next to eigenvalue k and takes Laguerre steps at once);
// otherwise the midpoint.
__device__ __forceinline__ double eigenvalue_k(const double* d, const double* esq, int N, int k, double gl, double gu,
                                              double pivmin, double atol, double x0 = 0.0, bool warm = false) {
  const double dn = (double)N;
  double lo = gl, hi = gu;
  double x = (warm && x0 > lo && x0 < hi) ? x0 : 0.5 * (lo + hi);
  for (int it = 0; it < 160; ++it) {
    double p, dp, ddp;
    const int c = sturm_poly(d, esq, N, x, pivmin, p, dp, ddp);
    if (c >= k + 1)
      hi = x;
    else
      lo = x;
    const double tol = 2.0 * DBL_EPSILON * fmax(fabs(lo), fabs(hi)) + atol;
    if (hi - lo <= tol) {
      x = 0.5 * (lo + hi);
      break;
    }
    double xn = 0.5 * (lo + hi);
    if (c == k || c == k + 1) {
      // u = p/p', w = p p''/p'^2; step = N u / (1 + sigma sqrt((N-1)(N(1-w)-1)))
      // with sigma chosen so that the step moves toward eigenvalue k.
      const double u = p / dp;
      const double w = (p * ddp) / (dp * dp);
      const double sq = sqrt((dn - 1.0) * (dn * (1.0 - w) - 1.0));
      const bool up = (c == k);
      const double sigma = ((u > 0.0) == up) ? -1.0 : 1.0;
      const double step = dn * u / (1.0 + sigma * sq);
      const double xt = x - step;
      // The Newton ratio u points to the nearest eigenvalue: when it points
      // away from eigenvalue k, x sits next to the neighbour on the other
      // side, where the Laguerre step is tiny and proves nothing.
      const bool nearest = up ? (u < 0.0) : (u > 0.0);
      if (nearest && fabs(step) <= 32.0 * tol) {  // cubic convergence: the step bounds the error
        x = fmin(fmax(xt, lo), hi);
        break;
      }
      if (xt > lo && xt < hi && (nearest || fabs(step) >= 0.125 * (hi - lo))) xn = xt;
    }
    if (xn <= lo || xn >= hi) break;
    x = xn;
  }
  return x;
}

// Eigenvalues k = 0..nneed-1 and N-1 by the whole CTA, one thread each (at most
// NT of them).  As eigenvalue_k, but every Sturm count serves every thread: the
// points and counts of a round are shared, so each bracket is the tightest that
// all of them allow, and a first round of evenly spread points isolates most
// eigenvalues of a cold start.  (One thread alone bisected its own way in from
// the Gerschgorin interval whenever its start was not next to its eigenvalue,
// and the slowest of a warp's 32 decided: about 30 evaluations at N = 128, here
// 4 to 8.)  warm: eps holds the previous SCC iteration's eigenvalues, the first
// points.  px, pc: N doubles of shared scratch.  Part: the CTA finds only NT of them
// from number `base` on; a cold start then takes two rounds of even points, the
// second over the interval that the first leaves to the CTA's eigenvalues, in two
// words of its own behind the NT of px (a thread that found its eigenvalue in the first
// round still has its point and count in px and pc for the others).
template <int NT, bool Part = false>
__device__ __forceinline__ void eigenvalues(const double* d, const double* esq, int N, int nneed, int nwarm, double gl,
                                            double gu, double pivmin, double atol, double* eps, double* px, double* pc,
                                            int base = 0) {
  const int tid = threadIdx.x;
  const int nall = (nneed < N) ? nneed + 1 : N;
  const int nlist = Part ? min(nall - base, NT) : nall;
  const int k = (base + tid < nneed) ? base + tid : N - 1;
  const double dn = (double)N;
  bool active = tid < nlist;
  double lo = gl, hi = gu, x = gl + (gu - gl) * ((tid + 0.5) / nlist);
  if (active && (k < nwarm || (nwarm > 0 && k == N - 1))) {
    const double x0 = eps[k];
    if (x0 > lo && x0 < hi) x = x0;
  }
  for (int it = 0; it < 160; ++it) {
    double p = 0.0, dp = 0.0, ddp = 0.0;
    int c = 0;
    if (active) {
      c = sturm_poly(d, esq, N, x, pivmin, p, dp, ddp);
      px[tid] = x;
      pc[tid] = (double)c;
    }
    __syncthreads();
    if (active) {
      // the first round takes every point, later ones those next in line
      const double kk = (double)(k + 1);
      const bool every = it == 0 || (Part && it == 1);
      const int j0 = every ? 0 : max(tid - 4, 0), j1 = every ? nlist : min(tid + 5, nlist);
#pragma unroll 4
      for (int j = j0; j < j1; ++j) {
        const double xj = px[j];
        if (pc[j] >= kk)
          hi = fmin(hi, xj);
        else
          lo = fmax(lo, xj);
      }
      const double tol = 2.0 * DBL_EPSILON * fmax(fabs(lo), fabs(hi)) + atol;
      double xn = 0.5 * (lo + hi);
      bool done = hi - lo <= tol;
      if (!done && (c == k || c == k + 1)) {  // the Laguerre step of eigenvalue_k
        const double u = p / dp;
        const double w = (p * ddp) / (dp * dp);
        const double sq = sqrt((dn - 1.0) * (dn * (1.0 - w) - 1.0));
        const bool up = (c == k);
        const double sigma = ((u > 0.0) == up) ? -1.0 : 1.0;
        const double step = dn * u / (1.0 + sigma * sq);
        const double xt = x - step;
        const bool nearest = up ? (u < 0.0) : (u > 0.0);
        if (nearest && fabs(step) <= 32.0 * tol) {
          xn = fmin(fmax(xt, lo), hi);
          done = true;
        } else if (xt > lo && xt < hi && (nearest || fabs(step) >= 0.125 * (hi - lo))) {
          xn = xt;
        }
      }
      if (!done && (xn <= lo || xn >= hi)) {
        xn = x;
        done = true;
      }
      x = xn;
      if (done) {
        eps[k] = x;
        active = false;
      }
    }
    if (!__syncthreads_or(active)) break;
    if (Part && it == 0 && nwarm == 0) {
      if (tid == 0) px[NT] = lo;
      if (tid == nlist - 1) px[NT + 1] = hi;
      __syncthreads();
      if (active) x = px[NT] + (px[NT + 1] - px[NT]) * ((tid + 0.5) / nlist);
    }
  }
  if (active) eps[k] = x;
  __syncthreads();
}

// Fermi occupations by bisection to the bracket fixed point (src/electronic.rs:
// 3853-3921), one warp.  Only eps[0..nneed) and eps[N-1] are known: orbitals in
// between lie at or above eps[nneed-1]; while a trial mu keeps them beyond the
// +80 kT clamp each contributes exactly 2/(1+e^80).  When a decision would need
// them, `ambiguous` is set and the caller computes every eigenvalue.
template <int CAP>
__device__ __noinline__ void fermi_warp(const double* eps, int N, int nneed, double nelec, double kt, double* occ, double& mu_out,
                           double& ts_out, bool& ambiguous) {
  constexpr double cap = CAP;  // electrons per orbital: 2, or 1 in a spin channel
  const int lane = threadIdx.x & 31;
  ambiguous = false;
  double mu = 0.0, ts = 0.0;
  if (kt <= 0.0) {  // aufbau (src/electronic.rs:3830-3851); needs every orbital up to the HOMO
    double rem = fmax(nelec, 0.0);
    int homo = 0;
    for (int i = 0; i < N; ++i) {
      const double fill = fmin(rem, cap);
      if (lane == 0) occ[i] = fill;
      rem -= fill;
      if (fill > 1e-12) homo = i;
    }
    if (homo >= nneed && nneed < N) ambiguous = true;
    mu = eps[homo];
  } else if (nelec <= 0.0) {
    for (int i = lane; i < N; i += 32) occ[i] = 0.0;
    mu = eps[0];
  } else if (nelec >= cap * N) {
    for (int i = lane; i < N; i += 32) occ[i] = cap;
    mu = eps[N - 1];
  } else {
    const double c80 = cap / (1.0 + exp(80.0));
    const double cm80 = cap / (1.0 + exp(-80.0));
    const int nunc = (nneed < N) ? (N - 1 - nneed) : 0;
    const double etop = eps[nneed - 1];
    const double ikt = 1.0 / kt;
    auto fo = [&](double ei, double m) {
      const double x = (ei - m) * ikt;
      if (x >= 80.0) return c80;
      if (x <= -80.0) return cm80;
      return cap / (1.0 + exp(x));
    };
    double lo = eps[0] - 100.0 * kt - 10.0, hi = eps[N - 1] + 100.0 * kt + 10.0;
    for (int it = 0; it < 200; ++it) {
      const double mid = 0.5 * (lo + hi);
      double s = 0.0;
      for (int i = lane; i < nneed; i += 32) s += fo(eps[i], mid);
      if (lane == 0 && nneed < N) s += fo(eps[N - 1], mid);
      s = warp_sum(s);
      if (nunc > 0) {
        if ((etop - mid) / kt >= 80.0) s += nunc * c80;
        else if (s < nelec) {
          ambiguous = true;
          break;
        }
      }
      double nlo = lo, nhi = hi;
      if (s < nelec) nlo = mid;
      else nhi = mid;
      if (nlo == lo && nhi == hi) break;
      lo = nlo;
      hi = nhi;
    }
    mu = 0.5 * (lo + hi);
    if (!ambiguous && nunc > 0 && !((etop - mu) / kt >= 80.0)) ambiguous = true;
    if (!ambiguous) {
      double t = 0.0;
      for (int i = lane; i < N; i += 32) {
        const bool known = i < nneed || i == N - 1;
        const double f = known ? fo(eps[i], mu) : c80;
        occ[i] = f;
        const double nn = fmin(1.0 - 1e-16, fmax(1e-16, f / cap));
        t += cap * kt * (nn * log(nn) + (1.0 - nn) * log(1.0 - nn));
      }
      ts = warp_sum(t);
    }
  }
  mu_out = mu;
  ts_out = ts;
}

// Finite-temperature occupations (kt > 0, 0 < nelec < 2N) by the whole CTA.
// The reference bisects [eps_0 - 100 kT - 10, eps_N-1 + 100 kT + 10] on
// "electron count < nelec" until the bracket stops shrinking
// (src/electronic.rs:3853-3921); here each round places one trial mu per thread,
// NT + 1 equal subintervals, and keeps the subinterval where the count crosses
// nelec, so the bracket converges to the same crossing in log_(NT+1) rounds, nine
// for 128 threads.  (One trial per warp, its sum over the lanes, took 26 rounds
// of a warp reduction and an exponential per orbital each.)  Orbitals more than
// 40 kT outside the bracket are full or empty to the last bit of the count, so a
// trial sums the few levels next to the gap.  Eigenvalues beyond
// eps[nneed-1] are unknown (apart from eps[N-1]); they are clamped at +80 kT like
// in fermi_warp, and a trial mu at which they would matter makes the result
// ambiguous (the caller then computes all of them).  Shared scratch: sh.first.
template <int NT, int CAP>
__device__ void fermi_cta(const double* eps, int N, int nneed, double nelec, double kt, double* occ, SccShared& sh,
                          double& mu_out, double& ts_out, bool& ambiguous) {
  constexpr int NW = NT / 32;
  constexpr double cap = CAP;  // electrons per orbital: 2, or 1 in a spin channel
  static_assert(NW <= 16, "one entry per warp");
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const double c80 = cap / (1.0 + exp(80.0));
  const double cm80 = cap / (1.0 + exp(-80.0));
  const int nunc = (nneed < N) ? (N - 1 - nneed) : 0;
  const double etop = eps[nneed - 1], elast = eps[N - 1];
  const double ikt = 1.0 / kt, w40 = 40.0 * kt;
  auto fo = [&](double ei, double m) {
    const double x = (ei - m) * ikt;
    if (x >= 80.0) return c80;
    if (x <= -80.0) return cm80;
    return cap / (1.0 + exp(x));
  };
  // The count crosses nelec within 40 kT of level k = ceil(nelec / cap) - 1: 40 kT
  // below it the levels from k on hold less than 1e-17 electrons each and those
  // before it cap k < nelec; 40 kT above it the first k + 1 levels are full to
  // the last bit.
  const int k = max(0, min(nneed - 1, (int)ceil(nelec / cap) - 1));
  double lo = eps[nelec - cap * k > 1e-6 ? k : max(k - 1, 0)] - w40, hi = eps[k] + w40;
  if ((nneed < N && k == nneed - 1) || !(hi > lo)) {
    lo = eps[0] - 100.0 * kt - 10.0;
    hi = elast + 100.0 * kt + 10.0;
  }
  bool amb = false;
  int i0 = k, i1 = k + 1;  // levels in reach of the bracket (eps ascends)
#pragma unroll 1
  while (i0 > 0 && eps[i0 - 1] >= lo - w40) --i0;
#pragma unroll 1
  while (i1 < nneed && eps[i1] <= hi + w40) ++i1;
  for (int round = 0; round < 64; ++round) {
    const double h = (hi - lo) * (1.0 / (NT + 1));
    const double mid = fmin(lo + (double)(tid + 1) * h, hi);
#pragma unroll 1
    while (i0 < k && eps[i0] < lo - w40) ++i0;
#pragma unroll 1
    while (i1 > k + 1 && eps[i1 - 1] > hi + w40) --i1;
    double sm = (double)i0 * cm80 + (double)(nneed - i1) * c80;
#pragma unroll 1
    for (int i = i0; i < i1; ++i) sm += fo(eps[i], mid);
    if (nneed < N) sm += fo(elast, mid);
    bool flag = false;
    if (nunc > 0) {
      if ((etop - mid) * ikt >= 80.0)
        sm += nunc * c80;
      else if (sm < nelec)
        flag = true;
    }
    const unsigned over = __ballot_sync(0xffffffffu, sm >= nelec);
    const unsigned bad = __ballot_sync(0xffffffffu, flag);
    int* first_at = sh.first[round & 1];  // two buffers: one barrier a round
    if (lane == 0) first_at[wid] = (over ? 32 * wid + __ffs(over) - 1 : NT) | (bad ? 1 << 30 : 0);
    __syncthreads();
    int j = NT;
#pragma unroll
    for (int q = 0; q < NW; ++q) {
      const int v = first_at[q];
      j = min(j, v & ~(1 << 30));
      amb = amb || (v >> 30);
    }
    const double nlo = (j == 0) ? lo : fmin(lo + (double)j * h, hi);
    const double nhi = (j == NT) ? hi : fmin(lo + (double)(j + 1) * h, hi);
    if (amb || (nlo == lo && nhi == hi)) break;
    lo = nlo;
    hi = nhi;
  }
  __syncthreads();
  const double mu = 0.5 * (lo + hi);
  if (!amb && nunc > 0 && !((etop - mu) / kt >= 80.0)) amb = true;
  double ts = 0.0;
  if (!amb) {
    double t = 0.0;
#pragma unroll 1
    for (int i = tid; i < N; i += NT) {
      const bool known = i < nneed || i == N - 1;
      const double f = known ? fo(eps[i], mu) : c80;
      occ[i] = f;
      const double nn = fmin(1.0 - 1e-16, fmax(1e-16, f / cap));
      t += cap * kt * (nn * log(nn) + (1.0 - nn) * log(1.0 - nn));
    }
    ts = block_sum(t, sh.red);
  }
  mu_out = mu;
  ts_out = ts;
  ambiguous = amb;
}

// A requested spin multiplicity fills the alpha and beta channels on their own,
// each orbital holding at most one electron per channel (src/electronic.rs:
// 3930-4045): occupation = alpha + beta, mu = their mean, TS = their sum.
// Every thread takes part; the results land in sh.scal[1] (mu), sh.scal[2]
// (TS) and sh.iscal[2] (ambiguous); `tmp` (N doubles) holds the beta channel.
// Kept out of line: inlined, this rarely used path changes how the compiler
// lays out the hot SCC loop (the closed-shell SCC stage measured 30% slower).
template <int NT>
__device__ __noinline__ void spin_channel_occupations(const double* eps, int N, int nneed, double nalpha,
                                                      double nbeta, double kt, double* occ, double* tmp,
                                                      SccShared& sh) {
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  auto channel = [&](double ne, double* o, double& fm, double& ft, bool& amb) {
    if (kt > 0.0 && ne > 0.0 && ne < (double)N) {
      fermi_cta<NT, 1>(eps, N, nneed, ne, kt, o, sh, fm, ft, amb);
    } else {
      if (wid == 0) {
        double m, t;
        bool a;
        fermi_warp<1>(eps, N, nneed, ne, kt, o, m, t, a);
        if (lane == 0) {
          sh.scal[4] = m;
          sh.scal[5] = t;
          sh.iscal[4] = a ? 1 : 0;
        }
      }
      __syncthreads();
      fm = sh.scal[4];
      ft = sh.scal[5];
      amb = sh.iscal[4] != 0;
      __syncthreads();
    }
  };
  double fa, ta, fb, tb;
  bool aa, ab;
  channel(nalpha, occ, fa, ta, aa);
  channel(nbeta, tmp, fb, tb, ab);
#pragma unroll 1
  for (int i = tid; i < N; i += NT) occ[i] += tmp[i];
  if (tid == 0) {
    sh.scal[1] = 0.5 * (fa + fb);
    sh.scal[2] = ta + tb;
    sh.iscal[2] = (aa || ab) ? 1 : 0;
  }
  __syncthreads();
}

// Index tables of one molecule (one thread): shell -> atom, shell -> index
// within its atom, shell -> first AO, AO -> shell, atom -> first shell.
__device__ void build_index_tables(const Batch& B, const Model& M, int a0, int nat, int* sh_atom, int* sh_k,
                                   int* sh_ao0, int* ao_sh, int* atom_sh) {
  int s = 0, o = 0;
  for (int a = 0; a < nat; ++a) {
    const ElemTable& el = M.elem[B.z[a0 + a]];
    atom_sh[a] = s;
    for (int k = 0; k < el.nsh; ++k) {
      sh_atom[s + k] = a;
      sh_k[s + k] = k;
      sh_ao0[s + k] = o + el.ao_first[k];
      for (int q = 0; q < 2 * el.l[k] + 1; ++q) ao_sh[o + el.ao_first[k] + q] = s + k;
    }
    s += el.nsh;
    o += el.nao;
  }
  atom_sh[nat] = s;
}

// Per-molecule view shared by the SCC stages: sizes, offsets and the index
// tables (shell -> atom, shell -> shell index within its atom, shell -> first
// AO, AO -> shell, atom -> first shell), plus the molecule's Coulomb matrix.
struct MolCtx {
  int m, a0, nat, sh0, nsh, N;
  const int *sh_atom, *sh_k, *sh_ao0, *ao_sh, *atom_sh;
  const double* G;
};

// (1) Shell potential of the input charges (src/coulomb.rs:140-193):
// w.qat, w.vsh and the AO potential vao.
template <int NT>
__device__ void stage_potential(const Batch& B, const Model& M, const MolCtx& c, CtaWs& w, double* vao) {
  const int tid = threadIdx.x;
  const int a0 = c.a0, nat = c.nat, nsh = c.nsh, N = c.N;
  const int *sh_atom = c.sh_atom, *ao_sh = c.ao_sh, *atom_sh = c.atom_sh;
  const double* G = c.G;
#pragma unroll 1
  for (int a = tid; a < nat; a += NT) {
    double q = 0.0;
    for (int s = atom_sh[a]; s < atom_sh[a + 1]; ++s) q += w.qin[s];
    w.qat[a] = q;
  }
  __syncthreads();
#pragma unroll 1
  for (int i = tid; i < nsh; i += NT) {
    double v = 0.0;
    for (int j = 0; j < nsh; ++j) v += G[(long long)j * nsh + i] * w.qin[j];  // G symmetric: coalesced column
    const int a = sh_atom[i];
    const double qa = w.qat[a];
    v += qa * qa * M.elem[B.z[a0 + a]].gam3;
    w.vsh[i] = v;
  }
  __syncthreads();
#pragma unroll 1
  for (int i = tid; i < N; i += NT) vao[i] = w.vsh[ao_sh[i]];
  __syncthreads();
}

// (9) Output shell and atomic charges, electronic energy, second- and
// third-order energies and the charge rms (src/electronic.rs:2173-2191,
// :3160-3200); also the output potential w.vout.
template <int NT>
__device__ void stage_charges_energy(const Batch& B, const Model& M, const MolCtx& c, CtaWs& w, const double* pop,
                                     const double* occ, const double* eps, const double* vao, int nocc, SccShared& sh,
                                     double& e_el, double& e2, double& e3, double& rms) {
  const int tid = threadIdx.x;
  const int a0 = c.a0, nat = c.nat, nsh = c.nsh, N = c.N;
  const int *sh_atom = c.sh_atom, *sh_k = c.sh_k, *sh_ao0 = c.sh_ao0, *atom_sh = c.atom_sh;
  const double* G = c.G;
#pragma unroll 1
  for (int s = tid; s < nsh; s += NT) {
    const ElemTable& el = M.elem[B.z[a0 + sh_atom[s]]];
    const int k = sh_k[s];
    double p = 0.0;
    for (int q = 0; q < 2 * el.l[k] + 1; ++q) p += pop[sh_ao0[s] + q];
    w.qout[s] = el.refocc[k] - p;
  }
  double part = 0.0;
#pragma unroll 1
  for (int i = tid; i < N; i += NT) part += (i < nocc ? occ[i] * eps[i] : 0.0) + vao[i] * pop[i];
  __syncthreads();
#pragma unroll 1
  for (int a = tid; a < nat; a += NT) {
    double q = 0.0;
    for (int s = atom_sh[a]; s < atom_sh[a + 1]; ++s) q += w.qout[s];
    w.qat[a] = q;
  }
  __syncthreads();
  double p2 = 0.0, p3 = 0.0, pr = 0.0;
#pragma unroll 1
  for (int i = tid; i < nsh; i += NT) {
    double v = 0.0;
    for (int j = 0; j < nsh; ++j) v += G[(long long)j * nsh + i] * w.qout[j];  // G symmetric: coalesced column
    p2 += w.qout[i] * v;
    const int a = sh_atom[i];
    const double qa = w.qat[a];
    const double g3 = M.elem[B.z[a0 + a]].gam3;
    w.vout[i] = v + qa * qa * g3;
    const double r = w.qout[i] - w.qin[i];
    pr += r * r;
  }
#pragma unroll 1
  for (int a = tid; a < nat; a += NT) {
    const double qa = w.qat[a];
    p3 += qa * qa * qa * M.elem[B.z[a0 + a]].gam3 / 3.0;
  }
  double sums[4] = {part, p2, p3, pr};
  block_sums<4>(sums, sh.red);
  e_el = sums[0];
  e2 = 0.5 * sums[1];
  e3 = sums[2];
  rms = nsh ? sqrt(sums[3] / nsh) : 0.0;
}

// (10) Charge mixing: modified Broyden (src/electronic.rs:3203-3309), linear
// damped step on the first iteration, a singular solve or an untrusted vector
// (:3311-3316, :3759-3761); the next input charges land in w.qin.
template <int NT>
__device__ void stage_mix(const SccOptions& opt, const MolCtx& c, CtaWs& w, int cap, int& bro_iter, SccShared& sh) {
  constexpr int NW = NT / 32;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int nsh = c.nsh;
  const double mixing = fmin(1.0, fmax(0.01, opt.mixing));
  const int memory = max(opt.broyden_size, 2);
  bool have_next = false;
  if (opt.broyden) {
    bro_iter += 1;
    if (bro_iter == 1) {
#pragma unroll 1
      for (int s = tid; s < nsh; s += NT) {
        const double r = w.qout[s] - w.qin[s];
        w.dqlast[s] = r;
        w.qlast[s] = w.qin[s];
        w.qnext[s] = w.qin[s] + mixing * r;
      }
      have_next = true;
      __syncthreads();
    } else {
      const int itn = bro_iter - 1;
      const int it1 = (itn - 1) % memory;
      const int slot = it1 % cap;
      double pn = 0.0, pd = 0.0;
#pragma unroll 1
      for (int s = tid; s < nsh; s += NT) {
        const double r = w.qout[s] - w.qin[s];
        pn += r * r;
        const double dfv = r - w.dqlast[s];
        pd += dfv * dfv;
      }
      double sums[2] = {pn, pd};
      block_sums<2>(sums, sh.red);
      const double dqn = sqrt(sums[0]), dfn = sqrt(sums[1]);
      const double inv = 1.0 / fmax(dfn, DBL_EPSILON);
      double* dfs = w.df + (long long)slot * nsh;
      double* us = w.u + (long long)slot * nsh;
#pragma unroll 1
      for (int s = tid; s < nsh; s += NT) {
        const double r = w.qout[s] - w.qin[s];
        const double dfv = (r - w.dqlast[s]) * inv;
        dfs[s] = dfv;
        us[s] = mixing * dfv + inv * (w.qin[s] - w.qlast[s]);
      }
      if (tid == 0) {
        double om = dqn > 0.01 / 100000.0 ? 0.01 / dqn : 100000.0;
        if (om < 1.0) om = 1.0;
        w.omega[slot] = om;
      }
      __syncthreads();
      const int start = itn > memory ? itn - memory + 1 : 1;
      const int mact = itn - start + 1;
      // dot products df_new . df_j for every active slot, and c_j = omega_j df_j . dq
#pragma unroll 1
      for (int r = wid; r < mact; r += NW) {
        const int sj = ((start + r - 1) % memory) % cap;
        const double* dj = w.df + (long long)sj * nsh;
        double s1 = 0.0, s2 = 0.0;
        for (int s = lane; s < nsh; s += 32) {
          s1 += dfs[s] * dj[s];
          s2 += dj[s] * (w.qout[s] - w.qin[s]);
        }
        s1 = warp_sum(s1);
        s2 = warp_sum(s2);
        if (lane == 0) {
          w.dots[(long long)slot * cap + sj] = s1;
          w.dots[(long long)sj * cap + slot] = s1;
          w.cvec[r] = s2;
        }
      }
      __syncthreads();
#pragma unroll 1
      for (int idx = tid; idx < mact * mact; idx += NT) {
        const int r = idx / mact, c = idx % mact;
        const int si = ((start + r - 1) % memory) % cap, sj = ((start + c - 1) % memory) % cap;
        double b = w.omega[si] * w.omega[sj] * w.dots[(long long)si * cap + sj];
        if (r == c) b += 0.01 * 0.01;
        w.beta[(long long)r * mact + c] = b;
      }
#pragma unroll 1
      for (int r = tid; r < mact; r += NT) {
        const int si = ((start + r - 1) % memory) % cap;
        w.cvec[r] *= w.omega[si];
      }
      __syncthreads();
      // Gauss-Jordan with partial pivoting (src/electronic.rs:3767-3806); up to 16
      // vectors by one warp, whose steps need no block barrier (six a column: most of the
      // mixing of a small molecule)
      const bool one = mact <= 16;
      const int t = one ? lane : tid, nt = one ? 32 : NT;
      auto sync = [&]() {
        if (one)
          __syncwarp();
        else
          __syncthreads();
      };
      bool ok = true;
      if (!one || wid == 0) {
#pragma unroll 1
        for (int col = 0; col < mact; ++col) {
          int piv = lane;
          if (wid == 0) {  // the first of the largest
            double pabs = lane >= col && lane < mact ? fabs(w.beta[(long long)lane * mact + col]) : -1.0;
#pragma unroll 4
            for (int r = lane + 32; r < mact; r += 32) {
              const double v = r >= col ? fabs(w.beta[(long long)r * mact + col]) : -1.0;
              if (v > pabs) {
                pabs = v;
                piv = r;
              }
            }
#pragma unroll 1
            for (int o = 16; o > 0; o >>= 1) {
              const double v = __shfl_xor_sync(0xffffffffu, pabs, o);
              const int at = __shfl_xor_sync(0xffffffffu, piv, o);
              if (v > pabs || (v == pabs && at < piv)) {
                pabs = v;
                piv = at;
              }
            }
            piv = pabs < 1e-18 ? -1 : piv;
          }
          if (one) {
            piv = __shfl_sync(0xffffffffu, piv, 0);
          } else {
            if (tid == 0) sh.iscal[1] = piv;
            __syncthreads();
            piv = sh.iscal[1];
          }
          if (piv < 0) {
            ok = false;
            break;
          }
          if (piv != col) {
#pragma unroll 1
            for (int j = t; j < mact; j += nt) {
              const double v = w.beta[(long long)piv * mact + j];
              w.beta[(long long)piv * mact + j] = w.beta[(long long)col * mact + j];
              w.beta[(long long)col * mact + j] = v;
            }
            if (t == 0) {
              const double v = w.cvec[piv];
              w.cvec[piv] = w.cvec[col];
              w.cvec[col] = v;
            }
            sync();
          }
          const double dg = w.beta[(long long)col * mact + col];
          sync();
#pragma unroll 1
          for (int j = col + t; j <= mact; j += nt) {  // the last one is the right-hand side
            double* at = j < mact ? w.beta + (long long)col * mact + j : w.cvec + col;
            *at /= dg;
          }
          sync();
#pragma unroll 1
          for (int r = t >> 4; r < mact; r += nt >> 4) {  // 16 threads a row; column `col` is zeroed below
            const double f = w.beta[(long long)r * mact + col];
            if (r == col || f == 0.0) continue;
            const double* from = w.beta + (long long)col * mact;
            double* to = w.beta + (long long)r * mact;
            int j = col + 1 + (t & 15);
#pragma unroll 1
            for (; j + 112 < mact; j += 128) {  // eight entries loaded before the first is stored
              double a[8], b[8];
#pragma unroll
              for (int u = 0; u < 8; ++u) {
                a[u] = to[j + 16 * u];
                b[u] = from[j + 16 * u];
              }
#pragma unroll
              for (int u = 0; u < 8; ++u) to[j + 16 * u] = a[u] - f * b[u];
            }
#pragma unroll 1
            for (; j <= mact; j += 16) {
              if (j < mact)
                to[j] -= f * from[j];
              else
                w.cvec[r] -= f * w.cvec[col];
            }
          }
          sync();
#pragma unroll 1
          for (int r = t; r < mact; r += nt)
            if (r != col) w.beta[(long long)r * mact + col] = 0.0;
          sync();
        }
        if (one && lane == 0) sh.iscal[1] = ok ? 1 : -1;
      }
      __syncthreads();
      if (one) ok = sh.iscal[1] > 0;
      if (ok) {
#pragma unroll 1
        for (int s = tid; s < nsh; s += NT) {
          const double r = w.qout[s] - w.qin[s];
          double qn = w.qin[s] + mixing * r;
#pragma unroll 2
          for (int rr = 0; rr < mact; ++rr) {
            const int si = ((start + rr - 1) % memory) % cap;
            qn -= w.omega[si] * w.cvec[rr] * w.u[(long long)si * nsh + s];
          }
          w.qnext[s] = qn;
          w.dqlast[s] = r;
          w.qlast[s] = w.qin[s];
        }
        have_next = true;
      }
      __syncthreads();
    }
    if (have_next) {  // trusted_charge_vector (src/electronic.rs:3759-3761)
      int bad = 0;
#pragma unroll 1
      for (int s = tid; s < nsh; s += NT)
        if (!isfinite(w.qnext[s]) || fabs(w.qnext[s]) >= 10.0) bad = 1;
      if (__syncthreads_or(bad)) have_next = false;
    }
  }
  if (!have_next)
#pragma unroll 1
    for (int s = tid; s < nsh; s += NT) w.qnext[s] = w.qin[s] + mixing * (w.qout[s] - w.qin[s]);
  __syncthreads();
#pragma unroll 1
  for (int s = tid; s < nsh; s += NT) w.qin[s] = w.qnext[s];
}

// Results of a finished SCC: energy terms, iterations, status, Fermi level,
// Mulliken dipole, shell charges and potential, atomic charges.
template <int NT>
__device__ void stage_results(const Batch& B, const MolCtx& c, CtaWs& w, int iter, bool converged, double e_el,
                              double e2, double e3, double ts, double mu) {
  const int tid = threadIdx.x;
  const int a0 = c.a0, nat = c.nat, nsh = c.nsh;
  const int m = c.m, sh0 = c.sh0;
  if (tid == 0) {
    double* t = B.terms + (long long)m * kTerms;
    const double erep = t[2], edisp = t[7], ehal = t[8];
    const double total_internal = e_el + e2 + e3 + erep + edisp + ehal;
    t[0] = total_internal + ts;
    t[1] = total_internal;
    t[3] = e_el;
    t[4] = e2;
    t[5] = e3;
    t[14] = ts;
    B.iterations[m] = iter;
    B.status[m] = converged ? kOk : kErrSccNotConverged;
    B.fermi[m] = mu;
    double dx = 0, dy = 0, dz = 0;
    for (int a = 0; a < nat; ++a) {
      dx += w.qat[a] * B.xyz[3 * (a0 + a)];
      dy += w.qat[a] * B.xyz[3 * (a0 + a) + 1];
      dz += w.qat[a] * B.xyz[3 * (a0 + a) + 2];
    }
    B.dipole[3 * m] = dx;
    B.dipole[3 * m + 1] = dy;
    B.dipole[3 * m + 2] = dz;
  }
#pragma unroll 1
  for (int s = tid; s < nsh; s += NT) {
    B.shell_q[sh0 + s] = w.qout[s];
    B.shell_pot[sh0 + s] = w.vout[s];
    if (B.shell_pot_in) B.shell_pot_in[sh0 + s] = w.vsh[s];
  }
#pragma unroll 1
  for (int a = tid; a < nat; a += NT) B.atom_q[a0 + a] = w.qat[a];
}

// ------------------------------------------------------------ one molecule per CTA
// Everything a launch of the SCC kernel needs.
struct SccArgs {
  Batch B;
  Model M;
  SccOptions opt;
  SccLaunch SL;
};

// State of the molecule a CTA works on, at the start of the dynamic shared
// memory.  The stages of the SCC are functions of their own that read it there:
// inlined into one kernel they shared a register budget that the largest of
// them needs alone, and each of them spilled.
struct MolState {
  int m, a0, nat, sh0, nsh, N, ld;  // molecule, first atom and shell, sizes, leading dimension
  int vec_at, tri_at;               // offsets (doubles) of the N-vectors and of the reduction's scratch
  int status, converged, iter, bro_iter, have_e, nneed, nneed0, nocc, spin;
  long long mo, go;  // offsets of the molecule's matrices and of its Coulomb matrix
  double nelec, nalpha, nbeta, kt, last_e, e_el, e2, e3, ts, mu, rms, onenrm;
};
struct alignas(16) SccCta {
  SccShared sh;
  MolState s;
};
__host__ __device__ constexpr size_t scc_cta_bytes() { return sizeof(SccCta); }

struct CtaView {
  SccShared& sh;
  MolState& s;
  MolCtx c;
  CtaWs w;
  double *d, *e, *tau, *eps, *occ, *pop, *vao, *esq;
};
__device__ __forceinline__ CtaView cta_view(const SccArgs& A) {
  extern __shared__ __align__(16) unsigned char smraw[];
  SccCta& cta = *reinterpret_cast<SccCta*>(smraw);
  MolState& s = cta.s;
  int* t = reinterpret_cast<int*>(smraw + scc_cta_bytes());
  double* v = reinterpret_cast<double*>(smraw) + s.vec_at;
  const int N = s.N, maxnsh = A.SL.maxnsh;
  const MolCtx c{s.m, s.a0, s.nat, s.sh0, s.nsh, N,
                 t, t + maxnsh, t + 2 * maxnsh, t + 3 * maxnsh, t + 3 * maxnsh + A.SL.maxn,
                 A.B.gam + s.go};
  return CtaView{cta.sh, s, c, cta_ws(A.SL.ws + (long long)blockIdx.x * A.SL.ws_stride, A.SL.maxn, maxnsh, A.SL.cap),
                 v, v + N, v + 2 * N, v + 3 * N, v + 4 * N, v + 5 * N, v + 6 * N, v + 7 * N};
}

// Molecule m: sizes, index tables, electron counts.
template <int KIND>
__device__ __noinline__ void scc_begin(const SccArgs& A, int m) {
  extern __shared__ __align__(16) unsigned char smraw[];
  MolState& s = reinterpret_cast<SccCta*>(smraw)->s;
  const Batch& B = A.B;
  if (threadIdx.x == 0) {
    s.m = m;
    s.a0 = B.atom_off[m];
    s.nat = B.atom_off[m + 1] - s.a0;
    s.sh0 = B.shell_off[m];
    s.nsh = B.shell_off[m + 1] - s.sh0;
    s.N = B.ao_off[m + 1] - B.ao_off[m];
    s.ld = work_ld(s.N);
    s.vec_at = (int)(scc_vec_bytes(A.SL.maxnsh, A.SL.maxn, A.SL.maxnat) / 8);
    s.tri_at = s.vec_at + ((kVecSlots * A.SL.maxn + 1) & ~1);
    s.mo = B.mat_off[m];
    s.go = B.gam_off[m];
    s.status = kOk;
    s.converged = 0;
    s.iter = 0;
    s.nocc = 0;
    s.e_el = s.e2 = s.e3 = s.ts = s.mu = s.rms = 0.0;
    const CtaView v = cta_view(A);
    build_index_tables(B, A.M, s.a0, s.nat, const_cast<int*>(v.c.sh_atom), const_cast<int*>(v.c.sh_k),
                       const_cast<int*>(v.c.sh_ao0), const_cast<int*>(v.c.ao_sh), const_cast<int*>(v.c.atom_sh));
    double nref = 0.0;
    for (int i = 0; i < s.nsh; ++i) nref += A.M.elem[B.z[s.a0 + v.c.sh_atom[i]]].refocc[v.c.sh_k[i]];
    s.nelec = nref - B.charge[m];
    // a requested spin multiplicity: alpha and beta electron counts (validated on the host)
    s.spin = A.opt.spin_mult > 0;
    s.nalpha = s.spin ? 0.5 * (rint(s.nelec) + (A.opt.spin_mult - 1)) : 0.0;
    s.nbeta = s.spin ? 0.5 * (rint(s.nelec) - (A.opt.spin_mult - 1)) : 0.0;
    s.nneed0 = min(s.N, max(1, (int)ceil(s.spin ? s.nalpha : 0.5 * s.nelec) + 8));
    s.nneed = s.nneed0;
  }
  __syncthreads();
}

// Cholesky S = L L^T, left-looking over panels of 8 columns: the panel minus
// (its rows of L) x (the panel's rows of L)^T over the finished columns on the
// FP64 tensor cores, the 8x8 diagonal block by one thread (registers; its
// factor and reciprocal pivots staged in shared memory), then the rows below by
// a triangular solve, one thread per row.
template <int KIND>
__device__ __noinline__ void scc_cholesky(const SccArgs& A) {
  constexpr int NT = kSccKinds[KIND].nt, NW = NT / 32;
  const CtaView v = cta_view(A);
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, g = lane >> 2, t4 = lane & 3;
  const int N = v.s.N, ld = v.s.ld;
  const double* S = A.B.S + v.s.mo;
  double* L = v.w.L;
  double(*Ld)[9] = v.sh.Ld;
#pragma unroll 1
  for (int idx = tid; idx < ld * ld; idx += NT) {  // zeros in the padding
    const int i = idx / ld, j = idx - i * ld;
    L[idx] = (i < N && j < N) ? S[(long long)i * N + j] : 0.0;
  }
  __syncthreads();
  for (int c0 = 0; c0 < N; c0 += 8) {
    const int nbc = min(8, N - c0);
    if (c0 > 0) {
      const int TR = (N - c0 + 7) >> 3;
      const bool jok = g < nbc;
      const double* lj = L + (long long)(jok ? c0 + g : 0) * ld;
      for (int RT = wid; RT < TR; RT += NW) {
        const int i = c0 + RT * 8 + g;
        const bool iok = i < N;
        const double* li = L + (long long)(iok ? i : 0) * ld;
        double d0 = 0.0, d1 = 0.0;
#pragma unroll 4
        for (int k0 = 0; k0 < c0; k0 += 4) {
          const int k = k0 + t4;
          dmma_m8n8k4(d0, d1, iok ? li[k] : 0.0, jok ? lj[k] : 0.0);
        }
        if (iok) {
          double* out = L + (long long)i * ld + c0 + 2 * t4;
          if (2 * t4 < nbc) out[0] -= d0;
          if (2 * t4 + 1 < nbc) out[1] -= d1;
        }
      }
      __syncthreads();
    }
    if (tid == 0) {
      double D[8][8];
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j <= i; ++j) D[i][j] = (i < nbc) ? L[(long long)(c0 + i) * ld + c0 + j] : (i == j ? 1.0 : 0.0);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        // the reference rejects overlaps with an eigenvalue <= eigen_tolerance (1e-12)
        if (j < nbc && !(D[j][j] > 1e-12)) v.s.status = kErrInvalidInput;
        const double r = sqrt(fmax(D[j][j], 1e-300));
        const double inv = 1.0 / r;
        D[j][j] = r;
        Ld[j][8] = inv;
#pragma unroll
        for (int i = j + 1; i < 8; ++i) D[i][j] *= inv;
#pragma unroll
        for (int k = j + 1; k < 8; ++k)
#pragma unroll
          for (int i = k; i < 8; ++i) D[i][k] -= D[i][j] * D[k][j];
      }
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j <= i; ++j) {
          Ld[i][j] = D[i][j];
          if (i < nbc) L[(long long)(c0 + i) * ld + c0 + j] = D[i][j];
        }
    }
    __syncthreads();
    for (int i = c0 + 8 + tid; i < N; i += NT) {  // rows below: x L_dd^T = row
      double* row = L + (long long)i * ld + c0;
      double x[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) x[j] = row[j];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
#pragma unroll
        for (int k = 0; k < j; ++k) x[j] -= x[k] * Ld[j][k];
        x[j] *= Ld[j][8];
        row[j] = x[j];
      }
    }
    __syncthreads();
  }
  for (int i = wid; i < N; i += NW)
    for (int j = i + 1 + lane; j < N; j += 32) L[(long long)i * ld + j] = 0.0;
  __syncthreads();
}

// L^-1, kept transposed, by 8 x 8 blocks: X = L^-1 has X_JJ = L_JJ^-1 and, down
// block column J, X_IJ = -L_II^-1 sum_{J <= K < I} L_IK X_KJ.  The block columns
// are independent, one warp each with the column (transposed) in tensor-core
// accumulators, as the occupied orbitals are; the inverses of the diagonal
// blocks go through the reduction's scratch.  (One thread per column of L^-1, a
// chain of N multiply-adds with a load each, took 1M cycles at N = 128.)
template <int KIND>
__device__ __noinline__ void scc_inverse(const SccArgs& A) {
  constexpr int NT = kSccKinds[KIND].nt, NW = NT / 32, P = kSccKinds[KIND].p, NB = P / 8;
  extern __shared__ __align__(16) unsigned char smraw[];
  const CtaView v = cta_view(A);
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, g = lane >> 2, t4 = lane & 3;
  const int N = v.s.N, ld = v.s.ld, nt = ld >> 3;
  const double* __restrict__ L = v.w.L;
  double* __restrict__ LiT = v.w.LiT;
  double* inv = reinterpret_cast<double*>(smraw) + v.s.tri_at;  // [nt][8][8] row-major
#pragma unroll 1
  for (int c = tid; c < ld; c += NT) {  // column c & 7 of the inverse of diagonal block c >> 3
    const int b = c >> 3, j = c & 7;
    double x[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int row = 8 * b + i;
      double t = i == j ? 1.0 : 0.0;
#pragma unroll
      for (int k = 0; k < 8; ++k)
        if (k < i) t -= L[(long long)row * ld + 8 * b + k] * x[k];
      x[i] = (row < N && c < N) ? t / L[(long long)row * ld + row] : 0.0;
      inv[64 * b + 8 * i + j] = x[i];
    }
  }
  __syncthreads();
  for (int J = wid; J < nt; J += NW) {
    double z[NB][2];
#pragma unroll
    for (int I = 0; I < NB; ++I) {
      z[I][0] = z[I][1] = 0.0;
      if (I < nt) {
        if (I == J) {
          z[I][0] = inv[64 * J + 8 * (2 * t4) + g];
          z[I][1] = inv[64 * J + 8 * (2 * t4 + 1) + g];
        } else if (I > J) {
          const double* lrow = L + (long long)(8 * I + g) * ld + 2 * t4;
          double s0[2] = {0.0, 0.0}, s1[2] = {0.0, 0.0};
#pragma unroll
          for (int q = 0; q < (I + 3) / 4; ++q)
            if (4 * q + 3 >= J) {
              double2 l[4];
#pragma unroll
              for (int u = 0; u < 4; ++u)
                if (4 * q + u < I) l[u] = *reinterpret_cast<const double2*>(lrow + 32 * q + 8 * u);
#pragma unroll
              for (int u = 0; u < 4; ++u)
                if (4 * q + u < I) {
                  dmma_m8n8k4(s0[u & 1], s1[u & 1], z[4 * q + u][0], l[u].x);
                  dmma_m8n8k4(s0[u & 1], s1[u & 1], z[4 * q + u][1], l[u].y);
                }
            }
          const double2 r = *reinterpret_cast<const double2*>(inv + 64 * I + 8 * g + 2 * t4);
          dmma_m8n8k4(z[I][0], z[I][1], -(s0[0] + s0[1]), r.x);
          dmma_m8n8k4(z[I][0], z[I][1], -(s1[0] + s1[1]), r.y);
        }
        *reinterpret_cast<double2*>(LiT + (long long)(8 * J + g) * ld + 8 * I + 2 * t4) = make_double2(z[I][0], z[I][1]);
      }
    }
  }
  __syncthreads();
}

// H0' = L^-1 H0 L^-T, one warp per block row: U = L^-1 H0 as tensor-core
// accumulators for all columns, which are then the A operand of U L^-T (blocks on
// and below the diagonal, written to both triangles so that H0' is exactly
// symmetric).
template <int KIND>
__device__ __noinline__ void scc_h0(const SccArgs& A) {
  constexpr int NT = kSccKinds[KIND].nt, NW = NT / 32, P = kSccKinds[KIND].p, NB = P / 8;
  const CtaView v = cta_view(A);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, g = lane >> 2, t4 = lane & 3;
  const int N = v.s.N, ld = v.s.ld, nt = ld >> 3;
  const double* __restrict__ H0 = A.B.H0 + v.s.mo;
  const double* __restrict__ LiT = v.w.LiT;
  double* __restrict__ Hp = v.w.Hp;
  for (int I0 = wid; I0 < nt; I0 += NW) {
    const int I = nt - 1 - I0;  // the longest rows first
    double u[NB][2];
#pragma unroll
    for (int t = 0; t < NB; ++t) u[t][0] = u[t][1] = 0.0;
#pragma unroll 2
    for (int k0 = 0; k0 < 8 * I + 8; k0 += 4) {
      const int k = k0 + t4;
      const double a = LiT[(long long)k * ld + 8 * I + g];
      const double* h = H0 + (long long)min(k, N - 1) * N;
#pragma unroll
      for (int t = 0; t < NB; ++t)
        if (t < nt) {
          const int j = 8 * t + g;
          dmma_m8n8k4(u[t][0], u[t][1], a, (k < N && j < N) ? h[j] : 0.0);
        }
    }
    for (int J = 0; J <= I; ++J) {
      double d0[2] = {0.0, 0.0}, d1[2] = {0.0, 0.0};
#pragma unroll
      for (int t = 0; t < NB; ++t)
        if (t <= J) {
          const double* b = LiT + (long long)(8 * t + 2 * t4) * ld + 8 * J + g;
          dmma_m8n8k4(d0[0], d1[0], u[t][0], b[0]);
          dmma_m8n8k4(d0[1], d1[1], u[t][1], b[ld]);
        }
      const int i = 8 * I + g, j = 8 * J + 2 * t4;
#pragma unroll
      for (int c = 0; c < 2; ++c)
        if (i < N && j + c <= i) {
          const double h = c ? d1[0] + d1[1] : d0[0] + d0[1];
          Hp[(long long)i * ld + j + c] = h;
          Hp[(long long)(j + c) * ld + i] = h;
        }
    }
  }
  __syncthreads();
}

// (1) shell potential from the input charges.
template <int KIND>
__device__ __noinline__ void scc_potential(const SccArgs& A) {
  CtaView v = cta_view(A);
  stage_potential<kSccKinds[KIND].nt>(A.B, A.M, v.c, v.w, v.vao);
}

// Level shift F += b (S - S P_prev S / 2) (src/electronic.rs:2125-2137); in the
// orthonormal basis F' += b (I - Z f Z^T / 2) with the previous iteration's
// eigenvectors Z and occupations f.
template <int KIND>
__device__ __noinline__ void scc_level_shift(const SccArgs& A, double lshift) {
  constexpr int NT = kSccKinds[KIND].nt;
  const CtaView v = cta_view(A);
  const int N = v.s.N, ld = v.s.ld, nocc = v.s.nocc;
  const double *Z = v.w.Z, *occ = v.occ;
  double* F = v.w.F;
  for (long long idx = threadIdx.x; idx < (long long)N * N; idx += NT) {
    const int i = (int)(idx / N), j = (int)(idx % N);
    if (j > i) continue;
    double sp = 0.0;
    for (int k = 0; k < nocc; ++k) sp += occ[k] * Z[(long long)i * ld + k] * Z[(long long)j * ld + k];
    const double val = lshift * ((i == j ? 1.0 : 0.0) - 0.5 * sp);
    F[(long long)i * ld + j] += val;
    if (i != j) F[(long long)j * ld + i] += val;
  }
  __syncthreads();
}

// (4) eigenvalues the occupations need and (5) the occupations
// (src/electronic.rs:3815-3921); when the known eigenvalues do not decide them,
// all eigenvalues and once more.  Also |T|_1 and the count of orbitals with
// occupation above 1e-30 (beyond which they do not matter at FP64 resolution).
// The marks: eigenvalues, occupations.
template <int KIND>
__device__ __noinline__ void scc_occupations(const SccArgs& A, StageClock* clk) {
  constexpr int NT = kSccKinds[KIND].nt;
  const CtaView v = cta_view(A);
  SccShared& sh = v.sh;
  MolState& s = v.s;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, N = s.N;
  const double *d = v.d, *e = v.e;
  double gl = INFINITY, gu = -INFINITY, onenrm = 0.0, emax2 = 0.0;
#pragma unroll 1
  for (int i = tid; i < N; i += NT) {
    const double off = (i > 0 ? fabs(e[i - 1]) : 0.0) + (i < N - 1 ? fabs(e[i]) : 0.0);
    gl = fmin(gl, d[i] - off);
    gu = fmax(gu, d[i] + off);
    onenrm = fmax(onenrm, fabs(d[i]) + off);
    if (i < N - 1) {
      v.esq[i] = e[i] * e[i];
      emax2 = fmax(emax2, v.esq[i]);
    }
  }
  {
    double v4[4] = {-gl, gu, onenrm, emax2};
    block_maxs<4>(v4, sh.red);
    gl = -v4[0];
    gu = v4[1];
    onenrm = v4[2];
    emax2 = v4[3];
  }
  const double pivmin = DBL_MIN * fmax(1.0, emax2);
  {
    const double span = gu - gl;
    gl -= 2.1 * DBL_EPSILON * fabs(gl) + 4.0 * DBL_EPSILON * span + pivmin;
    gu += 2.1 * DBL_EPSILON * fabs(gu) + 4.0 * DBL_EPSILON * span + pivmin;
  }
  const double nelec = s.nelec, kt = s.kt;
  const int nwarm = s.iter > 1 ? s.nneed : 0;  // from the previous iteration's eigenvalues once this rung has one
  int nneed = s.nneed0;
  for (int attempt = 0; attempt < 2; ++attempt) {
    eigenvalues<NT>(d, v.esq, N, nneed, attempt == 0 ? nwarm : 0, gl, gu, pivmin, 4.0 * DBL_EPSILON * onenrm, v.eps, v.occ,
                    v.pop);
    clk->mark(kStEigval);
    if (s.spin) {
      spin_channel_occupations<NT>(v.eps, N, nneed, s.nalpha, s.nbeta, kt, v.occ, v.pop, sh);
    } else if (kt > 0.0 && nelec > 0.0 && nelec < 2.0 * N) {
      double fm, ft;
      bool amb;
      fermi_cta<NT, 2>(v.eps, N, nneed, nelec, kt, v.occ, sh, fm, ft, amb);
      if (tid == 0) {
        sh.scal[1] = fm;
        sh.scal[2] = ft;
        sh.iscal[2] = amb ? 1 : 0;
      }
    } else if (wid == 0) {  // aufbau and the empty / full limits
      double fm, ft;
      bool amb;
      fermi_warp<2>(v.eps, N, nneed, nelec, kt, v.occ, fm, ft, amb);
      if (lane == 0) {
        sh.scal[1] = fm;
        sh.scal[2] = ft;
        sh.iscal[2] = amb ? 1 : 0;
      }
    }
    __syncthreads();
    clk->mark(kStFermi);
    if (!sh.iscal[2] || nneed == N) break;
    nneed = N;
  }
  int nocc_loc = 0;
#pragma unroll 1
  for (int i = tid; i < N; i += NT)
    if ((i < nneed || i == N - 1) && v.occ[i] > 1e-30) nocc_loc = max(nocc_loc, i + 1);
  nocc_loc = __reduce_max_sync(0xffffffffu, nocc_loc);
  if (lane == 0) sh.first[0][wid] = nocc_loc;
  __syncthreads();
  int nocc = 0;
#pragma unroll
  for (int q = 0; q < NT / 32; ++q) nocc = max(nocc, sh.first[0][q]);
  if (tid == 0) {
    s.mu = sh.scal[1];
    s.ts = sh.scal[2];
    s.nneed = nneed;
    s.nocc = nocc;
    s.onenrm = onenrm;
  }
  __syncthreads();
}

// Occupied eigenvectors of a cluster of eigenvalues j..jend-1, or of one that
// the twisted factorisation did not settle: inverse iteration with partial
// pivoting, modified Gram-Schmidt inside the cluster, one thread.
__device__ __noinline__ void inverse_iteration(const double* d, const double* e, int N, int ld, const double* eps, int j,
                                               int jend, double onenrm, double* iw, double* Z) {
  const double tiny = DBL_EPSILON * fmax(onenrm, 1e-300);
  double* ws = iw + j;  // column j of the interleaved factor arrays
  double lam_prev = -INFINITY;
  for (int jj = j; jj < jend; ++jj) {
    double lam = eps[jj];
    const double pert = 10.0 * DBL_EPSILON * fmax(fabs(lam), onenrm);
    if (jj > j && lam - lam_prev < pert) lam = lam_prev + pert;
    lam_prev = lam;
    double* x = Z + jj;  // column jj, stride ld
    if (jend - j == 1) {
      // the start vector's forward elimination runs with the factorisation, the
      // two solves are not normalised in between (growth below 1e40), and the
      // second one returns |x|^2
      const double cur = tri_factor_rhs(d, e, N, lam, tiny, ws, ld, x, ld, (unsigned)jj);
      tri_back(ws, N, ld, x, ld, cur);
      const double nrm = tri_solve(ws, N, ld, x, ld);
      const double inv = 1.0 / sqrt(fmax(nrm, 1e-300));
      for (int i = 0; i < N; ++i) x[(long long)i * ld] *= inv;
      continue;
    }
    tri_factor(d, e, N, lam, tiny, ws, ld);
    for (int i = 0; i < N; ++i) x[(long long)i * ld] = hash_unit(i, jj) + 1e-3;
    const int nit = 4;
    for (int it = 0; it < nit; ++it) {
      tri_solve(ws, N, ld, x, ld);
      for (int q = j; q < jj; ++q) {
        double dot = 0.0;
        for (int i = 0; i < N; ++i) dot += Z[(long long)i * ld + q] * x[(long long)i * ld];
        for (int i = 0; i < N; ++i) x[(long long)i * ld] -= dot * Z[(long long)i * ld + q];
      }
      double nrm = 0.0;
      for (int i = 0; i < N; ++i) nrm += x[(long long)i * ld] * x[(long long)i * ld];
      const double inv = 1.0 / sqrt(fmax(nrm, 1e-300));
      for (int i = 0; i < N; ++i) x[(long long)i * ld] *= inv;
    }
  }
}

// Eigenvector of an isolated eigenvalue lam of the tridiagonal (d, e) by one twisted
// factorisation (Parlett & Dhillon, "Fernando's solution to Wilkinson's problem", Linear
// Algebra Appl. 267, 1997) and one step of inverse iteration with its factors, by a pair
// of threads: T - lam = N_r D_r N_r^T with the pivots D+ from the top (thread `top`), D-
// from the bottom (the other) and gamma_r = D+_r + D-_r - (d_r - lam) in the row r where
// |gamma| is smallest.  N_r^T z = e_r (z_r = 1, z_{i-1} = -(e_{i-1} / D+_{i-1}) z_i upward
// and z_{i+1} = -(e_i / D-_{i+1}) z_i downward) solves (T - lam) z = gamma_r e_r, which
// leaves in z a part (error of lam) / gap of the neighbouring vectors, and so that much
// overlap of two vectors: 5e-12 at 128 AOs, 4e-11 at 2400.  The second solve squares it:
//   N_r y = z                 from both ends to r, where y_r = |z|^2,
//   N_r^T x = gamma_r D_r^-1 y from r to both ends, x_r = y_r / |z|^2 (scaled to 1),
// multiplied through by gamma_r, so that a gamma_r of zero needs no guard (x is z then).
// With the reciprocals of the pivots kept, both sweeps are multiply-adds; the chain of
// divides of the factorisation is the time.  (A Rayleigh quotient for lam and a second
// factorisation instead made lam better but squared nothing: 4e-11 at 2400 AOs.)
//   fac  five arrays `plane` apart: D+, then 1 / D and e / D (what couples a row to the next one
//        towards r) from the top and from the bottom; x the vector, up to the factor returned;
//        row i of each at [i * ld]
//   pa, pb, pc  a word each that the pair shares
// on: the pair has a column; every thread of the CTA calls (seven barriers).  Returns
// 1 / |x| in the top thread, or 0 where gamma_r is larger than the rounding of lam
// (limit) explains.  The lanes of a warp are at the same row in every sweep (their columns are
// side by side), U rows at a time loaded before the first of them is worked on.
template <int U>
__device__ __forceinline__ double twisted_vector(const double* d, const double* e, int N, double lam, double tiny,
                                                 double limit, bool on, bool top, double* __restrict__ fac,
                                                 long long plane, double* __restrict__ x, int ld, double* pa, double* pb,
                                                 double* pc) {
  double* __restrict__ dp = fac;
  double* __restrict__ rc = fac + (top ? 1 : 3) * plane;  // the thread's 1 / D and e / D
  double* __restrict__ cl = rc + plane;
  if (on) {
    // step s: row s from the top, N - 1 - s from the bottom
    const double* ep = top ? e : e + N - 2;
    const double* np = top ? d + 1 : d + N - 2;
    const int inc = top ? 1 : -1, step = inc * ld;
    double D = (top ? d[0] : d[N - 1]) - lam;
    int o = top ? 0 : (N - 1) * ld;
#pragma unroll 4
    for (int s = 0; s < N - 1; ++s, o += step, ep += inc, np += inc) {
      const double ei = *ep, dn = *np - lam;
      if (fabs(D) < tiny) D = D >= 0.0 ? tiny : -tiny;
      const double q = 1.0 / D, l = ei * q;
      if (top) dp[o] = D;
      rc[o] = q;
      cl[o] = l;
      D = dn - ei * l;
    }
    if (top) dp[o] = D;
  }
  __syncthreads();
  double best = INFINITY;  // the smallest gamma_i = D+_i - e_i (e_i / D-_{i+1}) of the thread's half of the rows
  int at = 0;
  if (on) {
    const double* cb = fac + 4 * plane;
    const int i0 = top ? 0 : N / 2, i1 = top ? N / 2 : N;
#pragma unroll 8
    for (int i = i0; i < i1; ++i) {
      double g = dp[i * ld];
      if (i < N - 1) g -= e[i] * cb[(i + 1) * ld];
      if (fabs(g) < fabs(best)) {
        best = g;
        at = i;
      }
    }
    if (!top) {
      *pa = best;
      *pb = (double)at;
    }
  }
  __syncthreads();
  if (on && top) {
    if (fabs(*pa) < fabs(best))
      best = *pa;
    else
      *pb = (double)at;
  }
  __syncthreads();
  const int r = on ? (int)*pb : 0;
  // Outward sweeps (from r to the thread's end) visit row N - 2 - s or s + 1 at step s and work from
  // step s_out on, inward ones row s or N - 1 - s before step s_in.
  const int s_out = top ? N - 1 - r : r, s_in = top ? r : N - 1 - r;
  const int o_out = top ? (N - 2) * ld : ld, o_in = top ? 0 : (N - 1) * ld, away = top ? -ld : ld;
  double nrm = top ? 1.0 : 0.0;
  if (on) {
    double z = 1.0;
    if (top) x[r * ld] = 1.0;
    auto row = [&](bool act, int o, double l) {
      if (act) {
        z *= -l;
        x[o] = z;
        nrm = fma(z, z, nrm);
      }
    };
    int s = 0, o = o_out;
    for (; s + U <= N - 1; s += U, o += U * away) {
      double lv[U];
#pragma unroll
      for (int q = 0; q < U; ++q) lv[q] = cl[o + q * away];
#pragma unroll
      for (int q = 0; q < U; ++q) row(s + q >= s_out, o + q * away, lv[q]);
    }
    for (; s < N - 1; ++s, o += away) row(s >= s_out, o, cl[o]);
    if (!top) *pc = nrm;
  }
  __syncthreads();
  bool good = false;
  double w = 0.0, g = 0.0;
  if (on && top) {
    nrm += *pc;
    good = fabs(best) <= limit * nrm && nrm < 1e200;
    w = 1.0 / nrm;
    g = best * w;
    *pa = g;
    *pb = w;
  }
  __syncthreads();
  if (on) {
    if (!top) {  // (the top thread does not look at pa again before its partner writes it)
      g = *pa;
      w = *pb;
    }
    double y = 0.0, l = 0.0;  // of the row before, and what couples it to this one
    auto row = [&](bool act, int o, double zi, double li, double ri) {
      if (act) {
        y = fma(-l, y, zi);
        l = li;
        x[o] = (g * ri) * y;
      }
    };
    int s = 0, o = o_in;
    for (; s + U <= N - 1; s += U, o -= U * away) {
      double xv[U], lv[U], rv[U];
#pragma unroll
      for (int q = 0; q < U; ++q) {
        xv[q] = x[o - q * away];
        lv[q] = cl[o - q * away];
        rv[q] = rc[o - q * away];
      }
#pragma unroll
      for (int q = 0; q < U; ++q) row(s + q < s_in, o - q * away, xv[q], lv[q], rv[q]);
    }
    for (; s < N - 1; ++s, o -= away) row(s < s_in, o, x[o], cl[o], rc[o]);
    *(top ? pc : pa) = l * y;
  }
  __syncthreads();
  if (on) {
    double v = w * ((1.0 - *pc) - *pa);
    nrm = top ? v * v : 0.0;
    if (top) x[r * ld] = v;
    auto row = [&](bool act, int o, double wi, double li) {
      if (act) {
        v = fma(-li, v, wi);
        x[o] = v;
        nrm = fma(v, v, nrm);
      }
    };
    int s = 0, o = o_out;
    for (; s + U <= N - 1; s += U, o += U * away) {
      double xv[U], lv[U];
#pragma unroll
      for (int q = 0; q < U; ++q) {
        xv[q] = x[o + q * away];
        lv[q] = cl[o + q * away];
      }
#pragma unroll
      for (int q = 0; q < U; ++q) row(s + q >= s_out, o + q * away, xv[q], lv[q]);
    }
    for (; s < N - 1; ++s, o += away) row(s >= s_out, o, x[o], cl[o]);
    if (!top) *pb = nrm;
  }
  __syncthreads();
  if (!on || !top || !good) return 0.0;
  nrm += *pb;
  return nrm > 0.0 && nrm < 1e300 ? 1.0 / sqrt(nrm) : 0.0;
}

// (6) occupied eigenvectors of the tridiagonal, columns of Z up to the factors
// scale[j] (in v.pop): twisted_vector for the eigenvalues farther than 1e-5 |T|_1 from
// their neighbours, a pair of threads each; clusters, and a column that it does not
// settle, by inverse iteration (a pivoted factorisation and two solves, five dependent
// passes over global memory, 147k cycles at N = 128, against 30k for the twisted
// factorisation with its first solve; the second solve adds 1.5% to the SCC at 128 AOs
// and 2% to the 4096-molecule batch).
template <int KIND>
__device__ __noinline__ void scc_vectors(const SccArgs& A) {
  constexpr int NT = kSccKinds[KIND].nt, HALF = NT / 2;
  const CtaView v = cta_view(A);
  const int tid = threadIdx.x, N = v.s.N, ld = v.s.ld, nocc = v.s.nocc;
  const double *d = v.d, *e = v.e, *eps = v.eps;
  const double onenrm = v.s.onenrm, ortol = 1e-5 * onenrm, tiny = DBL_EPSILON * fmax(onenrm, 1e-300);
  double* Z = v.w.Z;
  const long long n2 = (long long)ld * ld;
  const bool top = tid < HALF;
  for (int j0 = 0; j0 < nocc; j0 += HALF) {
    const int j = j0 + (top ? tid : tid - HALF);
    const bool col = j < nocc;
    const bool first = col && (j == 0 || eps[j] - eps[j - 1] > ortol);
    const bool single = first && (j + 1 >= nocc || eps[j + 1] - eps[j] > ortol);
    const int jc = col ? j : 0;
    // (tau and e^2 have served; the words are the pair's)
    const double scale = twisted_vector<8>(d, e, N, eps[jc], tiny, 64.0 * DBL_EPSILON * onenrm, single, top, v.w.iw + jc,
                                           n2, Z + jc, ld, v.pop + jc, v.esq + jc, v.tau + jc);
    if (top && first) {
      if (scale > 0.0) {
        v.pop[j] = scale;
      } else {
        int jend = j + 1;
        while (jend < nocc && eps[jend] - eps[jend - 1] <= ortol) ++jend;
        inverse_iteration(d, e, N, ld, eps, j, jend, onenrm, v.w.iw, Z);
        for (int q = j; q < jend; ++q) v.pop[q] = 1.0;
      }
    }
    __syncthreads();
  }
}

// (9) populations, output charges, energies and the convergence test.
template <int KIND, bool Robust>
__device__ __noinline__ void scc_energy(const SccArgs& A, double lshift) {
  constexpr int NT = kSccKinds[KIND].nt, NW = NT / 32;
  CtaView v = cta_view(A);
  MolState& s = v.s;
  const int tid = threadIdx.x, N = s.N, ld = s.ld;
#pragma unroll 1
  for (int i = tid; i < N; i += NT) {
    double p = 0.0;
#pragma unroll
    for (int q = 0; q < NW; ++q) p += v.w.popw[(long long)q * ld + i];
    v.pop[i] = p;
  }
  __syncthreads();
  double e_el, e2, e3, rms;
  stage_charges_energy<NT>(A.B, A.M, v.c, v.w, v.pop, v.occ, v.eps, v.vao, s.nocc, v.sh, e_el, e2, e3, rms);
  if (Robust && lshift != 0.0) {
    // with a shifted Fock matrix sum(f eps) is not tr(F P): E_el = tr(H0 P) = sum_k f_k z_k^T H0' z_k
    const double *Hp = v.w.Hp, *Z = v.w.Z;
    const int nocc = s.nocc;
    double part = 0.0;
#pragma unroll 1
    for (long long idx = tid; idx < (long long)N * nocc; idx += NT) {
      const int i = (int)(idx / nocc), k = (int)(idx % nocc);
      double hz = 0.0;
      for (int j = 0; j < N; ++j) hz += Hp[(long long)i * ld + j] * Z[(long long)j * ld + k];
      part += v.occ[k] * Z[(long long)i * ld + k] * hz;
    }
    e_el = block_sum(part, v.sh.red);
  }
  if (tid == 0) {
    const double escc = e_el + e2 + e3 + s.ts;
    const double err = s.have_e ? fabs(escc - s.last_e) : INFINITY;
    s.e_el = e_el;
    s.e2 = e2;
    s.e3 = e3;
    s.rms = rms;
    s.last_e = escc;
    s.have_e = 1;
    s.converged = err < A.opt.energy_tol && rms < A.opt.charge_tol;
  }
  __syncthreads();
}

// (10) charge mixing.
template <int KIND>
__device__ __noinline__ void scc_mix(const SccArgs& A, int broyden, double mixing) {
  CtaView v = cta_view(A);
  SccOptions ro = A.opt;
  ro.broyden = broyden;
  ro.mixing = mixing;
  int bro = v.s.bro_iter;
  __syncthreads();
  stage_mix<kSccKinds[KIND].nt>(ro, v.c, v.w, A.SL.cap, bro, v.sh);
  if (threadIdx.x == 0) v.s.bro_iter = bro;
  __syncthreads();
}

// Results, and the density and energy-weighted density of the last
// diagonalisation (src/linalg.rs:243-273), kept per molecule for the gradient
// kernel: P = C f C^T and W = C f eps C^T on the FP64 tensor cores, 16 x 16 tiles
// on and below the diagonal (eight accumulators share four operand loads)
// written to both triangles.
template <int KIND, bool Robust>
__device__ __noinline__ void scc_finish(const SccArgs& A, int rung) {
  constexpr int NT = kSccKinds[KIND].nt, NW = NT / 32;
  CtaView v = cta_view(A);
  const Batch& B = A.B;
  MolState& s = v.s;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, g = lane >> 2, t4 = lane & 3;
  const int m = s.m, N = s.N, ld = s.ld, nocc = s.nocc;
  if (!Robust && !s.converged && B.failed && tid == 0) B.failed[atomicAdd(B.queue + 3, 1)] = m;
  if constexpr (Robust) {  // rung-0 molecules keep the 0 the host wrote before the launches
    if (B.rung && tid == 0) B.rung[m] = s.converged ? rung : -1;
  }
  stage_results<NT>(B, v.c, v.w, s.iter, s.converged != 0, s.e_el, s.e2, s.e3, s.ts, s.mu);
  if (B.orb_eps) {  // orbital energies (NaN where the eigensolver did not need them) and occupations
    const int ao0 = B.ao_off[m];
#pragma unroll 1
    for (int i = tid; i < N; i += NT) {
      B.orb_eps[ao0 + i] = (i < s.nneed || i == N - 1) ? v.eps[i] : __longlong_as_double(0x7ff8000000000000LL);
      B.orb_occ[ao0 + i] = v.occ[i];
    }
  }
  const double* __restrict__ Ct = v.w.Ct;
  double* __restrict__ Pm = B.P + s.mo;
  double* __restrict__ Wm = B.W + s.mo;
  const int nt = ld >> 3, nt2 = (nt + 1) >> 1;
  for (int tile = wid; tile < nt2 * (nt2 + 1) / 2; tile += NW) {
    int I = 0;
    while ((I + 1) * (I + 2) / 2 <= tile) ++I;
    const int J = tile - I * (I + 1) / 2;
    const bool i1 = 2 * I + 1 < nt, j1 = 2 * J + 1 < nt;
    double p[2][2][2], q[2][2][2];
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
      for (int b = 0; b < 2; ++b) p[a][b][0] = p[a][b][1] = q[a][b][0] = q[a][b][1] = 0.0;
#pragma unroll 2
    for (int k0 = 0; k0 < nocc; k0 += 4) {
      const int k = k0 + t4;
      const bool kin = k < nocc;
      const double f = kin ? v.occ[k] : 0.0, ek = kin ? v.eps[k] : 0.0;
      const double* ck = Ct + (long long)(kin ? k : 0) * ld + g;
      double a[2], b[2];
      a[0] = f * ck[16 * I];
      a[1] = i1 ? f * ck[16 * I + 8] : 0.0;
      b[0] = ck[16 * J];
      b[1] = j1 ? ck[16 * J + 8] : 0.0;
#pragma unroll
      for (int x = 0; x < 2; ++x)
#pragma unroll
        for (int y = 0; y < 2; ++y) {
          dmma_m8n8k4(p[x][y][0], p[x][y][1], a[x], b[y]);
          dmma_m8n8k4(q[x][y][0], q[x][y][1], a[x] * ek, b[y]);
        }
    }
#pragma unroll
    for (int x = 0; x < 2; ++x)
#pragma unroll
      for (int y = 0; y < 2; ++y)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const int i = 16 * I + 8 * x + g, j = 16 * J + 8 * y + 2 * t4 + c;
          if (i < N && j <= i) {
            Pm[(long long)i * N + j] = p[x][y][c];
            Pm[(long long)j * N + i] = p[x][y][c];
            Wm[(long long)i * N + j] = q[x][y][c];
            Wm[(long long)j * N + i] = q[x][y][c];
          }
        }
  }
  __syncthreads();
}

template <int KIND, bool Robust>
__device__ __forceinline__ void scc_molecule(const SccArgs& A, int m) {
  constexpr int NT = kSccKinds[KIND].nt, P = kSccKinds[KIND].p, NW = NT / 32;
  extern __shared__ __align__(16) unsigned char smraw[];
  MolState& s = reinterpret_cast<SccCta*>(smraw)->s;
  const int tid = threadIdx.x;
  StageClock clk(A.B.stage_cycles);
  scc_begin<KIND>(A, m);
  scc_cholesky<KIND>(A);
  if (s.status != kOk) {
    if (tid == 0) {
      A.B.status[m] = s.status;
      A.B.iterations[m] = 0;
    }
    return;
  }
  clk.mark(kStChol);
  scc_inverse<KIND>(A);
  clk.mark(kStLinv);
  scc_h0<KIND>(A);
  // The reference's fallback ladder (src/electronic.rs:1390-1447): rung 0 is
  // the requested options (the main kernel); rungs 1-3 (the Robust kernel,
  // for molecules rung 0 left unconverged) restart from the initial charges
  // with linear mixing 0.2 and a level shift of max(requested, 0.2 Eh), then
  // 0.1 / max(requested, 0.1), then Broyden at T_el >= 3000 K without shift.
  // A requested level shift sends every molecule to the Robust kernel, which
  // then starts at rung 0 (the main kernel carries no level-shift code).
  const int rung_first = Robust ? (A.opt.level_shift != 0.0 ? 0 : 1) : 0, rung_last = Robust ? 3 : 0;
  int rung_used = rung_first;  // the rung whose SCC converged (reported by the ladder kernel)
  for (int rung = rung_first; rung <= rung_last && !s.converged; ++rung) {
    rung_used = rung;
    int broyden = A.opt.broyden, max_scc = A.opt.max_scc;
    double mixing = A.opt.mixing, etemp = A.opt.etemp, lshift = Robust ? A.opt.level_shift : 0.0;
    if (rung == 1 || rung == 2) {
      broyden = 0;
      mixing = rung == 1 ? 0.20 : 0.10;
      lshift = fmax(A.opt.level_shift, rung == 1 ? 0.20 : 0.10);
      max_scc = max(A.opt.max_scc, 800);
    } else if (rung == 3) {
      etemp = fmax(A.opt.etemp, 3000.0);
      max_scc = max(A.opt.max_scc, kLastRungScc);
      lshift = 0.0;
    }
    __syncthreads();
    {
      const CtaView v = cta_view(A);
#pragma unroll 1
      for (int i = tid; i < s.nsh; i += NT) v.w.qin[i] = A.B.init_q ? A.B.init_q[s.sh0 + i] : 0.0;
    }
    if (tid == 0) {
      s.kt = fmax(etemp, 0.0) * kBoltzmann;
      s.bro_iter = 0;
      s.have_e = 0;
      s.last_e = 0.0;
      s.iter = 1;
    }
    __syncthreads();
    clk.mark(kStPrologue);
    for (int iter = 1; iter <= max_scc; ++iter) {
      scc_potential<KIND>(A);
      {  // (2) F' = H0' - 1/2 (M + M^T), M = L^-1 diag(v) L
        const CtaView v = cta_view(A);
        fock_build<NW>(v.w.L, v.w.LiT, v.w.Hp, s.ld, s.vec_at + 6 * s.N, s.N, v.w.F, s.ld);
      }
      __syncthreads();
      if (Robust && lshift != 0.0 && iter > 1) scc_level_shift<KIND>(A, lshift);
      clk.mark(kStFock);
      {  // (3) Householder reduction: reflectors in the rows of w.V, their WY factors in its scratch
        const CtaView v = cta_view(A);
        const int N = s.N, ldv = refl_ld(N);
        if (P == 128 && N <= 96)  // every slot in registers
          tridiag_cta<NT, P == 128 ? 96 : P>(v.w.F, s.ld, N, s.vec_at, v.w.V, ldv, s.tri_at);
        else
          tridiag_cta<NT, P>(v.w.F, s.ld, N, s.vec_at, v.w.V, ldv, s.tri_at);
        wy_factors<NW>(v.w.V, ldv, N, s.vec_at + 2 * N, s.tri_at);
      }
      clk.mark(kStTridiag);
      scc_occupations<KIND>(A, &clk);
      scc_vectors<KIND>(A);
      clk.mark(kStInvIter);
      {  // (7) back-transformation, (8) C = L^-T Z and the AO populations
        const CtaView v = cta_view(A);
        const int N = s.N, ld = s.ld;
        occupied_orbitals<NW, P>(v.w.V, refl_ld(N), s.tri_at, N, v.w.Z, ld, s.nocc, s.vec_at + 4 * N, s.vec_at + 5 * N,
                                 v.w.L, v.w.LiT, ld, v.w.Ct, v.w.popw, Robust ? v.w.Z : nullptr);
      }
      __syncthreads();
      clk.mark(kStPop);
      scc_energy<KIND, Robust>(A, lshift);
      clk.mark(kStEnergy);
      if (s.converged || iter == max_scc) break;
      scc_mix<KIND>(A, broyden, mixing);
      if (tid == 0) s.iter = iter + 1;
      __syncthreads();
      clk.mark(kStMix);
    }
  }
  scc_finish<KIND, Robust>(A, rung_used);
  clk.mark(kStFinal);
}

// Persistent SCC kernel.  Robust = false: molecules q_begin..q_end of the
// processing order (rung 0 of the fallback ladder); Robust = true: the
// molecules the rung-0 launches left unconverged (rungs 1-3).
template <int KIND, bool Robust>
__global__ void __launch_bounds__(kSccKinds[KIND].nt, kSccKinds[KIND].ctas)
    scc_kernel(const __grid_constant__ SccArgs A) {
  __shared__ int next;
  const int nfailed = Robust ? A.B.queue[3] : 0;  // written by the rung-0 launches before this one
  for (;;) {
    if (threadIdx.x == 0) next = Robust ? atomicAdd(A.B.queue + 2, 1) : A.SL.q_begin + atomicAdd(A.SL.counter, 1);
    __syncthreads();
    const int idx = next;
    __syncthreads();
    int m;
    if (Robust) {
      if (idx >= nfailed) break;
      m = A.B.failed[idx];
    } else {
      if (idx >= A.SL.q_end) break;
      m = A.B.order[idx];
      if (A.B.status[m] != kOk) continue;  // rejected during setup
    }
    scc_molecule<KIND, Robust>(A, m);
  }
}

// ============================================================ large molecules
// Molecules too large for one SM run on many SMs: the kernels of wide.cuh
// (included at the end of this file) share the stage functions above.

__host__ __device__ inline size_t dense_table_bytes(int maxnsh, int maxn, int maxnat) {
  return ((size_t)4 * scc_ints(maxnsh, maxn, maxnat) + 15) & ~(size_t)15;
}

struct DenseTables {
  int *sh_atom, *sh_k, *sh_ao0, *ao_sh, *atom_sh;
};
__device__ DenseTables dense_tables(unsigned char* raw, int maxnsh, int maxn) {
  DenseTables t;
  t.sh_atom = (int*)raw;
  t.sh_k = t.sh_atom + maxnsh;
  t.sh_ao0 = t.sh_k + maxnsh;
  t.ao_sh = t.sh_ao0 + maxnsh;
  t.atom_sh = t.ao_sh + maxn;
  return t;
}

long long scc_workspace_doubles(int maxn, int maxnsh, int cap, int maxnat) {
  return cta_ws_size(maxn, maxnsh, cap, maxnat);
}

// The kernel a molecule of N AOs runs on: the first whose registers hold its
// matrix (the last one takes what a raised large-molecule threshold leaves).
int scc_kind(int N) { return N <= kSccKinds[0].p ? 0 : (N <= kSccKinds[1].p ? 1 : 2); }

// Dynamic shared memory of a launch: index tables, N-vectors and the scratch of
// the reduction.
size_t scc_smem_bytes(int kind, int maxnsh, int maxn, int maxnat) {
  const size_t tri = kind == 0   ? TriShape<kSccKinds[0].nt, kSccKinds[0].p>::kDoubles
                     : kind == 1 ? TriShape<kSccKinds[1].nt, kSccKinds[1].p>::kDoubles
                                 : TriShape<kSccKinds[2].nt, kSccKinds[2].p>::kDoubles;
  return scc_smem_fixed(maxnsh, maxn, maxnat) + sizeof(double) * tri;
}

template <int KIND, bool Robust>
static cudaError_t launch_scc_kind(int grid, size_t smem, cudaStream_t st, const Batch& B, const Model& M,
                                   const SccOptions& opt, const SccLaunch& SL) {
  cudaError_t e = cudaFuncSetAttribute(scc_kernel<KIND, Robust>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  scc_kernel<KIND, Robust><<<grid, kSccKinds[KIND].nt, smem, st>>>(SccArgs{B, M, opt, SL});
  return cudaGetLastError();
}

// Host launcher of one size class.
cudaError_t launch_scc(int kind, int grid, size_t smem, cudaStream_t st, const Batch& B, const Model& M,
                       const SccOptions& opt, const SccLaunch& SL) {
  if (kind == 0) return launch_scc_kind<0, false>(grid, smem, st, B, M, opt, SL);
  if (kind == 1) return launch_scc_kind<1, false>(grid, smem, st, B, M, opt, SL);
  if (kind == 2) return launch_scc_kind<2, false>(grid, smem, st, B, M, opt, SL);
  return cudaErrorInvalidValue;
}

// Host launcher of the fallback-ladder kernel (rungs 1-3 for the molecules
// listed in B.failed; returns at once when the list is empty).
cudaError_t launch_scc_robust(int kind, int grid, size_t smem, cudaStream_t st, const Batch& B, const Model& M,
                              const SccOptions& opt, const SccLaunch& SL) {
  if (kind == 0) return launch_scc_kind<0, true>(grid, smem, st, B, M, opt, SL);
  if (kind == 1) return launch_scc_kind<1, true>(grid, smem, st, B, M, opt, SL);
  if (kind == 2) return launch_scc_kind<2, true>(grid, smem, st, B, M, opt, SL);
  return cudaErrorInvalidValue;
}

}  // namespace gfn1

#include "wide.cuh"
