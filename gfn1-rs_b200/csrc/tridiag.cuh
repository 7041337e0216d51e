// Householder reduction of a symmetric matrix that one CTA keeps on chip.
//
// The reduction reads and updates the whole trailing matrix once per column, so
// what bounds it is where that matrix lives and how many instructions a column
// costs beyond its multiply-adds.  From L1-cached global memory a column of a
// 128 x 128 matrix took 7,000 cycles.  Here the full matrix is spread over the
// threads in cyclic order, element (i, j) in slot (i / TR, j / 8) of thread
// (i % TR, j % 8): the later columns (the ones that stay longest) in registers,
// the first ones, where the registers do not hold them all, in shared memory
// words of the thread's own.  (The lower triangle alone in registers needs a
// third fewer multiply-adds, but sums over both indices: 580 instructions per
// warp and column at N = 128, of which 114 were FP64, and 2,200 cycles.)  A column is
// two phases and two barriers:
//   M  the rank-2 update of the previous column fused with y = A22 x for the
//      unscaled column x; the eight lanes of a row reduce its sum by shuffles.
//      One warp forms the reflector's scalars from |x|^2 meanwhile.
//   C  one thread per entry: with v = x - alpha e_1,
//        A22 v = y - alpha A22 e_1,   v.A22 v = x.y - 2 alpha y_1 + alpha^2 A22_11
//      so that neither waited for alpha (no cancellation: alpha has the opposite
//      sign of x_1); w = beta A22 v - K v, K = beta^2 (v.A22 v) / 2, and the
//      next column of A22 - v w^T - w v^T, which lets the update wait for the
//      next phase M.
// The matrix sits at the end of the P x P slot grid (row N-1 in slot row P-1),
// so that the rows above an N x N matrix are slots already reduced and one
// instantiation serves every N <= P; phase M is instantiated for each number
// of live slot rows, straight-line code without a test per slot.
#pragma once

#include "common.cuh"
#include "orbitals.cuh"

namespace gfn1 {

template <int NT, int P>
struct TriShape {
  static constexpr int TR = NT / 8;               // thread rows; eight thread columns
  static constexpr int NA = P / TR, NB = P / 8;   // slots per thread
  static constexpr int CB = TR / 8;               // slot columns per slot row
  // slot columns in registers (the last ones); the rest in shared memory
  static constexpr int BR = NA * NB <= 36 ? NB : NB / 2;
  static constexpr int BS = NB - BR;
  static constexpr int NW = NT / 32;
  static_assert(P % TR == 0 && P <= NT && BS % 2 == 0, "slot grid");
  // x (two buffers), (v, w) pairs, next column, y, warp sums, scalars; then the slots
  static constexpr int kVec = 6 * P + 2 * NW + 4;
  // ... and afterwards the WY factors of the reflectors, 64 doubles per eight,
  // and the panels of the back-transformation
  static constexpr int kAfter = 8 * P + OrbitalPanels<P>::kDoubles;
  static constexpr int kDoubles = kVec + NA * BS * NT > kAfter ? kVec + NA * BS * NT : kAfter;
};

// Halves the values of a pair across lanes that differ in bit `mask`: the lane
// with the bit clear ends with the sum of `lo`, the other with the sum of `hi`.
__device__ __forceinline__ double pair_reduce(double lo, double hi, bool up, int mask) {
  const double keep = up ? hi : lo, send = up ? lo : hi;
  return keep + __shfl_xor_sync(0xffffffffu, send, mask);
}

template <int NW>
__device__ __forceinline__ double tree_sum(const double* p) {
  if constexpr (NW == 4)
    return (p[0] + p[1]) + (p[2] + p[3]);
  else
    return tree_sum<NW / 2>(p) + tree_sum<NW / 2>(p + NW / 2);
}

template <int NT, int P>
struct TriReg {
  double r[TriShape<NT, P>::NA][TriShape<NT, P>::BR];
};

// Columns k of the slot grid with k / TR == A0 (slot rows and columns before A0 are done).
template <int NT, int P, int A0>
__device__ __forceinline__ void tridiag_phase(TriReg<NT, P>& R, int N, double* d, double* e, double* tau,
                                              double* __restrict__ V, int ldv, double* sm) {
  using TS = TriShape<NT, P>;
  constexpr int TR = TS::TR, NA = TS::NA, NB = TS::NB, NW = TS::NW, BS = TS::BS, B0 = TS::CB * A0;
  constexpr int n = NA - A0;  // live slot rows
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int tc = lane & 7, tr = wid * 4 + (lane >> 3);
  const int off = P - N;
  double* xb = sm;
  double2* vw = reinterpret_cast<double2*>(sm + 2 * P);
  double* xn = sm + 4 * P;
  double* ys = sm + 5 * P;
  double* red = sm + 6 * P;
  double* scal = red + 2 * NW;
  double2* priv = reinterpret_cast<double2*>(sm + TS::kVec) + tid;  // slot pair s at priv[s * NT]
  const int kend = min(TR * (A0 + 1), P - 2);
  for (int k = max(off, TR * A0); k < kend; ++k) {
    const double* x = xb + (k & 1) * P;
    const int k1 = k + 1;
    // ---- phase M
    if (wid == NW - 1) {  // the reflector's scalars
      const double q = tree_sum<NW>(red);
      const double x0 = x[k1];
      double alpha = 0.0, beta = 0.0;
      if (q > 1e-280) {  // below: the column is zero next to any entry that matters
        const double nrm = sqrt(q);
        alpha = x0 >= 0.0 ? -nrm : nrm;
        beta = 1.0 / (q + fabs(x0) * nrm);  // 2 / |v|^2
      }
      if (lane == 0) {
        scal[0] = alpha;
        scal[1] = beta;
        e[k - off] = alpha;
        tau[k - off] = beta;
      }
    }
    double ra[n];
    {
      double vi[n], wi[n];
#pragma unroll
      for (int a = 0; a < n; ++a) {
        const double2 t = vw[tr + TR * (A0 + a)];
        vi[a] = -t.x;
        wi[a] = -t.y;
        ra[a] = 0.0;
      }
      // slot columns in shared memory: a pair's slots are all loaded, and the next
      // pair's are on their way, before any is stored back
      double2 c0, c1, u[n];
      double p0, p1;
      auto cols = [&](int b) {
        c0 = vw[tc + 8 * b];
        c1 = vw[tc + 8 * b + 8];
        p0 = x[tc + 8 * b];
        p1 = x[tc + 8 * b + 8];
      };
      auto slots = [&](int b) {
#pragma unroll
        for (int a = 0; a < n; ++a) u[a] = priv[((A0 + a) * (BS / 2) + b / 2) * NT];
      };
#pragma unroll
      for (int a = 0; a < n; ++a) u[a] = make_double2(0.0, 0.0);
      cols(B0);
      if (B0 < BS) slots(B0);
#pragma unroll
      for (int b = B0; b < NB; b += 2) {
        const double2 t0 = c0, t1 = c1;
        const double x0 = p0, x1 = p1;
        double2 t[n];
#pragma unroll
        for (int a = 0; a < n; ++a) t[a] = u[a];
        if (b + 2 < NB) cols(b + 2);
        if (b + 2 < BS) slots(b + 2);
#pragma unroll
        for (int a = 0; a < n; ++a) {
          if (b < BS) {
            double2 q;
            q.x = fma(wi[a], t0.x, fma(vi[a], t0.y, t[a].x));
            q.y = fma(wi[a], t1.x, fma(vi[a], t1.y, t[a].y));
            ra[a] = fma(q.y, x1, fma(q.x, x0, ra[a]));
            priv[((A0 + a) * (BS / 2) + b / 2) * NT] = q;
          } else {
            double& q = R.r[A0 + a][b - BS < 0 ? 0 : b - BS];
            double& w = R.r[A0 + a][b - BS < 0 ? 0 : b - BS + 1];
            q = fma(wi[a], t0.x, fma(vi[a], t0.y, q));
            w = fma(wi[a], t1.x, fma(vi[a], t1.y, w));
            ra[a] = fma(w, x1, fma(q, x0, ra[a]));
          }
        }
      }
    }
    if (tr == (k1 & (TR - 1))) {  // row (= column) k+1 of the trailing matrix
      if (k1 < TR * (A0 + 1)) {
#pragma unroll
        for (int b = B0; b < NB; ++b) {
          if (b < BS) {
            if ((b & 1) == 0) {
              const double2 u = priv[(A0 * (BS / 2) + b / 2) * NT];
              xn[tc + 8 * b] = u.x;
              xn[tc + 8 * b + 8] = u.y;
            }
          } else {
            xn[tc + 8 * b] = R.r[A0][b - BS < 0 ? 0 : b - BS];
          }
        }
      } else if constexpr (A0 + 1 < NA) {
#pragma unroll
        for (int b = B0 + TS::CB; b < NB; ++b) {
          if (b < BS) {
            if ((b & 1) == 0) {
              const double2 u = priv[((A0 + 1) * (BS / 2) + b / 2) * NT];
              xn[tc + 8 * b] = u.x;
              xn[tc + 8 * b + 8] = u.y;
            }
          } else {
            xn[tc + 8 * b] = R.r[A0 + 1][b - BS < 0 ? 0 : b - BS];
          }
        }
      }
    }
    // y of the rows over their eight lanes, and x.y over the warp (interleaved)
    double xy = 0.0;
#pragma unroll
    for (int a = 0; a < n; ++a) xy = fma(ra[a], x[tr + TR * (A0 + a)], xy);
    constexpr int n1 = (n + 1) / 2, n2 = (n1 + 1) / 2;
    double s1[n1], s2[n2], s3;
#pragma unroll
    for (int q = 0; q < n1; ++q)
      s1[q] = 2 * q + 1 < n ? pair_reduce(ra[2 * q], ra[2 * q + 1 < n ? 2 * q + 1 : 0], tc & 1, 1)
                            : ra[2 * q] + __shfl_xor_sync(0xffffffffu, ra[2 * q], 1);
    xy += __shfl_xor_sync(0xffffffffu, xy, 1);
#pragma unroll
    for (int q = 0; q < n2; ++q)
      s2[q] = 2 * q + 1 < n1 ? pair_reduce(s1[2 * q], s1[2 * q + 1 < n1 ? 2 * q + 1 : 0], tc & 2, 2)
                             : s1[2 * q] + __shfl_xor_sync(0xffffffffu, s1[2 * q], 2);
    xy += __shfl_xor_sync(0xffffffffu, xy, 2);
    if constexpr (n2 == 2)
      s3 = pair_reduce(s2[0], s2[1], tc & 4, 4);
    else
      s3 = s2[0] + __shfl_xor_sync(0xffffffffu, s2[0], 4);
    xy += __shfl_xor_sync(0xffffffffu, xy, 4);
    xy += __shfl_xor_sync(0xffffffffu, xy, 8);
    xy += __shfl_xor_sync(0xffffffffu, xy, 16);
    {  // the row whose sum this lane holds (lanes of an unpaired value hold copies)
      const int u = n2 == 2 ? (tc >> 2) : 0;
      const int q = 2 * u + 1 < n1 ? 2 * u + ((tc >> 1) & 1) : 2 * u;
      const int a = 2 * q + 1 < n ? 2 * q + (tc & 1) : 2 * q;
      ys[tr + TR * (A0 + a)] = s3;
      if (lane == 0) red[NW + wid] = xy;
    }
    __syncthreads();
    // ---- phase C
    if (wid < P / 32) {
      const double alpha = scal[0], beta = scal[1];
      const double y1 = ys[k1], a11 = xn[k1], v1 = x[k1] - alpha;
      const double vav = tree_sum<NW>(red + NW) + alpha * (alpha * a11 - 2.0 * y1);
      const double K = 0.5 * beta * beta * vav;
      const double w1 = beta * (y1 - alpha * a11) - K * v1;
      double v = 0.0, w = 0.0, xnext = 0.0;
      if (tid >= k1) {
        const double col = xn[tid];
        v = tid == k1 ? v1 : x[tid];
        w = beta * (ys[tid] - alpha * col) - K * v;
        const double t = col - (v * w1 + w * v1);
        if (tid == k1)
          d[k1 - off] = t;
        else
          xnext = t;
      }
      vw[tid] = make_double2(v, w);
      xb[((k + 1) & 1) * P + tid] = xnext;
      const double sq = warp_sum(xnext * xnext);
      if (lane == 0) red[wid] = sq;
      // row k of V; the threads above the matrix fill its padding columns
      const int col = tid >= off ? tid - off : N + (off - 1 - tid);
      if (col < ldv) V[(long long)(k - off) * ldv + col] = v;
    }
    __syncthreads();
  }
  if constexpr (A0 + 1 < NA) tridiag_phase<NT, P, A0 + 1>(R, N, d, e, tau, V, ldv, sm);
}

// F: the matrix (both triangles), row-major with leading dimension ldf.  Out: d, e, tau (e[k] = alpha, H_k = I - tau v v^T) and the
// reflectors, row k of V = v_k over columns 0..ldv-1 (zero outside k+1..N-1);
// rows N-2.. up to the next multiple of 16 are zeroed.  ldv <= P.
// d, e, tau: doubles `vec`, `vec` + N and `vec` + 2 N of the dynamic shared memory;
// scratch: TriShape::kDoubles doubles from `scratch`, 16-byte aligned.  They are
// passed as offsets, and the function is kept out of line, so that the compiler
// knows the address space and gives the loops the whole register budget: inlined
// into the SCC kernel they spilled (668k instead of 293k cycles at N = 128).
template <int NT, int P>
__device__ __noinline__ void tridiag_cta(const double* __restrict__ F, int ldf, int N, int vec,
                                         double* __restrict__ V, int ldv, int scratch) {
  extern __shared__ __align__(16) unsigned char smraw[];
  double* d = reinterpret_cast<double*>(smraw) + vec;
  double *e = d + N, *tau = d + 2 * N;
  double* sm = reinterpret_cast<double*>(smraw) + scratch;
  using TS = TriShape<NT, P>;
  constexpr int TR = TS::TR, NA = TS::NA, NB = TS::NB, BS = TS::BS;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int tc = lane & 7, tr = wid * 4 + (lane >> 3);
  const int off = P - N;
  double2* priv = reinterpret_cast<double2*>(sm + TS::kVec) + tid;
  TriReg<NT, P> R;
#pragma unroll
  for (int a = 0; a < NA; ++a) {
    const int i = tr + TR * a - off;
    const double* row = F + (long long)max(i, 0) * ldf + (tc - off);
#pragma unroll
    for (int b = 0; b < NB; b += 2) {
      double2 u = make_double2(0.0, 0.0);
      if (i >= 0) {
        if (tc + 8 * b >= off) u.x = row[8 * b];
        if (tc + 8 * b + 8 >= off) u.y = row[8 * b + 8];
      }
      if (b < BS) {
        priv[(a * (BS / 2) + b / 2) * NT] = u;
      } else {
        R.r[a][b - BS < 0 ? 0 : b - BS] = u.x;
        R.r[a][b - BS < 0 ? 0 : b - BS + 1] = u.y;
      }
    }
  }
  {
    double* red = sm + 6 * P;
    double sq = 0.0;
    if (tid < P) {
      const double x = tid > off ? F[(long long)(tid - off) * ldf] : 0.0;
      sm[(off & 1) * P + tid] = x;
      reinterpret_cast<double2*>(sm + 2 * P)[tid] = make_double2(0.0, 0.0);
      sq = x * x;
      if (tid == off) d[0] = F[0];
    }
    sq = warp_sum(sq);
    if (lane == 0) red[wid] = sq;  // zero for the warps beyond P, whose slots stay zero
  }
  const int nref = max(N - 2, 0), nz = (N + 13) & ~15;
  for (int idx = tid; idx < (nz - nref) * ldv; idx += NT) V[(long long)nref * ldv + idx] = 0.0;
  __syncthreads();
  tridiag_phase<NT, P, 0>(R, N, d, e, tau, V, ldv, sm);
  // the last 2 x 2 block
  if (tid == 0 && N >= 2) e[N - 2] = sm[((P - 2) & 1) * P + P - 1];
  if (tr == TR - 1 && tc == 7) {
    const double2 t = reinterpret_cast<double2*>(sm + 2 * P)[P - 1];
    if (N >= 2) {
      d[N - 1] = R.r[NA - 1][TS::BR - 1] - 2.0 * t.x * t.y;
      tau[N - 2] = 0.0;
    }
    e[N - 1] = 0.0;
    tau[N - 1] = 0.0;
  }
  __syncthreads();
}

}  // namespace gfn1
