// Householder reduction of a matrix that a cluster of C CTAs keeps on chip.
//
// The blocked reduction of the large-molecule path reads its matrix from L2 and
// synchronises its CTAs through global memory twice a column; at 768 AOs and 18
// CTAs a column took 28,000 cycles, of which the arithmetic is under 2,000.  A
// cluster of 16 SMs holds a 768 x 768 matrix in registers and shared memory, its
// barrier is a hardware one and its exchange goes through distributed shared
// memory.  The scheme is the one of tridiag.cuh with the rows dealt out to the
// CTAs in blocks of eight: row 8 (C a + r) + t is slot row a of thread row t of
// CTA r; column j is slot column j / 32 of thread column j % 32.  Per column
//   M  each CTA: the rank-2 update of the previous column fused with y = A22 x for
//      its rows; every row's y and its entry of the next column go to all CTAs,
//      with the CTA's share of x.y;
//   one cluster barrier;
//   C  every CTA forms w, the next column and |x|^2 for all rows from the gathered
//      values, the same in each, so that nothing else is exchanged.
// Measured on B200 (blocked reduction before): one matrix of 320 AOs 3.6 -> 0.47 ms
// (2,800 cycles a column: 600 the products, 580 the sums over lanes and warps, 1,150
// the exchange with its barrier, 730 phase C), eight of 768 AOs 10.1 -> 3.9 ms (4,980
// cycles a column, 1,890 of them the products).  The latencies of a column bound it.
// Eight CTAs up to 384 AOs: 15 such clusters run at once (7 of 16 CTAs), and a column
// is cheaper (2,996 cycles at 384 AOs, 3,209 at 385 with 16); 768 AOs is what the
// registers and the shared memory of 16 SMs hold.
#pragma once

#include <cooperative_groups.h>

#include "common.cuh"
#include "tridiag.cuh"

namespace gfn1 {

template <int C>
struct ClusterShape {
  static constexpr int NT = 256, NW = NT / 32;
  static constexpr int TR = 8, TC = 32;        // thread rows and columns of a CTA
  static constexpr int NA = 6;                 // slot rows
  static constexpr int P = TR * NA * C;        // largest matrix: 384 (C = 8), 768 (C = 16)
  static constexpr int NB = P / TC;            // slot columns: 12, 24
  static constexpr int CB = TR * C / TC;       // slot columns per slot row: 2, 4
  static constexpr int BR = 12, BS = NB - BR;  // slot columns in registers (the last ones) and in shared memory
  static constexpr int WC = NW / 2;            // warps across the columns; two across the thread rows
  static constexpr int kKeep = 16;             // columns kept in shared memory before they are written out
  static constexpr int kOut = TR * NA * (kKeep + 1) + 3 * kKeep;  // the CTA's rows of the reflectors; d, e, tau
  // x (two buffers), (v, w), gathered (y, next column) (two buffers), partial sums,
  // next column's entries, warp sums of |x|^2 (two buffers) and of x.y, x.y of the CTAs (two buffers);
  // then what waits to be written out, then the slots
  static constexpr int kVec = 8 * P + WC * TR * NA + TR * NA + 3 * NW + 2 * C + kOut;
  static constexpr size_t kBytes = sizeof(double) * (kVec + NA * BS * NT);
};

template <int C>
struct ClusterReg {
  double r[ClusterShape<C>::NA][ClusterShape<C>::BR];
};

// Where a molecule's reduction reads and writes: A (leading dimension ld) holds
// the matrix and then, in column k below the subdiagonal, reflector k scaled to
// v_{k+1} = 1.
struct ClusterOut {
  double *A, *d, *e, *tau;
  int N, ld;
};

// Writes the reflectors, d, e and tau up to column k that wait in shared memory.
// A store to global memory before a cluster barrier holds the barrier up until it
// is performed (about 800 cycles), so they go out once in kKeep columns.
template <int C>
__device__ __forceinline__ void cluster_write_out(const ClusterOut& O, int k, const double* sm) {
  using CS = ClusterShape<C>;
  constexpr int K = CS::kKeep, TR = CS::TR;
  const int tid = threadIdx.x, off = CS::P - O.N;
  const double* vk = sm + CS::kVec - CS::kOut;
  const double* det = vk + TR * CS::NA * (K + 1);
  const int rank = (int)cooperative_groups::this_cluster().block_rank();
  const int j0 = (k - off) & ~(K - 1), q = tid & (K - 1), j = j0 + q;
  if (j > k - off) return;
  for (int l = tid / K; l < TR * CS::NA; l += CS::NT / K) {
    const int i = TR * (C * (l / TR) + rank) + l % TR - off;
    if (i > j + 1) O.A[(long long)i * O.ld + j] = vk[l * (K + 1) + q];
  }
  if (rank == 0 && tid < K) {
    O.d[j + 1] = det[q];
    O.e[j] = det[K + q];
    O.tau[j] = det[2 * K + q];
  }
}

// Columns k of the slot grid with k / (TR C) == A0.
template <int C, int A0>
__device__ __forceinline__ void cluster_phase(ClusterReg<C>& R, const ClusterOut& O, double* sm) {
  namespace cg = cooperative_groups;
  using CS = ClusterShape<C>;
  constexpr int P = CS::P, NA = CS::NA, NB = CS::NB, NT = CS::NT, NW = CS::NW, TR = CS::TR, TC = CS::TC, BS = CS::BS,
                WC = CS::WC, B0 = CS::CB * A0;
  constexpr int n = NA - A0;  // live slot rows
  const cg::cluster_group cl = cg::this_cluster();
  const int rank = (int)cl.block_rank();
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int lc = lane & 7, wc = wid >> 1;
  const int tr = (wid & 1) * 4 + (lane >> 3), tc = wc * 8 + lc;
  const int off = P - O.N;
  double* xb = sm;                                             // [2][P]
  double2* vw = reinterpret_cast<double2*>(sm + 2 * P);        // [P]
  double2* gat = reinterpret_cast<double2*>(sm + 4 * P);       // [2][P]
  double* part = sm + 8 * P;                                   // [WC][TR NA]
  double* xnl = part + WC * TR * NA;                           // [TR NA]
  double* red = xnl + TR * NA;                                 // [2][NW] |x|^2, by the column's parity
  double* redxy = red + 2 * NW;                                // [NW] x.y
  double* xyc = redxy + NW;                                    // [2][C]
  double* vk = xyc + 2 * C;                                    // [TR NA][kKeep + 1]
  double* det = vk + TR * NA * (CS::kKeep + 1);                // [3][kKeep] d of column k + 1, e, tau
  double2* priv = reinterpret_cast<double2*>(sm + CS::kVec) + tid;
  auto row_of = [&](int a) { return TR * (C * a + rank) + tr; };
  const int kend = min(TR * C * (A0 + 1), P - 2);
  for (int k = max(off, TR * C * A0); k < kend; ++k) {
    const double* x = xb + (k & 1) * P;
    const int k1 = k + 1;
    // ---- phase M
    double ra[n];
    {
      double vi[n], wi[n];
#pragma unroll
      for (int a = 0; a < n; ++a) {
        const double2 t = vw[row_of(A0 + a)];
        vi[a] = -t.x;
        wi[a] = -t.y;
        ra[a] = 0.0;
      }
      double2 c0, c1, u[n];
      double p0, p1;
      auto cols = [&](int b) {
        c0 = vw[tc + TC * b];
        c1 = vw[tc + TC * b + TC];
        p0 = x[tc + TC * b];
        p1 = x[tc + TC * b + TC];
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
        // column k+1 of the trailing matrix for the CTA's rows (ranges, not b == k1 / TC: from the
        // equality the compiler derives an indexed access, which would put r in local memory)
        const bool next0 = TC * b <= k1 && k1 < TC * (b + 1) && tc == (k1 & (TC - 1));
        const bool next1 = TC * (b + 1) <= k1 && k1 < TC * (b + 2) && tc == (k1 & (TC - 1));
#pragma unroll
        for (int a = 0; a < n; ++a) {
          double2 q;
          if (b < BS) {
            q = t[a];
          } else {
            q.x = R.r[A0 + a][b - BS < 0 ? 0 : b - BS];
            q.y = R.r[A0 + a][b - BS < 0 ? 0 : b - BS + 1];
          }
          q.x = fma(wi[a], t0.x, fma(vi[a], t0.y, q.x));
          q.y = fma(wi[a], t1.x, fma(vi[a], t1.y, q.y));
          ra[a] = fma(q.y, x1, fma(q.x, x0, ra[a]));
          if (b < BS) {
            priv[((A0 + a) * (BS / 2) + b / 2) * NT] = q;
          } else {
            R.r[A0 + a][b - BS < 0 ? 0 : b - BS] = q.x;
            R.r[A0 + a][b - BS < 0 ? 0 : b - BS + 1] = q.y;
          }
          if (b < B0 + CS::CB + 2) {  // where column k+1 can be
            if (next0) xnl[TR * (A0 + a) + tr] = q.x;
            if (next1) xnl[TR * (A0 + a) + tr] = q.y;
          }
        }
      }
    }
    // rows over the eight lanes of a warp, and x.y over the warp
    double xy = 0.0;
#pragma unroll
    for (int a = 0; a < n; ++a) xy = fma(ra[a], x[row_of(A0 + a)], xy);
    constexpr int n1 = (n + 1) / 2, n2 = (n1 + 1) / 2;
    double s1[n1], s2[n2], s3;
#pragma unroll
    for (int q = 0; q < n1; ++q)
      s1[q] = 2 * q + 1 < n ? pair_reduce(ra[2 * q], ra[2 * q + 1 < n ? 2 * q + 1 : 0], lc & 1, 1)
                            : ra[2 * q] + __shfl_xor_sync(0xffffffffu, ra[2 * q], 1);
    xy += __shfl_xor_sync(0xffffffffu, xy, 1);
#pragma unroll
    for (int q = 0; q < n2; ++q)
      s2[q] = 2 * q + 1 < n1 ? pair_reduce(s1[2 * q], s1[2 * q + 1 < n1 ? 2 * q + 1 : 0], lc & 2, 2)
                             : s1[2 * q] + __shfl_xor_sync(0xffffffffu, s1[2 * q], 2);
    xy += __shfl_xor_sync(0xffffffffu, xy, 2);
    if constexpr (n2 == 2)
      s3 = pair_reduce(s2[0], s2[1], lc & 4, 4);
    else
      s3 = s2[0] + __shfl_xor_sync(0xffffffffu, s2[0], 4);
    xy += __shfl_xor_sync(0xffffffffu, xy, 4);
    xy += __shfl_xor_sync(0xffffffffu, xy, 8);
    xy += __shfl_xor_sync(0xffffffffu, xy, 16);
    {  // the row whose sum this lane holds (lanes of an unpaired value hold copies)
      const int u = n2 == 2 ? (lc >> 2) : 0;
      const int q = 2 * u + 1 < n1 ? 2 * u + ((lc >> 1) & 1) : 2 * u;
      const int a = 2 * q + 1 < n ? 2 * q + (lc & 1) : 2 * q;
      part[wc * TR * NA + TR * (A0 + a) + tr] = s3;
      if (lane == 0) redxy[wid] = xy;
    }
    __syncthreads();
    // the CTA's rows to every CTA
    constexpr int rows = TR * n, groups = NT / rows;
    if (tid < rows * groups) {
      const int l = TR * A0 + tid % rows, g = tid / rows;
      double y = part[l];
#pragma unroll
      for (int q = 1; q < WC; ++q) y += part[q * TR * NA + l];
      const double2 v = make_double2(y, xnl[l]);
      double2* at = gat + (k & 1) * P + TR * (C * (l / TR) + rank) + l % TR;
      for (int q = g; q < C; q += groups) *cl.map_shared_rank(at, q) = v;
    }
    if (wid == NW - 1 && lane < C) *cl.map_shared_rank(xyc + (k & 1) * C + rank, lane) = tree_sum<NW>(redxy);
    cl.barrier_arrive();
    // the reflector's scalars, in every thread while the barrier completes (a warp may read them after
    // the others are through it and have written the next column's |x|^2: hence the two buffers)
    const double xx = tree_sum<NW>(red + (k & 1) * NW), x0 = x[k1];
    double alpha = 0.0, beta = 0.0, iv = 0.0;
    if (xx > 1e-280) {  // below: the column is zero next to any entry that matters
      const double nrm = sqrt(xx);
      alpha = x0 >= 0.0 ? -nrm : nrm;
      beta = 1.0 / (xx + fabs(x0) * nrm);  // 2 / |v|^2
      iv = 1.0 / (x0 - alpha);
    }
    const int kq = (k - off) & (CS::kKeep - 1);
    if (tid == 0) {
      det[CS::kKeep + kq] = alpha;
      det[2 * CS::kKeep + kq] = beta * (x0 - alpha) * (x0 - alpha);
    }
    cl.barrier_wait();
    // ---- phase C
    const double2* gk = gat + (k & 1) * P;
    const double y1 = gk[k1].x, a11 = gk[k1].y, v1 = x0 - alpha;
    double vav = 0.0;
#pragma unroll
    for (int q = 0; q < C; q += 4)
      vav += (xyc[(k & 1) * C + q] + xyc[(k & 1) * C + q + 1]) + (xyc[(k & 1) * C + q + 2] + xyc[(k & 1) * C + q + 3]);
    vav += alpha * (alpha * a11 - 2.0 * y1);
    const double K = 0.5 * beta * beta * vav;
    const double w1 = beta * (y1 - alpha * a11) - K * v1;
    double sq = 0.0;
#pragma unroll
    for (int i0 = 0; i0 < P; i0 += NT) {
      const int i = i0 + tid;
      if (i0 + NT <= TR * C * A0 || i >= P) continue;
      double v = 0.0, w = 0.0, xnext = 0.0;
      if (i >= k1) {
        const double2 t = gk[i];
        v = i == k1 ? v1 : x[i];
        w = beta * (t.x - alpha * t.y) - K * v;
        const double q = t.y - (v * w1 + w * v1);
        if (i == k1) {
          det[kq] = q;
        } else {
          xnext = q;
          if ((i / TR) % C == rank) vk[(TR * (i / (TR * C)) + i % TR) * (CS::kKeep + 1) + kq] = v * iv;
        }
      }
      vw[i] = make_double2(v, w);
      xb[((k + 1) & 1) * P + i] = xnext;
      sq += xnext * xnext;
    }
    sq = warp_sum(sq);
    if (lane == 0) red[((k + 1) & 1) * NW + wid] = sq;
    __syncthreads();
    if (kq == CS::kKeep - 1 || k == P - 3) cluster_write_out<C>(O, k, sm);
  }
  if constexpr (A0 + 1 < NA) cluster_phase<C, A0 + 1>(R, O, sm);
}

template <int C>
__device__ __forceinline__ void cluster_tridiag(const ClusterOut& O, double* sm) {
  namespace cg = cooperative_groups;
  using CS = ClusterShape<C>;
  constexpr int P = CS::P, NA = CS::NA, NB = CS::NB, NT = CS::NT, TR = CS::TR, TC = CS::TC, BS = CS::BS;
  const cg::cluster_group cl = cg::this_cluster();
  const int rank = (int)cl.block_rank();
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int tr = (wid & 1) * 4 + (lane >> 3), tc = (wid >> 1) * 8 + (lane & 7);
  const int off = P - O.N;
  double2* priv = reinterpret_cast<double2*>(sm + CS::kVec) + tid;
  ClusterReg<C> R;
#pragma unroll
  for (int a = 0; a < NA; ++a) {
    const int i = TR * (C * a + rank) + tr - off;
    const double* row = O.A + (long long)max(i, 0) * O.ld + (tc - off);
#pragma unroll
    for (int b = 0; b < NB; b += 2) {
      double2 u = make_double2(0.0, 0.0);
      if (i >= 0) {
        if (tc + TC * b >= off) u.x = __ldcg(row + TC * b);
        if (tc + TC * b + TC >= off) u.y = __ldcg(row + TC * b + TC);
      }
      if (b < BS) {
        priv[(a * (BS / 2) + b / 2) * NT] = u;
      } else {
        R.r[a][b - BS < 0 ? 0 : b - BS] = u.x;
        R.r[a][b - BS < 0 ? 0 : b - BS + 1] = u.y;
      }
    }
  }
  double sq = 0.0;
  for (int i = tid; i < P; i += NT) {
    const double x = i > off ? __ldcg(O.A + (long long)(i - off) * O.ld) : 0.0;
    sm[(off & 1) * P + i] = x;
    reinterpret_cast<double2*>(sm + 2 * P)[i] = make_double2(0.0, 0.0);
    sq += x * x;
    if (i == off && rank == 0) O.d[0] = __ldcg(O.A);
  }
  sq = warp_sum(sq);
  double* red = sm + 8 * P + CS::WC * TR * NA + TR * NA;
  if (lane == 0) red[(off & 1) * CS::NW + wid] = sq;
  cl.sync();  // the matrix is read before the reflectors overwrite it
  cluster_phase<C, 0>(R, O, sm);
  // the last 2 x 2 block: its corner belongs to the last row's CTA
  if (tid == 0 && rank == 0 && O.N >= 2) O.e[O.N - 2] = sm[((P - 2) & 1) * P + P - 1];
  if (rank == C - 1 && tr == TR - 1 && tc == TC - 1) {
    const double2 t = reinterpret_cast<double2*>(sm + 2 * P)[P - 1];
    O.d[O.N - 1] = R.r[NA - 1][CS::BR - 1] - 2.0 * t.x * t.y;
    O.e[O.N - 1] = 0.0;
    O.tau[O.N - 1] = 0.0;
    if (O.N >= 2) O.tau[O.N - 2] = 0.0;
  }
  __threadfence();
  cl.sync();  // d, e of every CTA before CTA 0 reads them; no CTA leaves while others write to it
}

}  // namespace gfn1
