// Householder reduction of a matrix that G CTAs of a cooperative launch keep on chip.
//
// The scheme of tridiag_cluster.cuh for matrices beyond a cluster: the rows are dealt
// out to the CTAs in blocks of four (at most 16 rows a CTA), column j of thread column
// j % 128, the last slot columns in registers and the early ones in shared memory.  148 SMs hold 2368
// rows; of a larger matrix the blocked reduction does the first columns.  Per column
//   M  each CTA: the rank-2 update of the previous column fused with y = A22 x for
//      its rows, which it writes with their entries of the next column to a ring in
//      global memory;
//   C  every CTA reads all rows' values (16 bytes a row) and forms w, the next
//      column and its norm for all rows, the same in each.
// There is no barrier among the CTAs: the values are their own flags.  A ring slot
// holds the pattern "not written" (all ones, a NaN that no arithmetic yields) until
// its owner writes it, and the reader waits for every value to differ from it.  A
// barrier and a load after it are two round trips to L2, this is one.  Sixteen slots:
// once every CTA's values of column k, a multiple of eight, are there, all of them
// have read columns k - 8 .. k - 1; their owners mark those slots unwritten again and
// fence that before their values of column k + 2.  Every thread of a reader has its values
// of column k + 2 and fences in turn before it looks for those of column k + 8, the first to
// use these slots: with the two fences the marks happen before that look, so it finds the
// mark or a new value, never the number of sixteen columns ago.  (The loads and stores of the
// ring are relaxed; one fence by the readers in eight columns is all the order they need.)
// Every wait is bounded: after kSpinCycles, or when another CTA has raised the molecule's
// error flag, the CTA raises it and leaves.
//
// Measured on B200 (the blocked reduction before): 2368 AOs 42 -> 9.2 ms, 1296 -> 3.7 ms,
// 776 -> 2.0 ms.  (The fences of the readers are 3% of that.)  Of the other 7,250 cycles a column at 2368 AOs 1,840 are the products (660
// of the FP64 units, the rest shared memory), 360 the row sums, 550 the scalars, 2,900
// the exchange and its spread over the CTAs, 1,490 the vectors of phase C.  Rows singly
// 8,340 cycles (a line of the ring then has eight writers, each write takes the line
// from the readers that came early), in pairs 7,270, in eights 7,390 (the last rows of
// a block leave the CTA idle); values re-read one after the other 19,000; four slots
// with a fence a column 7,730 where rows were single.
#pragma once

#include <type_traits>

#include "common.cuh"
#include "tridiag.cuh"

namespace gfn1 {

struct GridShape {
  static constexpr int NT = 256, NW = NT / 32;
  static constexpr int TR = 2, TC = 128;         // thread rows and columns of a CTA
  static constexpr int NA = 8, NB = 19;          // slot rows and columns
  static constexpr int BR = 9, BS = NB - BR;     // slot columns in registers (the last ones) and in shared memory
  static constexpr int kRows = TR * NA;          // rows of a CTA: 16
  static constexpr int kBlock = 4;               // consecutive rows of a CTA
  static constexpr int P = TC * NB;              // columns: 2432
  static constexpr int NQ = (P + NT - 1) / NT;   // rows a thread of phase C holds
  static constexpr int WC = TC / 32;             // warps across the columns
  // A ring slot has N values, rounded up so that the rows of a block start on 64 bytes.
  static __host__ __device__ constexpr int ring_stride(int N) { return (N + 2 * kBlock - 1) & ~(kBlock - 1); }
  static constexpr int kRing = 16, kMark = 8;    // ring slots; slots marked unwritten at a time
  static constexpr int kRelease = 1, kAcquire = 2;  // columns after the marks: the owner's fence, the readers'
  // (v, w), x, partial sums, next column's entries, warp sums, scalars; then the slots
  static constexpr int kVec = 3 * P + WC * kRows + kRows + 2 * NW + 8;
  static constexpr size_t kBytes = sizeof(double) * (kVec + NA * BS * NT);
};

// Padded index of local row l of CTA c.
__device__ __forceinline__ int grid_row(int l, int c, int G) {
  constexpr int B = GridShape::kBlock;
  return B * (G * (l / B) + c) + l % B;
}

struct GridReg {
  double r[GridShape::NA][GridShape::BR];
};

// A (leading dimension ld) holds the matrix and then, in column k below the
// subdiagonal, reflector k scaled to v_{k+1} = 1; ring: kRing ring_stride(N) values,
// 128-byte aligned.
struct GridOut {
  double *A, *d, *e, *tau;
  double2* ring;
  int* err;
  int N, ld, G, c;
};

constexpr unsigned long long kUnwritten = ~0ull;

__device__ __forceinline__ void ring_store(double2* p, double a, double b) {
  asm volatile("st.relaxed.gpu.global.v2.f64 [%0], {%1, %2};" ::"l"(p), "d"(a), "d"(b) : "memory");
}
__device__ __forceinline__ double2 ring_load(const double2* p) {
  double2 v;
  asm volatile("ld.relaxed.gpu.global.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void ring_fence() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }
__device__ __forceinline__ bool unwritten(const double2& v) {
  return (unsigned long long)__double_as_longlong(v.x) == kUnwritten ||
         (unsigned long long)__double_as_longlong(v.y) == kUnwritten;
}

// Columns from k on for which slot rows before A0 are done; false if a wait gave up.
template <int A0>
__device__ __forceinline__ bool grid_phase(GridReg& R, const GridOut& O, double* sm, int k, double iv_prev,
                                           long long spin_cycles) {
  using GS = GridShape;
  constexpr int P = GS::P, NA = GS::NA, NB = GS::NB, NT = GS::NT, NW = GS::NW, TR = GS::TR, TC = GS::TC, BS = GS::BS,
                WC = GS::WC, NQ = GS::NQ;
  constexpr int n = NA - A0;  // live slot rows
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int wc = wid % WC, tr = wid / WC, tc = wc * 32 + lane;
  const int N = O.N, G = O.G, offr = GS::kRows * G - N, offc = P - N;
  double2* vw = reinterpret_cast<double2*>(sm);  // [P]
  double* x = sm + 2 * P;                        // [P]
  double* part = x + P;                          // [WC][kRows]
  double* xnl = part + WC * GS::kRows;           // [kRows]
  double* red = xnl + GS::kRows;                 // [NW] |x|^2, [NW] x.y
  double* scal = red + 2 * NW;                   // y and entry of the next column at row k + 1
  int* gave_up = reinterpret_cast<int*>(scal + 2);
  double2* priv = reinterpret_cast<double2*>(sm + GS::kVec) + tid;
  const int rs = GS::ring_stride(N);
  double2* ring0 = O.ring + (offr & (GS::kBlock - 1));
  const int kend = min(grid_row(TR * A0 + TR - 1, G - 1, G) - offr, N - 2);
  const int last = grid_row(GS::kRows - 1, O.c, G) - offr;  // the CTA's last row
  for (; k < kend; ++k) {
    const int k1 = k + 1, kk = k1 + offc;
    // ---- phase M
    const int q0 = kk / NT;  // slot columns before 2 q0 are done
    double ra[n];
    {
      double vi[n], wi[n];
#pragma unroll
      for (int a = 0; a < n; ++a) {
        const double2 t = vw[grid_row(TR * (A0 + a) + tr, O.c, G) - offr + offc];
        vi[a] = -t.x;
        wi[a] = -t.y;
        ra[a] = 0.0;
      }
      // Entered at the first live pair of slot columns, so that the code is a straight line
      // behind one jump; the operands of a pair are loaded before the arithmetic of the last.
      constexpr int h0 = (n + 1) / 2;  // rows of the first half
      double2 c0, c1, u[h0];
      double p0, p1;
      auto cols = [&](int b) {
        c0 = vw[tc + TC * b];
        c1 = vw[tc + TC * b + (b + 1 < NB ? TC : 0)];
        p0 = x[tc + TC * b];
        p1 = x[tc + TC * b + (b + 1 < NB ? TC : 0)];
      };
      auto half = [&](int b, int h) {  // slots of rows h h0 .. of columns b, b + 1
#pragma unroll
        for (int a = 0; a < h0; ++a)
          if (h * h0 + a < n) u[a] = priv[((A0 + h * h0 + a) * (BS / 2) + b / 2) * NT];
      };
      // the next column (a range, not b == kk / TC: from the equality the compiler derives an
      // indexed access, which would put r in local memory)
      auto is_next = [&](int b) { return TC * b <= kk && kk < TC * (b + 1) && tc == (kk & (TC - 1)); };
      auto shared_pair = [&](auto B) {
        constexpr int b = decltype(B)::value;
        const double2 d0 = c0, d1 = c1;
        const double x0 = p0, x1 = p1;
        const bool next0 = is_next(b), next1 = is_next(b + 1);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          double2 t[h0];
#pragma unroll
          for (int a = 0; a < h0; ++a) t[a] = u[a];
          if (h == 0) {
            half(b, 1);
          } else {
            cols(b + 2);
            if (b + 2 < BS) half(b + 2, 0);
          }
#pragma unroll
          for (int a = 0; a < h0; ++a) {
            if (h * h0 + a >= n) continue;
            const int i = h * h0 + a < n ? h * h0 + a : 0;
            t[a].x = fma(wi[i], d0.x, fma(vi[i], d0.y, t[a].x));
            t[a].y = fma(wi[i], d1.x, fma(vi[i], d1.y, t[a].y));
            ra[i] = fma(t[a].y, x1, fma(t[a].x, x0, ra[i]));
            priv[((A0 + i) * (BS / 2) + b / 2) * NT] = t[a];
          }
          if (next0 || next1) {
#pragma unroll
            for (int a = 0; a < h0; ++a)
              if (h * h0 + a < n) xnl[TR * (A0 + h * h0 + a) + tr] = next0 ? t[a].x : t[a].y;
          }
        }
      };
      auto reg_pair = [&](auto B) {
        constexpr int b = decltype(B)::value;
#pragma unroll
        for (int e = 0; e < 2 && b + e < NB; ++e) {
          const double2 cv = e ? c1 : c0;
          const double xv = e ? p1 : p0;
#pragma unroll
          for (int a = 0; a < n; ++a) {
            double& q = R.r[A0 + a][b + e - BS];
            q = fma(wi[a], cv.x, fma(vi[a], cv.y, q));
            ra[a] = fma(q, xv, ra[a]);
          }
          if (is_next(b + e)) {
#pragma unroll
            for (int a = 0; a < n; ++a) xnl[TR * (A0 + a) + tr] = R.r[A0 + a][b + e - BS];
          }
        }
      };
#pragma unroll
      for (int a = 0; a < h0; ++a) u[a] = make_double2(0.0, 0.0);
      {
        const int b = 2 * q0;
        const int d = b + 1 < NB ? TC : 0;
        c0 = vw[tc + TC * b];
        c1 = vw[tc + TC * b + d];
        p0 = x[tc + TC * b];
        p1 = x[tc + TC * b + d];
        if (b < BS) half(b, 0);
      }
#define GFN1_REG_PAIR(b)                                        \
  {                                                             \
    const double2 k0 = c0, k1 = c1;                             \
    const double m0 = p0, m1 = p1;                              \
    if (b + 2 < NB) cols(b + 2);                                \
    const double2 n0 = c0, n1 = c1;                             \
    const double o0 = p0, o1 = p1;                              \
    c0 = k0, c1 = k1, p0 = m0, p1 = m1;                         \
    reg_pair(std::integral_constant<int, b>());                 \
    c0 = n0, c1 = n1, p0 = o0, p1 = o1;                         \
  }
      static_assert(BS == 10 && NB == 19, "the cases below");
      switch (q0) {
        case 0: shared_pair(std::integral_constant<int, 0>());  // fall through, here and below
        case 1: shared_pair(std::integral_constant<int, 2>());
        case 2: shared_pair(std::integral_constant<int, 4>());
        case 3: shared_pair(std::integral_constant<int, 6>());
        case 4: shared_pair(std::integral_constant<int, 8>());
        case 5: GFN1_REG_PAIR(10)
        case 6: GFN1_REG_PAIR(12)
        case 7: GFN1_REG_PAIR(14)
        case 8: GFN1_REG_PAIR(16)
        default: GFN1_REG_PAIR(18)
      }
#undef GFN1_REG_PAIR
    }
    // row sums over the lanes of a warp
    const int lc = lane & 7;
    constexpr int n1 = (n + 1) / 2, n2 = (n1 + 1) / 2;
    double s1[n1], s2[n2], s3;
#pragma unroll
    for (int q = 0; q < n1; ++q)
      s1[q] = 2 * q + 1 < n ? pair_reduce(ra[2 * q], ra[2 * q + 1 < n ? 2 * q + 1 : 0], lc & 1, 1)
                            : ra[2 * q] + __shfl_xor_sync(0xffffffffu, ra[2 * q], 1);
#pragma unroll
    for (int q = 0; q < n2; ++q)
      s2[q] = 2 * q + 1 < n1 ? pair_reduce(s1[2 * q], s1[2 * q + 1 < n1 ? 2 * q + 1 : 0], lc & 2, 2)
                             : s1[2 * q] + __shfl_xor_sync(0xffffffffu, s1[2 * q], 2);
    if constexpr (n2 == 2)
      s3 = pair_reduce(s2[0], s2[1], lc & 4, 4);
    else
      s3 = s2[0] + __shfl_xor_sync(0xffffffffu, s2[0], 4);
    s3 += __shfl_xor_sync(0xffffffffu, s3, 8);
    s3 += __shfl_xor_sync(0xffffffffu, s3, 16);
    {  // the row whose sum this lane holds (lanes of an unpaired value hold copies)
      const int u = n2 == 2 ? (lc >> 2) : 0;
      const int q = 2 * u + 1 < n1 ? 2 * u + ((lc >> 1) & 1) : 2 * u;
      const int a = 2 * q + 1 < n ? 2 * q + (lc & 1) : 2 * q;
      if (lane < 8) part[wc * GS::kRows + TR * (A0 + a) + tr] = s3;
    }
    __syncthreads();
    double2* ring = ring0 + (size_t)(k & (GS::kRing - 1)) * rs;
    const int row = grid_row(lane, O.c, G) - offr;  // (warps 0 and 1) the CTA's row `lane`
    if (wid == 0) {
      if (lane < GS::kRows && row >= k1) {
        double y = part[lane];
#pragma unroll
        for (int q = 1; q < WC; ++q) y += part[q * GS::kRows + lane];
        ring_store(ring + row, y, xnl[lane]);
      }
    } else if (wid == 1) {  // the previous reflector
      if (lane < GS::kRows && row > k && k > 0) O.A[(long long)row * O.ld + k - 1] = vw[row + offc].x * iv_prev;
    }
    // A CTA whose last row is k + 1 has nothing left to do.  So a CTA that reads the values of a
    // column writes some at the next one, which is how the others know that it has read them.
    if (last <= k1) return true;
    // ---- phase C: the reflector's scalars, in every thread, before the values are there
    const double xx = tree_sum<NW>(red), x0 = x[kk];
    double alpha = 0.0, beta = 0.0, iv = 0.0;
    if (xx > 1e-280) {  // below: the column is zero next to any entry that matters
      const double nrm = sqrt(xx);
      alpha = x0 >= 0.0 ? -nrm : nrm;
      beta = 1.0 / (xx + fabs(x0) * nrm);  // 2 / |v|^2
      iv = 1.0 / (x0 - alpha);
    }
    double2 g[NQ];
    bool wait = false;
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      g[q] = make_double2(0.0, 0.0);
      if (q < q0) continue;
      const int i = tid + NT * q - offc;
      if (i >= k1 && i < N) g[q] = ring_load(ring + i);
    }
    // what was marked at the previous column, before the next column's values
    if (wid == 0 && (k & (GS::kMark - 1)) == GS::kRelease) ring_fence();
#pragma unroll
    for (int q = 0; q < NQ; ++q)
      if (q >= q0) wait |= unwritten(g[q]);
    if (wait) {  // all missing values at once: one after the other each costs a round trip to L2
      const long long t0 = clock64();
      for (int tries = 1; wait; ++tries) {
#pragma unroll
        for (int q = 0; q < NQ; ++q)
          if (q >= q0 && unwritten(g[q])) g[q] = ring_load(ring + (tid + NT * q - offc));
        wait = false;
#pragma unroll
        for (int q = 0; q < NQ; ++q)
          if (q >= q0) wait |= unwritten(g[q]);
        if (wait && (tries & 63) == 0 && (*(volatile int*)O.err != 0 || clock64() - t0 > spin_cycles)) {
          atomicExch(O.err, 1);
          *gave_up = 1;
          break;
        }
      }
    }
    // the owners' marks before the next look at those slots (each row's owner marks its slots, and
    // the thread that reads the row here is the one that will look there)
    if ((k & (GS::kMark - 1)) == GS::kAcquire) ring_fence();
    double xy = 0.0;
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      if (q < q0) continue;
      const int i = tid + NT * q - offc;
      if (i >= k1 && i < N) xy = fma(x[i + offc], g[q].x, xy);
      if (i == k1) {
        scal[0] = g[q].x;
        scal[1] = g[q].y;
      }
    }
    xy = warp_sum(xy);
    if (lane == 0) red[NW + wid] = xy;
    __syncthreads();
    if (*gave_up) return false;
    if ((k & (GS::kMark - 1)) == 0 && k > 0 && tid < GS::kMark * GS::kRows) {  // every CTA has read the columns before k
      const int s = k - GS::kMark + tid / GS::kRows, i = grid_row(tid % GS::kRows, O.c, G) - offr;
      if (i > s)
        ring_store(ring0 + (size_t)(s & (GS::kRing - 1)) * rs + i, __longlong_as_double((long long)kUnwritten),
                   __longlong_as_double((long long)kUnwritten));
    }
    const double y1 = scal[0], a11 = scal[1], v1 = x0 - alpha;
    const double vav = tree_sum<NW>(red + NW) + alpha * (alpha * a11 - 2.0 * y1);
    const double K = 0.5 * beta * beta * vav;
    const double w1 = beta * (y1 - alpha * a11) - K * v1;
    if (tid == 0 && O.c == G - 1) {
      O.d[k1] = a11 - 2.0 * v1 * w1;
      O.e[k] = alpha;
      O.tau[k] = beta * v1 * v1;
    }
    double sq = 0.0;
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      const int j = tid + NT * q, i = j - offc;
      if (q < q0 || j >= P) continue;
      double v = 0.0, w = 0.0, xnext = 0.0;
      if (i >= k1) {
        v = i == k1 ? v1 : x[j];
        w = beta * (g[q].x - alpha * g[q].y) - K * v;
        if (i > k1) xnext = g[q].y - (v * w1 + w * v1);
      }
      vw[j] = make_double2(v, w);
      x[j] = xnext;
      sq = fma(xnext, xnext, sq);
    }
    sq = warp_sum(sq);
    if (lane == 0) red[wid] = sq;
    iv_prev = iv;
    __syncthreads();
  }
  if constexpr (A0 + 1 < NA) {
    return grid_phase<A0 + 1>(R, O, sm, k, iv_prev, spin_cycles);
  } else {
    // the last reflector; then the last 2 x 2 block, whose corner belongs to the last row's CTA
    const int row = grid_row(lane, O.c, G) - offr;
    if (wid == 1 && lane < GS::kRows && row > k && k > 0) O.A[(long long)row * O.ld + k - 1] = vw[row + offc].x * iv_prev;
    if (tid == 0 && O.c == G - 1) O.e[N - 2] = x[P - 1];
    if (O.c == G - 1 && tr == TR - 1 && tc == TC - 1) {
      const double2 t = vw[P - 1];
      O.d[N - 1] = R.r[NA - 1][GS::BR - 1] - 2.0 * t.x * t.y;
      O.e[N - 1] = 0.0;
      O.tau[N - 1] = 0.0;
      O.tau[N - 2] = 0.0;
    }
    return true;
  }
}

// N >= 3.  The ring's values are all kUnwritten at the start.
__device__ __forceinline__ bool grid_tridiag(const GridOut& O, double* sm, long long spin_cycles) {
  using GS = GridShape;
  constexpr int P = GS::P, NA = GS::NA, NB = GS::NB, NT = GS::NT, NW = GS::NW, TR = GS::TR, TC = GS::TC, BS = GS::BS;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int tr = wid / GS::WC, tc = (wid % GS::WC) * 32 + lane;
  const int N = O.N, offr = GS::kRows * O.G - N, offc = P - N;
  double2* priv = reinterpret_cast<double2*>(sm + GS::kVec) + tid;
  double* red = sm + 3 * P + GS::WC * GS::kRows + GS::kRows;
  GridReg R;
#pragma unroll
  for (int a = 0; a < NA; ++a) {
    const int i = grid_row(TR * a + tr, O.c, O.G) - offr;
    const double* from = O.A + (long long)max(i, 0) * O.ld + (tc - offc);
    auto at = [&](int b) { return i >= 0 && tc + TC * b >= offc ? __ldcg(from + TC * b) : 0.0; };
#pragma unroll
    for (int b = 0; b < BS; b += 2) priv[(a * (BS / 2) + b / 2) * NT] = make_double2(at(b), at(b + 1));
#pragma unroll
    for (int b = BS; b < NB; ++b) R.r[a][b - BS] = at(b);
  }
  double sq = 0.0;
  for (int j = tid; j < P; j += NT) {
    const int i = j - offc;
    const double x = i > 0 ? __ldcg(O.A + i) : 0.0;  // row 0
    sm[2 * P + j] = x;
    reinterpret_cast<double2*>(sm)[j] = make_double2(0.0, 0.0);
    sq = fma(x, x, sq);
    if (i == 0 && O.c == 0) O.d[0] = __ldcg(O.A);
  }
  sq = warp_sum(sq);
  if (lane == 0) red[wid] = sq;
  if (tid == 0) *reinterpret_cast<int*>(red + 2 * NW + 2) = 0;
  __syncthreads();
  return grid_phase<0>(R, O, sm, 0, 0.0, spin_cycles);
}

}  // namespace gfn1
