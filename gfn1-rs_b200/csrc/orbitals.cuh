// Back-transformation of the occupied eigenvectors and the AO populations, one
// warp per eight orbitals with the orbitals in registers.
//
// Both steps multiply the orbitals by matrices every warp of the CTA reads
// (reflectors, L, L^-1), so the orbitals are what should stay put.  A warp
// keeps the transpose of its eight columns, Z^T (8 x N), as FP64 tensor-core
// accumulators (m8n8k4: lane (g, t) holds columns 2t and 2t+1 of row g of each
// 8 x 8 tile).  Read as an A operand of two k = 4 steps the same registers are
// rows g of Z^T with the contraction index taken in the order 2t | 2t + 1, so
// no value moves between lanes: W^T = Z^T V, W^T T^T and Z^T -= (W T^T)^T V^T chain
// on registers, without a barrier from the first reflector block to the
// populations.  The former form (tiles of Z staged through memory, three
// barriers per 16 reflectors, one load per tensor instruction and operand)
// spent 270k cycles on the back-transformation and 243k on the populations of
// a 128-AO molecule.
#pragma once

#include "common.cuh"

namespace gfn1 {

// D += A B for one 8x8x4 FP64 tile on the tensor cores (PTX mma.m8n8k4 .f64,
// row-major A, column-major B): lane l holds A[l/4][l%4], B[l%4][l/4] and
// D[l/4][2(l%4)], D[l/4][2(l%4)+1].
__device__ __forceinline__ void dmma_m8n8k4(double& d0, double& d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}

// Compact-WY factors of blocks of eight reflectors (rows of V, zero outside
// their range; rows from N-2 to the block's end are zero with tau = 0):
// H_kb ... H_kb+7 = I - V_b^T T V_b with T upper triangular, T_jj = tau_j,
// T[0:j, j] = -tau_j T[0:j, 0:j] (V V^T)[0:j, j].  One warp per block; T in
// row-major 8 x 8 blocks.  V V^T takes one load per tensor instruction (the A
// and the B operand are the same value).
// tau, T: offsets (doubles) into the dynamic shared memory.
template <int NW>
__device__ __noinline__ void wy_factors(const double* __restrict__ V, int ldv, int N, int tau_at, int t_at) {
  extern __shared__ __align__(16) unsigned char smraw[];
  const double* tau = reinterpret_cast<double*>(smraw) + tau_at;
  double* T = reinterpret_cast<double*>(smraw) + t_at;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, g = lane >> 2, t4 = lane & 3;
  const int nref = N - 2, nblk = (nref + 7) >> 3;
  for (int b = wid; b < nblk; b += NW) {
    const int kb = 8 * b;
    double g00 = 0.0, g01 = 0.0, g10 = 0.0, g11 = 0.0;
    const double* row = V + (long long)(kb + g) * ldv + t4;
#pragma unroll 4
    for (int r = kb; r < N; r += 8) {
      const double a0 = row[r], a1 = row[r + 4];
      dmma_m8n8k4(g00, g01, a0, a0);
      dmma_m8n8k4(g10, g11, a1, a1);
    }
    double* Tb = T + 64 * b;
    Tb[8 * g + 2 * t4] = g00 + g10;
    Tb[8 * g + 2 * t4 + 1] = g01 + g11;
    __syncwarp();
    double trow[8];
    if (lane < 8) {  // lane i forms row i of T
#pragma unroll
      for (int j = 0; j < 8; ++j) trow[j] = 0.0;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const double tj = kb + j < nref ? tau[kb + j] : 0.0;
        double s = 0.0;
#pragma unroll
        for (int l = 0; l < 8; ++l)
          if (l < j) s += trow[l] * Tb[8 * l + j];  // zero left of the diagonal
        trow[j] = j == lane ? tj : (j > lane ? -tj * s : 0.0);
      }
    }
    __syncwarp();
    if (lane < 8) {
#pragma unroll
      for (int j = 0; j < 8; ++j) Tb[8 * lane + j] = trow[j];
    }
  }
}

// 16 bytes from global to shared memory, in the background.
__device__ __forceinline__ void copy16_async(double* dst, const double* src) {
  const unsigned at = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(at), "l"(src) : "memory");
}

// Panels of occupied_orbitals in shared memory: eight rows each, three in turn.
// Row lengths that spread the operand loads over the banks: reflectors are read
// by rows (16 bytes) and by columns (8 bytes), L and L^-T by rows only.
template <int P>
struct OrbitalPanels {
  static constexpr int kVPitch = P + 2, kLPitch = P + 8;
  static constexpr int kPanel = 8 * kLPitch, kStages = 3;
  static constexpr int kDoubles = kStages * kPanel;
};

// For the occupied orbitals: Z := Q Z (Q = H_0 ... H_{N-3}), C = L^-T Z and the
// warp's share of the AO populations (S P)_mu,mu = sum_i f_i C_mu,i (L Z)_mu,i.
//   Zin  [N][ldz] tridiagonal eigenvectors in columns 0..nocc-1, to be scaled by
//        scale[0..nocc)
//   V, T reflectors and WY factors (above); ldv a multiple of 32, padding zero
//   L, LiT [8 ceil(N/8)][ld], ld = 8 ceil(N/8): the Cholesky factor and the
//        transpose of its inverse, zero in the padding (and above / below the
//        diagonal)
//   Ct   [8 ceil(nocc/8)][ld] orbitals by rows (C transposed)
//   popw [NW][ld] population sums of each warp
//   Zout [N][ldz] the transformed eigenvectors, or null
// Every warp needs all of V, L and L^-T, so they come to shared memory once per
// pass over the orbitals, in panels of eight reflectors and then of eight AOs
// copied two ahead of their use (each warp loading for itself kept the
// L2 busy: 1.4M cycles at 192 AOs with every SM at work).
// T, occ, scale: offsets (doubles) into the dynamic shared memory; the panels
// follow T's 8 P doubles.
template <int NW, int P>
__device__ __noinline__ void occupied_orbitals(const double* __restrict__ V, int ldv, int t_at, int N,
                                               const double* Zin, int ldz, int nocc, int occ_at, int scale_at,
                                               const double* __restrict__ L, const double* __restrict__ LiT, int ld,
                                               double* __restrict__ Ct, double* __restrict__ popw, double* Zout) {
  extern __shared__ __align__(16) unsigned char smraw[];
  using OP = OrbitalPanels<P>;
  constexpr int NQ = P / 32;  // groups of four row tiles
  const double* T = reinterpret_cast<double*>(smraw) + t_at;
  const double* occ = reinterpret_cast<double*>(smraw) + occ_at;
  const double* scale = reinterpret_cast<double*>(smraw) + scale_at;
  double* panels = reinterpret_cast<double*>(smraw) + t_at + 8 * P;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, g = lane >> 2, t4 = lane & 3;
  const int nblk = N > 2 ? (N - 2 + 7) >> 3 : 0;
  const int nt = (N + 7) >> 3, items = nblk + nt;
  // item q < nblk: reflector block b = nblk-1-q, its columns from the group of
  // row tiles it starts in; then the AO tiles m: L's row up to the diagonal tile
  // and, eight columns further on, L^-T's from it
  auto copy = [&](int q) {
    if (q < items) {
      double* dst = panels + (q % OP::kStages) * OP::kPanel;
      if (q < nblk) {
        const int kb = 8 * (nblk - 1 - q);
        for (int r = wid; r < 8; r += NW) {
          const double* src = V + (long long)(kb + r) * ldv;
          for (int c = (kb & ~31) + 2 * lane; c < ldv; c += 64) copy16_async(dst + r * OP::kVPitch + c, src + c);
        }
      } else {
        const int m = q - nblk;
        for (int r = wid; r < 8; r += NW) {
          const long long row = (long long)(8 * m + r) * ld;
          for (int c = 2 * lane; c < ld + 8; c += 64)
            copy16_async(dst + r * OP::kLPitch + c, c < 8 * m + 8 ? L + row + c : LiT + row + c - 8);
        }
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  double* pw = popw + (long long)wid * ld;
  for (int m = lane; m < ld; m += 32) pw[m] = 0.0;
  __syncwarp();
  for (int ct0 = 0; 8 * ct0 < nocc; ct0 += NW) {
    const int ct = ct0 + wid;
    const bool work = 8 * ct < nocc;
    const int col = 8 * ct + g;
    const double zs = col < nocc ? scale[col] : 0.0;
    __syncthreads();  // the panels of the pass before are done with
    copy(0);
    copy(1);
    double z[NQ][4][2];
    // (every element is set: one left undefined would be live from the function's entry on,
    // and its register taken from every caller's loop)
#pragma unroll
    for (int q = 0; q < NQ; ++q)
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const int row = 32 * q + 8 * u + 2 * t4 + c;
          z[q][u][c] = (row < N && col < nocc) ? zs * Zin[(long long)row * ldz + col] : 0.0;
        }
    const double f = col < nocc ? occ[col] : 0.0;
    for (int it = 0; it < nblk; ++it) {
      asm volatile("cp.async.wait_group 1;" ::: "memory");
      __syncthreads();
      copy(it + 2);
      if (!work) continue;
      const int b = nblk - 1 - it, kb = 8 * b;
      const double* pan = panels + (it % OP::kStages) * OP::kPanel;
      // W^T = Z^T V_b^T over the row groups from the block's own (V is zero above)
      double w0[4], w1[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) w0[u] = w1[u] = 0.0;
      const double* vrow = pan + g * OP::kVPitch + 2 * t4;
#pragma unroll
      for (int q = 0; q < NQ; ++q)
        if (32 * q + 31 > kb && 32 * q < N) {
          double2 v[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) v[u] = *reinterpret_cast<const double2*>(vrow + 32 * q + 8 * u);
#pragma unroll
          for (int u = 0; u < 4; ++u) dmma_m8n8k4(w0[u], w1[u], z[q][u][0], v[u].x);
#pragma unroll
          for (int u = 0; u < 4; ++u) dmma_m8n8k4(w0[u], w1[u], z[q][u][1], v[u].y);
        }
      const double s0 = (w0[0] + w0[1]) + (w0[2] + w0[3]), s1 = (w1[0] + w1[1]) + (w1[2] + w1[3]);
      double y0 = 0.0, y1 = 0.0;
      const double2 tt = *reinterpret_cast<const double2*>(T + 64 * b + 8 * g + 2 * t4);
      dmma_m8n8k4(y0, y1, s0, tt.x);
      dmma_m8n8k4(y0, y1, s1, tt.y);
      y0 = -y0;
      y1 = -y1;
      const double* v0 = pan + 2 * t4 * OP::kVPitch + g;
#pragma unroll
      for (int q = 0; q < NQ; ++q)
        if (32 * q + 31 > kb && 32 * q < N) {
          double a[4], c[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            a[u] = v0[32 * q + 8 * u];
            c[u] = v0[OP::kVPitch + 32 * q + 8 * u];
          }
#pragma unroll
          for (int u = 0; u < 4; ++u) dmma_m8n8k4(z[q][u][0], z[q][u][1], y0, a[u]);
#pragma unroll
          for (int u = 0; u < 4; ++u) dmma_m8n8k4(z[q][u][0], z[q][u][1], y1, c[u]);
        }
    }
    if (Zout && work) {
#pragma unroll
      for (int q = 0; q < NQ; ++q)
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            const int row = 32 * q + 8 * u + 2 * t4 + c;
            if (row < N && col < nocc) Zout[(long long)row * ldz + col] = z[q][u][c];
          }
    }
    // per 8 AOs: D^T = Z^T L^T (k up to the diagonal), C^T = Z^T L^-1 (k from it)
    double* crow = Ct + (long long)col * ld + 2 * t4;
    for (int m = 0; m < nt; ++m) {
      const int it = nblk + m;
      asm volatile("cp.async.wait_group 1;" ::: "memory");
      __syncthreads();
      copy(it + 2);
      if (!work) continue;
      const double* lrow = panels + (it % OP::kStages) * OP::kPanel + g * OP::kLPitch + 2 * t4;
      double d0[2] = {0.0, 0.0}, d1[2] = {0.0, 0.0}, c0[2] = {0.0, 0.0}, c1[2] = {0.0, 0.0};
#pragma unroll
      for (int q = 0; q < NQ; ++q)
        if (32 * q < N) {
          if (4 * q <= m) {
            double2 l[4];
#pragma unroll
            for (int u = 0; u < 4; ++u)
              l[u] = 4 * q + u <= m ? *reinterpret_cast<const double2*>(lrow + 32 * q + 8 * u) : make_double2(0.0, 0.0);
#pragma unroll
            for (int u = 0; u < 4; ++u) dmma_m8n8k4(d0[u & 1], d1[u & 1], z[q][u][0], l[u].x);
#pragma unroll
            for (int u = 0; u < 4; ++u) dmma_m8n8k4(d0[u & 1], d1[u & 1], z[q][u][1], l[u].y);
          }
          if (4 * q + 3 >= m) {
            double2 l[4];
#pragma unroll
            for (int u = 0; u < 4; ++u)
              l[u] = (4 * q + u >= m && 4 * q + u < nt) ? *reinterpret_cast<const double2*>(lrow + 32 * q + 8 * u + 8)
                                                       : make_double2(0.0, 0.0);
#pragma unroll
            for (int u = 0; u < 4; ++u) dmma_m8n8k4(c0[u & 1], c1[u & 1], z[q][u][0], l[u].x);
#pragma unroll
            for (int u = 0; u < 4; ++u) dmma_m8n8k4(c0[u & 1], c1[u & 1], z[q][u][1], l[u].y);
          }
        }
      const double ca = c0[0] + c0[1], cb = c1[0] + c1[1];
      *reinterpret_cast<double2*>(crow + 8 * m) = make_double2(ca, cb);
      double pa = f * ca * (d0[0] + d0[1]), pb = f * cb * (d1[0] + d1[1]);
#pragma unroll
      for (int o = 4; o < 32; o <<= 1) {  // over the eight orbitals
        pa += __shfl_xor_sync(0xffffffffu, pa, o);
        pb += __shfl_xor_sync(0xffffffffu, pb, o);
      }
      if (g == 0) {
        pw[8 * m + 2 * t4] += pa;
        pw[8 * m + 2 * t4 + 1] += pb;
      }
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// F' = H0' - (M + M^T) / 2 with M = L^-1 diag(v) L lower triangular, so
// F'_ij = H0'_ij - M_ij / 2 below the diagonal and H0'_ii - M_ii on it.  Each warp takes 16 x 16 tiles of M (four
// accumulator tiles share each pair of operand loads), k from the tile's first
// column to its last row.
// vao: offset (doubles) into the dynamic shared memory.
template <int NW>
__device__ __noinline__ void fock_build(const double* __restrict__ L, const double* __restrict__ LiT,
                                        const double* __restrict__ Hp, int ld, int vao_at, int N,
                                        double* __restrict__ F, int ldf) {
  extern __shared__ __align__(16) unsigned char smraw[];
  const double* vao = reinterpret_cast<double*>(smraw) + vao_at;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, g = lane >> 2, t4 = lane & 3;
  const int nt = (N + 7) >> 3, nt2 = (nt + 1) >> 1;
  int I = 0, base = 0;  // base: tiles of the tile rows before I
  for (int task = wid;; task += NW) {
    while (I < nt2 && task >= base + I + 1) {
      base += I + 1;
      ++I;
    }
    if (I >= nt2) break;
    const int J = task - base;
    const bool i1 = 2 * I + 1 < nt, j1 = 2 * J + 1 < nt;  // the second tile row / column exists
    const int kend = min(nt, 2 * I + 2);
    double acc[2][2][2];
#pragma unroll
    for (int p = 0; p < 2; ++p)
#pragma unroll
      for (int r = 0; r < 2; ++r) acc[p][r][0] = acc[p][r][1] = 0.0;
    const double* li = LiT + 16 * I + g;
    const double* lj = L + 16 * J + g;
#pragma unroll 2
    for (int kt = 2 * J; kt < kend; ++kt) {
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const int k = 8 * kt + 2 * t4 + c;
        const double vk = k < N ? vao[k] : 0.0;
        const double* pi = li + (long long)k * ld;
        const double* pj = lj + (long long)k * ld;
        const double a0 = pi[0], a1 = i1 ? pi[8] : 0.0;
        const double b0 = pj[0] * vk, b1 = j1 ? pj[8] * vk : 0.0;
        dmma_m8n8k4(acc[0][0][0], acc[0][0][1], a0, b0);
        dmma_m8n8k4(acc[0][1][0], acc[0][1][1], a0, b1);
        dmma_m8n8k4(acc[1][0][0], acc[1][0][1], a1, b0);
        dmma_m8n8k4(acc[1][1][0], acc[1][1][1], a1, b1);
      }
    }
#pragma unroll
    for (int p = 0; p < 2; ++p)
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const int i = 16 * I + 8 * p + g, j = 16 * J + 8 * r + 2 * t4;
#pragma unroll
        for (int c = 0; c < 2; ++c)
          if (i < N && j + c <= i) {
            const double f = Hp[(long long)i * ld + j + c] - (i == j + c ? acc[p][r][c] : 0.5 * acc[p][r][c]);
            F[(long long)i * ldf + j + c] = f;
            F[(long long)(j + c) * ldf + i] = f;
          }
      }
  }
}

}  // namespace gfn1
