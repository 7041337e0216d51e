// Analytic nuclear gradient of the converged SCC (gfn1-rs src/gradient.rs:122-531,
// stock terms only).
//
// Phase 1, the unordered atom pairs (one lane each, or eight):
//   * inside the 30 bohr integral cutoff, for every shell pair and AO pair the
//     overlap derivative dS/dR is contracted with
//       coeff = P (2 h_ij - v_mu - v_nu) - 2 W
//     plus the H0 polynomial term 2 P h_ij S dlnPi/dR and the dE/dCN accumulation
//     (src/gradient.rs:358-455);
//   * the Coulomb term q_i q_j d gamma_ij / dR over the shells of the two atoms
//     (src/gradient.rs:493-516, no cutoff).
//   Each pair writes its contributions to a scratch slot.
// Phase 2, one warp per atom: fixed-order sum over the atom's pairs plus the
//   diagonal CN term dsedcn * P_mu,mu (src/gradient.rs:464-469).
// Phase 3, one warp per atom: the CN chain (dE/dCN_i + dE/dCN_j) dCN/dr
//   (src/gradient.rs:470-490), then repulsion + dispersion from the setup kernel.
// Fixed-order reductions make the gradient bitwise reproducible.
#include "common.cuh"
#include "model.cuh"
#include "overlap.cuh"

#include <algorithm>
#include <type_traits>

namespace gfn1 {

using L0 = std::integral_constant<int, 0>;
using L1 = std::integral_constant<int, 1>;
using L2 = std::integral_constant<int, 2>;

// Overlap-derivative contraction of one shell pair (mu shell of angular
// momentum LB on atom b, nu shell LA on atom a), src/gradient.rs:358-455:
// gmu += dS/dR_b [P (2 h - v_mu - v_nu) - 2 W] + R 2 P h S dlnPi/dR, plus the
// dE/dCN accumulation of both atoms.  xs = {h, v_mu + v_nu, dlnPi/dR factor,
// -kcn_mu hscale Pi, -kcn_nu hscale Pi}.
// G lanes share the primitive pairs: everything is linear in S and dS, so a lane
// contracts its own share.
template <int LB, int LA, int G>
__device__ __forceinline__ void grad_shell_pair(int sub, const ElemTable& eb, int kb, const double* xb, const ElemTable& ea,
                                                int ka, const double* xa, const double* P, const double* W, int N,
                                                int mu0, int nu0, const double (&xs)[5], const double (&rv)[3],
                                                double (&gmu)[3], double& dcmu, double& dcnu) {
  double Sb[2 * LB + 1][2 * LA + 1], dA[2 * LB + 1][2 * LA + 1][3];
  overlap_block_any<LB, LA, true, G>(sub, eb.nprim[kb], eb.alpha[kb], eb.coef[kb], xb, ea.nprim[ka], ea.alpha[ka],
                                  ea.coef[ka], xa, 3, Sb, dA);
  const double hij = xs[0], vsum = xs[1], dlog = xs[2];
#pragma unroll
  for (int x = 0; x < 2 * LB + 1; ++x)
#pragma unroll
    for (int y = 0; y < 2 * LA + 1; ++y) {
      const long long idx = (long long)(mu0 + x) * N + (nu0 + y);
      const double pp = P[idx], ww = W[idx];
      const double coeff = pp * (2.0 * hij - vsum) - 2.0 * ww;
      const double pg = dlog * (2.0 * pp * hij * Sb[x][y]);
#pragma unroll
      for (int c = 0; c < 3; ++c) gmu[c] += dA[x][y][c] * coeff + rv[c] * pg;
      dcmu += xs[3] * pp * Sb[x][y];
      dcnu += xs[4] * pp * Sb[x][y];
    }
}

// What the atom pairs of a molecule need.
struct GradCtx {
  const int *zs, *atom_sh, *atom_ao, *ord;
  const double* xyz;
  const double *P, *W, *se, *pot, *q;  // density, energy-weighted density, per shell: self energy, potential, charge
  double* slots;
  int N, nat;
};

enum GradPhase : int { kGradPairs = 1, kGradSums = 2, kGradChain = 4, kGradAll = 7 };

// The pairs of atoms u from positions [u0, u0 + nu) and w from [w0, w0 + nw) of the
// order by kind (same: the unordered pairs of one range).
template <int MaxL, int G>
__device__ __forceinline__ void grad_pair_class(const Model& M, const GradCtx& X, int u0, int nu, int w0, int nw,
                                                bool same, int split, int nsplit) {
  const int n = same ? nu * (nu - 1) / 2 : nu * nw;
  constexpr int per = 32 / G;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nwarp = blockDim.x >> 5, sub = lane % G;
  for (int t0 = (split * nwarp + wid) * per; t0 < n; t0 += nsplit * nwarp * per) {
    const int t = min(t0 + lane / G, n - 1);
    const bool store = t0 + lane / G < n && sub == 0;
    int i, j;
    if (same) {
      tri_inverse(t, i, j);
      ++i;  // i > j
    } else {
      i = t / nw;
      j = t - i * nw;
    }
    const int a = X.ord[u0 + i], b = X.ord[w0 + j];
    const int za = X.zs[a], zb = X.zs[b];
    const ElemTable& ea = M.elem[za];
    const ElemTable& eb = M.elem[zb];
    const double* xa = X.xyz + 3 * a;
    const double* xb = X.xyz + 3 * b;
    const double rv[3] = {xb[0] - xa[0], xb[1] - xa[1], xb[2] - xa[2]};
    const double r2 = rv[0] * rv[0] + rv[1] * rv[1] + rv[2] * rv[2];
    double gmu[3] = {0, 0, 0};  // derivative with respect to atom b (mu on b, nu on a)
    double dcmu = 0.0, dcnu = 0.0;
    if (r2 <= 900.0 && r2 > 1e-12) {
      const double r = sqrt(r2);
      const double rr = sqrt(r / (ea.rad + eb.rad));
      for (int kb = 0; kb < eb.nsh; ++kb) {
        const int smu = X.atom_sh[b] + kb;
        const double semu = X.se[smu], vmu = X.pot[smu];
        for (int ka = 0; ka < ea.nsh; ++ka) {
          const int snu = X.atom_sh[a] + ka;
          const double senu = X.se[snu], vnu = X.pot[snu];
          const double fi = 1.0 + eb.poly[kb] * rr, fj = 1.0 + ea.poly[ka] * rr;
          const double poly = fi * fj;
          const double hs = hscale(M, zb, kb, za, ka) * poly;
          const double hij = 0.5 * (semu + senu) * hs;
          double dlog = 0.0;  // src/gradient.rs:1157-1175 (scalar factor of rvec)
          if (fabs(poly) > 1e-18) dlog = (fi * ea.poly[ka] + fj * eb.poly[kb]) * 0.5 * rr / r2 / poly;
          const int mu0 = X.atom_ao[b] + eb.ao_first[kb], nu0 = X.atom_ao[a] + ea.ao_first[ka];
          const double xs[5] = {hij, vmu + vnu, dlog, -eb.kcn[kb] * hs, -ea.kcn[ka] * hs};
          auto pair = [&](auto lb, auto la) {
            grad_shell_pair<decltype(lb)::value, decltype(la)::value, G>(sub, eb, kb, xb, ea, ka, xa, X.P, X.W, X.N, mu0, nu0,
                                                                         xs, rv, gmu, dcmu, dcnu);
          };
          const L0 s{};
          const L1 p{};
          if constexpr (MaxL < 2) {
            switch (eb.l[kb] * 2 + ea.l[ka]) {
              case 0: pair(s, s); break;
              case 1: pair(s, p); break;
              case 2: pair(p, s); break;
              default: pair(p, p); break;
            }
          } else {
            const L2 d{};
            switch (eb.l[kb] * 3 + ea.l[ka]) {
              case 0: pair(s, s); break;
              case 1: pair(s, p); break;
              case 2: pair(s, d); break;
              case 3: pair(p, s); break;
              case 4: pair(p, p); break;
              case 5: pair(p, d); break;
              case 6: pair(d, s); break;
              case 7: pair(d, p); break;
              default: pair(d, d); break;
            }
          }
        }
      }
    }
    if (sub == 0 && r2 > 1e-24) {  // Coulomb: shells of b with shells of a
      for (int kb = 0; kb < eb.nsh; ++kb) {
        const double qi = X.q[X.atom_sh[b] + kb];
        for (int ka = 0; ka < ea.nsh; ++ka) {
          const double qj = X.q[X.atom_sh[a] + ka];
          const double g = harmonic_avg(eb.hard[kb], ea.hard[ka]);
          const double den = r2 + 1.0 / (g * g);
          const double pref = -1.0 / (den * sqrt(den)) * qi * qj;
          for (int c = 0; c < 3; ++c) gmu[c] += rv[c] * pref;
        }
      }
    }
#pragma unroll
    for (int o = 1; o < G; o <<= 1) {
#pragma unroll
      for (int c = 0; c < 3; ++c) gmu[c] += __shfl_xor_sync(0xffffffffu, gmu[c], o);
      dcmu += __shfl_xor_sync(0xffffffffu, dcmu, o);
      dcnu += __shfl_xor_sync(0xffffffffu, dcnu, o);
    }
    if (store) {  // every term is a function of R_b - R_a: the derivative for atom a is -gmu
      const bool up = a < b;
      double* slot = X.slots + 8LL * tri_index(up ? a : b, up ? b : a, X.nat);
      const double sg = up ? 1.0 : -1.0;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        slot[c] = -sg * gmu[c];
        slot[3 + c] = sg * gmu[c];
      }
      slot[6] = up ? dcnu : dcmu;
      slot[7] = up ? dcmu : dcnu;
    }
  }
}

// Molecule blockIdx.x of `mols` (or of the batch when null).  A warp takes atom
// pairs whose atoms have the same highest angular momenta, so that its lanes run
// the same shell-pair code (pairs in atom order mixed four kinds of code in every
// warp: 7.0 ms for the 4096-molecule batch).  MaxL: the highest shell angular
// momentum of the batch; the s/p instantiation (MaxL = 1) leaves out the d-shell
// blocks and their registers.
template <int MaxL, int G>
__global__ void __launch_bounds__(kGradThreads, MaxL < 2 ? kGradMinBlocksSp : kGradMinBlocks)
    grad_kernel(Batch B, Model M, int max_nat, const int* mols, int phases) {
  extern __shared__ double gsm[];
  const int m = mols ? mols[blockIdx.x] : blockIdx.x;
  if (B.status[m] != kOk) return;
  const int split = blockIdx.y, nsplit = gridDim.y;
  const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, wid = tid >> 5, nw = nt >> 5;
  const int a0 = B.atom_off[m], nat = B.atom_off[m + 1] - a0;
  const int sh0 = B.shell_off[m];
  const int N = B.ao_off[m + 1] - B.ao_off[m];
  const int at0 = split * nw + wid, atn = nsplit * nw;  // atoms of the warp
  double* xyz = gsm;                 // 3*max_nat
  double* dedcn = xyz + 3 * max_nat; // max_nat
  double* gel = dedcn + max_nat;     // 3*max_nat
  int* zs = (int*)(gel + 3 * max_nat);
  int* atom_sh = zs + max_nat;       // max_nat+1
  int* atom_ao = atom_sh + max_nat + 1;
  int* ord = atom_ao + max_nat + 1;  // max_nat: atoms by their highest angular momentum
  int* kind = ord + max_nat;         // max_nat
  int* count = kind + max_nat;       // 3
  const double* P = B.P + B.mat_off[m];  // density of the converged SCC
  double* slots = B.pairbuf + 8 * B.pair_off[m];

  for (int i = tid; i < nat; i += nt) {
    zs[i] = B.z[a0 + i];
    for (int x = 0; x < 3; ++x) xyz[3 * i + x] = B.xyz[3 * (a0 + i) + x];
  }
  if (tid < 3) count[tid] = 0;
  __syncthreads();
  atom_offsets(M, zs, nat, atom_sh, atom_ao);

  if (phases & kGradPairs) {
    for (int i = tid; i < nat; i += nt) {
      const ElemTable& e = M.elem[zs[i]];
      int l = 0;
      for (int k = 0; k < e.nsh; ++k) l = max(l, e.l[k]);
      kind[i] = l;
      atomicAdd(count + l, 1);
    }
    __syncthreads();
    for (int i = tid; i < nat; i += nt) {
      int rank = 0;
      for (int q = 0; q < nat; ++q) rank += kind[q] < kind[i] || (kind[q] == kind[i] && q < i);
      ord[rank] = i;
    }
    __syncthreads();
    const GradCtx X{zs, atom_sh, atom_ao, ord, xyz, P, B.W + B.mat_off[m], B.se + sh0, B.shell_pot + sh0, B.shell_q + sh0,
                    slots, N, nat};
    const int n0 = count[0], n1 = count[1], n2 = count[2];
    const int first[3] = {0, n0, n0 + n1}, num[3] = {n0, n1, n2};
    for (int c = 0; c < 6; ++c) {  // the costliest kinds first
      const int u = c < 3 ? 2 : (c < 5 ? 1 : 0), w = c < 3 ? 2 - c : (c == 3 ? 1 : 0);
      grad_pair_class<MaxL, G>(M, X, first[u], num[u], first[w], num[w], u == w, split, nsplit);
    }
  }
  if (phases == kGradAll) __syncthreads();

  if (phases & kGradSums) {  // per-atom sums in a fixed pair order
    for (int i = at0; i < nat; i += atn) {
      double g0 = 0, g1 = 0, g2 = 0, dc = 0;
      for (int j = lane; j < nat; j += 32) {
        if (j == i) continue;
        const int lo = min(i, j), hi = max(i, j);
        const double* slot = slots + 8LL * tri_index(lo, hi, nat);
        const int o = (i == lo) ? 0 : 3;
        g0 += slot[o];
        g1 += slot[o + 1];
        g2 += slot[o + 2];
        dc += slot[(i == lo) ? 6 : 7];
      }
      const ElemTable& e = M.elem[zs[i]];
      for (int k = 0; k < e.nsh; ++k) {
        const int mu = atom_ao[i] + e.ao_first[k] + lane;
        if (lane < 2 * e.l[k] + 1) dc -= e.kcn[k] * P[(long long)mu * N + mu];
      }
      g0 = warp_sum(g0);
      g1 = warp_sum(g1);
      g2 = warp_sum(g2);
      dc = warp_sum(dc);
      if (lane == 0) {
        gel[3 * i] = g0;
        gel[3 * i + 1] = g1;
        gel[3 * i + 2] = g2;
        dedcn[i] = dc;
        if (!(phases & kGradChain)) {  // for the chain's own launch
          B.grad[3 * (a0 + i)] = g0;
          B.grad[3 * (a0 + i) + 1] = g1;
          B.grad[3 * (a0 + i) + 2] = g2;
          B.atom_tmp[4 * (a0 + i)] = dc;
        }
      }
    }
    __syncthreads();
  }

  if (phases & kGradChain) {  // CN chain (cutoff 30 bohr) and the classical terms
    if (!(phases & kGradSums)) {
      for (int i = tid; i < nat; i += nt) dedcn[i] = B.atom_tmp[4 * (a0 + i)];
      for (int i = at0; i < nat; i += atn)
        if (lane < 3) gel[3 * i + lane] = B.grad[3 * (a0 + i) + lane];
      __syncthreads();
    }
    for (int i = at0; i < nat; i += atn) {
      const double ri = M.elem[zs[i]].rcov;
      double g[3] = {0.0, 0.0, 0.0};
      for (int j = lane; j < nat; j += 32) {
        if (j == i) continue;
        const double d[3] = {xyz[3 * i] - xyz[3 * j], xyz[3 * i + 1] - xyz[3 * j + 1], xyz[3 * i + 2] - xyz[3 * j + 2]};
        const double r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2];
        if (r2 <= 1e-24 || r2 > 900.0) continue;
        const double r = sqrt(r2);
        if (r <= 1e-12) continue;
        double v, dv;
        exp_count(r, ri + M.elem[zs[j]].rcov, v, dv);
        const double pref = (dedcn[i] + dedcn[j]) * dv / r;
        for (int c = 0; c < 3; ++c) g[c] += d[c] * pref;
      }
      for (int c = 0; c < 3; ++c) g[c] = warp_sum(g[c]);
      if (lane == 0)
        for (int c = 0; c < 3; ++c)
          B.grad[3 * (a0 + i) + c] = gel[3 * i + c] + g[c] + B.grad_classic[3 * (a0 + i) + c];
    }
  }
}

size_t grad_smem_bytes(int max_nat) {
  return sizeof(double) * 7 * (size_t)max_nat + sizeof(int) * (5 * (size_t)max_nat + 2 + 4);
}

// Launches the gradient of `n` molecules (`mols`, or the batch when null) whose
// largest has max_nat atoms; max_l: the batch's highest shell angular momentum
// (the s/p instantiation below 2).  One CTA per molecule when they fill the GPU
// (four CTAs on each SM) or one CTA holds a molecule's pairs at once; otherwise
// eight lanes per atom pair, as many CTAs per molecule as fill it, and a launch
// each for the sums and the chain, whose warps take an atom at a time.  (The sums and
// the chain together by one CTA, a launch less, were slower from 18 atoms on: one molecule
// of 18 atoms 67 against 65 us, of 48 95 / 68, of 159 283 / 79; 64 of 24 atoms 78 / 73.)
static int grad_steps(int max_nat) { return (max_nat * (max_nat - 1) / 2 + 15) / 16; }  // 16 pairs per CTA and step
int grad_launches(int n, int max_nat, int num_sms) {
  if (n <= 0) return 0;
  return n >= 4 * num_sms || grad_steps(max_nat) <= 1 ? 1 : 3;
}
cudaError_t launch_grad(int max_l, int n, int max_nat, int num_sms, cudaStream_t st, const Batch& B, const Model& M,
                        const int* mols) {
  const size_t smem = grad_smem_bytes(max_nat);
  const bool few = n < 4 * num_sms;
  auto* k = max_l >= 2 ? (few ? grad_kernel<2, 8> : grad_kernel<2, 1>) : (few ? grad_kernel<1, 8> : grad_kernel<1, 1>);
  if (smem > 48 * 1024) {
    const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  const int fill = std::max(1, 8 * num_sms / n);
  const int steps = grad_steps(max_nat);
  if (!few || steps <= 1) {
    k<<<dim3(n, 1), kGradThreads, smem, st>>>(B, M, max_nat, mols, kGradAll);
  } else {
    k<<<dim3(n, std::min(fill, steps)), kGradThreads, smem, st>>>(B, M, max_nat, mols, kGradPairs);
    const int y = std::max(1, std::min(fill, (max_nat + 3) / 4));
    k<<<dim3(n, y), kGradThreads, smem, st>>>(B, M, max_nat, mols, kGradSums);
    k<<<dim3(n, y), kGradThreads, smem, st>>>(B, M, max_nat, mols, kGradChain);
  }
  return cudaGetLastError();
}

}  // namespace gfn1
