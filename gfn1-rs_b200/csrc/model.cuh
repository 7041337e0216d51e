// GFN1-xTB model functions shared by the device kernels: H0 shell-pair scaling,
// the distance polynomial, the coordination-number counting function and the
// Klopman-Ohno kernel.
#pragma once

#include "common.cuh"

namespace gfn1 {

struct Model {
  const ElemTable* elem;        // [kNZ]
  const double* pair_scaling;   // [kNZ*kNZ]
  const double* c6ref;          // [kNZ*kNZ*kMaxRef*kMaxRef], c6ref[(zi*kNZ+zj)*25 + ri*5 + rj]
  Globals g;
};

// k_shell / kshell_pair (src/params.rs:369-376, src/hamiltonian.rs:157-165)
__device__ __forceinline__ double k_shell(const Globals& g, int l) { return l == 0 ? g.ks : (l == 1 ? g.kp : g.kd); }
__device__ __forceinline__ double kshell_pair(const Globals& g, int li, int lj) {
  if ((li == 0 && lj == 1) || (li == 1 && lj == 0)) return g.ksp;
  return 0.5 * (k_shell(g, li) + k_shell(g, lj));
}

// hscale (src/hamiltonian.rs:140-155)
__device__ __forceinline__ double hscale(const Model& M, int za, int ka, int zb, int kb) {
  const ElemTable& ea = M.elem[za];
  const ElemTable& eb = M.elem[zb];
  const int va = ea.valence[ka], vb = eb.valence[kb];
  const int la = ea.l[ka], lb = eb.l[kb];
  if (va && vb) {
    const double den = (ea.en - eb.en) * (ea.en - eb.en);
    return M.pair_scaling[za * kNZ + zb] * kshell_pair(M.g, la, lb) * (1.0 + M.g.enscale * 0.01 * den);
  } else if (va) {
    return 0.5 * (kshell_pair(M.g, la, la) + M.g.kdiff);
  } else if (vb) {
    return 0.5 * (kshell_pair(M.g, lb, lb) + M.g.kdiff);
  }
  return M.g.kdiff;
}

// Exponential counting function and its radial derivative
// (src/coordination.rs:96-106), k = 16.
__device__ __forceinline__ void exp_count(double r, double rc, double& value, double& dvalue) {
  const double kcn = 16.0;
  const double raw = -kcn * (rc / r - 1.0);
  const double arg = fmin(80.0, fmax(-80.0, raw));
  const double e = exp(arg);
  value = 1.0 / (1.0 + e);
  dvalue = (raw < -80.0 || raw > 80.0) ? 0.0 : -kcn * rc * e / (r * r * (1.0 + e) * (1.0 + e));
}

// Klopman-Ohno effective kernel with exponent 2 (src/coulomb.rs:239-248)
__device__ __forceinline__ double harmonic_avg(double a, double b) { return 2.0 / (1.0 / a + 1.0 / b); }

// Exclusive prefix sums of the shell and AO counts of a molecule's atoms: the
// first shell and AO of each atom, [nat] the totals.  All threads of the CTA.
__device__ __forceinline__ void atom_offsets(const Model& M, const int* zs, int nat, int* atom_sh, int* atom_ao) {
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x;
    int s0 = 0, o0 = 0;
    for (int a0 = 0; a0 < nat; a0 += 32) {
      const int a = a0 + lane;
      int s = a < nat ? M.elem[zs[a]].nsh : 0, o = a < nat ? M.elem[zs[a]].nao : 0;
      const int ns = s, no = o;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int ts = __shfl_up_sync(0xffffffffu, s, d), to = __shfl_up_sync(0xffffffffu, o, d);
        if (lane >= d) {
          s += ts;
          o += to;
        }
      }
      if (a < nat) {
        atom_sh[a] = s0 + s - ns;
        atom_ao[a] = o0 + o - no;
      }
      s0 += __shfl_sync(0xffffffffu, s, 31);
      o0 += __shfl_sync(0xffffffffu, o, 31);
    }
    if (lane == 0) {
      atom_sh[nat] = s0;
      atom_ao[nat] = o0;
    }
  }
  __syncthreads();
}

// t-th unordered pair (i >= j) of a triangle with its diagonal.
__device__ __forceinline__ void tri_inverse(int t, int& i, int& j) {
  i = (int)((sqrtf(8.0f * (float)t + 1.0f) - 1.0f) * 0.5f);
  while ((long long)i * (i + 1) / 2 > t) --i;
  while ((long long)(i + 1) * (i + 2) / 2 <= t) ++i;
  j = t - i * (i + 1) / 2;
}

}  // namespace gfn1
