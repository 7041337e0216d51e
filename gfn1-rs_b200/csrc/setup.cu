// Per-molecule setup kernel: one CTA per molecule builds everything that depends
// on the geometry only.
//
//  * coordination numbers with the exponential count, k = 16, cutoff 30 bohr for
//    H0 and 25 bohr for D3 (src/coordination.rs:51-106, src/dispersion.rs:1245-1251);
//  * self energies se = h - kcn*CN (src/hamiltonian.rs:98-104);
//  * the overlap S and H0 = S * 1/2 (se_i + se_j) * hscale * Pi(R) for every shell
//    pair inside the 30 bohr integral cutoff (src/integrals.rs:133-243,
//    src/hamiltonian.rs:91-134).  Each unordered shell pair is evaluated once and
//    mirrored, where the reference evaluates both directed atom pairs;
//  * the shell-resolved Klopman-Ohno matrix (src/coulomb.rs:82-107);
//  * repulsion energy and gradient (src/repulsion.rs:39-59, :139-159);
//  * D3(BJ) two-body energy and gradient with its CN chain
//    (src/dispersion.rs:1232-1360, :1629-1692, :1753-1787);
//  * the halogen-bond correction, energy and gradient (src/halogen.rs:64-160).
//
// Per-atom sums run over all partners in a fixed order, so the results are bitwise
// reproducible (no floating-point atomics).
#include "common.cuh"
#include "model.cuh"
#include "overlap.cuh"

#include <algorithm>

namespace gfn1 {

// S and H0 entries of one shell pair (both triangles); LA, LB are the shells'
// angular momenta, so the overlap block stays in registers.  G lanes share the
// pair (its primitive pairs, then its elements).
template <int LA, int LB, int G>
__device__ __forceinline__ void shell_pair_sh0(int sub, const ElemTable& ea, int ka, const double* xa,
                                               const ElemTable& eb, int kb, const double* xb, bool zero, bool store,
                                               double hij, double* S, double* H0, int N, int mu0, int nu0) {
  double Sb[2 * LA + 1][2 * LB + 1];
  double dummy[2 * LA + 1][2 * LB + 1][3];
  overlap_block_any<LA, LB, false, G>(sub, zero ? 0 : ea.nprim[ka], ea.alpha[ka], ea.coef[ka], xa, eb.nprim[kb],
                                      eb.alpha[kb], eb.coef[kb], xb, 2, Sb, dummy);
#pragma unroll
  for (int x = 0; x < 2 * LA + 1; ++x)
#pragma unroll
    for (int y = 0; y < 2 * LB + 1; ++y) {
      double sv = Sb[x][y];
#pragma unroll
      for (int o = 1; o < G; o <<= 1) sv += __shfl_xor_sync(0xffffffffu, sv, o);
      if (store && (x * (2 * LB + 1) + y) % G == sub) {
        const long long i1 = (long long)(mu0 + x) * N + (nu0 + y);
        const long long i2 = (long long)(nu0 + y) * N + (mu0 + x);
        S[i1] = sv;
        S[i2] = sv;
        H0[i1] = sv * hij;
        H0[i2] = sv * hij;
      }
    }
}

// What the shell pairs of a molecule need, in shared memory.
struct PairCtx {
  const int *zs, *atom_ao, *sh_atom, *sh_k, *ord;
  const double *xyz, *se;
  double *S, *H0;
  int N;
};

// S and H0 for the pairs of one class: shells [a0, a0 + na) x [b0, b0 + nb) of the
// order by angular momentum, or the unordered pairs of one range (same).
template <int LA, int LB, int G>
__device__ __forceinline__ void shell_pair_class(const Model& M, const PairCtx& P, int a0, int na, int b0, int nb,
                                                 bool same, int split, int nsplit) {
  const int n = same ? na * (na + 1) / 2 : na * nb;
  constexpr int per = 32 / G;  // pairs of a warp
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5, sub = lane % G;
  for (int t0 = (split * nw + wid) * per; t0 < n; t0 += nsplit * nw * per) {
    const int t = min(t0 + lane / G, n - 1);
    const bool store = t0 + lane / G < n;
    int i, j;
    if (same) {
      tri_inverse(t, i, j);
    } else {
      i = t / nb;
      j = t - i * nb;
    }
    const int si = P.ord[a0 + i], sj = P.ord[b0 + j];
    const int a = P.sh_atom[si], b = P.sh_atom[sj];
    const int za = P.zs[a], zb = P.zs[b];
    const int ka = P.sh_k[si], kb = P.sh_k[sj];
    const ElemTable& ea = M.elem[za];
    const ElemTable& eb = M.elem[zb];
    const int mu0 = P.atom_ao[a] + ea.ao_first[ka], nu0 = P.atom_ao[b] + eb.ao_first[kb];
    const double sei = P.se[si], sej = P.se[sj];
    double hij = 0.0;
    bool zero = false;
    if (a == b) {
      hij = 0.5 * (sei + sej);
    } else {
      const double dx = P.xyz[3 * a] - P.xyz[3 * b], dy = P.xyz[3 * a + 1] - P.xyz[3 * b + 1],
                   dz = P.xyz[3 * a + 2] - P.xyz[3 * b + 2];
      const double r2 = dx * dx + dy * dy + dz * dz;
      if (r2 <= 1e-24 || r2 > 900.0) {
        zero = true;
      } else {
        const double rr = sqrt(sqrt(r2) / (ea.rad + eb.rad));
        const double poly = (1.0 + ea.poly[ka] * rr) * (1.0 + eb.poly[kb] * rr);
        hij = 0.5 * (sei + sej) * hscale(M, za, ka, zb, kb) * poly;
      }
    }
    shell_pair_sh0<LA, LB, G>(sub, ea, ka, &P.xyz[3 * a], eb, kb, &P.xyz[3 * b], zero, store, hij, P.S, P.H0, P.N, mu0, nu0);
  }
}

// Halogen-bond energy of one molecule; adds its gradient to gc [nat*3].  For
// each donor X with strength c = 0.1 CXB, K is the nearest other atom within
// 20 bohr and every acceptor J (N, O, P, S) within 20 bohr contributes
//   E = c b^6 (u^2 - xbdamp u) / (1 + u^2),  b = 1/2 - T/4,  u = (r0 / r_JX)^6,
// T = (r_KX^2 + r_JX^2 - r_JK^2) / (r_KX r_JX), r0 = xbrad (R_X + R_J), with the
// reference's +1e-18 on r_JX and r_KX.  The gradient is taken through the
// three squared distances.
__device__ double halogen_term(const Model& M, const int* zs, const double* xyz, int nat, double* gc) {
  const double cut2 = 400.0, eps = 1e-18;
  const double damp = M.g.xbdamp, rscale = M.g.xbrad;
  double e = 0.0;
  for (int x = 0; x < nat; ++x) {
    const int zx = zs[x];
    const double c = M.elem[zx].xb;
    if (c == 0.0 || !(zx == 17 || zx == 35 || zx == 53 || zx == 85)) continue;
    int k = -1;  // nearest other atom inside the cutoff (first of equals)
    double kr2 = 0.0;
    for (int j = 0; j < nat; ++j) {
      if (j == x) continue;
      const double dx = xyz[3 * j] - xyz[3 * x], dy = xyz[3 * j + 1] - xyz[3 * x + 1], dz = xyz[3 * j + 2] - xyz[3 * x + 2];
      const double r2 = dx * dx + dy * dy + dz * dz;
      if (r2 <= 1e-24 || r2 > cut2) continue;
      if (k < 0 || r2 < kr2) {
        k = j;
        kr2 = r2;
      }
    }
    if (k < 0) continue;
    for (int j = 0; j < nat; ++j) {
      const int zj = zs[j];
      if (j == x || !(zj == 7 || zj == 8 || zj == 15 || zj == 16)) continue;
      double vjx[3], vkx[3], vjk[3];
      for (int q = 0; q < 3; ++q) {
        vjx[q] = xyz[3 * j + q] - xyz[3 * x + q];
        vkx[q] = xyz[3 * k + q] - xyz[3 * x + q];
        vjk[q] = xyz[3 * j + q] - xyz[3 * k + q];
      }
      const double djx = vjx[0] * vjx[0] + vjx[1] * vjx[1] + vjx[2] * vjx[2];
      const double dkx = vkx[0] * vkx[0] + vkx[1] * vkx[1] + vkx[2] * vkx[2];
      const double djk = vjk[0] * vjk[0] + vjk[1] * vjk[1] + vjk[2] * vjk[2];
      if (djx <= 1e-24 || djx > cut2 || djx <= eps || dkx <= eps) continue;
      const double rjx = sqrt(djx) + eps, rkx = sqrt(dkx) + eps;
      const double xy = sqrt(dkx * djx);
      if (xy <= eps) continue;
      const double T = (dkx + djx - djk) / xy;
      const double b = 0.5 - 0.25 * T;
      const double b2 = b * b, b5 = b2 * b2 * b, b6 = b5 * b;
      const double r0 = rscale * (M.elem[zx].rad + M.elem[zj].rad);
      const double t1 = r0 / rjx, t3 = t1 * t1 * t1, u = t3 * t3;
      const double num = u * u - damp * u, den = 1.0 + u * u;
      const double L = num / den;
      e += c * b6 * L;
      const double dL = (6.0 * u * (damp - 2.0 * u) / den + 12.0 * u * u * num / (den * den)) / rjx;
      const double dET = -1.5 * c * b5 * L;  // dE/dT
      const double gjx = dET * (1.0 / (rkx * rjx) - 0.5 * T / (rjx * rjx)) + 0.5 * c * b6 * dL / rjx;
      const double gkx = dET * (1.0 / (rkx * rjx) - 0.5 * T / (rkx * rkx));
      const double gjk = -dET / xy;
      for (int q = 0; q < 3; ++q) {
        gc[3 * j + q] += 2.0 * (gjx * vjx[q] + gjk * vjk[q]);
        gc[3 * x + q] -= 2.0 * (gjx * vjx[q] + gkx * vkx[q]);
        gc[3 * k + q] += 2.0 * (gkx * vkx[q] - gjk * vjk[q]);
      }
    }
  }
  return e;
}

// Phases of the setup of one molecule.  One CTA does them all for a molecule of
// a large batch; for few molecules several CTAs (gridDim.y) share one.
enum SetupPhase : int {
  kSetupCn = 1,       // coordination numbers
  kSetupPairs = 2,    // self energies, S, H0, Coulomb matrix (after the coordination numbers)
  kSetupClassic = 4,  // repulsion and D3 pair terms (after the coordination numbers)
  kSetupSums = 8,     // D3 coordination-number chain and energies (after the pair terms)
  kSetupHalogen = 16, // halogen bonds (after the sums)
  kSetupAll = 31
};

// Molecule blockIdx.x of `mols` (or of the batch when null).  Each unordered
// shell pair is one work item; a warp takes pairs of one class of angular
// momenta, so that its lanes run the same code (pairs in shell order put ss, sp
// and pp pairs side by side, and every warp ran all of them: 8.6 ms for the
// 4096-molecule batch).  G lanes share a pair where the pairs of the batch do not
// fill the GPU.  Atoms with many partners are one warp each, lanes over partners.
// CTAs 0..pair_parts-1 of a molecule take its shell pairs, the rest (or, without
// any, the same) its classical terms; with all phases in one launch every CTA
// forms the coordination numbers and at most one takes the classical terms.
// MaxL: the highest shell angular momentum of the batch; the s/p instantiation
// (MaxL = 1) leaves out the d-shell blocks and their registers.  128-thread CTAs,
// four per SM (128 registers).
template <int MaxL, int G>
__global__ void __launch_bounds__(128, 4) setup_kernel(Batch B, Model M, int enable_dispersion, int max_nat,
                                                        int max_nsh, const int* mols, int phases, int pair_parts) {
  extern __shared__ double smem[];
  const int m = mols ? mols[blockIdx.x] : blockIdx.x;
  if (B.status[m] != kOk) return;  // rejected by the host-side validation
  const int split = blockIdx.y, nsplit = gridDim.y;
  const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, wid = tid >> 5, nw = nt >> 5;
  const int a0 = B.atom_off[m], nat = B.atom_off[m + 1] - a0;
  const int sh0 = B.shell_off[m], nsh = B.shell_off[m + 1] - sh0;
  const int N = B.ao_off[m + 1] - B.ao_off[m];
  const bool all = phases == kSetupAll;
  const bool do_pairs = (phases & kSetupPairs) && split < pair_parts;
  const bool classical = nsplit == pair_parts || split >= pair_parts;
  const bool do_classic = (phases & kSetupClassic) && classical, do_sums = (phases & kSetupSums) && classical;
  // the warp's atoms: all of them in one CTA, or shared by the CTAs of the phase
  const int part = all ? 0 : (split >= pair_parts ? split - pair_parts : split);
  const int at0 = part * nw + wid, atn = all ? nw : (nsplit > pair_parts ? nsplit - pair_parts : nsplit) * nw;
  // Shared memory bounds the size of a molecule (setup_max_atoms), so what is not needed at the same
  // time shares its words: the coordination numbers serve until the weights are formed, dE/dCN and the
  // repulsion energies come after them; the tables of the shell pairs stand where the weights come.
  double* xyz = smem;                    // 3*max_nat
  double* cn = xyz + 3 * max_nat;        // max_nat
  double* cnd = cn + max_nat;            // max_nat
  double* dedcn = cn;
  double* erep = cnd;                    // repulsion and dispersion energy of each atom
  double* edis = cnd + max_nat;          // max_nat
  double* gw = edis + max_nat;           // kMaxRef*max_nat
  double* dgw = gw + kMaxRef * max_nat;  // kMaxRef*max_nat
  int* zs = (int*)(dgw + kMaxRef * max_nat);  // max_nat
  int* atom_sh = zs + max_nat;           // max_nat+1
  int* atom_ao = atom_sh + max_nat + 1;  // max_nat+1
  int* lcount = atom_ao + max_nat + 1;   // 3
  static_assert(2 * kMaxRef * sizeof(double) >= kMaxShAtom * (sizeof(double) + 4 * sizeof(int)),
                "the pair tables stand where the weights come");
  double* se = gw;                       // max_nsh
  int* sh_atom = (int*)(se + max_nsh);   // max_nsh
  int* sh_k = sh_atom + max_nsh;         // max_nsh
  int* ord = sh_k + max_nsh;             // max_nsh
  int* key = ord + max_nsh;              // max_nsh

  for (int i = tid; i < nat; i += nt) {
    zs[i] = B.z[a0 + i];
    xyz[3 * i] = B.xyz[3 * (a0 + i)];
    xyz[3 * i + 1] = B.xyz[3 * (a0 + i) + 1];
    xyz[3 * i + 2] = B.xyz[3 * (a0 + i) + 2];
  }
  if (tid < 3) lcount[tid] = 0;
  __syncthreads();
  atom_offsets(M, zs, nat, atom_sh, atom_ao);
  if (phases & kSetupCn) {  // coordination numbers (both cutoffs)
    for (int i = at0; i < nat; i += atn) {
      const double ri = M.elem[zs[i]].rcov;
      double c30 = 0.0, c25 = 0.0;
      for (int j = lane; j < nat; j += 32) {
        if (j == i) continue;
        const double dx = xyz[3 * j] - xyz[3 * i], dy = xyz[3 * j + 1] - xyz[3 * i + 1], dz = xyz[3 * j + 2] - xyz[3 * i + 2];
        const double r2 = dx * dx + dy * dy + dz * dz;
        if (r2 <= 1e-24 || r2 > 900.0) continue;
        const double rc = ri + M.elem[zs[j]].rcov;
        double v, dv;
        exp_count(sqrt(r2), rc, v, dv);
        c30 += v;
        if (r2 <= 625.0) c25 += v;
      }
      c30 = warp_sum(c30);
      c25 = warp_sum(c25);
      if (lane == 0) {
        cn[i] = c30;
        cnd[i] = c25;
        if (!all || split == 0) {
          B.cn[a0 + i] = c30;
          B.atom_tmp[4 * (a0 + i)] = c25;
        }
      }
    }
  } else {
    for (int i = tid; i < nat; i += nt) {
      cn[i] = B.cn[a0 + i];
      cnd[i] = B.atom_tmp[4 * (a0 + i)];
    }
  }
  __syncthreads();

  if (do_pairs) {
    for (int i = tid; i < nat; i += nt) {  // shells, self energies, shells per angular momentum
      const ElemTable& e = M.elem[zs[i]];
      for (int k = 0; k < e.nsh; ++k) {
        const int s = atom_sh[i] + k;
        const double v = e.hdiag[k] - e.kcn[k] * cn[i];
        sh_atom[s] = i;
        sh_k[s] = k;
        se[s] = v;
        key[s] = 16 * e.l[k] + e.nprim[k];
        if (split == 0) B.se[sh0 + s] = v;
        atomicAdd(lcount + e.l[k], 1);
      }
    }
    __syncthreads();
    // order of the shells by angular momentum, then primitives, then index
    for (int s = tid; s < nsh; s += nt) {
      const int ks = key[s];
      int rank = 0;
      for (int q = 0; q < nsh; ++q) rank += key[q] < ks || (key[q] == ks && q < s);
      ord[rank] = s;
    }
    __syncthreads();
    const PairCtx P{zs, atom_ao, sh_atom, sh_k, ord, xyz, se, B.S + B.mat_off[m], B.H0 + B.mat_off[m], N};
    const int n0 = lcount[0], n1 = lcount[1], n2 = lcount[2], part = split, parts = pair_parts;
    if constexpr (MaxL >= 2) {
      shell_pair_class<2, 2, G>(M, P, n0 + n1, n2, n0 + n1, n2, true, part, parts);
      shell_pair_class<1, 2, G>(M, P, n0, n1, n0 + n1, n2, false, part, parts);
      shell_pair_class<0, 2, G>(M, P, 0, n0, n0 + n1, n2, false, part, parts);
    }
    shell_pair_class<1, 1, G>(M, P, n0, n1, n0, n1, true, part, parts);
    shell_pair_class<0, 1, G>(M, P, 0, n0, n0, n1, false, part, parts);
    shell_pair_class<0, 0, G>(M, P, 0, n0, 0, n0, true, part, parts);

    // ---- Klopman-Ohno matrix (exactly symmetric: G_ij and G_ji come from the
    // same commutative expression, which the SCC's column reads rely on)
    double* Gm = B.gam + B.gam_off[m];
    for (long long w = tid + (long long)part * nt; w < (long long)nsh * nsh; w += (long long)nt * parts) {
      const int i = (int)(w / nsh), j = (int)(w - (long long)i * nsh);
      const int a = sh_atom[i], b = sh_atom[j];
      const double g = harmonic_avg(M.elem[zs[a]].hard[sh_k[i]], M.elem[zs[b]].hard[sh_k[j]]);
      double v;
      if (a == b) v = g;
      else {
        const double dx = xyz[3 * a] - xyz[3 * b], dy = xyz[3 * a + 1] - xyz[3 * b + 1], dz = xyz[3 * a + 2] - xyz[3 * b + 2];
        const double r2 = dx * dx + dy * dy + dz * dz;
        v = rsqrt(r2 + 1.0 / (g * g));  // 1 ulp, as a square root and a divide
      }
      Gm[w] = v;
    }
  }

  if (do_classic) {
    if (do_pairs) __syncthreads();  // the pair tables have served
    if (enable_dispersion) {
      for (int i = tid; i < nat; i += nt) {  // reference weights, src/dispersion.rs:1629-1692
        const ElemTable& e = M.elem[zs[i]];
        const int nr = e.d3_nref;
        double logit[kMaxRef], mx = -INFINITY;
        for (int k = 0; k < nr; ++k) {
          const double d = cnd[i] - e.d3_cnref[k];
          logit[k] = -4.0 * d * d;
          mx = fmax(mx, logit[k]);
        }
        double raw[kMaxRef], norm = 0.0, dnorm = 0.0;
        for (int k = 0; k < nr; ++k) {
          raw[k] = exp(logit[k] - mx);
          norm += raw[k];
          dnorm += 8.0 * (e.d3_cnref[k] - cnd[i]) * raw[k];
        }
        const double ninv = 1.0 / norm;
        for (int k = 0; k < kMaxRef; ++k) {
          double gwk = 0.0, dgk = 0.0;
          if (k < nr) {
            const double expd = 8.0 * (e.d3_cnref[k] - cnd[i]) * raw[k];
            gwk = raw[k] * ninv;
            dgk = expd * ninv - raw[k] * dnorm * ninv * ninv;
            if (!isfinite(gwk)) gwk = 0.0;
            if (!isfinite(dgk)) dgk = 0.0;
          }
          gw[k * max_nat + i] = gwk;
          dgw[k * max_nat + i] = dgk;
        }
      }
    }
    __syncthreads();
    const double s6 = M.g.s6, s8 = M.g.s8, a1 = M.g.a1, a2 = M.g.a2;
    for (int i = at0; i < nat; i += atn) {
      const int zi = zs[i];
      const ElemTable& ei = M.elem[zi];
      double gx = 0, gy = 0, gz = 0, er = 0, ed = 0, dc = 0;
      for (int j = lane; j < nat; j += 32) {
        if (j == i) continue;
        const int zj = zs[j];
        const ElemTable& ej = M.elem[zj];
        const double dx = xyz[3 * j] - xyz[3 * i], dy = xyz[3 * j + 1] - xyz[3 * i + 1], dz = xyz[3 * j + 2] - xyz[3 * i + 2];
        const double r2 = dx * dx + dy * dy + dz * dz;
        double pref = 0.0;  // gradient along r_j - r_i
        if (r2 > 1e-24 && r2 <= 625.0) {  // repulsion (pairs within 25 bohr)
          const double r = sqrt(r2);
          const double alpha = sqrt(ei.repa * ej.repa);
          const double zeff = ei.repb * ej.repb;
          const double k = (zi <= 2 && zj <= 2) ? M.g.kexplight : M.g.kexp;
          const double rk = k == 1.5 ? r * sqrt(r) : pow(r, k);
          const double en = zeff * exp(-alpha * rk) / r;
          pref = (alpha * rk * k + 1.0) * en / r2;
          er += 0.5 * en;
        }
        if (enable_dispersion && r2 > 1e-14 && r2 <= 2500.0) {  // D3(BJ), src/dispersion.rs:1260-1297
          const double* c6r = M.c6ref + (long long)(zi * kNZ + zj) * (kMaxRef * kMaxRef);
          double c6 = 0.0, dc6 = 0.0;
          for (int ra = 0; ra < ei.d3_nref; ++ra) {
            double rowc = 0.0;
            for (int rb = 0; rb < ej.d3_nref; ++rb) rowc += gw[rb * max_nat + j] * c6r[ra * kMaxRef + rb];
            c6 += gw[ra * max_nat + i] * rowc;
            dc6 += dgw[ra * max_nat + i] * rowc;
          }
          const double r4r2ij = 3.0 * ei.r4r2 * ej.r4r2;
          const double r0 = a1 * sqrt(r4r2ij) + a2;
          const double r02 = r0 * r0, r06 = r02 * r02 * r02, r08 = r06 * r02;
          const double r4 = r2 * r2;
          const double t6 = 1.0 / (r4 * r2 + r06);
          const double t8 = 1.0 / (r4 * r4 + r08);
          const double d6 = -6.0 * r4 * t6 * t6;
          const double d8 = -8.0 * r4 * r2 * t8 * t8;
          const double e6 = s6 * t6 + s8 * r4r2ij * t8;
          ed -= 0.5 * c6 * e6;
          pref += c6 * (s6 * d6 + s8 * r4r2ij * d8);
          dc -= dc6 * e6;
        }
        gx += dx * pref;
        gy += dy * pref;
        gz += dz * pref;
      }
      gx = warp_sum(gx);
      gy = warp_sum(gy);
      gz = warp_sum(gz);
      er = warp_sum(er);
      ed = warp_sum(ed);
      dc = warp_sum(dc);
      if (lane == 0) {
        B.grad_classic[3 * (a0 + i)] = gx;
        B.grad_classic[3 * (a0 + i) + 1] = gy;
        B.grad_classic[3 * (a0 + i) + 2] = gz;
        dedcn[i] = dc;
        erep[i] = er;
        edis[i] = ed;
        if (!all) {
          B.atom_tmp[4 * (a0 + i) + 1] = dc;
          B.atom_tmp[4 * (a0 + i) + 2] = er;
          B.atom_tmp[4 * (a0 + i) + 3] = ed;
        }
      }
    }
    __syncthreads();
  }

  if (do_sums) {
    if (!all) {
      for (int i = tid; i < nat; i += nt) {
        dedcn[i] = B.atom_tmp[4 * (a0 + i) + 1];
        erep[i] = B.atom_tmp[4 * (a0 + i) + 2];
        edis[i] = B.atom_tmp[4 * (a0 + i) + 3];
      }
      __syncthreads();
    }
    if (enable_dispersion)
      for (int i = at0; i < nat; i += atn) {  // CN chain, src/dispersion.rs:1330-1342
        const double ri = M.elem[zs[i]].rcov;
        double gx = 0, gy = 0, gz = 0;
        for (int j = lane; j < nat; j += 32) {
          if (j == i) continue;
          const double dx = xyz[3 * i] - xyz[3 * j], dy = xyz[3 * i + 1] - xyz[3 * j + 1], dz = xyz[3 * i + 2] - xyz[3 * j + 2];
          const double r2 = dx * dx + dy * dy + dz * dz;
          if (r2 <= 1e-24 || r2 > 625.0) continue;
          const double r = sqrt(r2);
          double v, dv;
          exp_count(r, ri + M.elem[zs[j]].rcov, v, dv);
          const double pref = (dedcn[i] + dedcn[j]) * dv / r;
          gx += dx * pref;
          gy += dy * pref;
          gz += dz * pref;
        }
        gx = warp_sum(gx);
        gy = warp_sum(gy);
        gz = warp_sum(gz);
        if (lane == 0) {
          B.grad_classic[3 * (a0 + i)] += gx;
          B.grad_classic[3 * (a0 + i) + 1] += gy;
          B.grad_classic[3 * (a0 + i) + 2] += gz;
        }
      }
    __syncthreads();
    if (part == 0 && wid == 0) {
      double er = 0.0, ed = 0.0;
      for (int i = lane; i < nat; i += 32) {
        er += erep[i];
        ed += edis[i];
      }
      er = warp_sum(er);
      ed = warp_sum(ed);
      if (lane == 0) {
        double* t = B.terms + (long long)m * kTerms;
        for (int k = 0; k < kTerms; ++k) t[k] = 0.0;
        t[2] = er;
        t[7] = ed;
      }
    }
  }
  // ---- halogen bonds (src/halogen.rs:64-160, triples :716-786).  Donors (Cl, Br,
  // I, At with a CXB entry) are rare, so one thread sums every triple in atom
  // order after the per-atom terms.
  if ((phases & kSetupHalogen) && classical && tid == 0)
    B.terms[(long long)m * kTerms + 8] = halogen_term(M, zs, xyz, nat, B.grad_classic + 3LL * a0);
}

// 140 bytes an atom: 1660 atoms in the 227 KB of a CTA.
size_t setup_smem_bytes(int max_nat) {
  return sizeof(double) * (6 + 2 * kMaxRef) * (size_t)max_nat + sizeof(int) * (3 * (size_t)max_nat + 2 + 4);
}
// Atoms of the largest molecule whose set-up fits `smem` bytes of shared memory.
int setup_max_atoms(size_t smem) {
  int n = (int)(smem / (sizeof(double) * (6 + 2 * kMaxRef) + 3 * sizeof(int)));
  while (n > 0 && setup_smem_bytes(n) > smem) --n;
  return n;
}

// Launches the setup of `n` molecules (`mols`, or the batch when null) whose
// largest has max_nat atoms and max_nsh shells; max_l: the batch's highest shell
// angular momentum (the s/p instantiation below 2); halogens: some atom is a
// halogen-bond donor.
//  * one CTA per molecule when they fill the GPU (four CTAs on each SM);
//  * otherwise eight lanes per shell pair and as many CTAs per molecule as fill
//    it: one launch for up to kSetupOneLaunch atoms (whose classical terms one CTA
//    finishes while the others form the pairs), beyond that one launch each for
//    the coordination numbers, the pair terms and the sums.  Measured, us, one
//    launch / three: one molecule of 15 atoms 35 / 43, 18 37 / 42, 24 43 / 41, 48
//    90 / 46; 8 of 15 32 / 41, 18 37 / 41, 36 89 / 43; 64 of 15 50 / 47, 18 63 / 53.
constexpr int kSetupOneLaunch = 16;
int setup_launches(int n, int max_nat, bool halogens, int num_sms) {
  return n <= 0 ? 0 : (n >= 4 * num_sms || max_nat <= kSetupOneLaunch ? 1 : (halogens ? 4 : 3));
}
cudaError_t launch_setup(int max_l, int n, int max_nat, int max_nsh, bool halogens, int num_sms, cudaStream_t st,
                         const Batch& B, const Model& M, int enable_dispersion, const int* mols) {
  const size_t smem = setup_smem_bytes(max_nat);
  const bool few = n < 4 * num_sms;
  auto* k = max_l >= 2 ? (few ? setup_kernel<2, 8> : setup_kernel<2, 1>) : (few ? setup_kernel<1, 8> : setup_kernel<1, 1>);
  if (smem > 48 * 1024) {
    const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  const int fill = std::max(1, 8 * num_sms / n);
  const int yp = std::max(1, std::min(fill, (max_nsh * (max_nsh + 1) / 2 + 31) / 32));  // 16 pairs per CTA and step
  const int ya = std::max(1, std::min(fill, (max_nat + 3) / 4));                        // four atoms per CTA and step
  auto launch = [&](int y, int phases, int pair_parts) {
    k<<<dim3(n, y), 128, smem, st>>>(B, M, enable_dispersion, max_nat, max_nsh, mols, phases, pair_parts);
  };
  if (!few) {
    launch(1, kSetupAll, 1);
  } else if (max_nat <= kSetupOneLaunch) {
    launch(yp + 1, kSetupAll, yp);
  } else {
    launch(ya, kSetupCn, 0);
    launch(yp + ya, kSetupPairs | kSetupClassic, yp);
    launch(ya, kSetupSums, 0);
    if (halogens) launch(1, kSetupHalogen, 0);
  }
  return cudaGetLastError();
}

}  // namespace gfn1
