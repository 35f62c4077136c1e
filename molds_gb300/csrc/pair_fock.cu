// Kernels (a) and (b): one-time pair integrals and the NDDO Fock build.
//
// (a) pair_kernel -- one warp per atom pair of every molecule in the batch.
//     Evaluates the distinct diatomic-frame two-centre integrals from the term
//     table (a lane per term, then a lane per local integral sums its own), rotates the packed 10x10 block to the
//     molecular frame as T2 L T2^T (T2 = symmetrised product rotation), and
//     stores it with coalesced lane-strided stores.  The same warp computes the
//     Slater overlap of the pair (diatomic frame, then rotated), the resonance
//     block 1/2 (beta_mu + beta_nu) S_mu,nu of the core Hamiltonian, and the
//     core-core repulsion E_AB.
//     MolDS: Mndo::CalcTwoElecsTwoAtomCores (src/mndo/Mndo.cpp:3703-3820),
//     CalcDiatomicTwoElecsTwoCores (:3948-4025), RotateDiatomicTwoElecsTwoCores
//     ToSpaceFrame (:4223-4293), Cndo2::CalcOverlapAOs (src/cndo/Cndo2.cpp:
//     4030-4146), Mndo::GetDiatomCoreRepulsionEnergy (:319-327, :223-240) and
//     Am1::GetDiatomCoreRepulsionEnergy (src/am1/Am1.cpp:145-170).
//
// (b) hcore_kernel, a warp per atom, and fock_kernel, one CTA per atom.  Coulomb
//     terms of the diagonal block of atom A are gathered from all partner blocks
//     (Fock: a thread per partner and orbital pair) and summed in a fixed order, so
//     the result does not depend on scheduling (bitwise reproducible, alone or in a
//     batch).  The exchange block of a pair is written by the CTA of its first atom.
//     MolDS: Cndo2::CalcFockMatrix (src/cndo/Cndo2.cpp:1526-1636) with
//     Mndo::GetFockDiagElement (src/mndo/Mndo.cpp:422-488), GetFockOffDiagElement
//     (:490-580), GetCoulombInt/GetExchangeInt (:583-639), GetElectronCoreAttraction
//     (:643-650).
#include <cuda_runtime.h>
#include <algorithm>
#include <cmath>
#include "nddo_batch.cuh"
#include "kernels.h"
#include "nddo_dual.cuh"

namespace nddo {

__constant__ nddo_atom_params c_params[kNumParamSlots];
__constant__ double c_inv[128];   // c_inv[j] = 1 / j

void upload_primitives(const nddo_atom_params* p, cudaStream_t s);

void upload_params(const nddo_atom_params* p, cudaStream_t s) {
  static double inv[128];
  inv[0] = 0.0;
  for (int j = 1; j < 128; ++j) inv[j] = 1.0 / (double)j;
  cudaMemcpyToSymbolAsync(c_params, p, sizeof(nddo_atom_params) * kNumParamSlots, 0,
                          cudaMemcpyHostToDevice, s);
  cudaMemcpyToSymbolAsync(c_inv, inv, sizeof(inv), 0, cudaMemcpyHostToDevice, s);
  upload_primitives(p, s);
}

__device__ __forceinline__ double sel3(int i, double a, double b, double c) {
  return i == 0 ? a : (i == 1 ? b : c);
}

constexpr int kPairWarps = 4;

// E_AB of MNDO (Mndo.cpp:223-240, 319-327) plus the AM1/PM3 Gaussians
// (Am1.cpp:145-170); ssss = (s_A s_A | s_B s_B).
template <typename T>
__device__ __forceinline__ T core_core(const nddo_atom_params& pa, const nddo_atom_params& pb, T R, T ssss,
                                       int theory) {
  T f;
  const bool a_no = (pa.atomic_number == 7 || pa.atomic_number == 8);
  const bool b_no = (pb.atomic_number == 7 || pb.atomic_number == 8);
  if (pa.atomic_number == 1 && b_no)
    f = 1.0 + (R / NDDO_ANG2AU) * exp(-pb.alpha * R) + exp(-pa.alpha * R);
  else if (pb.atomic_number == 1 && a_no)
    f = 1.0 + (R / NDDO_ANG2AU) * exp(-pa.alpha * R) + exp(-pb.alpha * R);
  else
    f = 1.0 + exp(-pa.alpha * R) + exp(-pb.alpha * R);
  T e = (double)(pa.core_charge * pb.core_charge) * ssss * f;
  if (theory != NDDO_MNDO) {
    T t = 0.0;
    for (int i = 0; i < 4; ++i) {
      if (pa.gk[i] != 0.0) { const T d = R - pa.gm[i]; t += pa.gk[i] * exp(-pa.gl[i] * (d * d)); }
      if (pb.gk[i] != 0.0) { const T d = R - pb.gm[i]; t += pb.gk[i] * exp(-pb.gl[i] * (d * d)); }
    }
    e += (double)(pa.core_charge * pb.core_charge) * t * NDDO_ANG2AU / R;
  }
  if (theory == NDDO_PM3PDDG) {
    // PDDG term (Pm3Pddg.cpp:143-165, 239-245); n = valence electrons = core charge
    const double na = pa.core_charge, nb = pb.core_charge;
    T t = 0.0;
    for (int i = 0; i < 2; ++i)
      for (int k = 0; k < 2; ++k) {
        const T x = R - pa.pddg_da[i] - pb.pddg_da[k];
        t += (na * pa.pddg_pa[i] + nb * pb.pddg_pa[k]) * exp(-10.0 / (NDDO_ANG2AU * NDDO_ANG2AU) * (x * x));
      }
    e += t / (na + nb);
  }
  return e;
}

// core_core by a warp: the up to fourteen exponentials over the lanes, the sums
// in core_core's order by every lane
__device__ __forceinline__ double core_core_warp(const nddo_atom_params& pa, const nddo_atom_params& pb, double R,
                                                 double ssss, int theory, int lane) {
  // lanes 0-3 and 4-7: the Gaussians of A and B; 8, 9: e^{-alpha R}; 10-13: PDDG
  double x = 0.0;
  bool use = false;
  if (lane < 8) {
    const nddo_atom_params& p = lane < 4 ? pa : pb;
    const int i = lane & 3;
    use = theory != NDDO_MNDO && p.gk[i] != 0.0;
    const double d = R - p.gm[i];
    x = -p.gl[i] * (d * d);
  } else if (lane < 10) {
    use = true;
    x = -(lane == 8 ? pa : pb).alpha * R;
  } else if (lane < 14) {
    use = theory == NDDO_PM3PDDG;
    const double d = R - pa.pddg_da[(lane - 10) >> 1] - pb.pddg_da[(lane - 10) & 1];
    x = -10.0 / (NDDO_ANG2AU * NDDO_ANG2AU) * (d * d);
  }
  const double e = use ? exp(x) : 0.0;
  auto at = [&](int l) { return __shfl_sync(0xffffffffu, e, l); };
  const double ea = at(8), eb = at(9);
  const bool a_no = (pa.atomic_number == 7 || pa.atomic_number == 8);
  const bool b_no = (pb.atomic_number == 7 || pb.atomic_number == 8);
  double f;
  if (pa.atomic_number == 1 && b_no) f = 1.0 + (R / NDDO_ANG2AU) * eb + ea;
  else if (pb.atomic_number == 1 && a_no) f = 1.0 + (R / NDDO_ANG2AU) * ea + eb;
  else f = 1.0 + ea + eb;
  double s = (double)(pa.core_charge * pb.core_charge) * ssss * f;
  if (theory != NDDO_MNDO) {
    double t = 0.0;
    for (int i = 0; i < 4; ++i) {
      const double ga = at(i), gb = at(4 + i);
      if (pa.gk[i] != 0.0) t += pa.gk[i] * ga;
      if (pb.gk[i] != 0.0) t += pb.gk[i] * gb;
    }
    s += (double)(pa.core_charge * pb.core_charge) * t * NDDO_ANG2AU / R;
  }
  if (theory == NDDO_PM3PDDG) {
    const double na = pa.core_charge, nb = pb.core_charge;
    double t = 0.0;
    for (int i = 0; i < 2; ++i)
      for (int k = 0; k < 2; ++k) t += (na * pa.pddg_pa[i] + nb * pb.pddg_pa[k]) * at(10 + 2 * i + k);
    s += t / (na + nb);
  }
  return s;
}

// One overlap combination of the pair in the diatomic frame (thread-level):
// norm * ang * (R/2)^(na+nb+1) * sum_t c_t A_i(p) B_j(q).
template <typename T>
__device__ __forceinline__ T overlap_combo(const OverlapTable* __restrict__ ovt, int na, int nb, int c, double za,
                                           double zb, double norm, T R) {
  const int km = ovt->kmax[na - 1][nb - 1][c];
  T a[12], b[12];
  aux_a_all(0.5 * R * (za + zb), km, a);
  aux_b_all(0.5 * R * (za - zb), km, b, c_inv);
  T s = 0.0;
  const int nt = ovt->nterms[na - 1][nb - 1][c];
  for (int t = 0; t < nt; ++t)
    s += ovt->tc[na - 1][nb - 1][c][t] * a[ovt->ti[na - 1][nb - 1][c][t]] * b[ovt->tj[na - 1][nb - 1][c][t]];
  T rp = 1.0;
  for (int i = 0; i < na + nb + 1; ++i) rp *= 0.5 * R;
  return (norm * ovt->ang[c]) * rp * s;
}

__device__ __forceinline__ double slot_value(const EriTable* __restrict__ eri, int slot, double R,
                                             const nddo_atom_params& pa, const nddo_atom_params& pb) {
  double v = 0.0;
  const int nt = eri->nterms[slot];
  for (int t = 0; t < nt; ++t) {
    const EriTerm e = eri->terms[slot][t];
    const double da = e.la == 0 ? pa.d[0] : (e.la == 1 ? pa.d[1] : pa.d[2]);
    const double db = e.lb == 0 ? pb.d[0] : (e.lb == 1 ? pb.d[1] : pb.d[2]);
    const double ra = e.la == 0 ? pa.rho[0] : (e.la == 1 ? pa.rho[1] : pa.rho[2]);
    const double rb = e.lb == 0 ? pb.rho[0] : (e.lb == 1 ? pb.rho[1] : pb.rho[2]);
    const double l = R + (double)e.c1 * da + (double)e.c2 * db;
    const double u = (double)e.c3 * da + (double)e.c4 * db;
    const double w = (double)e.c5 * da + (double)e.c6 * db;
    const double a = ra + rb;
    v += e.coef * rsqrt(l * l + u * u + w * w + a * a);
  }
  return v;
}

// Pairs with at least one hydrogen, one thread per pair.  With X the atom
// carrying p orbitals (if any) and u the unit vector from X to H, the rotated
// block (X mu nu | H s s) of the local values s0 = (ss|ss), s3 = (xx|ss),
// s4 = (zz|ss), s10 = (sz|ss) is
//   (s s | s s) = s0,   (s p_mu | s s) = s10 u_mu,
//   (p_mu p_nu | s s) = s3 delta_mu,nu + (s4 - s3) u_mu u_nu,
// which is T2 L T2^T written out for this sparsity (the local z axis is u).
// Block layout is the same for both atom orders: 10 or 1 doubles.
__global__ void __launch_bounds__(128)
pair_light_kernel(const DevAtom* __restrict__ atoms, const DevPair* __restrict__ pairs,
                  const int* __restrict__ list, long long n, const DevMol* __restrict__ mols,
                  const EriTable* __restrict__ eri, const OverlapTable* __restrict__ ovt,
                  double* __restrict__ blocks, double* __restrict__ H, double* __restrict__ ecore_pair) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  const long long p = list ? list[t] : t;
  const DevPair pr = pairs[p];
  const DevAtom A = atoms[pr.a], B = atoms[pr.b];
  if (A.nao == 4 && B.nao == 4) return;   // no list: pair_kernel's
  const bool swap = (A.nao == 1 && B.nao == 4);
  const DevAtom X = swap ? B : A, Y = swap ? A : B;       // Y is a hydrogen
  const nddo_atom_params& px = c_params[X.pidx];
  const nddo_atom_params& py = c_params[Y.pidx];
  const DevMol mol = mols[pr.mol];
  const double dx = Y.x - X.x, dy = Y.y - X.y, dz = Y.z - X.z;
  const double R = sqrt(dx * dx + dy * dy + dz * dz);
  const double iR = 1.0 / R;
  const double u[4] = {0.0, dy * iR, dz * iR, dx * iR};   // orbital order s, py, pz, px
  const double s0 = slot_value(eri, 0, R, px, py);
  double* out = blocks + pr.blk;
  const long long ld = mol.nao;
  double Sss, Sps = 0.0;
  Sss = overlap_combo(ovt, px.principal_n, py.principal_n, 0, px.zeta[0], py.zeta[0],
                      px.sto_norm[0] * py.sto_norm[0], R);
  if (X.nao == 4) {
    const double s3 = slot_value(eri, 3, R, px, py);
    const double s4 = slot_value(eri, 4, R, px, py);
    const double s10 = slot_value(eri, 10, R, px, py);
    for (int P = 0; P < 10; ++P) {
      int m, k;
      unpack_index(P, &m, &k);
      double v;
      if (m == 0 && k == 0) v = s0;
      else if (m == 0) v = s10 * u[k];
      else v = (m == k ? s3 : 0.0) + (s4 - s3) * u[m] * u[k];
      out[P] = v;
    }
    Sps = overlap_combo(ovt, px.principal_n, py.principal_n, 2, px.zeta[1], py.zeta[0],
                        px.sto_norm[1] * py.sto_norm[0], R);
  } else {
    out[0] = s0;
  }
  // resonance entries 1/2 (beta_mu + beta_H) S_mu,H  (S_p,H = u_mu S_sigma-s)
  for (int mu = 0; mu < X.nao; ++mu) {
    const double sv = (mu == 0) ? Sss : u[mu] * Sps;
    const double h = 0.5 * (px.beta[mu == 0 ? 0 : 1] + py.beta[0]) * sv;
    const long long r = X.ao0 + mu, c = Y.ao0;
    H[mol.mat0 + r * ld + c] = h;
    H[mol.mat0 + c * ld + r] = h;
  }
  ecore_pair[p] = core_core(px, py, R, s0, mol.theory);
}

// Pairs of two atoms with s and p orbitals, one warp per pair.
__global__ void __launch_bounds__(kPairWarps * 32)
pair_kernel(const DevAtom* __restrict__ atoms, const DevPair* __restrict__ pairs, const int* __restrict__ list,
            long long npairs, const DevMol* __restrict__ mols, const EriTable* __restrict__ eri,
            const OverlapTable* __restrict__ ovt, double* __restrict__ blocks,
            double* __restrict__ H, double* __restrict__ ecore_pair) {
  __shared__ double s_val[kPairWarps][24];
  __shared__ double s_T2[kPairWarps][100];
  __shared__ double s_L[kPairWarps][100];
  __shared__ double s_M[kPairWarps][100];
  __shared__ double s_ab[kPairWarps][4][2][7];
  __shared__ double s_ov[kPairWarps][8];
  __shared__ double s_R[kPairWarps][16];
  __shared__ double s_term[kPairWarps][kMaxFlatTerms];
  const unsigned full = 0xffffffffu;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long pi = (long long)blockIdx.x * kPairWarps + warp;
  if (pi >= npairs) return;
  const long long p = list ? list[pi] : pi;

  const DevPair pr = pairs[p];
  const DevAtom A = atoms[pr.a], B = atoms[pr.b];
  if (!list && (A.nao == 1 || B.nao == 1)) return;   // no list: pair_light_kernel's
  const DevMol mol = mols[pr.mol];
  const nddo_atom_params& pa = c_params[A.pidx];
  const nddo_atom_params& pb = c_params[B.pidx];
  const double dx = B.x - A.x, dy = B.y - A.y, dz = B.z - A.z;
  const double R = sqrt(dx * dx + dy * dy + dz * dz);

  // ---- rotation matrix (lane 0) ------------------------------------------
  if (lane == 0) {
    double Rm[4][4];
    rotation_matrix(dx, dy, dz, Rm);
    for (int i = 0; i < 16; ++i) s_R[warp][i] = Rm[i >> 2][i & 3];
  }

  // ---- local two-centre integrals: lane = point-charge term, then lane = slot.
  // A warp instruction takes the FP64 pipe 64 clocks however few lanes it has:
  // by slot, 21 lanes walked up to 24 terms each.
  const int nterm = eri->nflat;
  for (int t = lane; t < nterm; t += 32) {
    const EriTerm e = eri->flat[t];
    const double da = sel3(e.la, pa.d[0], pa.d[1], pa.d[2]);
    const double db = sel3(e.lb, pb.d[0], pb.d[1], pb.d[2]);
    const double ra = sel3(e.la, pa.rho[0], pa.rho[1], pa.rho[2]);
    const double rb = sel3(e.lb, pb.rho[0], pb.rho[1], pb.rho[2]);
    const double l = R + (double)e.c1 * da + (double)e.c2 * db;
    const double u = (double)e.c3 * da + (double)e.c4 * db;
    const double v = (double)e.c5 * da + (double)e.c6 * db;
    const double a = ra + rb;
    const double arg = l * l + u * u + v * v + a * a;
    s_term[warp][t] = e.coef * rsqrt(arg);
  }
  __syncwarp();
  double val = 0.0;
  if (lane < 21) {
    const int first = eri->flat_first[lane], nt = eri->nterms[lane];
    for (int t = 0; t < nt; ++t) val += s_term[warp][first + t];
  }
  const double s5 = __shfl_sync(full, val, 5), s6 = __shfl_sync(full, val, 6);
  if (lane == 21) val = 0.5 * (s5 - s6);
  if (lane < 22) s_val[warp][lane] = val;

  // ---- overlap auxiliary integrals: lane zc computes A_0..6 of zeta combination
  //      zc, lane 4 + zc its B_0..6 (zc: ss, s-p, p-s, p-p exponents) ----------
  const int na = pa.principal_n, nb = pb.principal_n;
  if (lane < 8) {
    const int zc = lane & 3;
    const double za = (zc >= 2) ? pa.zeta[1] : pa.zeta[0];
    const double zb = (zc & 1) ? pb.zeta[1] : pb.zeta[0];
    double v[7];
    if (lane < 4) aux_a_all(0.5 * R * (za + zb), 6, v);
    else aux_b_all(0.5 * R * (za - zb), 6, v, c_inv);
#pragma unroll
    for (int k = 0; k < 7; ++k) s_ab[warp][zc][lane >> 2][k] = v[k];
  }
  __syncwarp();

  // ---- T2 (pair rotation) and local block L ---------------------------------
  for (int e = lane; e < 100; e += 32) {
    const int P = e / 10, Q = e % 10;
    int m, n, i, j;
    unpack_index(P, &m, &n);
    unpack_index(Q, &i, &j);
    const double* Rm = s_R[warp];
    s_T2[warp][e] = (i == j) ? Rm[m * 4 + i] * Rm[n * 4 + i]
                             : Rm[m * 4 + i] * Rm[n * 4 + j] + Rm[m * 4 + j] * Rm[n * 4 + i];
    const int sl = eri->slot_of[P][Q];
    s_L[warp][e] = sl >= 0 ? s_val[warp][sl] : 0.0;
  }
  // overlap sums, lane = combination (ss, s-sigma, sigma-s, sigma-sigma, pi-pi)
  if (lane < 5) {
    const int c = lane, zc = (c == 4) ? 3 : c;
    const int nt = ovt->nterms[na - 1][nb - 1][c];
    double s = 0.0;
    for (int t = 0; t < nt; ++t)
      s += ovt->tc[na - 1][nb - 1][c][t] * s_ab[warp][zc][0][ovt->ti[na - 1][nb - 1][c][t]] *
           s_ab[warp][zc][1][ovt->tj[na - 1][nb - 1][c][t]];
    const double norm = pa.sto_norm[c >= 2 ? 1 : 0] * pb.sto_norm[(c == 1 || c >= 3) ? 1 : 0];
    double rp = 1.0;
    for (int i = 0; i < na + nb + 1; ++i) rp *= 0.5 * R;
    s_ov[warp][c] = s * (norm * ovt->ang[c] * rp);
  }
  __syncwarp();

  // ---- M = L T2^T,  W = T2 M ----------------------------------------------
  for (int e = lane; e < 100; e += 32) {
    const int P = e / 10, Qp = e % 10;
    double s = 0.0;
    for (int Q = 0; Q < 10; ++Q) s += s_L[warp][P * 10 + Q] * s_T2[warp][Qp * 10 + Q];
    s_M[warp][e] = s;
  }
  __syncwarp();
  double* out = blocks + pr.blk;
  for (int e = lane; e < 100; e += 32) {
    const int Pp = e / 10, Qp = e % 10;
    double s = 0.0;
    for (int P = 0; P < 10; ++P) s += s_T2[warp][Pp * 10 + P] * s_M[warp][P * 10 + Qp];
    out[e] = s;
  }

  // ---- resonance block of H:  1/2 (beta_mu + beta_nu) S_mu,nu --------------
  if (lane < 16) {
    const int mu = lane >> 2, nu = lane & 3;
    double Ls[4][4] = {};
    Ls[0][0] = s_ov[warp][0];
    Ls[0][2] = s_ov[warp][1];
    Ls[2][0] = s_ov[warp][2];
    Ls[2][2] = s_ov[warp][3];
    Ls[1][1] = s_ov[warp][4];
    Ls[3][3] = s_ov[warp][4];
    const double* Rm = s_R[warp];
    double s = 0.0;
    for (int i = 0; i < 4; ++i)
      for (int j = 0; j < 4; ++j) s += Rm[mu * 4 + i] * Ls[i][j] * Rm[nu * 4 + j];
    const double h = 0.5 * (pa.beta[mu == 0 ? 0 : 1] + pb.beta[nu == 0 ? 0 : 1]) * s;
    const long long ld = mol.nao;
    const long long r0 = A.ao0 + mu, c0 = B.ao0 + nu;
    H[mol.mat0 + r0 * ld + c0] = h;
    H[mol.mat0 + c0 * ld + r0] = h;
  }

  // ---- core-core repulsion --------------------------------------------------
  const double ec = core_core_warp(pa, pb, R, s_val[warp][0], mol.theory, lane);
  if (lane == 0) ecore_pair[p] = ec;
}

// warp-wide sum with a fixed tree (bitwise reproducible)
__device__ __forceinline__ double warp_sum(double v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// block (a,b) of the molecule, with a flag telling whether atom `self` owns the rows
__device__ __forceinline__ const double* partner_block(const DevPair* __restrict__ pairs, const double* blocks,
                                                       const DevMol& mol, int self, int other, bool* self_rows) {
  const int a = self < other ? self : other, b = self < other ? other : self;
  *self_rows = self < other;
  return blocks + pairs[mol.pair0 + pair_index(a, b, mol.natoms)].blk;
}

constexpr int kFockThreads = 256;

// Local integral (A's multipoles | a bare point charge): the slot's terms with
// both rho set to zero (MolDS Mndo::GetSemiEmpiricalMultipoleInteraction,
// src/mndo/Mndo.cpp:6602-6613, for an atom-EPC pair) and no charge separation
// on the point charge, whose only multipole is its monopole.
__device__ __forceinline__ double epc_slot_value(const EriTable* __restrict__ eri, int slot, double R,
                                                 const nddo_atom_params& pa) {
  double v = 0.0;
  const int nt = eri->nterms[slot];
  for (int t = 0; t < nt; ++t) {
    const EriTerm e = eri->terms[slot][t];
    const double da = e.la == 0 ? pa.d[0] : (e.la == 1 ? pa.d[1] : pa.d[2]);
    const double l = R + (double)e.c1 * da;
    const double u = (double)e.c3 * da;
    const double w = (double)e.c5 * da;
    v += e.coef * rsqrt(l * l + u * u + w * w);
  }
  return v;
}

// One-centre block of H (U on the diagonal plus the attraction of every other
// core, -Z_B (mu nu|s_B s_B)).  With
// environmental point charges each adds -q (mu nu|s s) to the block (MolDS
// Mndo::GetFockDiagElement / GetFockOffDiagElement, src/mndo/Mndo.cpp:474-484,
// 546-556, present in every non-guess Fock matrix and so in H = F(P = 0) of
// the energy, src/cndo/Cndo2.cpp:1324-1416), the block rotated from the local
// values exactly as a pair with a hydrogen (pair_light_kernel); the
// cores' energy in their field, sum Z_A q / R (Mndo.cpp:329-331,
// Cndo2.cpp:418-426), is ecore_kernel's.  CTAs over the atoms of every molecule
// (one CTA per molecule, its pair energies summed by one warp, took 1.7 ms for
// (H2O)180).
__global__ void __launch_bounds__(kFockThreads)
hcore_kernel(const DevAtom* __restrict__ atoms, const DevPair* __restrict__ pairs, const DevMol* __restrict__ mols,
             const int* __restrict__ mol_list, const double* __restrict__ blocks,
             const double* __restrict__ ecore_pair, double* __restrict__ ecore_row, const EriTable* __restrict__ eri,
             const double* __restrict__ epc, double* __restrict__ H) {
  const int m = mol_list[blockIdx.y];
  const DevMol mol = mols[m];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
  const long long ld = mol.nao;
  // a warp per atom
  for (int ia = blockIdx.x * nwarps + warp; ia < mol.natoms; ia += gridDim.x * nwarps) {
    // the row's core-core energies, sum over B > A
    if (ia + 1 < mol.natoms) {
      const double* row = ecore_pair + mol.pair0 + pair_index(ia, ia + 1, mol.natoms);
      double e = 0.0;
      for (int k = lane; k < mol.natoms - 1 - ia; k += 32) e += row[k];
      e = warp_sum(e);
      if (lane == 0) ecore_row[mol.vec0 + ia] = e;
    }
    const DevAtom A = atoms[mol.atom0 + ia];
    const int dA = A.nao == 4 ? 10 : 1;
    double acc[10];
#pragma unroll
    for (int k = 0; k < 10; ++k) acc[k] = 0.0;
    for (int ib = lane; ib < mol.natoms; ib += 32) {
      if (ib == ia) continue;
      const DevAtom Bt = atoms[mol.atom0 + ib];
      const double zb = c_params[Bt.pidx].core_charge;
      bool rows;
      const double* blk = partner_block(pairs, blocks, mol, ia, ib, &rows);
      const int dB = Bt.nao == 4 ? 10 : 1;
#pragma unroll
      for (int k = 0; k < 10; ++k)
        if (k < dA) acc[k] -= zb * (rows ? blk[k * dB] : blk[k]);
    }
    if (mol.nepc > 0) {
      const nddo_atom_params& pa = c_params[A.pidx];
      for (int i = lane; i < mol.nepc; i += 32) {
        const double* pc = epc + 4 * (mol.epc0 + i);
        const double dx = pc[0] - A.x, dy = pc[1] - A.y, dz = pc[2] - A.z, q = pc[3];
        const double R = sqrt(dx * dx + dy * dy + dz * dz);
        const double iR = 1.0 / R;
        acc[0] -= q * epc_slot_value(eri, 0, R, pa);
        if (dA == 10) {
          const double s3 = epc_slot_value(eri, 3, R, pa);
          const double s4 = epc_slot_value(eri, 4, R, pa);
          const double s10 = epc_slot_value(eri, 10, R, pa);
          const double u[4] = {0.0, dy * iR, dz * iR, dx * iR};   // orbital order s, py, pz, px
#pragma unroll
          for (int k = 1; k < 10; ++k) {
            int mu, nu;
            unpack_index(k, &mu, &nu);
            const double v = mu == 0 ? s10 * u[nu] : (mu == nu ? s3 : 0.0) + (s4 - s3) * u[mu] * u[nu];
            acc[k] -= q * v;
          }
        }
      }
    }
#pragma unroll
    for (int k = 0; k < 10; ++k) acc[k] = warp_sum(acc[k]);
    if (lane < dA) {
      int mu, nu;
      unpack_index(lane, &mu, &nu);
      double v = 0.0;
#pragma unroll
      for (int k = 0; k < 10; ++k) if (k == lane) v = acc[k];
      if (mu == nu) v += c_params[A.pidx].u[mu == 0 ? 0 : 1];
      const long long r = A.ao0 + mu, c = A.ao0 + nu;
      H[mol.mat0 + r * ld + c] = v;
      H[mol.mat0 + c * ld + r] = v;
    }
  }
}

// The molecule's core-core energy from its rows' sums, and the cores' energy
// in the field of the point charges
__global__ void __launch_bounds__(kFockThreads)
ecore_kernel(const DevAtom* __restrict__ atoms, const DevMol* __restrict__ mols, const int* __restrict__ mol_list,
             const double* __restrict__ ecore_row, const double* __restrict__ epc, MolState* __restrict__ st) {
  __shared__ double red[2][kFockThreads / 32];
  const int m = mol_list[blockIdx.x];
  const DevMol mol = mols[m];
  const int tid = threadIdx.x;
  double e = 0.0, q = 0.0;
  for (int ia = tid; ia + 1 < mol.natoms; ia += kFockThreads)
    e += ecore_row[mol.vec0 + ia];
  for (long long t = tid; t < (long long)mol.natoms * mol.nepc; t += kFockThreads) {
    const DevAtom& A = atoms[mol.atom0 + t / mol.nepc];
    const double* pc = epc + 4 * (mol.epc0 + t % mol.nepc);
    const double dx = pc[0] - A.x, dy = pc[1] - A.y, dz = pc[2] - A.z;
    q += c_params[A.pidx].core_charge * pc[3] / sqrt(dx * dx + dy * dy + dz * dz);
  }
  e = warp_sum(e);
  q = warp_sum(q);
  if ((tid & 31) == 0) { red[0][tid >> 5] = e; red[1][tid >> 5] = q; }
  __syncthreads();
  if (tid < 2) {
    double v = 0.0;
    for (int w = 0; w < kFockThreads / 32; ++w) v += red[tid][w];
    if (tid == 0) st[m].ecore = v; else st[m].ecore_epc = v;
  }
}

__device__ __forceinline__ double g_one(const nddo_atom_params& p, int m, int n) {   // coulomb
  if (m == 0 && n == 0) return p.gss;
  if (m == 0 || n == 0) return p.gsp;
  return m == n ? p.gpp : p.gp2;
}
__device__ __forceinline__ double h_one(const nddo_atom_params& p, int m, int n) {   // exchange
  if (m == n) return g_one(p, m, n);
  if (m == 0 || n == 0) return p.hsp;
  return p.hpp;
}

// packed index of an orbital pair of one atom as a nibble table: pack_index(m, n)
__device__ __forceinline__ int pack_lut(int m, int n) {
  constexpr unsigned long long kTable = 0x9863875265413210ULL;   // [4 m + n]
  return (int)(kTable >> (16 * m + 4 * n)) & 15;
}

constexpr int kFockAtomThreads = 128;
constexpr int kFockStage = 256;   // atoms whose densities are staged at a time (20 KB)

// F = H + G(P) (mode 0) or the MolDS guess Fock (mode 1: U on the diagonal,
// zero one-centre off-diagonal, resonance blocks between atoms).  P_old <- P
// is copied on the way when copy_old is set.
// One CTA per atom A.  Coulomb: a thread per (B, orbital pair of A), its dot
// product over B's orbital pairs against B's one-centre densities, staged packed
// in shared memory; the threads of one orbital pair are summed in a fixed order.
// Exchange with B > A: a thread per element of the A-B block.
// What bounds it: latency and the number of loads in flight (the blocks of one
// molecule are L2-resident).  A warp per atom, with a lane walking whole 10 x 10
// blocks, left a single molecule on natoms / 8 CTAs.  Staging where each partner's
// block lies takes a dependent load off every one of them: 650 -> 568 us a build
// for 256 (H2O)32.
__global__ void __launch_bounds__(kFockAtomThreads)
fock_kernel(const DevAtom* __restrict__ atoms, const DevPair* __restrict__ pairs, const DevMol* __restrict__ mols,
            const int* __restrict__ mol_list, const double* __restrict__ blocks, const double* __restrict__ H,
            const double* __restrict__ P, double* __restrict__ F, double* __restrict__ Pold,
            const MolState* __restrict__ st, int mode_override, int copy_old, int require_active) {
  __shared__ double s_p[kFockStage * 10];
  __shared__ double s_red[kFockAtomThreads];
  __shared__ short s_list[kFockStage];
  __shared__ int s_ao[kFockStage];          // 2 * first orbital + (sp atom)
  __shared__ long long s_blk[kFockStage];
  __shared__ int s_n[4];
  const int m = mol_list[blockIdx.y], ia = blockIdx.x;
  const DevMol mol = mols[m];
  if (ia >= mol.natoms) return;
  const int status = st[m].status;
  if (require_active && status != kActive) return;
  int mode = mode_override;
  if (mode < 0) mode = (st[m].iter == 0 && st[m].requires_guess) ? 1 : 0;
  const int tid = threadIdx.x;
  const long long ld = mol.nao;
  const double* Pm = P + mol.mat0;
  const double* Hm = H + mol.mat0;
  double* Fm = F + mol.mat0;
  const DevAtom* am = atoms + mol.atom0;
  const DevAtom A = am[ia];
  const nddo_atom_params& pa = c_params[A.pidx];
  const int nA = A.nao, dA = nA == 4 ? 10 : 1, fa = A.ao0;
  if (copy_old) {
    const double* from = Pm + fa * ld;
    double* to = Pold + mol.mat0 + fa * ld;
    for (long long i = tid; i < nA * ld; i += kFockAtomThreads) to[i] = from[i];
  }
  // threads k + dA j share orbital pair k
  const int per = kFockAtomThreads / dA, k = tid % dA, j0 = tid / dA;
  double acc = 0.0;
  for (int b0 = 0; b0 < mol.natoms; b0 += kFockStage) {
    const int nb = min(kFockStage, mol.natoms - b0);
    __syncthreads();
    // where each partner's orbitals and block are: one round of loads here instead
    // of a dependent one before every block
    for (int i = tid; i < nb; i += kFockAtomThreads) {
      const int ib = b0 + i;
      s_ao[i] = am[ib].ao0 * 2 + (am[ib].nao == 4 ? 1 : 0);
      if (ib != ia) s_blk[i] = pairs[mol.pair0 + pair_index(min(ia, ib), max(ia, ib), mol.natoms)].blk;
    }
    __syncthreads();
    // heavy atoms first in the list, hydrogens from its end: a warp then works
    // on one kind, and the FP64 pipe, which takes 64 clocks a warp instruction,
    // is not spent on lanes that sit out
    if (tid < 32) {
      int h = 0, l = 0, h0 = 0, l0 = 0;
      for (int base = 0; base < nb; base += 32) {
        const int i = base + tid;
        const bool in = i < nb, heavy = in && (s_ao[i] & 1);
        const unsigned mh = __ballot_sync(0xffffffffu, heavy), ml = __ballot_sync(0xffffffffu, in && !heavy);
        const unsigned below = (1u << tid) - 1u;
        if (heavy) s_list[h + __popc(mh & below)] = (short)i;
        else if (in) s_list[kFockStage - 1 - (l + __popc(ml & below))] = (short)i;
        const unsigned upto = __ballot_sync(0xffffffffu, in && b0 + i <= ia);
        h0 += __popc(mh & upto);
        l0 += __popc(ml & upto);
        h += __popc(mh);
        l += __popc(ml);
      }
      if (tid == 0) { s_n[0] = h; s_n[1] = l; s_n[2] = h0; s_n[3] = l0; }   // counts, those up to atom A
    }
    if (mode == 0)
      for (int e = tid; e < nb * 10; e += kFockAtomThreads) {
        const int ao = s_ao[e / 10], o = ao >> 1;
        int l, sg;
        unpack_index(e % 10, &l, &sg);
        double v = 0.0;
        if ((ao & 1) || e % 10 == 0) v = Pm[(o + l) * ld + o + sg] * (l == sg ? 1.0 : 2.0);
        s_p[e] = v;
      }
    __syncthreads();
    const int nh = s_n[0], nl = s_n[1], h0 = s_n[2], l0 = s_n[3];
    if (mode == 0 && j0 < per) {
      for (int t = j0; t < nh; t += per) {
        const int i = s_list[t], ib = b0 + i;
        if (ib == ia) continue;
        const bool rows = ia < ib;
        const double* x = blocks + s_blk[i] + (rows ? k * 10 : k);
        const int step = rows ? 1 : dA;
        double v = 0.0;
#pragma unroll
        for (int q = 0; q < 10; ++q) v += x[q * step] * s_p[i * 10 + q];
        acc += v;
      }
      for (int t = j0; t < nl; t += per) {
        const int i = s_list[kFockStage - 1 - t], ib = b0 + i;
        if (ib == ia) continue;
        acc += blocks[s_blk[i] + k] * s_p[i * 10];
      }
    }
    // two-centre blocks (A, B > A): resonance + exchange -1/2 sum P_nu,si (mu nu|la si);
    // a thread per (B, mu, la)
    const int sh = nA == 4 ? 4 : 2;
    for (int t = h0 + (tid >> sh); t < nh; t += kFockAtomThreads >> sh) {
      const int i = s_list[t], fb = s_ao[i] >> 1, mu = (tid >> 2) & (nA - 1), la = tid & 3;
      double v = Hm[(fa + mu) * ld + fb + la];
      if (mode == 0) {
        const double* blk = blocks + s_blk[i];
        const double* Pab = Pm + fa * ld + fb;
        double x = 0.0;
        if (nA == 4) {
#pragma unroll
          for (int n = 0; n < 4; ++n) {
            const double* row = blk + pack_lut(mu, n) * 10;
#pragma unroll
            for (int sg = 0; sg < 4; ++sg) x += Pab[n * ld + sg] * row[pack_lut(la, sg)];
          }
        } else {
#pragma unroll
          for (int sg = 0; sg < 4; ++sg) x += Pab[sg] * blk[pack_lut(la, sg)];
        }
        v -= 0.5 * x;
      }
      Fm[(fa + mu) * ld + fb + la] = v;
      Fm[(fb + la) * ld + fa + mu] = v;
    }
    const int sl = nA == 4 ? 2 : 0;
    for (int t = l0 + (tid >> sl); t < nl; t += kFockAtomThreads >> sl) {
      const int i = s_list[kFockStage - 1 - t], fb = s_ao[i] >> 1, mu = tid & (nA - 1);
      double v = Hm[(fa + mu) * ld + fb];
      if (mode == 0) {
        const double* blk = blocks + s_blk[i];
        const double* Pab = Pm + fa * ld + fb;
        double x = 0.0;
        for (int n = 0; n < nA; ++n) x += Pab[n * ld] * blk[pack_lut(mu, n)];
        v -= 0.5 * x;
      }
      Fm[(fa + mu) * ld + fb] = v;
      Fm[fb * ld + fa + mu] = v;
    }
  }
  if (mode == 0) {
    s_red[tid] = j0 < per ? acc : 0.0;
    __syncthreads();
  }
  // one-centre block
  if (tid < dA) {
    int mu, nu;
    unpack_index(tid, &mu, &nu);
    double v;
    if (mode == 1) {
      v = (mu == nu) ? pa.u[mu == 0 ? 0 : 1] : 0.0;
    } else {
      double j = 0.0;
      for (int i = 0; i < per; ++i) j += s_red[i * dA + tid];
      v = Hm[(fa + mu) * ld + fa + nu];
      if (mu == nu) {
        double t = 0.0;
        for (int n = 0; n < nA; ++n) t += Pm[(fa + n) * ld + fa + n] * (g_one(pa, mu, n) - 0.5 * h_one(pa, mu, n));
        v += t;
      } else {
        v += (1.5 * h_one(pa, mu, nu) - 0.5 * g_one(pa, mu, nu)) * Pm[(fa + mu) * ld + fa + nu];
      }
      v += j;
    }
    Fm[(fa + mu) * ld + fa + nu] = v;
    Fm[(fa + nu) * ld + fa + mu] = v;
  }
}

// All pairs without index lists (each kernel skips the other's): a warp per
// pair with a hydrogen as well took 1.9 of 3.1 ms for 450 atoms.
void launch_pair_kernel(const DevAtom* atoms, const DevPair* pairs, long long npairs, const DevMol* mols,
                        const EriTable* eri, const OverlapTable* ovt, double* blocks, double* H,
                        double* ecore_pair, cudaStream_t s) {
  if (npairs <= 0) return;
  const long long grid = (npairs + kPairWarps - 1) / kPairWarps;
  pair_kernel<<<(unsigned)grid, kPairWarps * 32, 0, s>>>(atoms, pairs, nullptr, npairs, mols, eri, ovt, blocks, H,
                                                         ecore_pair);
  pair_light_kernel<<<(unsigned)((npairs + 127) / 128), 128, 0, s>>>(atoms, pairs, nullptr, npairs, mols, eri, ovt,
                                                                     blocks, H, ecore_pair);
}

void launch_pair_kernels_split(const DevAtom* atoms, const DevPair* pairs, const int* heavy_list, long long n_heavy,
                               const int* light_list, long long n_light, const DevMol* mols, const EriTable* eri,
                               const OverlapTable* ovt, double* blocks, double* H, double* ecore_pair,
                               cudaStream_t s) {
  if (n_heavy > 0) {
    const long long grid = (n_heavy + kPairWarps - 1) / kPairWarps;
    pair_kernel<<<(unsigned)grid, kPairWarps * 32, 0, s>>>(atoms, pairs, heavy_list, n_heavy, mols, eri, ovt, blocks,
                                                           H, ecore_pair);
  }
  if (n_light > 0) {
    const long long grid = (n_light + 127) / 128;
    pair_light_kernel<<<(unsigned)grid, 128, 0, s>>>(atoms, pairs, light_list, n_light, mols, eri, ovt, blocks, H,
                                                     ecore_pair);
  }
}

void launch_hcore_kernel(const DevAtom* atoms, const DevPair* pairs, const DevMol* mols, const int* mol_list,
                         int nlist, int max_atoms, const double* blocks, const double* ecore_pair,
                         double* ecore_row, const EriTable* eri, const double* epc, double* H, MolState* st,
                         cudaStream_t s) {
  if (nlist <= 0) return;
  constexpr int kWarps = kFockThreads / 32;
  hcore_kernel<<<dim3((max_atoms + kWarps - 1) / kWarps, nlist), kFockThreads, 0, s>>>(
      atoms, pairs, mols, mol_list, blocks, ecore_pair, ecore_row, eri, epc, H);
  ecore_kernel<<<nlist, kFockThreads, 0, s>>>(atoms, mols, mol_list, ecore_row, epc, st);
}

void launch_fock_kernel(const DevAtom* atoms, const DevPair* pairs, const DevMol* mols, const int* mol_list,
                        int nlist, int max_atoms, const double* blocks, const double* H, const double* P, double* F,
                        double* Pold, const MolState* st, int mode_override, int copy_old, int require_active,
                        cudaStream_t s) {
  if (nlist <= 0) return;
  fock_kernel<<<dim3(max_atoms, nlist), kFockAtomThreads, 0, s>>>(atoms, pairs, mols, mol_list, blocks, H, P, F, Pold,
                                                                  st, mode_override, copy_old, require_active);
}

// E = 1/2 sum P (F + H) + E_core + E_vdW (Cndo2::CalcElecSCFEnergy, src/cndo/Cndo2.cpp:1324-1416),
// Mulliken charges q_A = Z_A - sum_{mu in A} P_mu,mu (Cndo2.cpp:1187-1199, 1733-1747)
// and, for MNDO, the heat of formation (Mndo::CalcHeatsFormation, src/mndo/Mndo.cpp:395-404).
// E_vdW: the empirical dispersion energy of Cndo2::CalcVdWCorrectionEnergy
// (Cndo2.cpp:464-513), on when requested or for AM1-D / PM3-D (which fix
// s6 = 1.40, d = 23).
// Partial sums over fixed chunks of each molecule's matrix (their number depends
// on N alone), then one CTA per molecule: a single CTA walking N^2 took 1.26 ms
// for (H2O)180.
__host__ __device__ __forceinline__ int energy_chunks(long long n2) {
  const long long c = (n2 + 2047) / 2048;
  return (int)(c < 1 ? 1 : (c > kDipChunks ? kDipChunks : c));
}

__global__ void __launch_bounds__(kFockThreads)
energy_partial_kernel(const DevAtom* __restrict__ atoms, const DevPair* __restrict__ pairs,
                      const DevMol* __restrict__ mols, const int* __restrict__ mol_list, const double* __restrict__ P,
                      const double* __restrict__ F, const double* __restrict__ H, double* __restrict__ partial,
                      VdwParams vdw) {
  __shared__ double red[2][kFockThreads / 32];
  const DevMol mol = mols[mol_list[blockIdx.y]];
  const long long n2 = (long long)mol.nao * mol.nao;
  const int chunks = energy_chunks(n2);
  if ((int)blockIdx.x >= chunks) return;
  const long long step = (long long)chunks * kFockThreads, first = (long long)blockIdx.x * kFockThreads + threadIdx.x;
  double acc = 0.0;
  for (long long i = first; i < n2; i += step) acc += P[mol.mat0 + i] * (F[mol.mat0 + i] + H[mol.mat0 + i]);
  acc = warp_sum(acc);
  const bool dtheory = mol.theory == NDDO_AM1D || mol.theory == NDDO_PM3D;
  const bool vdw_on = vdw.on || dtheory;
  const double s6 = dtheory ? NDDO_VDW_S6_D : vdw.s6, dd = dtheory ? NDDO_VDW_DAMP_D : vdw.d;
  double ev = 0.0;
  if (vdw_on)
    for (long long t = first; t < mol.npairs; t += step) {
      const DevPair pr = pairs[mol.pair0 + t];
      const DevAtom A = atoms[pr.a], B = atoms[pr.b];
      const nddo_atom_params& pa = c_params[A.pidx];
      const nddo_atom_params& pb = c_params[B.pidx];
      const double csum = pa.vdw_c6 + pb.vdw_c6;
      if (csum <= 0.0) continue;
      const double dx = A.x - B.x, dy = A.y - B.y, dz = A.z - B.z;
      const double R = sqrt(dx * dx + dy * dy + dz * dz);
      const double c6 = 2.0 * pa.vdw_c6 * pb.vdw_c6 / csum;
      const double damp = 1.0 / (1.0 + exp(-1.0 * dd * (R / (pa.vdw_r0 + pb.vdw_r0) - 1.0)));
      ev += -1.0 * s6 * c6 * damp / (R * R * R * R * R * R);
    }
  ev = warp_sum(ev);
  if ((threadIdx.x & 31) == 0) { red[0][threadIdx.x >> 5] = acc; red[1][threadIdx.x >> 5] = ev; }
  __syncthreads();
  if (threadIdx.x < 2) {
    double v = 0.0;
    for (int w = 0; w < kFockThreads / 32; ++w) v += red[threadIdx.x][w];
    partial[((long long)blockIdx.y * gridDim.x + blockIdx.x) * 2 + threadIdx.x] = v;
  }
}

__global__ void __launch_bounds__(kFockThreads)
energy_kernel(const DevAtom* __restrict__ atoms, const DevMol* __restrict__ mols, const int* __restrict__ mol_list,
              int grid_chunks, const double* __restrict__ P, const double* __restrict__ partial,
              MolState* __restrict__ st, double* __restrict__ charges) {
  __shared__ double red[3][kFockThreads / 32];
  const int m = mol_list[blockIdx.x], tid = threadIdx.x;
  const DevMol mol = mols[m];
  const int chunks = energy_chunks((long long)mol.nao * mol.nao);
  double e = 0.0, v = 0.0, f = 0.0;
  for (int c = tid; c < chunks; c += kFockThreads) {
    e += partial[((long long)blockIdx.x * grid_chunks + c) * 2];
    v += partial[((long long)blockIdx.x * grid_chunks + c) * 2 + 1];
  }
  for (int a = tid; a < mol.natoms; a += kFockThreads) {
    const DevAtom A = atoms[mol.atom0 + a];
    const nddo_atom_params& pa = c_params[A.pidx];
    double pop = 0.0;
    for (int k = 0; k < A.nao; ++k) pop += P[mol.mat0 + (long long)(A.ao0 + k) * mol.nao + A.ao0 + k];
    charges[mol.atom0 + a] = pa.core_charge - pop;
    f += pa.dhf_atom - pa.e_atom;
  }
  e = warp_sum(e);
  v = warp_sum(v);
  f = warp_sum(f);
  if ((tid & 31) == 0) { red[0][tid >> 5] = e; red[1][tid >> 5] = v; red[2][tid >> 5] = f; }
  __syncthreads();
  if (tid == 0) {
    e = v = f = 0.0;
    for (int w = 0; w < kFockThreads / 32; ++w) { e += red[0][w]; v += red[1][w]; f += red[2][w]; }
    e *= 0.5;
    MolState* s = st + m;
    s->energy_electronic = e;
    s->vdw_energy = v;
    s->energy = e + s->ecore + s->ecore_epc + v;
    s->heat_of_formation = s->energy + f;
  }
}

void launch_energy_kernel(const DevAtom* atoms, const DevPair* pairs, const DevMol* mols, const int* mol_list,
                          int nlist, int max_n, const double* P, const double* F, const double* H, double* partial,
                          MolState* st, double* charges, VdwParams vdw, cudaStream_t s) {
  if (nlist <= 0) return;
  const int chunks = energy_chunks((long long)max_n * max_n);   // the largest molecule's count sets the grid
  energy_partial_kernel<<<dim3(chunks, nlist), kFockThreads, 0, s>>>(atoms, pairs, mols, mol_list, P, F, H, partial,
                                                                     vdw);
  energy_kernel<<<nlist, kFockThreads, 0, s>>>(atoms, mols, mol_list, chunks, P, partial, st, charges);
}

// ---------------------------------------------------------------------------
// (c) Dipole moment after convergence.
//
// MolDS builds the Cartesian matrix X_k,mu,nu = <mu| r_k |nu> of every AO pair
// (same atom included) from the STO-6G expansion of each Slater orbital
// (Cndo2::CalcCartesianMatrixByGTOExpansion, src/cndo/Cndo2.cpp:1946-2130) and
// then forms mu_elec = -sum P X + c sum P S with c the centre of core mass,
// and mu_core = sum_A Z_A (R_A - c) (Cndo2.cpp:1871-1944).  Here the matrix is
// never stored: one warp takes one atom pair (or one atom), its lanes take the
// 6 x 6 primitive pairs of each shell pair, and every primitive block is
// contracted with P at once.
//
// Primitive integrals: normalised Cartesian Gaussians, s = N e^{-a|r-A|^2},
// p_i = 2 sqrt(a) (r_i - A_i) s.  With p = a + b, the product centre Pc,
// PA = Pc - A, PB = Pc - B and h = 1/(2p), the one-dimensional moments of
// (x-A)^i (x-B)^j follow from the Obara-Saika recurrence:
//   s10 = PA, s01 = PB, s11 = PA PB + h, s02 = PB^2 + h, s12 = PA PB^2 + (PA + 2 PB) h,
// and x = (x - B) + B turns them into moments of the position operator:
//   m00 = Pc, m10 = s11 + B PA, m01 = s02 + B PB, m11 = s12 + B s11.
// The three-dimensional integral is (s|s) times the product over directions,
// (s|s) = (2 sqrt(ab) / p)^{3/2} e^{-mu R^2}, mu = ab / p.
//
// Screen: a primitive pair with mu R^2 > 46 (e^{-46} = 1e-20) is skipped.
// Its elements are below 1e-17 (coefficients, normalisation and moments are
// O(1..100)), far below the FP64 rounding of the sums they would join.
// ---------------------------------------------------------------------------
constexpr int kDipThreads = 256;
constexpr double kDipScreen = 46.0;

// Per parameter slot and shell (s, p): the six primitive exponents a_i =
// zeta^2 alpha_i and factors f_i = d_i (2 sqrt(a_i) for p) a_i^{3/4}, so that a
// primitive pair's weight is 2^{3/2} f_i f_j p^{-3/2} e^{-mu R^2}.
__device__ double g_prim[kNumParamSlots][2][2][6];

void upload_primitives(const nddo_atom_params* p, cudaStream_t s) {
  static double prim[kNumParamSlots][2][2][6];
  for (int slot = 0; slot < kNumParamSlots; ++slot)
    for (int l = 0; l < 2; ++l)
      for (int i = 0; i < 6; ++i) {
        const int sh = p[slot].principal_n - 1;
        const double z = p[slot].zeta[l];
        const bool ok = sh >= 0 && sh < 3 && (l == 0 || p[slot].n_ao > 1) && z > 0.0;
        const double a = ok ? z * z * nddo_sto6g_exp[sh][l][i] : 0.0;
        double f = ok ? nddo_sto6g_coef[sh][l][i] * std::pow(a, 0.75) : 0.0;
        if (ok && l == 1) f *= 2.0 * std::sqrt(a);
        prim[slot][l][0][i] = a;
        prim[slot][l][1][i] = f;
      }
  cudaMemcpyToSymbolAsync(g_prim, prim, sizeof(prim), 0, cudaMemcpyHostToDevice, s);
}

// One primitive pair's X block (weighted), out[k][i][j]: k the axis of r, i / j
// the p axis (0 for an s shell).  Returns false when the pair is screened.
template <int LA, int LB>
__device__ __forceinline__ bool prim_block(const double* ra, const double* rb, const double* d, double R2, double a,
                                           double fa, double b, double fb,
                                           double (&out)[3][LA ? 3 : 1][LB ? 3 : 1]) {
  constexpr int NA = LA ? 3 : 1, NB = LB ? 3 : 1;
  const double r = rsqrt(a + b);          // p^{-1/2}
  const double ip = r * r;
  const double x = a * b * ip * R2;
  if (x > kDipScreen) return false;
  const double w = 2.8284271247461903 * fa * fb * (r * ip) * exp(-x);
  const double h = 0.5 * ip;
  double Pc[3], PA[3], PB[3];
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    Pc[q] = (a * ra[q] + b * rb[q]) * ip;
    PA[q] = -b * ip * d[q];
    PB[q] = a * ip * d[q];
  }
#pragma unroll
  for (int k = 0; k < 3; ++k)
#pragma unroll
    for (int i = 0; i < NA; ++i)
#pragma unroll
      for (int j = 0; j < NB; ++j) {
        double v;
        if (!LA && !LB) {
          v = Pc[k];
        } else if (!LA) {
          v = (k == j) ? PB[j] * PB[j] + h + rb[j] * PB[j] : PB[j] * Pc[k];
        } else if (!LB) {
          v = (k == i) ? PA[i] * PB[i] + h + rb[i] * PA[i] : PA[i] * Pc[k];
        } else if (i == j) {
          const double s11 = PA[i] * PB[i] + h;
          v = (k == i) ? PA[i] * PB[i] * PB[i] + (PA[i] + 2.0 * PB[i]) * h + rb[i] * s11 : s11 * Pc[k];
        } else {
          v = (k == i)   ? (PA[i] * PB[i] + h + rb[i] * PA[i]) * PB[j]
              : (k == j) ? PA[i] * (PB[j] * PB[j] + h + rb[j] * PB[j])
                         : PA[i] * PB[j] * Pc[k];
        }
        out[k][i][j] = w * v;
      }
  return true;
}

// AO index within an atom of p axis i (MolDS order s, py, pz, px)
__device__ __forceinline__ int ao_of_axis(int i) { return i == 0 ? 3 : i; }

// acc[k] += sum_{i, j} Wa_ij X_k,ij of one primitive pair, Wa in axis order
// (Wa[0][*] for an s shell on A, Wa[*][0] for an s shell on B).  The sums over
// i, j are folded into row / column sums: with U_k = sum_j Wa_kj PB_j,
// V_k = sum_i Wa_ik PA_i, Q = sum_k PA_k U_k, D = sum_i Wa_ii PA_i PB_i and
// T = sum_i Wa_ii s11_i, the p-p contraction for axis k is
//   Wa_kk m11_k + (T - Wa_kk s11_k) Pc_k + U'_k m10_k + V'_k m01_k
//   + (Q - D - PA_k U'_k - PB_k V'_k) Pc_k,  U'_k = U_k - Wa_kk PB_k, V'_k = V_k - Wa_kk PA_k,
// the terms of the block with k = i = j, i = j != k, k = i != j, k = j != i and
// i, j, k all different.
template <int LA, int LB>
__device__ __forceinline__ void prim_contract(const double* ra, const double* rb, const double* d, double R2,
                                              double a, double fa, double b, double fb, const double (&Wa)[3][3],
                                              double* acc) {
  const double r = rsqrt(a + b);          // p^{-1/2}
  const double ip = r * r;
  const double x = a * b * ip * R2;
  const double w = 2.8284271247461903 * fa * fb * (r * ip) * exp(-x);
  const double h = 0.5 * ip;
  double Pc[3], PA[3], PB[3];
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    Pc[q] = (a * ra[q] + b * rb[q]) * ip;
    PA[q] = -b * ip * d[q];
    PB[q] = a * ip * d[q];
  }
  if (!LA && !LB) {
    const double ws = w * Wa[0][0];
#pragma unroll
    for (int k = 0; k < 3; ++k) acc[k] += ws * Pc[k];
  } else if (!LA) {
    const double sPB = Wa[0][0] * PB[0] + Wa[0][1] * PB[1] + Wa[0][2] * PB[2];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const double m01 = PB[k] * PB[k] + h + rb[k] * PB[k];
      acc[k] += w * (Wa[0][k] * m01 + Pc[k] * (sPB - Wa[0][k] * PB[k]));
    }
  } else if (!LB) {
    const double sPA = Wa[0][0] * PA[0] + Wa[1][0] * PA[1] + Wa[2][0] * PA[2];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const double m10 = PA[k] * PB[k] + h + rb[k] * PA[k];
      acc[k] += w * (Wa[k][0] * m10 + Pc[k] * (sPA - Wa[k][0] * PA[k]));
    }
  } else {
    double s11[3], U[3], V[3];
    double T = 0.0, D = 0.0;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      s11[i] = PA[i] * PB[i] + h;
      T += Wa[i][i] * s11[i];
      D += Wa[i][i] * PA[i] * PB[i];
      U[i] = Wa[i][0] * PB[0] + Wa[i][1] * PB[1] + Wa[i][2] * PB[2];
      V[i] = Wa[0][i] * PA[0] + Wa[1][i] * PA[1] + Wa[2][i] * PA[2];
    }
    const double Q = PA[0] * U[0] + PA[1] * U[1] + PA[2] * U[2];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const double m10 = s11[k] + rb[k] * PA[k];
      const double m01 = PB[k] * PB[k] + h + rb[k] * PB[k];
      const double m11 = PA[k] * PB[k] * PB[k] + (PA[k] + 2.0 * PB[k]) * h + rb[k] * s11[k];
      const double Ur = U[k] - Wa[k][k] * PB[k];
      const double Vr = V[k] - Wa[k][k] * PA[k];
      acc[k] += w * (Wa[k][k] * m11 + (T - Wa[k][k] * s11[k]) * Pc[k] + Ur * m10 + Vr * m01 +
                     (Q - D - PA[k] * Ur - PB[k] * Vr) * Pc[k]);
    }
  }
}

// acc[k] += sum_{mu, nu} W_mu,nu X_k,mu,nu of the shell pair (LA, LB).  The
// warp screens the 36 primitive pairs (mu R^2 > 46, tested without a divide
// as a b R^2 > 46 (a + b)) and hands the survivors out lane by lane, so a
// distant atom pair with few survivors takes one pass.  Called by all lanes.
template <int LA, int LB>
__device__ __forceinline__ void shell_contract_warp(const double* ra, const double* rb, const double* d, double R2,
                                                    const double* pa_a, const double* pa_f, const double* pb_a,
                                                    const double* pb_f, const double (&W)[4][4], int lane,
                                                    double* acc) {
  double Wa[3][3];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) Wa[i][j] = W[LA ? ao_of_axis(i) : 0][LB ? ao_of_axis(j) : 0];
  const double a0 = pa_a[lane / 6], b0 = pb_a[lane % 6];
  const bool keep0 = !(a0 * b0 * R2 > kDipScreen * (a0 + b0));
  bool keep1 = false;
  if (lane < 4) {
    const double a1 = pa_a[(lane + 32) / 6], b1 = pb_a[(lane + 32) % 6];
    keep1 = !(a1 * b1 * R2 > kDipScreen * (a1 + b1));
  }
  const unsigned m0 = __ballot_sync(0xffffffffu, keep0);
  const unsigned m1 = __ballot_sync(0xffffffffu, keep1);
  const int n0 = __popc(m0), n = n0 + __popc(m1);
  for (int slot = lane; slot < n; slot += 32) {
    // position of the (slot)-th set bit (0-based) of m0, then of m1
    unsigned m = slot < n0 ? m0 : m1;
    for (int q = slot < n0 ? slot : slot - n0; q > 0; --q) m &= m - 1;
    const int e = (slot < n0 ? 0 : 32) + __ffs(m) - 1;
    const int i6 = e / 6, j6 = e - 6 * (e / 6);
    prim_contract<LA, LB>(ra, rb, d, R2, pa_a[i6], pa_f[i6], pb_a[j6], pb_f[j6], Wa, acc);
  }
}

// CTAs of one molecule's dipole sums: a function of the molecule alone, so a
// molecule's result does not depend on the batch it runs in.
__host__ __device__ __forceinline__ int dipole_chunks(int natoms) {
  const long long items = (long long)natoms + (long long)natoms * (natoms - 1) / 2;
  const long long c = (items + 4LL * (kDipThreads / 32) - 1) / (4LL * (kDipThreads / 32));   // four items a warp
  return (int)(c < 1 ? 1 : (c > kDipChunks ? kDipChunks : c));
}

size_t reduce_scratch_doubles(int slots, int cap_n) {
  return (size_t)slots * std::max(2 * energy_chunks((long long)cap_n * cap_n), 4 * dipole_chunks(cap_n));
}

// One work item: atom t of the molecule (t < natoms, the same-atom block) or
// atom pair t - natoms (a < b).  Returns the batch-global atom indices.
__device__ __forceinline__ void dipole_item(const DevMol& mol, const DevPair* __restrict__ pairs, long long t,
                                            int* ia, int* ib) {
  if (t < mol.natoms) {
    *ia = *ib = mol.atom0 + (int)t;
  } else {
    const DevPair pr = pairs[mol.pair0 + (t - mol.natoms)];
    *ia = pr.a;
    *ib = pr.b;
  }
}

// Partial sums per CTA: sum W X (x, y, z) and sum P S.  W = P_mu,nu + P_nu,mu
// for two different atoms (both triangles of MolDS's full-matrix dot product),
// P_mu,nu within one atom.  The inter-atom block of H is exactly
// 1/2 (beta_mu + beta_nu) S_mu,nu, so S is read back from H; within an atom S
// is the identity (Cndo2.cpp:4135-4140).  One warp per item.
__global__ void __launch_bounds__(kDipThreads, 2)
dipole_partial_kernel(const DevAtom* __restrict__ atoms, const DevPair* __restrict__ pairs,
                      const DevMol* __restrict__ mols, const int* __restrict__ mol_list,
                      const double* __restrict__ P, const double* __restrict__ H, double* __restrict__ partial) {
  __shared__ double s_prim[kNumParamSlots][2][2][6];
  __shared__ double red[kDipThreads / 32][4];
  const DevMol mol = mols[mol_list[blockIdx.y]];
  const int chunks = dipole_chunks(mol.natoms);
  if ((int)blockIdx.x >= chunks) return;
  for (int i = threadIdx.x; i < kNumParamSlots * 24; i += blockDim.x) (&s_prim[0][0][0][0])[i] = (&g_prim[0][0][0][0])[i];
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int kWarps = kDipThreads / 32;
  const long long items = (long long)mol.natoms + mol.npairs;
  const long long ld = mol.nao;
  const double* Pm = P + mol.mat0;
  const double* Hm = H + mol.mat0;
  double acc[4] = {0.0, 0.0, 0.0, 0.0};
  for (long long t = (long long)blockIdx.x * kWarps + warp; t < items; t += (long long)chunks * kWarps) {
    int ia, ib;
    dipole_item(mol, pairs, t, &ia, &ib);
    const DevAtom A = atoms[ia], B = atoms[ib];
    const bool same = ia == ib;
    double W[4][4];
#pragma unroll
    for (int mu = 0; mu < 4; ++mu)
#pragma unroll
      for (int nu = 0; nu < 4; ++nu) {
        double w = 0.0;
        if (mu < A.nao && nu < B.nao) {
          const long long r = A.ao0 + mu, c = B.ao0 + nu;
          w = Pm[r * ld + c];
          if (!same) w += Pm[c * ld + r];
        }
        W[mu][nu] = w;
      }
    // sum P S: lane e takes element (e / 4, e % 4) of the block
    if (lane < 16) {
      const int mu = lane >> 2, nu = lane & 3;
      if (mu < A.nao && nu < B.nao) {
        const long long r = A.ao0 + mu, c = B.ao0 + nu;
        if (!same) {
          const double bs = c_params[A.pidx].beta[mu == 0 ? 0 : 1] + c_params[B.pidx].beta[nu == 0 ? 0 : 1];
          acc[3] += (Pm[r * ld + c] + Pm[c * ld + r]) * (2.0 * Hm[r * ld + c] / bs);
        } else if (mu == nu) {
          acc[3] += Pm[r * ld + c];
        }
      }
    }
    const double ra[3] = {A.x, A.y, A.z}, rb[3] = {B.x, B.y, B.z};
    const double d[3] = {ra[0] - rb[0], ra[1] - rb[1], ra[2] - rb[2]};
    const double R2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2];
    const double* As = s_prim[A.pidx][0][0];
    const double* Af = s_prim[A.pidx][0][1];
    const double* Bs = s_prim[B.pidx][0][0];
    const double* Bf = s_prim[B.pidx][0][1];
    const double* Ap = s_prim[A.pidx][1][0];
    const double* Apf = s_prim[A.pidx][1][1];
    const double* Bp = s_prim[B.pidx][1][0];
    const double* Bpf = s_prim[B.pidx][1][1];
    shell_contract_warp<0, 0>(ra, rb, d, R2, As, Af, Bs, Bf, W, lane, acc);
    if (B.nao > 1) shell_contract_warp<0, 1>(ra, rb, d, R2, As, Af, Bp, Bpf, W, lane, acc);
    if (A.nao > 1) shell_contract_warp<1, 0>(ra, rb, d, R2, Ap, Apf, Bs, Bf, W, lane, acc);
    if (A.nao > 1 && B.nao > 1) shell_contract_warp<1, 1>(ra, rb, d, R2, Ap, Apf, Bp, Bpf, W, lane, acc);
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const double v = warp_sum(acc[q]);
    if (lane == 0) red[warp][q] = v;
  }
  __syncthreads();
  if (threadIdx.x < 4) {
    double v = 0.0;
    for (int w = 0; w < kWarps; ++w) v += red[w][threadIdx.x];
    partial[((long long)blockIdx.y * gridDim.x + blockIdx.x) * 4 + threadIdx.x] = v;
  }
}

// Sums over a CTA of kFinishThreads, the result in every thread
constexpr int kFinishThreads = 128;
__device__ __forceinline__ double finish_sum(double v, double* red) {
  v = warp_sum(v);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  double t = 0.0;
  for (int w = 0; w < kFinishThreads / 32; ++w) t += red[w];
  return t;
}

// One CTA per molecule: chunk sums in a fixed order, the centre of core
// mass (src/base/Molecule.cpp:396-419), the core dipole and the electronic
// dipole; MolState::dipole = total, electronic, core (x, y, z each).  (A thread
// per molecule walked its atoms twice: 270 us for (H2O)180.)
__global__ void __launch_bounds__(kFinishThreads)
dipole_finish_kernel(const DevAtom* __restrict__ atoms, const DevMol* __restrict__ mols,
                     const int* __restrict__ mol_list, int grid_chunks, const double* __restrict__ partial,
                     MolState* __restrict__ st) {
  __shared__ double red[kFinishThreads / 32];
  const int li = blockIdx.x, m = mol_list[li], tid = threadIdx.x;
  const DevMol mol = mols[m];
  const int chunks = dipole_chunks(mol.natoms);
  double v[12];
#pragma unroll
  for (int q = 0; q < 12; ++q) v[q] = 0.0;
  for (int c = tid; c < chunks; c += kFinishThreads)
    for (int q = 0; q < 4; ++q) v[q] += partial[((long long)li * grid_chunks + c) * 4 + q];
  for (int a = tid; a < mol.natoms; a += kFinishThreads) {
    const DevAtom A = atoms[mol.atom0 + a];
    const double cm = c_params[A.pidx].core_mass;
    v[4] += cm;
    v[5] += A.x * cm;
    v[6] += A.y * cm;
    v[7] += A.z * cm;
  }
#pragma unroll
  for (int q = 0; q < 8; ++q) v[q] = finish_sum(v[q], red);
  const double center[3] = {v[5] / v[4], v[6] / v[4], v[7] / v[4]};
  for (int a = tid; a < mol.natoms; a += kFinishThreads) {
    const DevAtom A = atoms[mol.atom0 + a];
    const double z = c_params[A.pidx].core_charge;
    v[8] += z * (A.x - center[0]);
    v[9] += z * (A.y - center[1]);
    v[10] += z * (A.z - center[2]);
  }
#pragma unroll
  for (int q = 8; q < 11; ++q) v[q] = finish_sum(v[q], red);
  if (tid == 0) {
    MolState* s = st + m;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const double elec = -v[k] + center[k] * v[3];
      s->dipole[k] = elec + v[8 + k];
      s->dipole[3 + k] = elec;
      s->dipole[6 + k] = v[8 + k];
    }
  }
}

void launch_dipole(const DevAtom* atoms, const DevPair* pairs, const DevMol* mols, const int* mol_list, int nlist,
                   int max_atoms, const double* P, const double* H, double* partial, MolState* st, cudaStream_t s) {
  if (nlist <= 0) return;
  const int chunks = dipole_chunks(max_atoms);   // the largest molecule's count sets the grid
  dipole_partial_kernel<<<dim3(chunks, nlist), kDipThreads, 0, s>>>(atoms, pairs, mols, mol_list, P, H, partial);
  dipole_finish_kernel<<<nlist, kFinishThreads, 0, s>>>(atoms, mols, mol_list, chunks, partial, st);
}

// X[k][mu][nu] of molecule m (3 x N x N doubles, row-major), both triangles:
// the matrix MolDS keeps as cartesianMatrix (Cndo2.cpp:1946-2057).  One thread
// per atom pair (or atom) and shell pair; not on the SCF path.
template <int LA, int LB>
__device__ __forceinline__ void shell_store(const double* ra, const double* rb, const double* d, double R2,
                                            const double* pa_a, const double* pa_f, const double* pb_a,
                                            const double* pb_f, int ao0A, int ao0B, long long N,
                                            double* __restrict__ X) {
  constexpr int NA = LA ? 3 : 1, NB = LB ? 3 : 1;
  double sum[3][NA][NB] = {};
  for (int i6 = 0; i6 < 6; ++i6)
    for (int j6 = 0; j6 < 6; ++j6) {
      double blk[3][NA][NB];
      if (!prim_block<LA, LB>(ra, rb, d, R2, pa_a[i6], pa_f[i6], pb_a[j6], pb_f[j6], blk)) continue;
      for (int k = 0; k < 3; ++k)
        for (int i = 0; i < NA; ++i)
          for (int j = 0; j < NB; ++j) sum[k][i][j] += blk[k][i][j];
    }
  const long long NN = N * N;
  for (int k = 0; k < 3; ++k)
    for (int i = 0; i < NA; ++i)
      for (int j = 0; j < NB; ++j) {
        const long long r = ao0A + (LA ? ao_of_axis(i) : 0), c = ao0B + (LB ? ao_of_axis(j) : 0);
        X[k * NN + r * N + c] = sum[k][i][j];
        X[k * NN + c * N + r] = sum[k][i][j];
      }
}

__global__ void __launch_bounds__(kDipThreads)
cartesian_matrix_kernel(const DevAtom* __restrict__ atoms, const DevPair* __restrict__ pairs,
                        const DevMol* __restrict__ mols, int m, double* __restrict__ X) {
  const DevMol mol = mols[m];
  const long long items = (long long)mol.natoms + mol.npairs;
  const long long N = mol.nao;
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < items;
       t += (long long)gridDim.x * blockDim.x) {
    int ia, ib;
    dipole_item(mol, pairs, t, &ia, &ib);
    const DevAtom A = atoms[ia], B = atoms[ib];
    const double ra[3] = {A.x, A.y, A.z}, rb[3] = {B.x, B.y, B.z};
    const double d[3] = {ra[0] - rb[0], ra[1] - rb[1], ra[2] - rb[2]};
    const double R2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2];
    const double* As = g_prim[A.pidx][0][0];
    const double* Af = g_prim[A.pidx][0][1];
    const double* Bs = g_prim[B.pidx][0][0];
    const double* Bf = g_prim[B.pidx][0][1];
    const double* Ap = g_prim[A.pidx][1][0];
    const double* Apf = g_prim[A.pidx][1][1];
    const double* Bp = g_prim[B.pidx][1][0];
    const double* Bpf = g_prim[B.pidx][1][1];
    shell_store<0, 0>(ra, rb, d, R2, As, Af, Bs, Bf, A.ao0, B.ao0, N, X);
    if (B.nao > 1) shell_store<0, 1>(ra, rb, d, R2, As, Af, Bp, Bpf, A.ao0, B.ao0, N, X);
    if (A.nao > 1) shell_store<1, 0>(ra, rb, d, R2, Ap, Apf, Bs, Bf, A.ao0, B.ao0, N, X);
    if (A.nao > 1 && B.nao > 1) shell_store<1, 1>(ra, rb, d, R2, Ap, Apf, Bp, Bpf, A.ao0, B.ao0, N, X);
  }
}

void launch_cartesian_matrix(const DevAtom* atoms, const DevPair* pairs, const DevMol* mols, int m, int natoms,
                             double* X, cudaStream_t s) {
  const long long items = (long long)natoms + (long long)natoms * (natoms - 1) / 2;
  const int blocks = (int)std::max(1LL, std::min<long long>(4096, (items + kDipThreads - 1) / kDipThreads));
  cartesian_matrix_kernel<<<blocks, kDipThreads, 0, s>>>(atoms, pairs, mols, m, X);
}

// ---------------------------------------------------------------------------
// Analytic energy gradient (forces) of a converged SCF, for the molecules of
// a list (Mndo::CalcForce, src/mndo/Mndo.cpp:2711-2986, ground state).
//
// With the density P fixed at convergence (the SCF energy is stationary in
// the orbitals and NDDO has no basis-overlap terms) the energy depends on the
// geometry only through the pair terms, each a function of the pair's
// relative position d = R_B - R_A:
//   E_AB = sum_PQ C_PQ W_PQ(d) + sum_{mu in A, la in B} P_mu,la (beta_mu + beta_la) S_mu,la(d)
//          + E_core(d) [+ E_vdW(d)]
// with W = T2 L T2^T the rotated (mu nu|la si) block, C_PQ = m_P m_Q P_P P_Q
// - 1/2 X_PQ (Coulomb and exchange, m = 2 for mu != nu, X summed over both
// orbital orders) plus the electron-core attractions -Z_B (mu nu|s_B s_B) on
// the (mu nu, ss) column and -Z_A on the (ss, la si) row.
//
// The derivative is taken in the pair's local frame (z along d).  With
// C' = T2^T C T2 the density factors of that frame, E = sum C'_PQ L_PQ(R):
//   along z:  sum C'_PQ dL_PQ/dR (each local integral's terms differentiated);
//   along x:  moving B by delta turns the frame by delta / R about y, so the
//             columns of T2 change by T2 G with the generator G of that
//             rotation on orbital products, and dE = (delta / R) sum C'_PQ
//             (G L + L G^T)_PQ; y alike.
// Resonance: the same with the 4 x 4 overlap block and w' = Rm^T w Rm; core-core
// and dispersion depend on R alone.  These are the exact derivatives of the
// formulas the pair kernels evaluate, for any azimuth of the frame (the local
// integrals are cylindrically symmetric).  One warp per pair: lane = local
// integral, then lane = (P, Q).  The gradient of atom i is then
//   g_i = sum_{a < i} dE_ai/dd - sum_{b > i} dE_ib/dd   (fixed order).
// What bounds it: latency, a few thousand clocks of dependent FP64 per pair.
// One thread per pair in three-component dual numbers kept its 10 x 10 matrices
// in local memory: 1.30 ms for octane's 325 pairs.
// ---------------------------------------------------------------------------
constexpr int kGradWarps = 4;

struct GradShared {
  double T2[100], C[100], M[100];
  double val[24], dval[24];
  double ab[4][2][9];      // per exponent combination: A_0..8, B_0..8
  double Rm[16], w[16], ls[8], dls[8], pA[10], pB[10], pab[16];
};

// where the generator of a frame rotation takes local orbital i (s, y, z, x):
// axis 0 turns z towards x, axis 1 turns z towards y; sign 0: nowhere
__device__ __forceinline__ double turned(int axis, int i, int* k) {
  const int to = axis == 0 ? 3 : 1;
  if (i == 2) { *k = to; return 1.0; }
  if (i == to) { *k = 2; return -1.0; }
  *k = 0;
  return 0.0;
}

__global__ void __launch_bounds__(kGradWarps * 32)
pair_grad_kernel(const DevAtom* __restrict__ atoms, const DevPair* __restrict__ pairs, long long pair0,
                 long long npairs, const DevMol* __restrict__ mols, const EriTable* __restrict__ eri,
                 const OverlapTable* __restrict__ ovt, const double* __restrict__ P, VdwParams vdw,
                 double* __restrict__ grad) {
  __shared__ GradShared shared[kGradWarps];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long t = (long long)blockIdx.x * kGradWarps + warp;
  if (t >= npairs) return;
  GradShared& sh = shared[warp];
  const DevPair pr = pairs[pair0 + t];
  const DevAtom A = atoms[pr.a], B = atoms[pr.b];
  const DevMol mol = mols[pr.mol];
  const nddo_atom_params& pa = c_params[A.pidx];
  const nddo_atom_params& pb = c_params[B.pidx];
  const int nA = A.nao, nB = B.nao, dA = nA == 4 ? 10 : 1, dB = nB == 4 ? 10 : 1;
  const double dx = B.x - A.x, dy = B.y - A.y, dz = B.z - A.z;
  const double R = sqrt(dx * dx + dy * dy + dz * dz);
  const double* Pm = P + mol.mat0;
  const long long ld = mol.nao;

  if (lane == 0) {
    double Rm[4][4];
    rotation_matrix(dx, dy, dz, Rm);
    for (int i = 0; i < 16; ++i) sh.Rm[i] = Rm[i >> 2][i & 3];
  }
  // density of both atoms and between them
  if (lane < 10 && lane < dA) {
    int m, n;
    unpack_index(lane, &m, &n);
    sh.pA[lane] = Pm[(A.ao0 + m) * ld + A.ao0 + n];
  }
  if (lane >= 10 && lane - 10 < dB) {
    int m, n;
    unpack_index(lane - 10, &m, &n);
    sh.pB[lane - 10] = Pm[(B.ao0 + m) * ld + B.ao0 + n];
  }
  if (lane < 16) {
    const int mu = lane >> 2, la = lane & 3;
    sh.pab[lane] = mu < nA && la < nB ? Pm[(A.ao0 + mu) * ld + B.ao0 + la] : 0.0;
  }
  // local integrals and their derivatives in R: lane = slot
  double val = 0.0, dval = 0.0;
  if (lane < 21) {
    bool need;
    if (nA == 4 && nB == 4) need = true;
    else if (nA == 4) need = (lane == 0 || lane == 3 || lane == 4 || lane == 10);
    else if (nB == 4) need = (lane == 0 || lane == 1 || lane == 2 || lane == 13);
    else need = (lane == 0);
    if (need) {
      const int nt = eri->nterms[lane];
      for (int k = 0; k < nt; ++k) {
        const EriTerm e = eri->terms[lane][k];
        const double da = sel3(e.la, pa.d[0], pa.d[1], pa.d[2]);
        const double db = sel3(e.lb, pb.d[0], pb.d[1], pb.d[2]);
        const double a = sel3(e.la, pa.rho[0], pa.rho[1], pa.rho[2]) + sel3(e.lb, pb.rho[0], pb.rho[1], pb.rho[2]);
        const double l = R + (double)e.c1 * da + (double)e.c2 * db;
        const double u = (double)e.c3 * da + (double)e.c4 * db;
        const double v = (double)e.c5 * da + (double)e.c6 * db;
        const double r = rsqrt(l * l + u * u + v * v + a * a);
        const double w = e.coef * r;
        val += w;
        dval -= w * l * (r * r);
      }
    }
  }
  {
    const double s5 = __shfl_sync(0xffffffffu, val, 5), s6 = __shfl_sync(0xffffffffu, val, 6);
    const double d5 = __shfl_sync(0xffffffffu, dval, 5), d6 = __shfl_sync(0xffffffffu, dval, 6);
    if (lane == 21 && nA == 4 && nB == 4) { val = 0.5 * (s5 - s6); dval = 0.5 * (d5 - d6); }
  }
  if (lane < 22) { sh.val[lane] = val; sh.dval[lane] = dval; }
  // overlap auxiliary integrals (as pair_kernel), one order more for the
  // derivatives: A_k' = -A_{k+1}, B_k' = -B_{k+1}
  const int na = pa.principal_n, nb = pb.principal_n;
  if (lane < 8) {
    const int zc = lane & 3;
    const bool need = (zc == 0) || (zc == 1 && nB == 4) || (zc == 2 && nA == 4) || (zc == 3 && nA == 4 && nB == 4);
    if (need) {
      const double za = (zc >= 2) ? pa.zeta[1] : pa.zeta[0];
      const double zb = (zc & 1) ? pb.zeta[1] : pb.zeta[0];
      double v[9];
      if (lane < 4) aux_a_all(0.5 * R * (za + zb), 8, v);
      else aux_b_all(0.5 * R * (za - zb), 8, v, c_inv);
#pragma unroll
      for (int k = 0; k < 9; ++k) sh.ab[zc][lane >> 2][k] = v[k];
    }
  }
  __syncwarp();
  // rotation of orbital products, density factors of the space-frame integrals
  for (int e = lane; e < 100; e += 32) {
    int m, n, i, j;
    unpack_index(e / 10, &m, &n);
    unpack_index(e % 10, &i, &j);
    const double* Rm = sh.Rm;
    sh.T2[e] = (i == j) ? Rm[m * 4 + i] * Rm[n * 4 + i] : Rm[m * 4 + i] * Rm[n * 4 + j] + Rm[m * 4 + j] * Rm[n * 4 + i];
  }
  for (int e = lane; e < dA * dB; e += 32) {
    const int q = e / dB, r = e % dB;
    int a, b, c, d;
    unpack_index(q, &a, &b);
    unpack_index(r, &c, &d);
    const double mA = a == b ? 1.0 : 2.0, mB = c == d ? 1.0 : 2.0;
    // exchange: both orders of (a b) and of (c d)
    double x = sh.pab[a * 4 + c] * sh.pab[b * 4 + d];
    if (a != b) x += sh.pab[b * 4 + c] * sh.pab[a * 4 + d];
    if (c != d) x += sh.pab[a * 4 + d] * sh.pab[b * 4 + c];
    if (a != b && c != d) x += sh.pab[b * 4 + d] * sh.pab[a * 4 + c];
    double f = mA * mB * sh.pA[q] * sh.pB[r] - 0.5 * x;
    if (r == 0) f -= (double)pb.core_charge * mA * sh.pA[q];
    if (q == 0) f -= (double)pa.core_charge * mB * sh.pB[r];
    sh.C[q * 10 + r] = f;
  }
  // overlaps and their derivatives (ss, s-sigma, sigma-s, sigma-sigma, pi-pi)
  if (lane < 5) {
    const int c = lane;
    const bool need = (c == 0) || (c == 1 && nB == 4) || (c == 2 && nA == 4) || (c >= 3 && nA == 4 && nB == 4);
    double s = 0.0, ds = 0.0;
    if (need) {
      const int zc = (c == 4) ? 3 : c;
      const double za = (zc >= 2) ? pa.zeta[1] : pa.zeta[0], zb = (zc & 1) ? pb.zeta[1] : pb.zeta[0];
      const double dp = 0.5 * (za + zb), dq = 0.5 * (za - zb);
      const double* a = sh.ab[zc][0];
      const double* b = sh.ab[zc][1];
      const int nt = ovt->nterms[na - 1][nb - 1][c];
      for (int k = 0; k < nt; ++k) {
        const double tc = ovt->tc[na - 1][nb - 1][c][k];
        const int i = ovt->ti[na - 1][nb - 1][c][k], j = ovt->tj[na - 1][nb - 1][c][k];
        s += tc * a[i] * b[j];
        ds -= tc * (dp * a[i + 1] * b[j] + dq * a[i] * b[j + 1]);
      }
      const double norm = pa.sto_norm[c >= 2 ? 1 : 0] * pb.sto_norm[(c == 1 || c >= 3) ? 1 : 0] * ovt->ang[c];
      double rp = 1.0;
      for (int i = 0; i < na + nb + 1; ++i) rp *= 0.5 * R;
      ds = norm * rp * (ds + (double)(na + nb + 1) / R * s);
      s *= norm * rp;
    }
    sh.ls[c] = s;
    sh.dls[c] = ds;
  }
  // w' = Rm^T w Rm of the resonance energy sum w_mu,la S_mu,la
  if (lane < 16) {
    const int i = lane >> 2, j = lane & 3;
    double s = 0.0;
    for (int mu = 0; mu < 4; ++mu)
      for (int la = 0; la < 4; ++la)
        s += sh.Rm[mu * 4 + i] * sh.pab[mu * 4 + la] * (pa.beta[mu == 0 ? 0 : 1] + pb.beta[la == 0 ? 0 : 1]) *
             sh.Rm[la * 4 + j];
    sh.w[lane] = s;
  }
  __syncwarp();
  // C' = T2^T C T2
  for (int e = lane; e < dA * dB; e += 32) {
    const int q = e / dB, r = e % dB;
    double s = 0.0;
    for (int k = 0; k < dB; ++k) s += sh.C[q * 10 + k] * sh.T2[k * 10 + r];
    sh.M[q * 10 + r] = s;
  }
  __syncwarp();
  for (int e = lane; e < dA * dB; e += 32) {
    const int q = e / dB, r = e % dB;
    double s = 0.0;
    for (int k = 0; k < dA; ++k) s += sh.T2[k * 10 + q] * sh.M[k * 10 + r];
    sh.C[q * 10 + r] = s;
  }
  __syncwarp();
  double gr = 0.0, g[2] = {0.0, 0.0};
  for (int e = lane; e < dA * dB; e += 32) {
    const int q = e / dB, r = e % dB;
    const int sl = eri->slot_of[q][r];
    if (sl < 0) continue;
    gr += sh.C[q * 10 + r] * sh.dval[sl];
    const double L = sh.val[sl];
    int i, j, k;
#pragma unroll
    for (int axis = 0; axis < 2; ++axis) {
      double f = 0.0, sg;
      if (dA == 10) {
        unpack_index(q, &i, &j);
        sg = turned(axis, i, &k);
        if (sg != 0.0) f += sg * (i != j && k == j ? 2.0 : 1.0) * sh.C[pack_index(k, j) * 10 + r];
        if (i != j) {
          sg = turned(axis, j, &k);
          if (sg != 0.0) f += sg * (k == i ? 2.0 : 1.0) * sh.C[pack_index(k, i) * 10 + r];
        }
      }
      if (dB == 10) {
        unpack_index(r, &i, &j);
        sg = turned(axis, i, &k);
        if (sg != 0.0) f += sg * (i != j && k == j ? 2.0 : 1.0) * sh.C[q * 10 + pack_index(k, j)];
        if (i != j) {
          sg = turned(axis, j, &k);
          if (sg != 0.0) f += sg * (k == i ? 2.0 : 1.0) * sh.C[q * 10 + pack_index(k, i)];
        }
      }
      g[axis] += L * f;
    }
  }
  if (lane < 16) {
    const int i = lane >> 2, j = lane & 3;
    const int c = (i == 0 && j == 0) ? 0 : (i == 0 && j == 2) ? 1 : (i == 2 && j == 0) ? 2 : (i == 2 && j == 2) ? 3
                  : ((i == 1 && j == 1) || (i == 3 && j == 3)) ? 4 : -1;
    if (c >= 0) {
      gr += sh.w[lane] * sh.dls[c];
      int k;
#pragma unroll
      for (int axis = 0; axis < 2; ++axis) {
        double sg = turned(axis, i, &k);
        if (sg != 0.0) g[axis] += sh.ls[c] * sg * sh.w[k * 4 + j];
        sg = turned(axis, j, &k);
        if (sg != 0.0) g[axis] += sh.ls[c] * sg * sh.w[i * 4 + k];
      }
    }
  }
  if (lane == 31) {
    // core-core repulsion (with the AM1 / PM3 Gaussians and the PDDG term) and
    // the empirical dispersion (energy_kernel's pair term): functions of R
    const Dual3 Rd(R, 1.0, 0.0, 0.0);
    Dual3 e = core_core(pa, pb, Rd, Dual3(sh.val[0], sh.dval[0], 0.0, 0.0), mol.theory);
    const bool dtheory = mol.theory == NDDO_AM1D || mol.theory == NDDO_PM3D;
    if (vdw.on || dtheory) {
      const double s6 = dtheory ? NDDO_VDW_S6_D : vdw.s6, dd = dtheory ? NDDO_VDW_DAMP_D : vdw.d;
      const double csum = pa.vdw_c6 + pb.vdw_c6;
      if (csum > 0.0) {
        const double c6 = 2.0 * pa.vdw_c6 * pb.vdw_c6 / csum;
        const Dual3 damp = 1.0 / (1.0 + exp(-1.0 * dd * (Rd / (pa.vdw_r0 + pb.vdw_r0) - 1.0)));
        const Dual3 R2 = Rd * Rd;
        e += (-1.0 * s6 * c6) * damp / (R2 * R2 * R2);
      }
    }
    gr += e.d[0];
  }
  gr = warp_sum(gr);
  g[0] = warp_sum(g[0]) / R;
  g[1] = warp_sum(g[1]) / R;
  if (lane < 3) {
    // rows of Rm: s, py, pz, px; columns: local s, y, z, x
    const int row = lane == 0 ? 3 : lane;
    grad[3 * t + lane] = sh.Rm[row * 4 + 2] * gr + sh.Rm[row * 4 + 3] * g[0] + sh.Rm[row * 4 + 1] * g[1];
  }
}

// forces F_i = -g_i of one molecule's atoms from its pair gradients: a warp per atom
__global__ void __launch_bounds__(128)
force_reduce_kernel(const DevMol* __restrict__ mols, int m, const double* __restrict__ grad,
                    double* __restrict__ forces) {
  const DevMol mol = mols[m];
  const int i = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (i >= mol.natoms) return;
  double g[3] = {0.0, 0.0, 0.0};
  for (int a = lane; a < mol.natoms; a += 32) {
    if (a == i) continue;
    const double sg = a < i ? 1.0 : -1.0;
    const double* q = grad + 3 * (a < i ? pair_index(a, i, mol.natoms) : pair_index(i, a, mol.natoms));
    for (int k = 0; k < 3; ++k) g[k] += sg * q[k];
  }
  for (int k = 0; k < 3; ++k) g[k] = warp_sum(g[k]);
  if (lane < 3) forces[3 * i + lane] = -(lane == 0 ? g[0] : lane == 1 ? g[1] : g[2]);
}

void launch_forces(const DevAtom* atoms, const DevPair* pairs, const DevMol* mols, int m, long long pair0,
                   long long npairs, int natoms, const EriTable* eri, const OverlapTable* ovt, const double* P,
                   VdwParams vdw, double* grad, double* forces, cudaStream_t s) {
  if (npairs > 0)
    pair_grad_kernel<<<(unsigned)((npairs + kGradWarps - 1) / kGradWarps), kGradWarps * 32, 0, s>>>(
        atoms, pairs, pair0, npairs, mols, eri, ovt, P, vdw, grad);
  force_reduce_kernel<<<(natoms + 3) / 4, 128, 0, s>>>(mols, m, grad, forces);
}

}  // namespace nddo
