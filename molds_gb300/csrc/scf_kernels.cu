// Kernels (c) and (e): batched dense contractions and the density-DIIS step.
//
// (c) gemm_kernel -- one launch multiplies a list of per-molecule matrices of
//     different shapes ("jobs"); each CTA computes one 64x64 tile of one job.
//     Used for the warm-start transform G = C_prev F C_prev^T, the density
//     P = 2 C_occ^T C_occ (MolDS Cndo2::CalcOrbitalElectronPopulation,
//     src/cndo/Cndo2.cpp:1702-1719 via Blas::Dsyrk) and the FP64 subspace
//     refinement of the mixed-precision path.  The arithmetic type is a template
//     parameter: FP32 in the early iterations, FP64 after the switch and on the
//     plain FP64 path.
//
// (e) DIIS -- partial (with the solve) / apply kernels: RMS density change and convergence
//     test (Cndo2::SatisfyConvergenceCriterion, src/cndo/Cndo2.cpp:1472-1517),
//     density DIIS with MolDS's exact window/acceptance rules (Cndo2::DoDIIS,
//     :920-1028) and damping (Cndo2::DoDamp, :1030-1061).  The DIIS history is
//     a ring buffer instead of MolDS's memmove shift; the linear system is
//     assembled in chronological order so it is the same system.  All
//     reductions use fixed-order trees.
#include <cuda_runtime.h>
#include <algorithm>
#include "nddo_batch.cuh"
#include "kernels.h"

namespace nddo {

constexpr int kTile = 64, kTileK = 16, kGemmThreads = 256;

template <typename TA, typename TB, typename TC, typename TAcc, bool TA_, bool TB_>
__global__ void __launch_bounds__(kGemmThreads)
gemm_kernel(const GemmJob* __restrict__ jobs, int njobs, const TA* __restrict__ A, const TB* __restrict__ B,
            TC* __restrict__ C, const MolState* __restrict__ st, int require_active, int require_phase) {
  __shared__ TAcc As[kTileK][kTile + 1];
  __shared__ TAcc Bs[kTileK][kTile + 1];
  // job of this tile (jobs sorted by tile0)
  int lo = 0, hi = njobs - 1;
  const int t = blockIdx.x;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (jobs[mid].tile0 <= t) lo = mid; else hi = mid - 1;
  }
  const GemmJob job = jobs[lo];
  if (mol_skipped(st[job.mol], require_active)) return;
  if (require_phase >= 0 && st[job.mol].phase != require_phase) return;
  const int local = t - job.tile0;
  int tm, tn;
  if (job.sym) {
    // upper-triangle tile order: row tm holds tiles tm..T-1
    const int T = job.tiles_n;
    tm = 0;
    int rem = local;
    while (rem >= T - tm) { rem -= T - tm; ++tm; }
    tn = tm + rem;
  } else {
    tm = local / job.tiles_n;
    tn = local % job.tiles_n;
  }
  const int row0 = tm * kTile, col0 = tn * kTile;
  const TA* Aj = A + job.a_off;
  const TB* Bj = B + job.b_off;
  TC* Cj = C + job.c_off;
  const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
  TAcc acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0;

  for (int k0 = 0; k0 < job.K; k0 += kTileK) {
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int e = tid + r * kGemmThreads;
      int ii, kk;
      if (TA_) { kk = e >> 6; ii = e & 63; } else { ii = e >> 4; kk = e & 15; }
      const int gi = row0 + ii, gk = k0 + kk;
      TAcc v = 0;
      if (gi < job.M && gk < job.K) v = (TAcc)(TA_ ? Aj[(long long)gk * job.lda + gi] : Aj[(long long)gi * job.lda + gk]);
      As[kk][ii] = v;
      int jj, kb;
      if (TB_) { jj = e >> 4; kb = e & 15; } else { kb = e >> 6; jj = e & 63; }
      const int gj = col0 + jj, gkb = k0 + kb;
      TAcc w = 0;
      if (gj < job.N && gkb < job.K) w = (TAcc)(TB_ ? Bj[(long long)gj * job.ldb + gkb] : Bj[(long long)gkb * job.ldb + gj]);
      Bs[kb][jj] = w;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < kTileK; ++kk) {
      TAcc a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = As[kk][ty * 4 + i];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = Bs[kk][tx * 4 + j];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] += a[i] * b[j];
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int gi = row0 + ty * 4 + i;
    if (gi >= job.M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int gj = col0 + tx * 4 + j;
      if (gj >= job.N) continue;
      TC* c = Cj + (long long)gi * job.ldc + gj;
      double v = job.alpha * (double)acc[i][j];
      if (gi == gj) v += job.diag;
      *c = (TC)(job.beta != 0.0 ? v + job.beta * (double)(*c) : v);
      if (job.sym && tm != tn) {   // mirror (beta is zero for symmetric jobs)
        TC* cm = Cj + (long long)gj * job.ldc + gi;
        *cm = (TC)v;
      }
    }
  }
}

int gemm_tiles(int M, int N) { return ((M + kTile - 1) / kTile) * ((N + kTile - 1) / kTile); }
int gemm_tiles_n(int N) { return (N + kTile - 1) / kTile; }
int gemm_tiles_sym(int N) { const int T = (N + kTile - 1) / kTile; return T * (T + 1) / 2; }

#define GEMM_LAUNCH(TA, TB, TC, TACC)                                                                        \
  void launch_gemm(const GemmJob* jobs, int njobs, int ntiles, const TA* A, const TB* B, TC* C, bool ta,      \
                   bool tb, TACC /*acc tag*/, const MolState* st, int require_active, int require_phase,        \
                   cudaStream_t s) {                                                                         \
    if (ntiles <= 0 || njobs <= 0) return;                                                                   \
    if (!ta && !tb) gemm_kernel<TA, TB, TC, TACC, false, false><<<ntiles, kGemmThreads, 0, s>>>(jobs, njobs, A, B, C, st, require_active, require_phase); \
    else if (ta && !tb) gemm_kernel<TA, TB, TC, TACC, true, false><<<ntiles, kGemmThreads, 0, s>>>(jobs, njobs, A, B, C, st, require_active, require_phase); \
    else if (!ta && tb) gemm_kernel<TA, TB, TC, TACC, false, true><<<ntiles, kGemmThreads, 0, s>>>(jobs, njobs, A, B, C, st, require_active, require_phase); \
    else gemm_kernel<TA, TB, TC, TACC, true, true><<<ntiles, kGemmThreads, 0, s>>>(jobs, njobs, A, B, C, st, require_active, require_phase); \
  }
GEMM_LAUNCH(double, double, double, double)
GEMM_LAUNCH(double, double, double, float)
GEMM_LAUNCH(double, double, float, float)
GEMM_LAUNCH(float, double, float, float)
GEMM_LAUNCH(double, float, float, float)
GEMM_LAUNCH(float, double, double, float)
#undef GEMM_LAUNCH

// ---------------------------------------------------------------------------
// One SCF bookkeeping step per molecule, after the new density P is formed, in
// two launches.  (1) partial sums over fixed chunks of the molecule's matrix
// (sum e^2, max |e|, the new B row) while the new history entry is written; the
// molecule's last CTA to finish reduces the chunks in a fixed order and one warp
// runs the convergence test, the DIIS solve, damping and the phase switch;
// (2) the extrapolation and damping over the same chunks.  The chunking depends
// only on N, so a molecule's result does not depend on the rest of the batch.
// What bounds it: latency for one molecule (a launch, two passes of block
// reductions and a 6 x 6 solve), HBM for a batch.  A CTA per 4096 elements with
// a block reduction per sum and the solve on one thread of a launch of its own
// took 75 us for octane in an iteration of 420.
// ---------------------------------------------------------------------------
constexpr int kDiisThreads = 256;
constexpr int kDiisChunksMax = 128;
constexpr int kDiisPart = 2 + kMaxDiis;     // sum e^2, max |e|, dots

__host__ __device__ __forceinline__ int diis_chunks(long long n2) {
  const long long c = (n2 + 2047) / 2048;
  return (int)(c < kDiisChunksMax ? (c < 1 ? 1 : c) : kDiisChunksMax);
}

struct DiisStep {          // decisions of kernel (1) read by kernel (2)
  double coef[kMaxDiis];
  int apply, damp, active, pad;
};

// The molecule's bookkeeping by one warp, from its summed quantities.
// a: (kMaxDiis + 1) x (kMaxDiis + 2) doubles, f: kMaxDiis + 1, in shared memory.
__device__ void diis_decide(MolState* s, const ScfParamsDev& prm, long long n2, const double* sum, TraceEntry* trace,
                            int trace_len, DiisStep* step, double* a, double* f) {
  const int lane = threadIdx.x & 31;
  const int iter = s->iter;
  const bool is_guess = (iter == 0 && s->requires_guess);
  const int M = prm.diis_m;
  const bool do_diis = !is_guess && M > 0;
  const int slot = do_diis ? (s->diis_count % M) : 0;
  const int count = do_diis ? min(s->diis_count + 1, M) : 0;
  const double rms = sqrt(sum[0] / (double)n2), maxe = sum[1];
  const bool converged = rms < prm.rms_density;
  const bool apply = do_diis && !converged && (M <= iter) && (prm.diis_end < maxe) && (maxe < prm.diis_start) &&
                     (count == M);
  __syncwarp();
  if (lane == 0) {
    if (trace && iter < trace_len) {
      TraceEntry te;
      te.rms = rms; te.diis_err = s->diis_err; te.diis_on = s->diis_on; te.damp_on = s->damp_on;
      trace[iter] = te;
    }
    s->rms = rms;
    step->apply = step->damp = 0;
    step->active = converged ? 0 : 1;
    if (converged) s->status = kConverged;
  }
  if (lane < kMaxDiis) step->coef[lane] = 0.0;
  if (converged) return;
  bool solved = false;
  if (do_diis) {
    if (lane < count) { s->B[lane * kMaxDiis + slot] = sum[2 + lane]; s->B[slot * kMaxDiis + lane] = sum[2 + lane]; }
    __syncwarp();
    if (lane == 0) {
      s->diis_count += 1;
      s->diis_head = slot;
      s->diis_err = maxe;
    }
    if (apply) {
      // augmented matrix in chronological order: oldest ... newest
      const int n = M + 1, ld = kMaxDiis + 2;
      for (int e = lane; e < n * (n + 1); e += 32) {
        const int i = e / (n + 1), j = e % (n + 1);
        double v;
        if (j == n) v = i == M ? -1.0 : 0.0;
        else if (i < M && j < M) v = s->B[((slot + 1 + i) % M) * kMaxDiis + (slot + 1 + j) % M];
        else v = i == M && j == M ? 0.0 : -1.0;
        a[i * ld + j] = v;
      }
      __syncwarp();
      // Gaussian elimination with partial pivoting; an exactly zero pivot
      // means a singular system, which MolDS answers by skipping the step
      bool singular = false;
      for (int c = 0; c < n && !singular; ++c) {
        int piv = c;
        for (int r = c + 1; r < n; ++r) if (fabs(a[r * ld + c]) > fabs(a[piv * ld + c])) piv = r;
        if (a[piv * ld + c] == 0.0) { singular = true; break; }
        __syncwarp();
        if (piv != c && lane <= n) {
          const double t = a[c * ld + lane];
          a[c * ld + lane] = a[piv * ld + lane];
          a[piv * ld + lane] = t;
        }
        __syncwarp();
        if (lane > c && lane < n) f[lane] = a[lane * ld + c] / a[c * ld + c];
        __syncwarp();
        const int w = n + 1 - c;
        for (int e = lane; e < (n - 1 - c) * w; e += 32) {
          const int r = c + 1 + e / w, j = c + e % w;
          a[r * ld + j] -= f[r] * a[c * ld + j];
        }
        __syncwarp();
      }
      if (!singular) {
        if (lane == 0) {
          for (int c = n - 1; c >= 0; --c) {
            double v = a[c * ld + n];
            for (int j = c + 1; j < n; ++j) v -= a[c * ld + j] * f[j];
            f[c] = v / a[c * ld + c];
          }
          for (int k = 0; k < M; ++k) step->coef[k] = f[k];
          step->apply = 1;
        }
        solved = true;
      }
    }
  }
  if (lane == 0) {
    if (!is_guess) {
      if (do_diis) s->diis_on = solved ? 1 : 0;
      const int damp = (prm.damping_weight > 0.0 && prm.damping_thresh < rms) ? 1 : 0;
      step->damp = damp;
      s->damp_on = damp;
      if (prm.precision == 1 && s->phase == 0 && do_diis && maxe < prm.switch_error) s->phase = 1;
    }
    s->iter = iter + 1;
    if (iter + 1 >= prm.max_iter) s->status = kNotConverged;
  }
}

__global__ void __launch_bounds__(kDiisThreads, 3)
diis_partial_kernel(const DevMol* __restrict__ mols, const int* __restrict__ mol_list, MolState* __restrict__ st,
                    ScfParamsDev prm, const double* __restrict__ P, const double* __restrict__ Pold,
                    double* __restrict__ hist_dens, double* __restrict__ hist_err, long long hist_stride,
                    double* __restrict__ part, DiisStep* __restrict__ steps, int* __restrict__ ticket,
                    TraceEntry* __restrict__ trace, int trace_len) {
  constexpr int kWarps = kDiisThreads / 32;
  __shared__ double s_red[kWarps][kDiisPart];
  __shared__ double s_a[(kMaxDiis + 1) * (kMaxDiis + 2)], s_f[kMaxDiis + 1], s_sum[kDiisPart];
  __shared__ int s_last;
  const int li = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int m = mol_list[li];
  MolState* s = st + m;
  if (s->status != kActive || ((s->flags & kNeedEigen) && !prm.eigen_ran)) {
    if (blockIdx.x == 0 && tid == 0) steps[li].active = 0;
    return;
  }
  const DevMol mol = mols[m];
  const long long n2 = (long long)mol.nao * mol.nao;
  const int chunks = diis_chunks(n2);
  if ((int)blockIdx.x >= chunks) return;
  const long long len = (n2 + chunks - 1) / chunks;
  const long long lo = blockIdx.x * len, hi = (lo + len < n2) ? lo + len : n2;
  const bool is_guess = (s->iter == 0 && s->requires_guess);
  const int M = prm.diis_m;
  const bool do_diis = !is_guess && M > 0;
  const int slot = do_diis ? (s->diis_count % M) : 0;
  const int count = do_diis ? min(s->diis_count + 1, M) : 0;
  const double* Pm = P + mol.mat0;
  const double* Po = Pold + mol.mat0;
  double* dslot = hist_dens + slot * hist_stride + mol.mat0;
  double* eslot = hist_err + slot * hist_stride + mol.mat0;
  double v[kDiisPart];
#pragma unroll
  for (int k = 0; k < kDiisPart; ++k) v[k] = 0.0;
  // two elements' loads before the first store: the history is read and written
  // through one pointer, so the compiler keeps their order.  A launch takes 24 us for
  // (H2O)33, 55 for (H2O)180 and 266 for 256 (H2O)32; with one element 27, 69 and 234,
  // with four (142 registers) 386 for the batch.
  constexpr int kU = 2;
  for (long long i0 = lo + tid; i0 < hi; i0 += kU * kDiisThreads) {
    double p[kU], e[kU], x[kMaxDiis][kU];
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      const long long i = i0 + u * kDiisThreads;
      p[u] = i < hi ? Pm[i] : 0.0;
      e[u] = i < hi ? p[u] - Po[i] : 0.0;
    }
    if (do_diis) {
#pragma unroll
      for (int k = 0; k < kMaxDiis; ++k)
        if (k < count && k != slot)
#pragma unroll
          for (int u = 0; u < kU; ++u) {
            const long long i = i0 + u * kDiisThreads;
            x[k][u] = i < hi ? hist_err[k * hist_stride + mol.mat0 + i] : 0.0;
          }
    }
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      const long long i = i0 + u * kDiisThreads;
      v[0] += e[u] * e[u];
      v[1] = fmax(v[1], fabs(e[u]));
      if (do_diis && i < hi) {
        dslot[i] = p[u];
        eslot[i] = e[u];
#pragma unroll
        for (int k = 0; k < kMaxDiis; ++k)
          if (k < count) v[2 + k] += (k == slot ? e[u] : x[k][u]) * e[u];
      }
    }
  }
#pragma unroll
  for (int k = 0; k < kDiisPart; ++k) {
    if (k < 2 + count)
      for (int o = 16; o > 0; o >>= 1) {
        const double t = __shfl_xor_sync(0xffffffffu, v[k], o);
        v[k] = k == 1 ? fmax(v[k], t) : v[k] + t;
      }
    if (lane == 0) s_red[warp][k] = v[k];
  }
  __syncthreads();
  double* out = part + (long long)li * gridDim.x * kDiisPart;
  if (tid < kDiisPart) {
    double t = s_red[0][tid];
    for (int w = 1; w < kWarps; ++w) t = tid == 1 ? fmax(t, s_red[w][tid]) : t + s_red[w][tid];
    out[blockIdx.x * kDiisPart + tid] = t;
    __threadfence();
  }
  __syncthreads();
  if (tid == 0) s_last = atomicAdd(ticket + li, 1) == chunks - 1;
  __syncthreads();
  if (!s_last || warp != 0) return;
  __threadfence();
#pragma unroll
  for (int k = 0; k < kDiisPart; ++k) {
    double t = 0.0;
    if (k < 2 + count) {
      for (int c = lane; c < chunks; c += 32) {
        const double x = __ldcg(out + c * kDiisPart + k);
        t = k == 1 ? fmax(t, x) : t + x;
      }
      for (int o = 16; o > 0; o >>= 1) {
        const double x = __shfl_xor_sync(0xffffffffu, t, o);
        t = k == 1 ? fmax(t, x) : t + x;
      }
    }
    if (lane == 0) s_sum[k] = t;
  }
  if (lane == 0) {
    ticket[li] = 0;
    if (mol.natoms > 1) s->flags &= ~kNeedEigen;
  }
  __syncwarp();
  diis_decide(s, prm, n2, s_sum, trace ? trace + (long long)m * trace_len : nullptr, trace_len, steps + li, s_a, s_f);
}

__global__ void __launch_bounds__(kDiisThreads)
diis_apply_kernel(const DevMol* __restrict__ mols, const int* __restrict__ mol_list, const MolState* __restrict__ st,
                  ScfParamsDev prm, double* __restrict__ P, const double* __restrict__ Pold,
                  const double* __restrict__ hist_dens, long long hist_stride, const DiisStep* __restrict__ steps) {
  const int li = blockIdx.y;
  const DiisStep* d = steps + li;
  const int apply = d->apply, damp = d->damp;
  if (!d->active || (!apply && !damp)) return;
  const int m = mol_list[li];
  const DevMol mol = mols[m];
  const long long n2 = (long long)mol.nao * mol.nao;
  const int chunks = diis_chunks(n2);
  if ((int)blockIdx.x >= chunks) return;
  const long long len = (n2 + chunks - 1) / chunks;
  const long long lo = blockIdx.x * len, hi = (lo + len < n2) ? lo + len : n2;
  const int M = prm.diis_m;
  double* Pm = P + mol.mat0;
  const double* Po = Pold + mol.mat0;
  // the newest entry is the one this iteration pushed (diis_head); oldest first
  // (MolDS sums the stored densities in slot order through Dgemv)
  const int newest = st[m].diis_head;
  double coef[kMaxDiis];
  long long off[kMaxDiis];
#pragma unroll
  for (int k = 0; k < kMaxDiis; ++k)
    if (apply && k < M) {
      coef[k] = d->coef[k];
      off[k] = ((newest + 1 + k) % M) * hist_stride + mol.mat0;
    }
  for (long long i = lo + threadIdx.x; i < hi; i += kDiisThreads) {
    double v = Pm[i];
    if (apply) {
      v = 0.0;
#pragma unroll
      for (int k = 0; k < kMaxDiis; ++k)
        if (k < M) v += coef[k] * hist_dens[off[k] + i];
    }
    if (damp) v = v * (1.0 - prm.damping_weight) + prm.damping_weight * Po[i];
    Pm[i] = v;
  }
}

void launch_diis(const DevMol* mols, const int* mol_list, int nlist, int max_n, MolState* st, const ScfParamsDev& prm,
                 double* P, const double* Pold, double* hist_dens, double* hist_err, long long hist_stride,
                 TraceEntry* trace, int trace_len, void* scratch, int slots, int cap_n, cudaStream_t s) {
  if (nlist <= 0) return;
  double* part = static_cast<double*>(scratch);
  DiisStep* steps = reinterpret_cast<DiisStep*>(part + (size_t)slots * diis_chunks((long long)cap_n * cap_n) * kDiisPart);
  int* ticket = reinterpret_cast<int*>(steps + slots);
  const int chunks = diis_chunks((long long)max_n * max_n);
  diis_partial_kernel<<<dim3(chunks, nlist), kDiisThreads, 0, s>>>(mols, mol_list, st, prm, P, Pold, hist_dens, hist_err,
                                                                  hist_stride, part, steps, ticket, trace, trace_len);
  diis_apply_kernel<<<dim3(chunks, nlist), kDiisThreads, 0, s>>>(mols, mol_list, st, prm, P, Pold, hist_dens,
                                                                hist_stride, steps);
}

// partial sums, decisions and tickets (zero between launches) of `slots` list entries
// of up to cap_n basis functions
size_t diis_scratch_bytes(int slots, int cap_n) {
  const size_t part = (size_t)diis_chunks((long long)cap_n * cap_n) * kDiisPart * sizeof(double);
  return (size_t)slots * (part + sizeof(DiisStep) + sizeof(int)) + 256;
}

// ---------------------------------------------------------------------------
// small elementwise helpers
// ---------------------------------------------------------------------------
// FP64 refinement (one Newton step of Ogita & Aishima's eigenvector refinement,
// restricted to the occupied columns): with approximate eigenvectors x and
// eigenvalues lam, K_ai = -(x_a^T F x_i - lam_i x_a^T x_i) / (lam_a - lam_i),
// a virtual, i occupied.  The overlap term removes the first-order error left
// by the non-orthogonality of FP32 eigenvectors.
__global__ void newton_scale_kernel(const DevMol* __restrict__ mols, const int* __restrict__ mol_list,
                                    const MolState* __restrict__ st, int require_phase, double* __restrict__ K,
                                    const double* __restrict__ O, const double* __restrict__ eps) {
  const int m = mol_list[blockIdx.y];
  if (st[m].status != kActive || (require_phase >= 0 && st[m].phase != require_phase)) return;
  const DevMol mol = mols[m];
  const int n = mol.nao, o = mol.nocc, v = n - o;
  const long long cnt = (long long)v * o;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < cnt; e += (long long)gridDim.x * blockDim.x) {
    const int a = (int)(e / o), i = (int)(e % o);
    const double li = eps[mol.vec0 + i];
    const double gap = eps[mol.vec0 + o + a] - li;
    K[mol.mat0 + e] = -(K[mol.mat0 + e] - li * O[mol.mat0 + e]) / gap;
  }
}

void launch_newton_scale(const DevMol* mols, const int* mol_list, int nlist, const MolState* st, int require_phase,
                         double* K, const double* O, const double* eps, cudaStream_t s) {
  if (nlist <= 0) return;
  newton_scale_kernel<<<dim3(8, nlist), 256, 0, s>>>(mols, mol_list, st, require_phase, K, O, eps);
}

// D = M - I in place (o x o): the first-order (Y^T Y)^-1 = I - D is applied by
// the caller as Z = Y - D Y.
__global__ void neumann_kernel(const DevMol* __restrict__ mols, const int* __restrict__ mol_list,
                               const MolState* __restrict__ st, int require_phase, double* __restrict__ Mm) {
  const int m = mol_list[blockIdx.y];
  if (st[m].status != kActive || (require_phase >= 0 && st[m].phase != require_phase)) return;
  const DevMol mol = mols[m];
  const int o = mol.nocc;
  const long long cnt = (long long)o * o;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < cnt; e += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(e / o), j = (int)(e % o);
    if (i == j) Mm[mol.mat0 + e] -= 1.0;
  }
}

void launch_neumann(const DevMol* mols, const int* mol_list, int nlist, const MolState* st, int require_phase,
                    double* M, cudaStream_t s) {
  if (nlist <= 0) return;
  neumann_kernel<<<dim3(8, nlist), 256, 0, s>>>(mols, mol_list, st, require_phase, M);
}

// copy the first `rows` rows of C (n x n, row-major) into dst (rows x n)
__global__ void copy_rows_kernel(const DevMol* __restrict__ mols, const int* __restrict__ mol_list,
                                 const MolState* __restrict__ st, int require_phase, const double* __restrict__ src,
                                 double* __restrict__ dst) {
  const int m = mol_list[blockIdx.y];
  if (st[m].status != kActive || (require_phase >= 0 && st[m].phase != require_phase)) return;
  const DevMol mol = mols[m];
  const long long cnt = (long long)mol.nocc * mol.nao;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < cnt; e += (long long)gridDim.x * blockDim.x)
    dst[mol.mat0 + e] = src[mol.mat0 + e];
}

void launch_copy_occ_rows(const DevMol* mols, const int* mol_list, int nlist, const MolState* st, int require_phase,
                          const double* src, double* dst, cudaStream_t s) {
  if (nlist <= 0) return;
  copy_rows_kernel<<<dim3(8, nlist), 256, 0, s>>>(mols, mol_list, st, require_phase, src, dst);
}

// FP32 shadows of the basis C (twice: operand and Newton-Schulz output) and of
// F for the tensor-core chain of the FP32 phase: one conversion per element
// and iteration instead of one per tile that loads it
__global__ void tc_shadows_kernel(const DevMol* __restrict__ mols, const int* __restrict__ mol_list,
                                  const MolState* __restrict__ st, const double* __restrict__ C,
                                  const double* __restrict__ F, float* __restrict__ Cf, float* __restrict__ Cf2,
                                  float* __restrict__ Ff) {
  const int m = mol_list[blockIdx.y];
  if (st[m].status != kActive) return;
  const DevMol mol = mols[m];
  const long long cnt = (long long)mol.nao * mol.nao;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < cnt; e += (long long)gridDim.x * blockDim.x) {
    const float c = (float)C[mol.mat0 + e];
    Cf[mol.mat0 + e] = c;
    Cf2[mol.mat0 + e] = c;
    Ff[mol.mat0 + e] = (float)F[mol.mat0 + e];
  }
}

void launch_tc_shadows(const DevMol* mols, const int* mol_list, int nlist, const MolState* st, const double* C,
                       const double* F, float* Cf, float* Cf2, float* Ff, cudaStream_t s) {
  if (nlist <= 0) return;
  tc_shadows_kernel<<<dim3(16, nlist), 256, 0, s>>>(mols, mol_list, st, C, F, Cf, Cf2, Ff);
}

// copy each listed active molecule's N x N block (src -> dst, same offsets)
__global__ void copy_matrices_kernel(const DevMol* __restrict__ mols, const int* __restrict__ mol_list,
                                     const MolState* __restrict__ st, const double* __restrict__ src,
                                     double* __restrict__ dst) {
  const int m = mol_list[blockIdx.y];
  if (st[m].status != kActive) return;
  const DevMol mol = mols[m];
  const long long cnt = (long long)mol.nao * mol.nao;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < cnt; e += (long long)gridDim.x * blockDim.x)
    dst[mol.mat0 + e] = src[mol.mat0 + e];
}

void launch_copy_matrices(const DevMol* mols, const int* mol_list, int nlist, const MolState* st, const double* src,
                          double* dst, cudaStream_t s) {
  if (nlist <= 0) return;
  copy_matrices_kernel<<<dim3(16, nlist), 256, 0, s>>>(mols, mol_list, st, src, dst);
}

}  // namespace nddo
