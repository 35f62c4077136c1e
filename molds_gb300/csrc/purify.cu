// Density matrix by spectral purification on the tensor cores.
//
// The SCF needs P = 2 (projector on the nocc lowest eigenvectors of F).  The
// SP2 iteration (A. M. N. Niklasson, Phys. Rev. B 66, 155115 (2002)) reaches
// the projector from X_0 = (hi - F) / (hi - lo), [lo, hi] a Gershgorin
// interval of F, by X <- X^2 when tr X > nocc and X <- 2 X - X^2 otherwise:
// one symmetric matrix product per step, 18 to 24 steps for the HOMO-LUMO gaps
// of converging molecules.
//
// Why: GB300 issues two FP64 FMAs per clock and SM but 4096 FP16 ones on its
// tensor cores.  X has its spectrum in [0, 1], so |X_ij| <= 1 and it can be
// held in fixed point: 64-bit integers with 55 fraction bits.  Each is split
// into seven signed 8-bit digits, X = sum_i d_i 2^(-7-8i), which FP16 holds
// exactly.  A product of two digits has 14 bits; sums of up to 512 terms (a level
// of a K segment) stay integers of about 2^22, which FP32 holds exactly and a range
// check guards, so tcgen05 MMAs with FP32 accumulators multiply the digit matrices
// without any rounding (the error-free splitting of
// Ozaki, Ogita, Oishi & Rump, Numer. Algorithms 59, 95 (2012)).  Level l sums
// the digit products with i + j = l, levels 0 to 7 are kept (34 products) and
// recombined in 64-bit integers, rounded to 2^-55 (half a step is 2^-56): finer than
// FP64's rounding of entries of order one.  What is dropped, levels 8 to 12, is at
// most 2^-64 a term of a level-8 product.  For a dense X it sums to 2^-57 at N = 256;
// on the diagonal the squares of digit 4 make it a positive bias of about N 2^-65.6,
// half a rounding step at N = 770 and two at 3072.  Integer sums do not depend on
// their order, so X stays exactly symmetric and a molecule's result does not depend
// on its batch.
//
// The error of the last step is known from the traces: tr X_{k+1} - tr X_k is
// +- tr(X_k - X_k^2), the sum of lambda (1 - lambda).  Once that is below 2^-30
// one step of each kind squares what is left on both sides (4e-18).  A molecule
// that does not get there, or to the wrong rank (a vanishing gap, a non-finite
// F), is flagged and waits for an iteration with the Householder eigensolver
// (tridiag.cu).
//
// MolDS's counterpart: Dsyevd and CalcOrbitalElectronPopulation
// (src/cndo/Cndo2.cpp:652-656, 1702-1719).
#include <cuda_runtime.h>
#include <stdint.h>
#include <algorithm>
#include <mutex>
#include "nddo_batch.cuh"
#include "kernels.h"

namespace nddo {

constexpr int kDigits = 7, kLevels = 8;
constexpr int kPurSmallThreads = 17 * 32;
constexpr int kPurSmallSteps = 100;                // the one-CTA kernel stops by itself; its steps are cheap
constexpr int kTraceShift = 12;                    // traces are summed in units of 2^-43
constexpr long long kTraceOne = 1LL << (55 - kTraceShift);
constexpr long long kTraceTol = kTraceOne >> 30;   // tr(X - X^2) that two more steps square away

__device__ __forceinline__ uint32_t pu_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Operand descriptors: K-major, no swizzle; core matrices of 8 rows x 16 bytes,
// K-adjacent ones 128 bytes apart, 8-row groups sbo apart.  Only the low word
// depends on the address: the issuing thread adds to it and nothing else, since
// its instruction stream has to keep up with one MMA per few dozen clocks.
__device__ __forceinline__ uint32_t pu_desc_lo(uint32_t addr) { return (addr >> 4) | (128u >> 4) << 16; }
__device__ __forceinline__ uint32_t pu_desc_hi(uint32_t sbo) { return (sbo >> 4) | 1u << 14; }

__device__ __forceinline__ void pu_mma(uint32_t tmem, uint32_t a, uint32_t b, uint32_t hi, uint32_t idesc, uint32_t acc) {
  asm volatile("{\n .reg .pred p;\n .reg .b64 da, db;\n setp.ne.b32 p, %5, 0;\n mov.b64 da, {%1, %3};\n"
               " mov.b64 db, {%2, %3};\n tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %4, p;\n}"
               :: "r"(tmem), "r"(a), "r"(b), "r"(hi), "r"(idesc), "r"(acc) : "memory");
}

// kind::f16: D = F32, A = B = F16, both K-major, M = 128
__device__ __forceinline__ uint32_t pu_idesc(int ncols) {
  return (1u << 4) | ((uint32_t)(ncols >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
}

// The digit products of levels [L0, L1) over `steps` K steps of 16, by one
// thread.  The digits of B lie behind one another (stride sb, cols rows each) and
// so do the level accumulators (cols columns each), so one MMA multiplies digit i
// of A with up to MOST = 256 / cols digits j, j + 1, .. of B into levels i + j,
// i + j + 1, ..: 12 MMAs of up to 256 columns per K step at 64 columns instead of
// 34.  Reading A costs an MMA 32 clocks of shared memory whatever its width, so
// a 64-column one runs at half the tensor rate and a 256-column one at all of it.
// Unrolled: the issuing thread has about a hundred clocks per MMA.
template <int MOST, int L0, int L1>
__device__ __forceinline__ void pu_products(uint32_t tmem, uint32_t a, uint32_t sa, uint32_t b, uint32_t sb, uint32_t hi,
                                            int cols, int steps, bool fresh) {
#pragma unroll
  for (int i = 0; i < kDigits; ++i) {
    const int j0 = L0 > i ? L0 - i : 0, top = L1 - 1 - i < kDigits - 1 ? L1 - 1 - i : kDigits - 1;
    // the first product into a level overwrites it: digit 0 of A for levels
    // 0 .. 6, product (1, 6), by itself, for level 7
    const int j1 = i == 1 && L1 == kLevels ? top - 1 : top;
#pragma unroll
    for (int t = 0; t < kDigits; ++t) {
      const bool extra = t == kDigits - 1;
      const int j = extra ? kDigits - 1 : j0 + t * MOST;
      if (extra ? !(i == 1 && L1 == kLevels) : j > j1) continue;
      const int w = extra ? 1 : (MOST < j1 - j + 1 ? MOST : j1 - j + 1);
      const uint32_t d = tmem + (i + j - L0) * cols, idesc = pu_idesc(w * cols);
      uint32_t ai = a + ((i * sa) >> 4), bj = b + ((j * sb) >> 4), acc = (i == 0 || extra) && fresh ? 0u : 1u;
      for (int s = 0; s < steps; ++s, ai += 256 >> 4, bj += 256 >> 4) {
        pu_mma(d, ai, bj, hi, idesc, acc);
        acc = 1;
      }
    }
  }
}

// whether a phase came within `limit` clocks
__device__ __forceinline__ bool pu_wait(uint32_t bar, uint32_t parity, long long limit) {
  uint32_t done = 0;
  const long long t0 = clock64();
  while (!done && clock64() - t0 < limit)
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
                 : "=r"(done) : "r"(bar), "r"(parity) : "memory");
  return done != 0;
}
// After a wait that ran out: no copy and no MMA that a CTA has set going may outlive
// it, so what was waited for is waited for once more, with the usual limit.
__device__ __noinline__ void pu_drain(uint32_t bar, uint32_t parity) { pu_wait(bar, parity, kPurWaitCycles); }

__device__ __forceinline__ void pu_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" :: "r"(bar) : "memory");
}

// Accumulators as integers.  They are integers, so adding 1.375 * 2^23 leaves
// those from -0.75 * 2^22 up to 1.25 * 2^22 in the low mantissa bits: a full-rate
// FP32 add where the conversion instruction runs at a quarter of it (5390 -> 1800
// clocks for a 128 x 64 tile).  range collects the bits that would show one outside.
// The interval lies off zero because the sums do: a digit's squares on the diagonal
// have a mean of 0.67 * 2^22 at K = 512 where the digits are spread evenly (a dense
// X), with a standard deviation of 0.09 * 2^22; everything else has none and 0.08.
// That leaves 6.4 deviations above; an interval of +-2^22 left 3.8, and from N = 512
// on a dense molecule went to the eigensolver every few iterations.
__device__ __forceinline__ void pu_ld8(uint32_t addr, float* v) {
  uint32_t u[8];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7])
               : "r"(addr));
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(u[i]);
}
constexpr int kMagic = 0x4B300000;   // 1.375 * 2^23
__device__ __forceinline__ int pu_int(float f, uint32_t& range) {
  const int b = __float_as_int(f + 11534336.0f);
  range |= (uint32_t)(b ^ kMagic);
  return b - kMagic;
}
__device__ __forceinline__ bool pu_in_range(uint32_t range) { return range < (1u << 23); }

__device__ __forceinline__ long long pu_mad(int a, int b, long long c) {
  long long r;
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
  return r;
}

// x += sgn * (levels L .. END - 1), units of 2^-55: level l weighs 2^(41 - 8 l);
// an even level and the next one make one 32-bit number, the last two are rounded
template <int L, int END, int NL>
__device__ __forceinline__ void pu_add(const float (&v)[NL][8], int i, int sgn, long long& x, uint32_t& range) {
  constexpr int w = 41 - 8 * L, at = L - (END - NL);
  if constexpr (L + 2 == kLevels) {
    x = pu_mad((pu_int(v[at][i], range) + (pu_int(v[at + 1][i], range) >> 8) + 64) >> 7, sgn, x);
  } else if constexpr ((L & 1) == 0 && L + 1 < END) {
    const int t = pu_int(v[at][i], range) * 256 + pu_int(v[at + 1][i], range);
    if constexpr (L == 0) x += (long long)((unsigned long long)(unsigned)(t * sgn * 2) << 32);
    else x = pu_mad(t, sgn * (1 << (w - 8)), x);
    if constexpr (L + 2 < END) pu_add<L + 2, END, NL>(v, i, sgn, x, range);
  } else {
    if constexpr (w < 31) x = pu_mad(pu_int(v[at][i], range), sgn * (1 << w), x);
    if constexpr (L + 1 < END) pu_add<L + 1, END, NL>(v, i, sgn, x, range);
  }
}
template <int L0, int NL>
__device__ __forceinline__ void pu_levels8(uint32_t addr, int stride, int sgn, long long* x, uint32_t& range) {
  float v[NL][8];
#pragma unroll
  for (int l = 0; l < NL; ++l) pu_ld8(addr + l * stride, v[l]);
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 8; ++i) pu_add<L0, L0 + NL, NL>(v, i, sgn, x[i], range);
}

// Balanced base-256 digits of eight values as FP16, most significant slice
// first.  With 128 added to every digit they are the bytes of one 64-bit word
// (the top one up to 256), and 0x6400 | byte is the FP16 number 1024 + byte.
__device__ __forceinline__ void pu_split8(const long long* x, uint4* out) {
  uint32_t w[kDigits][4];
  constexpr uint32_t kBias = 0x64806480u;   // two times 1024 + 128
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    const unsigned long long a = (unsigned long long)x[2 * p] + 0x0080808080808080ull;
    const unsigned long long b = (unsigned long long)x[2 * p + 1] + 0x0080808080808080ull;
    const uint32_t al = (uint32_t)a, ah = (uint32_t)(a >> 32), bl = (uint32_t)b, bh = (uint32_t)(b >> 32);
#pragma unroll
    for (int d = 0; d < kDigits; ++d) {
      const int byte = 6 - d;
      uint32_t v;
      if (d == 0) v = (ah >> 16) | (bh & 0xFFFF0000u);   // 0 .. 256: nine bits
      else if (byte >= 4) v = __byte_perm(ah, bh, (byte - 4) | (byte << 8)) & 0x00FF00FFu;
      else v = __byte_perm(al, bl, byte | ((byte + 4) << 8)) & 0x00FF00FFu;
      v += 0x64006400u;
      asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(w[d][p]) : "r"(v), "r"(kBias));
    }
  }
#pragma unroll
  for (int d = 0; d < kDigits; ++d) out[d] = make_uint4(w[d][0], w[d][1], w[d][2], w[d][3]);
}

// eight values back from their digits
__device__ __forceinline__ void pu_join8(const uint4* in, long long* x) {
  constexpr uint32_t kBias = 0x64806480u;
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    uint32_t b[kDigits];   // digit + 128 of both values in the halves
#pragma unroll
    for (int d = 0; d < kDigits; ++d) {
      const uint32_t u = p == 0 ? in[d].x : p == 1 ? in[d].y : p == 2 ? in[d].z : in[d].w;
      asm("add.rn.f16x2 %0, %1, %2;" : "=r"(b[d]) : "r"(u), "r"(kBias));
    }
    // low halves, then high halves; the top digit keeps nine bits
    const uint32_t lo0 = __byte_perm(__byte_perm(b[6], b[5], 0x0040), __byte_perm(b[4], b[3], 0x0040), 0x5410);
    const uint32_t hi0 = (__byte_perm(b[2], b[1], 0x0040) & 0xFFFFu) | ((b[0] - 0x6400u) << 16);
    const uint32_t lo1 = __byte_perm(__byte_perm(b[6], b[5], 0x0062), __byte_perm(b[4], b[3], 0x0062), 0x5410);
    const uint32_t hi1 = (__byte_perm(b[2], b[1], 0x0062) & 0xFFFFu) | (((b[0] >> 16) - 0x6400u) << 16);
    x[2 * p] = (long long)((unsigned long long)hi0 << 32 | lo0) - 0x0080808080808080LL;
    x[2 * p + 1] = (long long)((unsigned long long)hi1 << 32 | lo1) - 0x0080808080808080LL;
  }
}

// a double cut to FP32 by integer instructions (0 below 2^-126, huge above 2^127)
__device__ __forceinline__ float pu_float(double v) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(v);
  const int e = (int)(b >> 52) & 0x7ff;
  const uint32_t s = (uint32_t)(b >> 32) & 0x80000000u;
  if (e < 897) return __uint_as_float(s);
  if (e > 1150) return __uint_as_float(s | 0x7f000000u);
  return __uint_as_float(s | ((uint32_t)(e - 896) << 23) | (uint32_t)((b >> 29) & 0x7fffffu));
}
__device__ __forceinline__ long long pu_fixed(double v) { return __double2ll_rn(v * 36028797018963968.0); }   // 2^55
__device__ __forceinline__ double pu_density(long long x) {   // 2 * 2^-55 x: the exponent by an integer instruction
  const double v = (double)x;
  return x ? __hiloint2double(__double2hiint(v) - (54 << 20), __double2loint(v)) : 0.0;
}

// Where the iteration stands at X_k, with t0, t1 the traces of X_k and X_{k-1}:
// the step to take (1: X^2, 0: 2 X - X^2), or -1 when X_k is the projector.
// first = the first step j whose tr(X_j - X_j^2) was below the tolerance (-1:
// none yet).
__device__ __forceinline__ int pu_step(long long t0, long long t1, int k, int first, long long occ) {
  if (first >= 0 && k >= first + 3) return -1;
  if (first >= 0 && k == first + 2) return t1 > occ ? 0 : 1;   // the other kind than step k - 1
  return t0 > occ ? 1 : 0;
}
__device__ __forceinline__ bool pu_traced(long long a, long long b) {
  const long long d = a > b ? a - b : b - a;
  return d < kTraceTol;
}

// the projector has rank nocc (a level that is degenerate across the gap moves
// to 0 or 1 as a whole)
__device__ __forceinline__ bool pu_counted(long long t, long long occ) {
  const long long d = t > occ ? t - occ : occ - t;
  return d < kTraceOne / 2;
}

// ---------------------------------------------------------------------------
// N <= 128: one CTA per molecule, everything on the SM.  The seven digit
// matrices (K-major core-matrix tiles, the same copy serves as A and as B
// because X is symmetric: 224 KB at N = 128) in shared memory, X itself in
// registers: thread (row r, columns 16 g .. of each 64) with r its TMEM lane.
// A step is 34 digit products over all N columns (an MMA costs its 4 KB of A
// whatever its width: 50 clocks, so few wide ones).  The eight accumulators do
// not fit tensor memory together above N = 64, so the levels go in groups of L
// through two buffers of it: the issuing warp fills one while the others
// recombine the other.
// Measured (clocks a step, N = 50 / 72 / 120): 18000 / 32000 / 50000 with all
// levels of 64 columns at a time, conversions by instruction and the trace by
// shared atomics; 11000 / 16000 / 29000 now.  At small N the interval was as dear
// as the steps: in FP32 with weights it took (H2O)2 from 2.18 to 1.84 ms and
// C14H30 with 900 external charges from 18.5 to 15.2 ms.
// ---------------------------------------------------------------------------
constexpr int kPurSmallWarps = 16;   // recombining; one more issues the MMAs

template <int H, int L, int J>
__device__ __forceinline__ void pu_group(uint32_t taddr, int np, int g, int sgn, long long (&x)[H][16],
                                         uint32_t& range) {
  constexpr int L0 = J * L, NL = L0 + L <= kLevels ? L : kLevels - L0;
#pragma unroll
  for (int h = 0; h < H; ++h) {
    const int c0 = 64 * h + 16 * g;
    if (c0 < np) {
#pragma unroll
      for (int s = 0; s < 2; ++s)
        pu_levels8<L0, NL>(taddr + (J & 1) * L * np + c0 + 8 * s, np, sgn, &x[h][8 * s], range);
    }
  }
}

template <int L, int J>
__device__ __forceinline__ void pu_level_group(uint32_t to, uint32_t lo, uint32_t slice, uint32_t hi, int np) {
  constexpr int L0 = J * L, L1 = L0 + L < kLevels ? L0 + L : kLevels;
  const int k = np / 16;
  if (L == 2) pu_products<2, L0, L1>(to, lo, slice, lo, slice, hi, np, k, true);
  else if (L == 3) pu_products<3, L0, L1>(to, lo, slice, lo, slice, hi, np, k, true);
  else if (np <= 32) pu_products<7, L0, L1>(to, lo, slice, lo, slice, hi, np, k, true);
  else pu_products<4, L0, L1>(to, lo, slice, lo, slice, hi, np, k, true);
}

// The recombining warps have read level group j (buffer j of a step's first two
// groups).  A named barrier per group: a warp that runs ahead reaches the next
// group's while others are still to arrive at this one.
__device__ __forceinline__ void pu_drained(int j, bool issuer) {
  constexpr int kAll = (kPurSmallWarps + 1) * 32;
  if (issuer) asm volatile("bar.sync %0, %1;" :: "r"(1 + j), "n"(kAll) : "memory");
  else asm volatile("bar.arrive %0, %1;" :: "r"(1 + j), "n"(kAll) : "memory");
}

template <int H, int L>
__global__ void __launch_bounds__(kPurSmallThreads, 1)
purify_small_kernel(const DevMol* __restrict__ mols, const int* __restrict__ list, MolState* __restrict__ st,
                    const double* __restrict__ F, double* __restrict__ P, int np_max, long long limit,
                    PurState* __restrict__ pur, int* __restrict__ err) {
  constexpr int G = (kLevels + L - 1) / L;   // level groups
  extern __shared__ __align__(1024) unsigned char pu_sm[];
  const int mi = list[blockIdx.x];
  if (st[mi].status != kActive) return;
  const DevMol mol = mols[mi];
  const int n = mol.nao, np = (n + 15) & ~15;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, q = warp & 3, g = warp >> 2;
  const bool issuer = warp == kPurSmallWarps;
  const int r = issuer ? 128 : q * 32 + lane;
  // behind the digits (the last one padded to the MMA's 128 rows)
  unsigned char* tail = pu_sm + (size_t)(kDigits - 1) * 2 * np_max * np_max + (size_t)256 * np_max;
  const uint32_t bar = pu_smem(tail);                                      // two, one per buffer
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tail + 16);
  long long* diag = reinterpret_cast<long long*>(tail + 32);               // 2 x 128
  const double* Fm = F + mol.mat0;

  // Interval of the eigenvalues: Gershgorin's circles with positive weights,
  // F_ii +- sum_j |F_ij| w_j / w_i, bound the spectrum for any w; two rounds of
  // power iteration bring w towards the best one, for each end its own.  Plain
  // circles (w = 1) make the interval two to three times as wide as the spectrum,
  // which costs two of about 22 steps.  In FP32, widened by far more than its
  // rounding: an FP64 instruction of a warp takes the SM 16 clocks.
  float flo = -3e37f, fhi = 3e37f;
  {
    float* w = reinterpret_cast<float*>(pu_sm);   // two buffers of (upper, lower) weights, where the digits come later
    float* fred = reinterpret_cast<float*>(diag);
    for (int i = tid; i < 256; i += kPurSmallThreads) w[i] = 1.0f;
    float dmin = 0.0f, dmax = 0.0f, eps = 0.0f;
    for (int pass = 0; pass < 3; ++pass) {
      __syncthreads();
      const float* wu = w + (pass & 1) * 256;
      const float* wl = wu + 128;
      float* nu = w + ((pass & 1) ^ 1) * 256;
      float bl = 3e37f, bu = -3e37f, d0 = 3e37f, d1 = -3e37f;
      for (int i = warp; i < n; i += kPurSmallWarps + 1) {
        float su = 0.0f, sl = 0.0f, d = 0.0f;
        bool big = false;
        for (int j = lane; j < n; j += 32) {
          const float f = pu_float(Fm[(long long)i * n + j]);
          big = big || !(fabsf(f) < 1e30f);
          if (j == i) d = f;
          else { su += fabsf(f) * wu[j]; sl += fabsf(f) * wl[j]; }
        }
        for (int o = 16; o > 0; o >>= 1) {
          su += __shfl_xor_sync(0xffffffffu, su, o);
          sl += __shfl_xor_sync(0xffffffffu, sl, o);
        }
        d = __shfl_sync(0xffffffffu, d, i & 31);
        if (__any_sync(0xffffffffu, big)) bl = -3e38f;
        d0 = fminf(d0, d);
        d1 = fmaxf(d1, d);
        bl = fminf(bl, d - sl / wl[i]);
        bu = fmaxf(bu, d + su / wu[i]);
        if (lane == 0) {   // products with dmin and dmax shifting the diagonal, known from pass 1 on
          nu[i] = su + (pass ? (d - dmin + eps) * wu[i] : 0.0f);
          nu[128 + i] = sl + (pass ? (dmax - d + eps) * wl[i] : 0.0f);
          if (!pass) w[512 + i] = d;
        }
      }
      if (lane == 0) { fred[warp] = bl; fred[32 + warp] = bu; fred[64 + warp] = d0; fred[96 + warp] = d1; }
      __syncthreads();
      const bool in = lane < kPurSmallWarps + 1;
      bl = in ? fred[lane] : 3e37f;
      bu = in ? fred[32 + lane] : -3e37f;
      d0 = in ? fred[64 + lane] : 3e37f;
      d1 = in ? fred[96 + lane] : -3e37f;
      for (int o = 16; o > 0; o >>= 1) {
        bl = fminf(bl, __shfl_xor_sync(0xffffffffu, bl, o));
        bu = fmaxf(bu, __shfl_xor_sync(0xffffffffu, bu, o));
        d0 = fminf(d0, __shfl_xor_sync(0xffffffffu, d0, o));
        d1 = fmaxf(d1, __shfl_xor_sync(0xffffffffu, d1, o));
      }
      flo = pass ? fmaxf(flo, bl) : bl;
      fhi = pass ? fminf(fhi, bu) : bu;
      if (pass) continue;
      if (!(bl > -1e37f && bu > bl)) break;
      dmin = d0;
      dmax = d1;
      eps = 0.02f * (bu - bl);
      for (int i = tid; i < n; i += kPurSmallThreads) {
        nu[i] += w[512 + i] - dmin + eps;
        nu[128 + i] += dmax - w[512 + i] + eps;
      }
    }
    __syncthreads();
  }
  for (int i = tid; i < 256; i += kPurSmallThreads) diag[i] = 0;
  int ncols = 32;
  while (ncols < 2 * L * np) ncols <<= 1;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 :: "r"(pu_smem(tmem_slot)), "r"(ncols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(bar));
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(bar + 8));
    asm volatile("fence.mbarrier_init.release.cluster;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = *tmem_slot;
  const bool usable = flo > -1e37f && fhi > flo;
  const float pad = 1e-4f * (fhi - flo) + 1e-5f * (fabsf(flo) + fabsf(fhi));
  const double scale = usable ? 36028797018963968.0 / ((double)(fhi - flo) + 2.0 * pad) : 0.0;   // 2^55 / width
  const double top = ((double)fhi + pad) * scale;

  long long x[H][16];
#pragma unroll
  for (int h = 0; h < H; ++h) {
    const int c0 = 64 * h + 16 * g;
#pragma unroll
    for (int c = 0; c < 16; ++c) x[h][c] = 0;
    if (q * 32 < n && c0 < n && !issuer) {
#pragma unroll
      for (int c = 0; c < 16; ++c) {
        const int col = c0 + c;
        if (r < n && col < n)
          x[h][c] = __double2ll_rn(fma(-Fm[(long long)max(r, col) * n + min(r, col)], scale, r == col ? top : 0.0));
      }
    }
  }

  const long long occ = (long long)mol.nocc * kTraceOne;
  const uint32_t slice = 2u * np * np, sbo = 16u * np;
  const uint32_t taddr = tmem + ((uint32_t)((q * 32) & 127) << 16);
  const bool work = !issuer && q * 32 < n;
  uint32_t parity[2] = {0, 0}, range = 0;
  bool ok = true, done = false;
  int first = -1;
  long long t0 = 0, t1 = 0;   // traces of X_k and X_{k-1}
  int k = 0;
  for (; usable; ++k) {
    // digits of X_k into shared memory, its diagonal
#pragma unroll
    for (int h = 0; h < H; ++h) {
      const int c0 = 64 * h + 16 * g;
      if (r < np && c0 < np) {
#pragma unroll
        for (int s = 0; s < 2; ++s) {
          uint4 dg[kDigits];
          pu_split8(&x[h][8 * s], dg);
          unsigned char* to = pu_sm + (r >> 3) * sbo + ((c0 >> 3) + s) * 128 + (r & 7) * 16;
#pragma unroll
          for (int d = 0; d < kDigits; ++d) *reinterpret_cast<uint4*>(to + d * slice) = dg[d];
        }
#pragma unroll
        for (int c = 0; c < 16; ++c)
          if (c0 + c == r) diag[(k & 1) * 128 + r] = x[h][c] >> kTraceShift;
      }
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;");
    if (!__syncthreads_and(ok)) { ok = false; break; }
    t1 = t0;
    t0 = 0;
    for (int i = lane; i < n; i += 32) t0 += diag[(k & 1) * 128 + i];
    for (int o = 16; o > 0; o >>= 1) t0 += __shfl_xor_sync(0xffffffffu, t0, o);
    if (first < 0 && k > 0 && pu_traced(t0, t1)) first = k - 1;
    const int op = pu_step(t0, t1, k, first, occ);
    if (op < 0) { done = pu_counted(t0, occ); break; }
    if (k == kPurSmallSteps) break;
    if (issuer) {
      asm volatile("tcgen05.fence::after_thread_sync;");
      const uint32_t lo = pu_desc_lo(pu_smem(pu_sm));
#pragma unroll
      for (int j = 0; j < G; ++j) {
        if (j >= 2) {
          pu_drained(j - 2, true);
          asm volatile("tcgen05.fence::after_thread_sync;");
        }
        if (lane == 0) {
          const uint32_t to = tmem + (j & 1) * L * np, hi = pu_desc_hi(sbo);
          if (j == 0) pu_level_group<L, 0>(to, lo, slice, hi, np);
          else if (j == 1) pu_level_group<L, 1>(to, lo, slice, hi, np);
          else if (j == 2) pu_level_group<L, (G > 2 ? 2 : 0)>(to, lo, slice, hi, np);
          else pu_level_group<L, (G > 3 ? 3 : 0)>(to, lo, slice, hi, np);
          pu_commit(bar + 8 * (j & 1));
        }
        __syncwarp();
      }
    } else {
      const int sgn = op ? 1 : -1;
#pragma unroll
      for (int h = 0; h < H; ++h)
#pragma unroll
        for (int c = 0; c < 16; ++c) x[h][c] = op ? 0 : 2 * x[h][c];
#pragma unroll
      for (int j = 0; j < G; ++j) {
        if (!pu_wait(bar + 8 * (j & 1), parity[j & 1], limit)) {
          ok = false;
          pu_drain(bar + 8 * (j & 1), parity[j & 1]);
        }
        parity[j & 1] ^= 1;
        asm volatile("tcgen05.fence::after_thread_sync;");
        if (work) {
          if (j == 0) pu_group<H, L, 0>(taddr, np, g, sgn, x, range);
          else if (j == 1) pu_group<H, L, 1>(taddr, np, g, sgn, x, range);
          else if (j == 2) pu_group<H, L, (G > 2 ? 2 : 0)>(taddr, np, g, sgn, x, range);
          else pu_group<H, L, (G > 3 ? 3 : 0)>(taddr, np, g, sgn, x, range);
        }
        asm volatile("tcgen05.fence::before_thread_sync;");
        if (j + 2 < G) pu_drained(j, false);
      }
      // rows past the basis came from whatever lies behind the digits
      if (r >= n) {
        range = 0;
#pragma unroll
        for (int h = 0; h < H; ++h)
#pragma unroll
          for (int c = 0; c < 16; ++c) x[h][c] = 0;
      }
    }
  }
  done = __syncthreads_and(ok && done && pu_in_range(range));
  if (done && !issuer) {
    double* Pm = P + mol.mat0;
#pragma unroll
    for (int h = 0; h < H; ++h)
#pragma unroll
      for (int c = 0; c < 16; ++c) {
        const int col = 64 * h + 16 * g + c;
        if (r < n && col < n) Pm[(long long)r * n + col] = pu_density(x[h][c]);
      }
  }
  if (tid == 0) {
    if (!ok) atomicExch(err, 1);
    st[mi].flags = done ? 0 : kNeedEigen;
    atomicAdd(&pur[mi].steps, (unsigned long long)k);
  }
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(ncols));
}

// ---------------------------------------------------------------------------
// N > 128: one launch per step over the 128 x TN tiles of every molecule's
// upper triangle, TN = 64, or 32 where the wider tiles would leave half of the
// SMs without one (a single molecule below N ~ 900, see Batch::build_jobs): half
// the work on a CTA's path for twice the CTAs ((H2O)33: 22.0 -> 17.7 ms, (H2O)101:
// 55.6 -> 43.6 ms; for 256 (H2O)32, where every SM has wide tiles, narrow ones cost
// 87 -> 95 ms).  The sums are exact, so the choice changes no bit.  The digit
// matrices live in global memory (L2) in the layout
// of the MMA operands, [K chunk of 32][8-row group][4 k-blocks][8 rows][8 k], so a
// tile's rows of one K chunk are one contiguous bulk copy per digit; two
// buffers alternate between steps.  They share the eigensolver's scratch
// matrices: two digits per N x N doubles (Np = N rounded up to 32 has
// Np^2 <= 2 N^2 from N = 79 on).
// ---------------------------------------------------------------------------
constexpr int kPurTileThreads = 512;
constexpr int kTileM = 128, kChunkK = 32, kStages = 2;
constexpr uint32_t kStageA = kTileM * kChunkK * 2;        // bytes per digit
constexpr uint32_t stage_bytes(int tn) { return kDigits * (kStageA + (uint32_t)tn * kChunkK * 2); }
constexpr int kSegChunks = 16;                            // K = 512: see pu_int
constexpr int kXPitch = kTileM + 1;                       // transposed tile, 8-byte elements: no bank conflicts either way
constexpr size_t tile_smem(int tn) { return kStages * stage_bytes(tn) + 256; }

__device__ __forceinline__ unsigned char* pu_plane(const PurScratch& ws, const DevMol& mol, int buf, int d) {
  const int s = buf * kDigits + d;
  const long long n2 = ((long long)mol.nao * mol.nao + 31) / 32 * 32;
  return reinterpret_cast<unsigned char*>(ws.m[s >> 1] + mol.mat0) + (s & 1) * (n2 * 4);
}
__device__ __forceinline__ int pu_np(int n) { return (n + 31) & ~31; }
// byte offset of (row r, k-block k / 8) in a plane; k a multiple of 8
__device__ __forceinline__ size_t pu_at(int np, int r, int k) {
  return (size_t)(k >> 5) * (64 * (size_t)np) + (size_t)(r >> 3) * 512 + ((k >> 3) & 3) * 128 + (r & 7) * 16;
}

__device__ __forceinline__ unsigned long long pu_key(double v) {   // order-preserving
  const unsigned long long b = (unsigned long long)__double_as_longlong(v);
  return (b >> 63) ? ~b : b | 0x8000000000000000ull;
}
__device__ __forceinline__ double pu_unkey(unsigned long long k) {
  return __longlong_as_double((long long)((k >> 63) ? k & 0x7fffffffffffffffull : ~k));
}

// Gershgorin interval of every molecule: a warp per row
__global__ void __launch_bounds__(256)
purify_bounds_kernel(const DevMol* __restrict__ mols, const int* __restrict__ list, const MolState* __restrict__ st,
                     const double* __restrict__ F, PurState* __restrict__ pur) {
  const int mi = list[blockIdx.y];
  if (st[mi].status != kActive) return;
  const DevMol mol = mols[mi];
  const int n = mol.nao, lane = threadIdx.x & 31;
  const int i = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (i >= n) return;
  const double* row = F + mol.mat0 + (long long)i * n;
  double s = 0.0;
  for (int j = lane; j < n; j += 32)
    if (j != i) s += fabs(row[j]);
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) {
    const double d = row[i];
    const bool bad = !(s + fabs(d) < 1e290);
    atomicMin(&pur[mi].lo, pu_key(bad ? -1e300 : d - s));
    if (!bad) atomicMax(&pur[mi].hi, pu_key(d + s));
  }
}

__device__ __forceinline__ bool pu_interval(const PurState& s, double* lo, double* hi) {
  *lo = pu_unkey(s.lo);
  *hi = pu_unkey(s.hi);
  return *lo > -1e299 && *hi > *lo;
}

// X_0 and its digits: a thread per row and eight columns
__global__ void __launch_bounds__(256)
purify_init_kernel(const DevMol* __restrict__ mols, const int* __restrict__ list, const MolState* __restrict__ st,
                   const double* __restrict__ F, PurState* __restrict__ pur, PurScratch ws) {
  const int mi = list[blockIdx.y];
  if (st[mi].status != kActive) return;
  const DevMol mol = mols[mi];
  const int n = mol.nao, np = pu_np(n), kb = np >> 3;
  double lo, hi;
  if (!pu_interval(pur[mi], &lo, &hi)) return;
  const double scale = 1.0 / (hi - lo);
  const double* Fm = F + mol.mat0;
  // eight consecutive rows (the rows of a core matrix) by consecutive threads
  for (long long e = (long long)blockIdx.x * 256 + threadIdx.x; e < (long long)np * kb; e += (long long)gridDim.x * 256) {
    const int r = (int)(e / (8 * kb)) * 8 + (int)(e & 7), c0 = (int)((e >> 3) % kb) * 8;
    long long x[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const int col = c0 + c;
      x[c] = 0;
      if (r < n && col < n) {
        const double f = Fm[(long long)max(r, col) * n + min(r, col)];
        x[c] = pu_fixed(((r == col ? hi : 0.0) - f) * scale);
        if (r == col)
          atomicAdd(reinterpret_cast<unsigned long long*>(&pur[mi].trace[0]),
                    (unsigned long long)(x[c] >> kTraceShift));
      }
    }
    uint4 dg[kDigits];
    pu_split8(x, dg);
    const size_t at = pu_at(np, r, c0);
#pragma unroll
    for (int d = 0; d < kDigits; ++d) *reinterpret_cast<uint4*>(pu_plane(ws, mol, 0, d) + at) = dg[d];
  }
}

// first step whose tr(X - X^2) was below the tolerance, from T_0 .. T_k (k < 64)
__device__ __forceinline__ int pu_first(const long long* T, int k) {
  const int lane = threadIdx.x & 31;
  const unsigned a = __ballot_sync(0xffffffffu, lane < k && pu_traced(T[lane + 1], T[lane]));
  const unsigned b = __ballot_sync(0xffffffffu, lane + 32 < k && pu_traced(T[lane + 33], T[lane + 32]));
  return a ? __ffs(a) - 1 : (b ? __ffs(b) + 31 : -1);
}

// A tile of step k failed: the molecule's X is lost.  The steps after k learn it from
// the trace that they read anyway (a flag of its own cost them 0.3 %; written during
// the step, it would also let the threads of one CTA decide differently).
constexpr long long kTraceFailed = 1LL << 60;   // traces are below N 2^43
__device__ __forceinline__ void pu_failed(PurState& s, int k) {
  atomicExch(&s.bad, 1);
  atomicExch(reinterpret_cast<unsigned long long*>(&s.trace[k + 1]), (unsigned long long)(2 * kTraceFailed));
}

// One step of the molecules that still need one.  tiles: (molecule, row block,
// column block, 0).  Warp 0 copies, warp 1 issues the MMAs, all sixteen
// recombine.
template <int TN>
__global__ void __launch_bounds__(kPurTileThreads, 1)
purify_step_kernel(const DevMol* __restrict__ mols, const int4* __restrict__ tiles, const MolState* __restrict__ st,
                   PurState* __restrict__ pur, PurScratch ws, int k, long long limit, int* __restrict__ err) {
  constexpr int kCW = TN / 4, kGroups = kCW / 8;   // columns of a warp, groups of eight of them
  constexpr uint32_t kStageBytes = stage_bytes(TN);
  constexpr int kTmem = kLevels * TN;
  extern __shared__ __align__(1024) unsigned char pu_sm[];
  // what no step changes is read while the previous step still runs (programmatic
  // dependent launch); every CTA waits for it before it looks at anything else,
  // or returns, so that the next step's wait covers all earlier ones
  const int4 tile = tiles[blockIdx.x];
  const int mi = tile.x;
  const DevMol mol = mols[mi];
  cudaTriggerProgrammaticLaunchCompletion();
  cudaGridDependencySynchronize();
  // every load before the first branch: one trip to L2 instead of three
  const int status = st[mi].status;
  const long long t0 = pur[mi].trace[k], t1 = pur[mi].trace[k > 0 ? k - 1 : 0];
  double lo, hi;
  const bool usable = pu_interval(pur[mi], &lo, &hi);
  const int n = mol.nao, np = pu_np(n), first = pu_first(pur[mi].trace, k);
  const long long occ = (long long)mol.nocc * kTraceOne;
  const int op = pu_step(t0, t1, k, first, occ);   // the same in every CTA of the molecule
  const bool failed = t0 >= kTraceFailed;
  if (status != kActive || !usable || op < 0 || failed) {
    if (failed && threadIdx.x == 0) pur[mi].trace[k + 1] = 2 * kTraceFailed;
    return;
  }
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int r0 = tile.y * kTileM, c0 = tile.z * TN;
  const int rows = min(kTileM, np - r0), cols = min(TN, np - c0);
  const int chunks = np / kChunkK;
  unsigned char* tail = pu_sm + kStages * kStageBytes;
  const uint32_t full = pu_smem(tail), empty = full + 8 * kStages, last = empty + 8 * kStages;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tail + 64);
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 :: "r"(pu_smem(tmem_slot)), "r"(kTmem));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 0) {
    for (int s = 0; s < kStages; ++s) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(full + 8 * s));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(empty + 8 * s));
    }
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(last));
    asm volatile("fence.mbarrier_init.release.cluster;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = *tmem_slot;
  const uint32_t sm = pu_smem(pu_sm);
  const int buf = k & 1;
  const int q = warp & 3, r = r0 + q * 32 + lane;
  const int cw = (warp >> 2) * kCW;   // this warp's first column of the tile
  const uint32_t taddr = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)cw;
  const int groups = q * 32 < rows ? max(0, min(kGroups, (cols - cw) >> 3)) : 0;   // of eight columns
  long long v[kGroups][8];
#pragma unroll
  for (int s = 0; s < kGroups; ++s)
#pragma unroll
    for (int i = 0; i < 8; ++i) v[s][i] = 0;
  uint32_t range = 0;
  bool ok = true;
  int issued = 0;   // K chunks whose copies (thread 0) or MMAs (thread 32) this thread has issued
  // K in segments whose digit sums pu_int covers
  for (int seg = 0, cb = 0; cb < chunks && ok; ++seg, cb += kSegChunks) {
    const int ce = min(chunks, cb + kSegChunks);
    if (warp == 0 && lane == 0) {
      const uint32_t ba = (uint32_t)rows * kChunkK * 2, bb = (uint32_t)cols * kChunkK * 2;
      for (int c = cb; c < ce; ++c) {
        const int s = c % kStages;
        if (c >= kStages && !pu_wait(empty + 8 * s, ((c / kStages) - 1) & 1, limit)) { ok = false; break; }
        issued = c + 1;
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;"
                     :: "r"(full + 8 * s), "r"((ba + bb) * kDigits) : "memory");
        for (int d = 0; d < kDigits; ++d) {
          const unsigned char* p = pu_plane(ws, mol, buf, d) + (size_t)c * (64 * (size_t)np);
          const uint32_t to = sm + s * kStageBytes;
          asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                       :: "r"(to + d * kStageA), "l"(p + (size_t)r0 * 64), "r"(ba), "r"(full + 8 * s) : "memory");
          asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                       :: "r"(to + kDigits * kStageA + d * bb), "l"(p + (size_t)c0 * 64), "r"(bb), "r"(full + 8 * s)
                       : "memory");
        }
      }
    } else if (warp == 1 && lane == 0) {
      asm volatile("tcgen05.fence::after_thread_sync;");
      for (int c = cb; c < ce; ++c) {
        const int s = c % kStages;
        if (!pu_wait(full + 8 * s, (c / kStages) & 1, limit)) { ok = false; break; }
        asm volatile("tcgen05.fence::after_thread_sync;");
        const uint32_t base = pu_desc_lo(sm + s * kStageBytes);
        const uint32_t bb = base + (kDigits * kStageA >> 4), sb = (uint32_t)cols * kChunkK * 2;
        if (TN == 64 && cols == TN)
          pu_products<4, 0, kLevels>(tmem, base, kStageA, bb, sb, pu_desc_hi(512), cols, kChunkK / 16, c == cb);
        else
          pu_products<7, 0, kLevels>(tmem, base, kStageA, bb, sb, pu_desc_hi(512), cols, kChunkK / 16, c == cb);
        pu_commit(empty + 8 * s);
        issued = c + 1;
      }
      if (ok) pu_commit(last);
    }
    __syncwarp();
    ok = pu_wait(last, seg & 1, limit) && ok;
    asm volatile("tcgen05.fence::after_thread_sync;");
    ok = __syncthreads_and(ok);
    if (ok) {
#pragma unroll
      for (int s = 0; s < kGroups; ++s)
        if (s < groups) {
          pu_levels8<0, 4>(taddr + 8 * s, cols, 1, v[s], range);
          pu_levels8<4, 4>(taddr + 4 * cols + 8 * s, cols, 1, v[s], range);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
  }
  if (!ok) {
    // a wait ran out: this tile of X_{k+1} is missing, the molecule goes to the
    // eigensolver
    for (int c = max(0, issued - kStages); c < issued; ++c)
      pu_drain((warp == 0 ? full : empty) + 8 * (c % kStages), (c / kStages) & 1);
    if (tid == 0) {
      pu_failed(pur[mi], k);
      atomicExch(err, 1);
    }
  } else {
    // X_{k+1}: row r, the digits of eight columns at a time
    const bool mirror = tile.z >= (kTileM / TN) * (tile.y + 1);   // the transposed block is no tile of its own
    long long* xt = reinterpret_cast<long long*>(pu_sm);   // the operand stages are free now
    // rows past the padded basis are whatever the stage held before
    if (r < np && !pu_in_range(range)) pu_failed(pur[mi], k);
    long long tr = 0;
#pragma unroll
    for (int s = 0; s < kGroups; ++s) {
      if (s >= groups) continue;
      const int cl = cw + 8 * s, c = c0 + cl;
      const size_t at = pu_at(np, r, c);
      uint4 dg[kDigits];
      if (!op) {
        long long x[8];
#pragma unroll
        for (int d = 0; d < kDigits; ++d) dg[d] = *reinterpret_cast<const uint4*>(pu_plane(ws, mol, buf, d) + at);
        pu_join8(dg, x);
#pragma unroll
        for (int i = 0; i < 8; ++i) v[s][i] = 2 * x[i] - v[s][i];
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        if (c + i == r) tr += v[s][i] >> kTraceShift;
        if (mirror) xt[(cl + i) * kXPitch + q * 32 + lane] = v[s][i];
      }
      pu_split8(v[s], dg);
#pragma unroll
      for (int d = 0; d < kDigits; ++d) *reinterpret_cast<uint4*>(pu_plane(ws, mol, buf ^ 1, d) + at) = dg[d];
    }
    if (tr != 0) atomicAdd(reinterpret_cast<unsigned long long*>(&pur[mi].trace[k + 1]), (unsigned long long)tr);
    if (mirror) {
      __syncthreads();
      // rows c0 + j, columns r0 + 8 t ..: eight consecutive rows by consecutive threads
      for (int e = tid; e < cols * (rows >> 3); e += kPurTileThreads) {
        const int t = e / cols, j = e - t * cols;
        uint4 dg[kDigits];
        long long x[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) x[i] = xt[j * kXPitch + 8 * t + i];
        pu_split8(x, dg);
        const size_t at = pu_at(np, c0 + j, r0 + 8 * t);
#pragma unroll
        for (int d = 0; d < kDigits; ++d) *reinterpret_cast<uint4*>(pu_plane(ws, mol, buf ^ 1, d) + at) = dg[d];
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(kTmem));
}

// P = 2 X of the molecules whose iteration ended; the others are flagged
__global__ void __launch_bounds__(256)
purify_store_kernel(const DevMol* __restrict__ mols, const int* __restrict__ list, MolState* __restrict__ st,
                    PurState* __restrict__ pur, PurScratch ws, int steps, double* __restrict__ P) {
  const int mi = list[blockIdx.y];
  if (st[mi].status != kActive) return;
  const DevMol mol = mols[mi];
  const int n = mol.nao, np = pu_np(n), kb = np >> 3;
  double lo, hi;
  const int first = pu_first(pur[mi].trace, steps);
  const bool done = !pur[mi].bad && pu_interval(pur[mi], &lo, &hi) && first >= 0 && first + 3 <= steps &&
                    pu_counted(pur[mi].trace[first + 3], (long long)mol.nocc * kTraceOne);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    st[mi].flags = done ? 0 : kNeedEigen;
    atomicAdd(&pur[mi].steps, (unsigned long long)(first >= 0 && first + 3 < steps ? first + 3 : steps));
  }
  if (!done) return;
  const int buf = (first + 3) & 1;
  double* Pm = P + mol.mat0;
  for (long long e = (long long)blockIdx.x * 256 + threadIdx.x; e < (long long)n * kb; e += (long long)gridDim.x * 256) {
    const int r = (int)(e / kb), c0 = (int)(e % kb) * 8;
    uint4 dg[kDigits];
    const size_t at = pu_at(np, r, c0);
#pragma unroll
    for (int d = 0; d < kDigits; ++d) dg[d] = *reinterpret_cast<const uint4*>(pu_plane(ws, mol, buf, d) + at);
    long long x[8];
    pu_join8(dg, x);
#pragma unroll
    for (int c = 0; c < 8; ++c)
      if (c0 + c < n) Pm[(long long)r * n + c0 + c] = pu_density(x[c]);
  }
}

// traces and bounds of the next call
__global__ void purify_reset_kernel(const int* __restrict__ list, PurState* __restrict__ pur) {
  PurState& s = pur[list[blockIdx.x]];
  for (int i = threadIdx.x; i <= kPurBigSteps; i += blockDim.x) s.trace[i] = 0;
  if (threadIdx.x == 0) { s.lo = ~0ull; s.hi = 0ull; s.bad = 0; }
}

// ---------------------------------------------------------------------------
static size_t small_smem(int np) {
  return (size_t)(kDigits - 1) * 2 * np * np + (size_t)256 * np + 32 + 2 * 128 * 8;
}

void purify_prepare() {
  static std::once_flag once;
  std::call_once(once, [] {
    cudaFuncSetAttribute(purify_small_kernel<1, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)small_smem(64));
    cudaFuncSetAttribute(purify_small_kernel<2, 3>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)small_smem(80));
    cudaFuncSetAttribute(purify_small_kernel<2, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)small_smem(128));
    cudaFuncSetAttribute(purify_step_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tile_smem(64));
    cudaFuncSetAttribute(purify_step_kernel<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tile_smem(32));
  });
}

int purify_tiles(int mol, int n, int tn, int4* out) {
  const int np = (n + 31) / 32 * 32, nr = (np + kTileM - 1) / kTileM, nc = (np + tn - 1) / tn;
  int t = 0;
  for (int i = 0; i < nr; ++i)
    for (int j = kTileM / tn * i; j < nc; ++j, ++t)
      if (out) out[t] = make_int4(mol, i, j, 0);
  return t;
}

// 34 digit products, M = 128 rows whatever the basis
double purify_step_flops(int n, int tn) {
  if (n <= kPurSmallMaxN) {
    const double np = (n + 15) / 16 * 16;
    return 34.0 * 2.0 * kTileM * np * np;
  }
  const int np = (n + 31) / 32 * 32;
  double cols = 0.0;
  for (int i = 0; i * kTileM < np; ++i)
    for (int j = kTileM / tn * i; j * tn < np; ++j) cols += std::min(tn, np - j * tn);
  return 34.0 * 2.0 * kTileM * cols * np;
}

void launch_purify_small(const DevMol* mols, const int* list, int nlist, int max_n, MolState* st, const double* F,
                         double* P, PurState* pur, int* err, long long limit, cudaStream_t s) {
  if (nlist <= 0) return;
  purify_prepare();
  const int np = (max_n + 15) / 16 * 16;
  const size_t sm = small_smem(np);
  // levels per group: two buffers of L x np of the 512 columns of tensor memory
  if (np <= 64) purify_small_kernel<1, 4><<<nlist, kPurSmallThreads, sm, s>>>(mols, list, st, F, P, np, limit, pur, err);
  else if (np <= 80) purify_small_kernel<2, 3><<<nlist, kPurSmallThreads, sm, s>>>(mols, list, st, F, P, np, limit, pur, err);
  else purify_small_kernel<2, 2><<<nlist, kPurSmallThreads, sm, s>>>(mols, list, st, F, P, np, limit, pur, err);
}

int launch_purify_big(const DevMol* mols, const int* list, int nlist, int max_n, const int4* tiles, int ntiles, int tn,
                      MolState* st, const double* F, double* P, PurState* pur, const PurScratch& ws, int steps,
                      bool alone, int* err, long long limit, cudaStream_t s) {
  if (nlist <= 0) return 0;
  purify_prepare();
  const int np = (max_n + 31) / 32 * 32;
  const int blocks = std::max(1, std::min(512, np * (np / 8) / 512));
  purify_reset_kernel<<<nlist, 64, 0, s>>>(list, pur);
  purify_bounds_kernel<<<dim3((max_n + 7) / 8, nlist), 256, 0, s>>>(mols, list, st, F, pur);
  purify_init_kernel<<<dim3(blocks, nlist), 256, 0, s>>>(mols, list, st, F, pur, ws);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ntiles);
  cfg.blockDim = dim3(kPurTileThreads);
  cfg.dynamicSmemBytes = tile_smem(tn);
  cfg.stream = s;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  for (int k = 0; k < steps; ++k) {
    // CTAs launched ahead hold an SM while they wait: only where no other stream
    // has work for it (a server's burst took 104 ms without and 119 with them)
    cfg.numAttrs = alone && k > 0 ? 1 : 0;
    cudaLaunchKernelEx(&cfg, tn == 64 ? purify_step_kernel<64> : purify_step_kernel<32>, mols, tiles,
                       (const MolState*)st, pur, ws, k, limit, err);
  }
  purify_store_kernel<<<dim3(blocks, nlist), 256, 0, s>>>(mols, list, st, pur, ws, steps, P);
  return steps + 4;
}

}  // namespace nddo
