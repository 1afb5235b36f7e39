// Acceptance of a contraction in residues (mu_rns.cu), which gathers the statistics; mu_gemm.cu
// checks by them and commits the sum or the FP64 kernel's.
#pragma once

#include "internal.cuh"

namespace linqt {

constexpr int kMaxParts = 8;  // parts of a row chunk (k_residues)

// What the acceptance of a contraction is decided by, zero between contractions (the last block of
// k_commit clears it).  Maxima are taken on the bits of non-negative doubles, whose order is
// that of the numbers: the same in any order of arrival.
struct RnsSide {
  unsigned long long unit;             // largest unit 2^(e - 53) of a row
  unsigned long long sq[kMaxParts];    // largest sum of squares of a row's part
};
struct RnsStats {
  unsigned long long top;              // largest |re| or |im| of the sum
  unsigned done;                       // blocks of k_commit
  int rejected;
};
// The error allowed, of the sum's largest value.  Moments: 8 units of FP64 rounding.  Tables for sigma: one,
// since the Bastin integrand multiplies a table's errors by 1e6 (1024 energies, band edge) and the
// bar of 1e-10 is that of a table rounded to FP64.  The estimate for random states is 5 / sqrt(K)
// units, and about one in a table that is noise alone (operators whose products average out).
constexpr double kAcceptMoments = 8.8817841970012523e-16;  // 2^-50
constexpr double kAcceptSigma = 1.1102230246251565e-16;    // 2^-53

__device__ __forceinline__ void raise_to(unsigned long long *a, double v) {
  atomicMax(a, (unsigned long long)__double_as_longlong(v));
}

// Whether the sum may be off by more than `accept` of its largest value `top`.  A value of a row is
// off by up to half its unit, as if at random, so a sum with the rows' units ua, ub and norms |a|,
// |b| by (ua |b| (+) ub |a|) / sqrt(6), (+) and the chunks in quadrature; the largest of the rows
// stand for all.  By one warp of a CTA, through L1: with every warp of a few hundred CTAs reading these few
// lines from L2, their one slice took 10 to 20 us.  Not finite: rejected.
__device__ __forceinline__ bool rns_rejected(const RnsSide *side, int nchunk, double top, double accept) {
  const double allowed = accept * top;
  double sum = 0.0;
  for (int c = threadIdx.x & 31; c < nchunk; c += 32) {
    double u[2], n[2];
#pragma unroll
    for (int z = 0; z < 2; ++z) {
      const RnsSide &sd = side[2 * c + z];
      double t = 0.0;
#pragma unroll
      for (int p = 0; p < kMaxParts; ++p) t += __longlong_as_double((long long)sd.sq[p]);
      u[z] = __longlong_as_double((long long)sd.unit);
      n[z] = sqrt(t);
    }
    const double x = u[0] * n[1], y = u[1] * n[0];
    if (x != 0.0) sum += (x / allowed) * (x / allowed);
    if (y != 0.0) sum += (y / allowed) * (y / allowed);
  }
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  return !(sum <= 6.0 && top < INFINITY);
}

}  // namespace linqt
