// Acceptance of a contraction in residues (mu_rns.cu), which gathers the statistics; mu_gemm.cu
// judges by them and commits the sum or the FP64 kernel's.
#pragma once

#include "internal.cuh"

namespace linqt {

constexpr int kMaxParts = 8;  // parts of a row chunk (k_residues)

// What the acceptance of a contraction is judged by, zero between contractions (the last block of
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
// The error allowed, of the sum's largest value: 8 units of FP64 rounding.  The estimate for random
// states is a tenth of it and less, and at most about one unit in a table that is noise alone
// (operators whose products average out).
constexpr double kAccept = 8.8817841970012523e-16;  // 2^-50

__device__ __forceinline__ void raise_to(unsigned long long *a, double v) {
  atomicMax(a, (unsigned long long)__double_as_longlong(v));
}

// Whether the sum may be off by more than kAccept of its largest value `top`.  A value of a row is
// off by up to half its unit, as if at random, so a sum with the rows' units ua, ub and norms |a|,
// |b| by (ua |b| (+) ub |a|) / sqrt(6), (+) and the chunks in quadrature; the largest of the rows
// stand for all.  By one block; not finite: rejected.
__device__ inline bool judge(const RnsSide *side, int nchunk, double top) {
  __shared__ double red[256];
  double big = 0.0, sum = 0.0;
  for (int pass = 0; pass < 2; ++pass) {
    for (int c = threadIdx.x; c < nchunk; c += blockDim.x) {
      double u[2], n[2];
      for (int z = 0; z < 2; ++z) {
        const RnsSide &sd = side[2 * c + z];
        double t = 0.0;
        for (int p = 0; p < kMaxParts; ++p) t += __longlong_as_double((long long)__ldcg(&sd.sq[p]));
        u[z] = __longlong_as_double((long long)__ldcg(&sd.unit));
        n[z] = sqrt(t);
      }
      double x = u[0] * n[1], y = u[1] * n[0];
      if (!(x < INFINITY && y < INFINITY)) x = y = INFINITY;
      big = fmax(big, fmax(x, y));
      if (pass) sum += (x / red[0]) * (x / red[0]) + (y / red[0]) * (y / red[0]);
    }
    if (pass) {
      big = red[0];
      __syncthreads();
    }
    red[threadIdx.x] = pass ? sum : big;
    __syncthreads();
    for (int o = blockDim.x / 2; o > 0; o >>= 1) {
      if ((int)threadIdx.x < o)
        red[threadIdx.x] = pass ? red[threadIdx.x] + red[threadIdx.x + o] : fmax(red[threadIdx.x], red[threadIdx.x + o]);
      __syncthreads();
    }
    if (pass == 0 && red[0] == 0.0) return false;  // a side is zero
    if (pass == 0 && red[0] == INFINITY) return true;
  }
  return !(big * sqrt(red[0] / 6.0) <= kAccept * top);
}

}  // namespace linqt
