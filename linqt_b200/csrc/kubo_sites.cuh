// The weights of Kubo_solver_FFT's transforms, for the site transforms (kubo_fft.cu) and the sums from the
// moment table (kubo_table.cu).
#pragma once

#include "internal.cuh"

namespace linqt {

// Jackson-damped amplitude a_m (include/Kubo_solver_FFT.hpp:99-107)
__device__ __forceinline__ double site_amplitude(int m, int M) {
  const double g = 1 / (M + 1.0) *
                   ((M - m + 1.0) * cos(M_PI * m / (M + 1.0)) + sin(M_PI * m / (M + 1.0)) / tan(M_PI / (M + 1.0)));
  return (2 - (m == 0)) * g;
}
// prefactor pf_m = a_m e^(i pi m / (2 nump)) (src/Bastin_FFTs.cpp:20-21)
__device__ __forceinline__ double2 site_prefactor(int m, int M, int nump) {
  const double amp = site_amplitude(m, M);
  double sn, cs;
  sincos(M_PI * m / (2.0 * nump), &sn, &cs);
  return make_double2(amp * cs, amp * sn);
}
// root of unity of the direct transforms
__device__ __forceinline__ double2 site_root(int t, int nump) {
  double sn, cs;
  sincospi(2.0 * t / nump, &sn, &cs);
  return make_double2(cs, sn);
}

// The buffers of both: pf [M], and tw [nump] where the transforms are direct (else NULL).
struct SiteTables {
  double2 *pf, *tw;
};
SiteTables site_tables(Session *s, int M, int nump, int formula);

}  // namespace linqt
