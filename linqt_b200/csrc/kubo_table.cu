// Kubo_solver_FFT's site sums from the moment table.
//
// The reference transforms every site's Chebyshev vectors and sums products of the transforms
// over the sites (kubo_fft.cu).  With C_m = a_m cos(m phi), S_m = a_m sin(m phi), a_m the
// Jackson-damped amplitude, phi the angle of a frequency folded into (0, pi], and U the raw
// table sum_sites conj(bra_m) ket_m', the two sums that reach sigma are bilinear forms of U:
//
//   Bastin:     p = 2 sum_m C_m Re Z(m),   w = -2 sum_m C_m Im D(m)
//   Greenwood:  p =   sum_m C_m sum_m' Re U_s(m, m') C_m'
//   Z(m) = sum_m' U_s(m, m') a_m' e^(i m' phi),   D(m) = sum_m' m' U_s(m, m') a_m' e^(i m' phi)
//
// (src/Bastin_FFTs.cpp:128-163 and src/Greenwood_FFTs.cpp:252-257 written out; U_s = (U + U^H)/2;
// only Re p and Im w are used, src/Kubo_solver_FFT_postProcess.cpp:192).  The Bastin integrand
// divides by (1 - E^2)^2, which multiplies errors near the band edges by 1e11 at 1024
// energies: a table rounded to FP64 leaves sigma at 3e-11 to 1e-10 of its maximum.  So U comes
// in double-double from the residue contraction (mu_rns.cu) and everything up to p and w
// stays in double-double; sigma then differs from the site-by-site transforms by what those
// round (1e-13).
//
// Work: with m' = a + A b and A a divisor of 2 n (n energies), e^(i A b phi_i) depends on i
// mod P = 2 n / A only, so each row takes n (2 M / A) + n A terms in two steps instead of
// n M.  The cost no longer grows with the number of sites.  Measured: graphene 128 x 128, R = 8,
// M = 512, 1024 energies: 8.60 ms of site transforms -> 0.26 ms; Greenwood of 15360 sites at 1000
// energies (M = 300): 9.5 ms of direct transforms -> 0.39 ms with the contraction.
#include <cmath>

#include "dd.cuh"
#include "internal.cuh"
#include "kubo_sites.cuh"

namespace linqt {

namespace {

// All that depends on the sizes alone, in one launch: cos(pi q / (2 n)) for q < 4 n in double-double
// (Taylor series of sine and cosine on [0, pi/4]), the amplitudes, and the weights of the site
// transforms, which take the blocks whose table is rejected.
__global__ void k_table_setup(int n, int M, double2 *__restrict__ tab, double *__restrict__ amp,
                              double2 *__restrict__ pf, double2 *__restrict__ tw) {
  const int t0 = blockIdx.x * blockDim.x + threadIdx.x, st = gridDim.x * blockDim.x;
  for (int m = t0; m < M; m += st) {
    amp[m] = site_amplitude(m, M);
    pf[m] = site_prefactor(m, M, n);
  }
  for (int t = t0; tw && t < n; t += st) tw[t] = site_root(t, n);
  for (int q = t0; q < 4 * n; q += st) {
    const int quad = q / n;
    int r = q % n;
    const bool swap = 2 * r > n;  // use the complement
    if (swap) r = n - r;
    const double2 pi = make_double2(3.141592653589793116, 1.2246467991473532072e-16);
    const double2 x = dd_div(dd_scale(pi, (double)r), 2.0 * n);
    const double2 x2 = dd_neg(dd_mul(x, x));
    double2 c = make_double2(1.0, 0.0), s = x, tc = c, ts = x;
    for (int k = 1; k <= 14; ++k) {
      tc = dd_div(dd_mul(tc, x2), (2.0 * k - 1.0) * (2.0 * k));
      ts = dd_div(dd_mul(ts, x2), (2.0 * k) * (2.0 * k + 1.0));
      c = dd_add(c, tc);
      s = dd_add(s, ts);
    }
    if (swap) {
      const double2 t = c;
      c = s;
      s = t;
    }
    tab[q] = quad == 0 ? c : quad == 1 ? dd_neg(s) : quad == 2 ? dd_neg(c) : s;
  }
}

// h(m, m') = a_m' U_s(m, m') as two dd numbers (re, im)
__global__ void k_table_coef(const double2 *__restrict__ hi, const double2 *__restrict__ lo,
                             const double *__restrict__ amp, int M, double2 *__restrict__ re,
                             double2 *__restrict__ im) {
  const long tot = (long)M * M;
  for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < tot; t += (long)gridDim.x * blockDim.x) {
    const int i = (int)(t / M), j = (int)(t % M);
    const size_t tt = (size_t)j * M + i;
    const double f = 0.5 * amp[j];
    re[t] = dd_scale(dd_add(make_double2(hi[t].x, lo[t].x), make_double2(hi[tt].x, lo[tt].x)), f);
    im[t] = dd_scale(dd_add(make_double2(hi[t].y, lo[t].y), make_double2(-hi[tt].y, -lo[tt].y)), f);
  }
}

constexpr int kTabThreads = 256;
constexpr int kTabItems = 4;         // outputs per thread at most
constexpr int kTabPairs = 1024;      // (a, i') pairs of a block at most: 64 KB of shared memory

// CTA (ib, g): the outputs i = i' + P t (i <= n: odd n reaches i = n) of the IB residues i' of
// block ib, summed over the rows m = g, g + gridDim.y, ...  Per row: G(a, i') = sum_b h(a + A b)
// e^(i A b phi) and its derivative part sum_b (a + A b) h e^(...) (by suffix sums over b)
// into shared memory, then sum_a G e^(i a phi) and the product with C_m.
//
// Bound by FP64 instructions: about 68 per (a, b, i') and 48 per (a, i) for Bastin; 233 us at
// M = 512, n = 1024, 8.4e12 of them a second.
template <bool BASTIN>
__global__ void __launch_bounds__(kTabThreads)
    k_table_rows(const double2 *__restrict__ hre, const double2 *__restrict__ him, const double *__restrict__ amp,
                 const double2 *__restrict__ cosines, int M, int n, int A, int P, int IB, double2 *__restrict__ part) {
  extern __shared__ double2 sm[];
  const int pairs = A * IB;
  double2 *gzr = sm, *gzi = sm + pairs, *gdr = sm + 2 * pairs, *gdi = sm + 3 * pairs;
  const int i0 = blockIdx.x * IB, nb = min(IB, P - i0);
  const int T = n / P + 1;  // values of t with i' + P t <= n
  const int n4 = 4 * n;
  double2 p[kTabItems], w[kTabItems];
#pragma unroll
  for (int k = 0; k < kTabItems; ++k) p[k] = w[k] = make_double2(0.0, 0.0);
  for (int m = blockIdx.y; m < M; m += gridDim.y) {
    const double2 *hr = hre + (size_t)m * M, *hi = him + (size_t)m * M;
    for (int e = threadIdx.x; e < nb * A; e += kTabThreads) {
      const int a = e % A, il = e / A;
      const int o = 2 * (i0 + il) + 1;
      // b from the top: S_b = sum_{b' >= b} x_b', sum_b b x_b = sum_{b >= 1} S_b
      double2 zr = make_double2(0.0, 0.0), zi = zr, dr = zr, di = zr;
      const long step = (long)A * o % n4;
      const int bmax = a < M ? (M - 1 - a) / A : -1;
      int q = bmax < 0 ? 0 : (int)(step * bmax % n4);
      for (int b = bmax; b >= 0; --b) {
        const double2 c = cosines[q], s = cosines[q < n ? q + 3 * n : q - n];
        const double2 xr = hr[a + A * b];
        dd_fma(xr, c, zr);
        if (BASTIN) {
          const double2 xi = hi[a + A * b];
          dd_fma(dd_neg(xi), s, zr);
          dd_fma(xr, s, zi);
          dd_fma(xi, c, zi);
          if (b > 0) {
            dd_acc(zr, dr);
            dd_acc(zi, di);
          }
        } else {
          dd_fma(xr, s, zi);
        }
        q -= (int)step;
        if (q < 0) q += n4;
      }
      zr = dd_norm(zr);
      zi = dd_norm(zi);
      gzr[a * IB + il] = zr;
      gzi[a * IB + il] = zi;
      if (BASTIN) {
        gdr[a * IB + il] = dd_add(dd_scale(dd_norm(dr), A), dd_scale(zr, a));
        gdi[a * IB + il] = dd_add(dd_scale(dd_norm(di), A), dd_scale(zi, a));
      }
    }
    __syncthreads();
    const double am = amp[m] * (BASTIN ? 2.0 : 1.0);
#pragma unroll
    for (int k = 0; k < kTabItems; ++k) {
      const int e = threadIdx.x + k * kTabThreads;
      const int il = e % IB, t = e / IB, i = i0 + il + P * t;
      if (t < T && il < nb && i <= n) {
        const int o = 2 * i + 1;  // below 4 n
        double2 z = make_double2(0.0, 0.0), d = z;
        int q = 0;
        for (int a = 0; a < A; ++a) {
          const double2 c = cosines[q], s = cosines[q < n ? q + 3 * n : q - n];
          dd_fma(gzr[a * IB + il], c, z);
          dd_fma(dd_neg(gzi[a * IB + il]), s, z);
          if (BASTIN) {
            dd_fma(gdr[a * IB + il], s, d);
            dd_fma(gdi[a * IB + il], c, d);
          }
          q += o;
          if (q >= n4) q -= n4;
        }
        const double2 cm = dd_scale(cosines[(long)m * o % n4], am);
        dd_fma(cm, dd_norm(z), p[k]);
        if (BASTIN) dd_fma(dd_neg(cm), dd_norm(d), w[k]);
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int k = 0; k < kTabItems; ++k) {
    const int e = threadIdx.x + k * kTabThreads;
    const int il = e % IB, t = e / IB, i = i0 + il + P * t;
    if (t < T && il < nb && i <= n) {
      double2 *out = part + ((size_t)blockIdx.y * (n + 1) + i) * 2;
      out[0] = dd_norm(p[k]);
      out[1] = dd_norm(w[k]);
    }
  }
}

// acc[k].x += p, acc[n + k].y += w of frequency k (angle pi (4 k + 1) / (2 n) below n / 2, its
// reflection above), the row groups summed in order; one warp per frequency
__global__ void k_table_sum(const double2 *__restrict__ part, int groups, int n, double2 *__restrict__ acc) {
  const int k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (k >= n) return;
  const int i = k < n / 2 ? 2 * k : 2 * (n - k) - 1;
  double2 p = make_double2(0.0, 0.0), w = p;
  for (int g = lane; g < groups; g += 32) {
    const double2 *in = part + ((size_t)g * (n + 1) + i) * 2;
    dd_acc(in[0], p);
    dd_acc(in[1], w);
  }
  for (int o = 16; o > 0; o >>= 1) {
    dd_acc(make_double2(__shfl_down_sync(0xffffffffu, p.x, o), __shfl_down_sync(0xffffffffu, p.y, o)), p);
    dd_acc(make_double2(__shfl_down_sync(0xffffffffu, w.x, o), __shfl_down_sync(0xffffffffu, w.y, o)), w);
  }
  if (lane == 0) {
    acc[k].x += p.x + p.y;
    acc[n + k].y += w.x + w.y;
  }
}

// FP64 instructions per row and energy with the split A (k_table_rows).
double split_cost(int M, int A) { return 2.0 * ((M + A - 1) / A) * 68 + 48.0 * A; }

// The divisor A of 2 n (2 to 256) with the fewest.
int best_split(int M, int n) {
  int best = 2;
  double cost = 1e300;
  for (int A = 2; A <= 256 && A <= 2 * n; ++A) {
    if (2 * n % A) continue;
    const double c = split_cost(M, A);
    if (c < cost) {
      cost = c;
      best = A;
    }
  }
  return best;
}

}  // namespace

// 40 us of launches, then the FP64 instructions at the rate measured for k_table_rows.
double kubo_table_us(int M, int nump, int formula) {
  const double work = (double)M * nump * split_cost(M, best_split(M, nump));
  return 40 + work * (formula == LINQT_KUBO_BASTIN ? 1.0 : 0.5) / 8.8e6;
}

namespace {
struct TableGrid {
  int A, P, IB, blocks, groups;
};
TableGrid table_grid(const Session *s, int M, int n) {
  TableGrid g;
  g.A = best_split(M, n);
  g.P = 2 * n / g.A;
  g.IB = std::max(1, std::min(g.P, kTabPairs / g.A));
  g.blocks = (g.P + g.IB - 1) / g.IB;
  g.groups = std::max(1, std::min(M, 4 * s->sm_count / g.blocks));
  return g;
}
struct TableBuffers {
  double2 *cosines, *coef, *part, *table;
  double *amp;
};
TableBuffers table_buffers(Session *s, int M, int n) {
  const size_t MM = (size_t)M * M;
  TableBuffers b;
  b.cosines = (double2 *)s->get("kt_cos", sizeof(double2) * 4 * (size_t)n);
  b.amp = (double *)s->get("kt_amp", sizeof(double) * (size_t)M);
  b.coef = (double2 *)s->get("kt_coef", sizeof(double2) * 2 * MM);
  b.part = (double2 *)s->get("kt_part", sizeof(double2) * 2 * (size_t)table_grid(s, M, n).groups * (n + 1));
  b.table = (double2 *)s->get("kt_table", sizeof(double2) * 2 * MM);
  return b;
}
}  // namespace

// The raw table's buffer, with all that kubo_table_sums needs beside it, its weights and those of the site
// transforms formed; NULL where memory is short (the site transforms do without).
double2 *kubo_table_reserve(Session *s, int M, int nump, int formula) {
  const SiteTables t = site_tables(s, M, nump, formula);
  try {
    const TableBuffers b = table_buffers(s, M, nump);
    k_table_setup<<<(std::max(M, 4 * nump) + 127) / 128, 128, 0, s->stream>>>(nump, M, b.cosines, b.amp, t.pf, t.tw);
    LQ_LAUNCHED();
    return b.table;
  } catch (const Error &e) {
    if (e.code != LINQT_ERR_NOMEM || s->strict_memory) throw;
    s->release("kt_");
    return nullptr;
  }
}

// acc += what kubo_fft_sites gives (the parts of p and w that reach sigma), from the raw table
// hi + lo [M][M].
void kubo_table_sums(Session *s, const double2 *hi, const double2 *lo, int M, int nump, int formula, double2 *acc) {
  const int n = nump;
  const TableGrid tg = table_grid(s, M, n);
  const int A = tg.A, P = tg.P, IB = tg.IB, blocks = tg.blocks, groups = tg.groups;
  const TableBuffers b = table_buffers(s, M, n);
  double2 *tab = b.cosines, *re = b.coef, *im = re + (size_t)M * M, *part = b.part;
  double *amp = b.amp;
  const long tot = (long)M * M;
  const int g = (int)std::max(1L, std::min((tot + 255) / 256, (long)s->sm_count * 8));
  k_table_coef<<<g, 256, 0, s->stream>>>(hi, lo, amp, M, re, im);
  LQ_LAUNCHED();
  const size_t smem = sizeof(double2) * 4 * (size_t)A * IB;
  const bool bastin = formula == LINQT_KUBO_BASTIN;
  const void *f = bastin ? (const void *)k_table_rows<true> : (const void *)k_table_rows<false>;
  raise_smem_limit(f, smem);
  if (bastin)
    k_table_rows<true><<<dim3(blocks, groups), kTabThreads, smem, s->stream>>>(re, im, amp, tab, M, n, A, P, IB, part);
  else
    k_table_rows<false><<<dim3(blocks, groups), kTabThreads, smem, s->stream>>>(re, im, amp, tab, M, n, A, P, IB, part);
  LQ_LAUNCHED();
  k_table_sum<<<(n * 32 + 255) / 256, 256, 0, s->stream>>>(part, groups, n, acc);
  LQ_LAUNCHED();
}

}  // namespace linqt
