// FP64 post-processing on the device: Jackson damping, the DOS on the Chebyshev
// grid, the Kubo-Bastin energy sum, and Gershgorin spectral bounds.
#include <cmath>

#include "internal.cuh"

namespace linqt {

namespace {

// Jackson factor g_m for a table of Mom moments
// (src/chebyshev_moments1D.cpp:79-86, src/chebyshev_moments2D.cpp:105-116)
__device__ __host__ inline double jackson_g(int m, int Mom) {
  const double phi = M_PI / (double)(Mom + 1.0);
  return ((Mom - m + 1) * cos(phi * m) + sin(phi * m) * cos(phi) / sin(phi)) * phi / M_PI;
}

// out[M0t x M1t] = mu[:M0t, :M1t] * g0 * g1  (truncation keeps the top-left block,
// src/chebyshev_moments2D.cpp:4-13)
__global__ void k_jackson2d(const double2 *__restrict__ mu, int M1, int M0t, int M1t, double2 *__restrict__ out) {
  const long tot = (long)M0t * M1t;
  for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < tot; t += (long)gridDim.x * blockDim.x) {
    const int i = (int)(t / M1t), j = (int)(t % M1t);
    out[t] = cscale(mu[(size_t)i * M1 + j], jackson_g(i, M0t) * jackson_g(j, M1t));
  }
}

// The spectral function N/a sum_m delta(E_i, m) Re mu_m (delta_chebF of
// include/chebyshev_coefficients.hpp:9-14) on num_div energies, one block per energy:
//   grid 0: x_i = -1 + i 2/(num_div - 1), the sum as it is (src/spectralFunctionFromChebmom.cpp:35-72;
//           the end points divide by zero and come out non-finite there and here);
//   grid 1: x_i = cos(pi (i+1/2)/num_div), its absolute value
//           (src/spectralFunctionFromChebmom_FFTgrid.cpp:35-75).
__global__ void k_dos(const double2 *__restrict__ mu, int M, double N, double a, double bc, int grid, int num_div,
                      double *__restrict__ E, double *__restrict__ dos) {
  const int i = blockIdx.x;
  const double x = grid == 0 ? -1.0 + i * (2 * 1.0) / (num_div - 1) : cos(M_PI * (i + 0.5) / num_div);
  const double f0 = sqrt(1.0 - x * x), th = acos(x);
  double acc = 0.0;
  for (int m = threadIdx.x; m < M; m += blockDim.x) acc += cos(m * th) / f0 / M_PI * mu[m].x;
  __shared__ double sh[256];
  sh[threadIdx.x] = acc;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    E[i] = x * a + bc;
    const double v = sh[0] * N / a;
    dos[i] = grid == 0 ? v : fabs(v);
  }
}

// ---------------------------------------------------------------------------
// The energy sums of LinQT's post-processors (kuboBastinFromChebmom{,_FFTgrid},
// kuboGreenwoodFromChebmom{,_FFTgrid}, kuboBastin{I,II,Sea,Surf}FromChebmom) on a
// Jackson-damped table mu[M0][M1]:  kernel(x) = pref * sum_{m0,m1} f(x, m0, m1, mu).
// Each is evaluated as Y(i, m0) = sum_m1 B(x_i, m1) mu(m0, m1) (an FP64 GEMM against a
// coefficient table) and a per-energy sum over m0 with the left coefficient, in the GEMM's epilogue
// but for Bastin II.  The
// coefficient functions are those of include/chebyshev_coefficients.hpp:9-32:
//   delta(x, m)  = cos(m acos x) / f0 / pi,            f0 = sqrt(1 - x^2)
//   G(x, m)      = -i (x - i f0)^m / f0,                (x - i f0)^m = exp(-i m acos x)
//   DG(x, m)     = -i (x - i f0)^m (x + i m f0) / f0^3
// ---------------------------------------------------------------------------
enum CoefKind { COEF_DELTA = 0, COEF_G = 1, COEF_DG = 2, COEF_REDG2 = 3 };

// energy i of the grid: 0 uniform in [-xbound, xbound]; 1 cos(pi (2i + 1/2)/n); 2 grid 1 in
// the ascending order of rearrange_crescent_order (src/kuboBastinFromChebmom_FFTgrid.cpp:18-36)
__device__ __host__ inline double grid_energy(int grid, int i, int n, double xbound) {
  if (grid == 0) return -xbound + i * (2 * xbound) / (n - 1);
  if (grid == 2) i = rearranged_source(i, n);
  return cos(M_PI * (2 * i + 0.5) / n);
}

// An energy with its angle and sqrt(1 - x^2).
struct Node {
  double x, th, f0, unused;
};
__device__ inline Node node_of(double x) { return Node{x, acos(x), sqrt(1.0 - x * x), 0.0}; }
__global__ void k_energy_nodes(int grid, int num_div, double xbound, Node *__restrict__ nodes) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < num_div; i += gridDim.x * blockDim.x)
    nodes[i] = node_of(grid_energy(grid, i, num_div, xbound));
}

__device__ inline double2 coef(int kind, const Node &e, int m) {
  const double f0 = e.f0;
  double sn, cs;
  sincos(m * e.th, &sn, &cs);
  if (kind == COEF_DELTA) return make_double2(cs / f0 / M_PI, 0.0);
  const double2 p = make_double2(cs, -sn);  // (x - i f0)^m
  if (kind == COEF_G) return make_double2(p.y / f0, -p.x / f0);  // -i p / f0
  const double2 q = cmul(p, make_double2(e.x, m * f0));           // * (x + i m f0)
  const double inv = 1.0 / (f0 * f0 * f0);
  const double2 dg = make_double2(q.y * inv, -q.x * inv);          // -i q / f0^3
  if (kind == COEF_DG) return dg;
  return make_double2(dg.x + dg.x, 0.0);                           // Re DG + conj(Re DG)
}

// Coefficient rows of all energies.  parts 2: B(x_i, m) as (re, im); 1: its real part (the others
// are real); conjugate: conj(B), for zgemm_cn.  Rows of ld numbers, zero past parts * M1.
__global__ void k_coef_table(int kind, int num_div, int M1, int ld, int parts, int conjugate,
                             const Node *__restrict__ nodes, double *__restrict__ tab) {
  const int per = (ld + parts - 1) / parts;
  const long tot = (long)num_div * per;
  for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < tot; t += (long)gridDim.x * blockDim.x) {
    const int i = (int)(t / per), m = (int)(t % per);
    double2 c = m < M1 ? coef(kind, nodes[i], m) : make_double2(0.0, 0.0);
    if (conjugate) c = cconj(c);
    double *o = tab + (size_t)i * ld + (size_t)m * parts;
    o[0] = c.x;
    if (parts == 2) o[1] = c.y;
  }
}

// Right-hand rows of the real sums: parts 2 (Im of B mu = Br Im mu + Bi Re mu): (Im, Re) of mu;
// parts 1: Im mu or Re mu.
__global__ void k_table_rows_real(const double2 *__restrict__ mu, int M0, int M1, int ld, int parts, int imag,
                                  double *__restrict__ q) {
  const int per = (ld + parts - 1) / parts;
  const long tot = (long)M0 * per;
  for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < tot; t += (long)gridDim.x * blockDim.x) {
    const int i = (int)(t / per), m = (int)(t % per);
    const double2 v = m < M1 ? mu[(size_t)i * M1 + m] : make_double2(0.0, 0.0);
    double *o = q + (size_t)i * ld + (size_t)m * parts;
    o[0] = imag ? v.y : v.x;
    if (parts == 2) o[1] = v.x;
  }
}

// part[bx][i] = sum over the m0 of column block bx of left(i, m0) Y(i, m0),  Y = P Q^T: P [num_div][ld],
// Q [M0][ld], real, ld a multiple of 16.  Only one real number per (energy, m0) reaches the
// output of five of the six sums, so they take one real product (K = 2 M1, or M1 where B is real)
// in place of a complex one, and Y never leaves the registers: 512 x 512 moments at 15360 energies
// 0.61 ms (27 of 36 TFLOP/s), where the complex product, its reduction and the sums took 0.94.  FP64 tensor cores (m8n8k4),
// 128 x 64 outputs per CTA, 8 warps of 32 x 32, K slices of 16 in three cp.async stages (pitch 20:
// the fragment loads are free of bank conflicts).  left: variant 4 (sea) 2 Im G(m0), else delta(m0).
constexpr int EBM = 128, EBN = 64, EBK = 16, ELD = EBK + 4, EST = 3;

__device__ __forceinline__ void ecp16(void *smem, const void *g, bool ok) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(g), "r"(ok ? 16 : 0));
}

__global__ void __launch_bounds__(256, 2)
    k_energy_gemm(int variant, const double *__restrict__ P, const double *__restrict__ Q, int num_div, int M0, int ld,
                  const Node *__restrict__ nodes, double *__restrict__ part) {
  extern __shared__ __align__(16) double esm[];
  double(*As)[EBM][ELD] = reinterpret_cast<double(*)[EBM][ELD]>(esm);
  double(*Bs)[EBN][ELD] = reinterpret_cast<double(*)[EBN][ELD]>(esm + EST * EBM * ELD);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, wm = warp >> 1, wn = warp & 1;
  const int fr = lane >> 2, fk = lane & 3;
  const int i0 = blockIdx.y * EBM, n0 = blockIdx.x * EBN;
  const auto load = [&](int st, int k0) {
#pragma unroll
    for (int q = 0; q < (EBM + EBN) * EBK / 2 / 256; ++q) {  // 16-byte pieces, 8 a row
      const int e = threadIdx.x + 256 * q, r = e >> 3, c = (e & 7) * 2;
      if (r < EBM) {
        const bool ok = i0 + r < num_div;
        ecp16(&As[st][r][c], P + (ok ? (size_t)(i0 + r) * ld + k0 + c : 0), ok);
      } else {
        const bool ok = n0 + r - EBM < M0;
        ecp16(&Bs[st][r - EBM][c], Q + (ok ? (size_t)(n0 + r - EBM) * ld + k0 + c : 0), ok);
      }
    }
  };
  double acc[4][4][2];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
  const int nk = ld / EBK;
#pragma unroll
  for (int st = 0; st < EST - 1; ++st) {
    if (st < nk) load(st, st * EBK);
    asm volatile("cp.async.commit_group;\n" ::);
  }
  for (int it = 0; it < nk; ++it) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(EST - 2));
    __syncthreads();  // slice `it` has landed, and everyone is done with the one before it
    if (it + EST - 1 < nk) load((it + EST - 1) % EST, (it + EST - 1) * EBK);
    asm volatile("cp.async.commit_group;\n" ::);
    const int cur = it % EST;
#pragma unroll
    for (int ks = 0; ks < EBK; ks += 4) {
      double a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = As[cur][wm * 32 + i * 8 + fr][ks + fk];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = Bs[cur][wn * 32 + j * 8 + fr][ks + fk];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
          asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                       : "+d"(acc[i][j][0]), "+d"(acc[i][j][1])
                       : "d"(a[i]), "d"(b[j]));
    }
  }
  asm volatile("cp.async.wait_group 0;\n" ::);
  __shared__ double rows[2][EBM];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = wm * 32 + i * 8 + fr, e = i0 + r;
    double sum = 0.0;
    if (e < num_div) {
      const Node nd = nodes[e];
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int m0 = n0 + wn * 32 + j * 8 + 2 * fk + h;
          if (m0 < M0) {
            const double c = cos(m0 * nd.th);
            sum += (variant == 4 ? -2.0 * c / nd.f0 : c / nd.f0 / M_PI) * acc[i][j][h];
          }
        }
    }
    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
    sum += __shfl_xor_sync(0xffffffffu, sum, 2);
    if (fk == 0) rows[wn][r] = sum;
  }
  __syncthreads();
  if (threadIdx.x < EBM && i0 + threadIdx.x < num_div)
    part[(size_t)blockIdx.x * num_div + i0 + threadIdx.x] = rows[0][threadIdx.x] + rows[1][threadIdx.x];
}

// kern[i] = pref * sum_b part[b][i]  (fixed order)
__global__ void k_energy_parts(const double *__restrict__ part, int blocks, int num_div, double pref,
                               double *__restrict__ kern) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < num_div; i += gridDim.x * blockDim.x) {
    double s = 0.0;
    for (int b = 0; b < blocks; ++b) s += part[(size_t)b * num_div + i];
    kern[i] = s * pref;
  }
}

// Bastin II: kernel_i = pref * sum_m0 -Re(G(m0) DG(m1) mu - DG(m0) G(m1) mu), one warp per energy,
// fixed order (Y1 = DG mu, Y2 = G mu, complex)
__global__ void k_energy_sums2(const double2 *__restrict__ Y1, const double2 *__restrict__ Y2,
                               const Node *__restrict__ nodes, int num_div, int M0, double pref,
                               double *__restrict__ kern) {
  const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, l = threadIdx.x & 31;
  if (w >= num_div) return;
  const Node nd = nodes[w];
  double acc = 0.0;
  for (int m0 = l; m0 < M0; m0 += 32) {
    const double2 y1 = Y1[(size_t)w * M0 + m0], y2 = Y2[(size_t)w * M0 + m0];
    const double2 t = csub(cmul(coef(COEF_G, nd, m0), y1), cmul(coef(COEF_DG, nd, m0), y2));
    acc += -t.x;
  }
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
  if (l == 0) kern[w] = acc * pref;
}

// The drivers' output columns (num_div - 1 points): E and the kernel, the mean of its neighbours, or
// its running integral.  One CTA, every thread a run of consecutive points; the integrals are each
// thread's sums on top of the prefix of the threads before it, in a fixed order.  On one thread
// the 15360 points of a 512-moment table took 4.2 ms, four times the energy sums before it.
__global__ void __launch_bounds__(1024)
    k_energy_output(int variant, int grid, const double *__restrict__ kern, int num_div, double xbound, double a,
                    double bc, double *__restrict__ E, double *__restrict__ out) {
  const int n = num_div - 1, per = (n + blockDim.x - 1) / blockDim.x;
  const int lo = min(n, (int)threadIdx.x * per), hi = min(n, lo + per);
  const bool integral = variant == 0 || variant == 3 || variant == 4;
  auto term = [&](int i, double de) {
    return variant == 0 ? kern[i] * de : (variant == 3 ? 1.0 : 0.5) * (kern[i] + kern[i + 1]) * de;
  };
  double e0 = grid_energy(grid, lo, num_div, xbound), sum = 0.0;
  if (integral) {
    for (int i = lo; i < hi; ++i) {
      const double e1 = grid_energy(grid, i + 1, num_div, xbound);
      sum += term(i, e1 - e0);
      e0 = e1;
    }
    sum = exclusive_prefix(sum);
    e0 = grid_energy(grid, lo, num_div, xbound);
  }
  for (int i = lo; i < hi; ++i) {
    const double e1 = grid_energy(grid, i + 1, num_div, xbound);
    E[i] = e0 * a + bc;
    if (integral) {
      sum += term(i, e1 - e0);
      out[i] = sum;
    } else if (variant == 1) {
      out[i] = kern[i];
    } else {
      out[i] = variant == 2 ? 0.5 * (kern[i] + kern[i + 1]) : (kern[i + 1] + kern[i]) / 2.0;
    }
    e0 = e1;
  }
}

// Gershgorin: per-block min(center - radius), max(center + radius)
__global__ void k_gershgorin(int n, const int *__restrict__ rp, const int *__restrict__ ci,
                             const double2 *__restrict__ v, double2 *__restrict__ part) {
  double lo = INFINITY, hi = -INFINITY;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    double c = 0.0, r = 0.0;
    for (int k = rp[i]; k < rp[i + 1]; ++k) {
      if (ci[k] == i)
        c += v[k].x;
      else
        r += hypot(v[k].x, v[k].y);
    }
    lo = fmin(lo, c - r);
    hi = fmax(hi, c + r);
  }
  __shared__ double sl[256], sh[256];
  sl[threadIdx.x] = lo;
  sh[threadIdx.x] = hi;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o) {
      sl[threadIdx.x] = fmin(sl[threadIdx.x], sl[threadIdx.x + o]);
      sh[threadIdx.x] = fmax(sh[threadIdx.x], sh[threadIdx.x + o]);
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) part[blockIdx.x] = make_double2(sl[0], sh[0]);
}

__global__ void k_minmax(const double2 *__restrict__ part, int nb, double2 *__restrict__ out) {
  if (threadIdx.x || blockIdx.x) return;
  double lo = INFINITY, hi = -INFINITY;
  for (int b = 0; b < nb; ++b) {
    lo = fmin(lo, part[b].x);
    hi = fmax(hi, part[b].y);
  }
  *out = make_double2(lo, hi);
}

}  // namespace

namespace {
// C(t_n) = scale * sum_{m < T} delta(x, m) (g_m Re mu(m, n)), one thread per time step
__global__ void k_time_correlation(const double2 *__restrict__ mu, int NT, int T, double x, double scale, double dt,
                                   double *__restrict__ t_out, double *__restrict__ c_out) {
  const double phi = M_PI / (double)(T + 1.0);
  const Node e = node_of(x);
  for (int n = blockIdx.x * blockDim.x + threadIdx.x; n < NT; n += gridDim.x * blockDim.x) {
    double out = 0.0;
    for (int m = 0; m < T; ++m) {
      const double g = ((T - m + 1) * cos(phi * m) + sin(phi * m) * cos(phi) / sin(phi)) * phi / M_PI;
      out += coef(COEF_DELTA, e, m).x * (mu[(size_t)m * NT + n].x * g);
    }
    t_out[n] = n * dt;
    c_out[n] = out * scale;
  }
}
}  // namespace

void time_correlation(Session *s, const double2 *mu, int M, int NT, int N, double band_width, double band_center,
                      double dt, double broad_meV, double energy, double *t_out, double *c_out, int *T_out) {
  const int T = jackson_cut(M, band_width, broad_meV);
  const double hw = band_width / 2;
  k_time_correlation<<<(NT + 127) / 128, 128, 0, s->stream>>>(mu, NT, T, (energy - band_center) / hw, N / hw, dt,
                                                               t_out, c_out);
  LQ_LAUNCHED();
  *T_out = T;
}

int jackson_cut(int M, double band_width, double broad) {
  const double eta = 2.0 * broad / 1000 / band_width;
  const int maxMom = (int)ceil(M_PI / eta);
  return maxMom > M ? M : maxMom;
}

double jackson_factor(int m, int Mom) { return jackson_g(m, Mom); }

void jackson2d_dev(Session *s, const double2 *mu, int M0, int M1, int M0t, int M1t, double2 *out) {
  (void)M0;
  const long tot = (long)M0t * M1t;
  const int g = (int)std::max(1L, std::min((tot + 255) / 256, (long)s->sm_count * 8));
  k_jackson2d<<<g, 256, 0, s->stream>>>(mu, M1, M0t, M1t, out);
  LQ_LAUNCHED();
}

void dos_grid(Session *s, const double2 *mu, int M, int N, double band_width, double band_center, double *E,
              double *dos) {
  spectral_grid(s, mu, M, N, band_width, band_center, 1, M, E, dos);
}

void spectral_grid(Session *s, const double2 *mu, int M, int N, double band_width, double band_center, int grid,
                   int num_div, double *E, double *out) {
  LQ_REQUIRE((grid == 0 || grid == 1) && num_div >= 2, "spectral function: bad grid");
  k_dos<<<num_div, 256, 0, s->stream>>>(mu, M, (double)N, band_width / 2.0, band_center, grid, num_div, E, out);
  LQ_LAUNCHED();
}

void energy_sums(Session *s, const double2 *mu, int M0, int M1, int N, double band_width, double band_center,
                 int variant, int grid, double xbound, int num_div, double *E, double *out) {
  LQ_REQUIRE(variant >= 0 && variant <= 5 && grid >= 0 && grid <= 2 && num_div >= 2, "energy sums: bad argument");
  static const int kind1[6] = {COEF_DG, COEF_G, COEF_G, COEF_DG, COEF_REDG2, COEF_DELTA};
  const double a = band_width / 2.0, w = N / a / a;
  const double pref[6] = {-2.0 * w, -w, -w, w / 2 / M_PI, w / 2 / M_PI, M_PI * w};
  double *kern = (double *)s->get("esum_kern", sizeof(double) * (size_t)num_div);
  Node *nodes = (Node *)s->get("esum_nodes", sizeof(Node) * (size_t)num_div);
  k_energy_nodes<<<(num_div + 127) / 128, 128, 0, s->stream>>>(grid, num_div, xbound, nodes);
  LQ_LAUNCHED();
  const auto blocks_of = [&](long tot) { return (int)std::max(1L, std::min((tot + 255) / 256, (long)s->sm_count * 16)); };
  if (variant == 3) {
    double2 *tab = (double2 *)s->get("esum_tab", sizeof(double2) * (size_t)num_div * M1);
    double2 *Y1 = (double2 *)s->get("esum_y1", sizeof(double2) * (size_t)num_div * M0);
    double2 *Y2 = (double2 *)s->get("esum_y2", sizeof(double2) * (size_t)num_div * M0);
    for (double2 *Y : {Y1, Y2}) {
      // Y(i, m0) = sum_m1 conj(tab(i, m1)) mu(m0, m1) = sum_m1 B(x_i, m1) mu(m0, m1)
      k_coef_table<<<blocks_of((long)num_div * M1), 256, 0, s->stream>>>(Y == Y1 ? COEF_DG : COEF_G, num_div, M1,
                                                                         2 * M1, 2, 1, nodes, (double *)tab);
      LQ_LAUNCHED();
      zgemm_cn(s, tab, num_div, mu, M0, M1, Y, false);
    }
    k_energy_sums2<<<(num_div * 32 + 255) / 256, 256, 0, s->stream>>>(Y1, Y2, nodes, num_div, M0, pref[3], kern);
    LQ_LAUNCHED();
  } else {
    // Im(B mu) for the Bastin and Greenwood kernels; B is real for the sea (Im) and surface (Re) terms
    const int parts = variant <= 2 ? 2 : 1, ld = (parts * M1 + EBK - 1) / EBK * EBK;
    double *P = (double *)s->get("esum_tab", sizeof(double) * (size_t)num_div * ld);
    double *Q = (double *)s->get("esum_q", sizeof(double) * (size_t)M0 * ld);
    const dim3 g((M0 + EBN - 1) / EBN, (num_div + EBM - 1) / EBM);
    double *part = (double *)s->get("esum_part", sizeof(double) * (size_t)g.x * num_div);
    k_coef_table<<<blocks_of((long)num_div * ld / parts), 256, 0, s->stream>>>(kind1[variant], num_div, M1, ld, parts, 0,
                                                                              nodes, P);
    LQ_LAUNCHED();
    k_table_rows_real<<<blocks_of((long)M0 * ld / parts), 256, 0, s->stream>>>(mu, M0, M1, ld, parts, variant != 5, Q);
    LQ_LAUNCHED();
    const size_t smem = sizeof(double) * EST * (EBM + EBN) * ELD;
    raise_smem_limit((const void *)k_energy_gemm, smem);
    k_energy_gemm<<<g, 256, smem, s->stream>>>(variant, P, Q, num_div, M0, ld, nodes, part);
    LQ_LAUNCHED();
    k_energy_parts<<<blocks_of(num_div), 256, 0, s->stream>>>(part, (int)g.x, num_div, pref[variant], kern);
    LQ_LAUNCHED();
  }
  k_energy_output<<<1, 1024, 0, s->stream>>>(variant, grid, kern, num_div, xbound, a, band_center, E, out);
  LQ_LAUNCHED();
}

void bastin_grid(Session *s, const double2 *mu, int M0, int M1, int N, double band_width, double band_center,
                 double xbound, int num_div, double *E, double *sigma) {
  energy_sums(s, mu, M0, M1, N, band_width, band_center, 0, 0, xbound, num_div, E, sigma);
}

void gershgorin(Session *s, const DeviceOp &A, double *lo, double *hi) {
  const int nb = (int)std::max(1L, std::min(((long)A.n + 255) / 256, (long)s->sm_count * 4));
  double2 *part = (double2 *)s->get("gersh_part", sizeof(double2) * (nb + 1));
  k_gershgorin<<<nb, 256, 0, s->stream>>>(A.n, A.d_rowptr, A.d_col, A.d_val64, part);
  LQ_LAUNCHED();
  k_minmax<<<1, 1, 0, s->stream>>>(part, nb, part + nb);
  LQ_LAUNCHED();
  double2 h;
  LQ_CUDA(cudaMemcpyAsync(&h, part + nb, sizeof(double2), cudaMemcpyDeviceToHost, s->stream));
  LQ_CUDA(cudaStreamSynchronize(s->stream));
  *lo = h.x;
  *hi = h.y;
}

}  // namespace linqt
