// The recursions of small lattices in one thread-block cluster, vectors and operators on chip.
//
// A step of the persistent grid kernels (recur.cu) costs about 2.3 us however small the lattice
// is: the grid barrier and the gathers after it are L2 round trips.  When two (1D), three
// (evolution series) or four (L/R) blocks of N x R values and the operators' rows fit the
// shared memory of up to 16 SMs, one cluster of CTAs holds them: a row's neighbours are read from
// the owners' shared memory (ld.shared::cluster), the steps are separated by the hardware
// cluster barrier, and global memory only takes what the solve keeps (the L/R stores).  The
// barrier cannot be left waiting for a CTA that is not resident: a cluster is launched whole.
//
// Bound by latency: a remote shared-memory read, a row's dependent FMAs and the cluster barrier, about
// 1.2 us a step (2.3 on the grid).  1024 threads with 4 reads in flight each measured as fast or
// faster than 512 with 8.
//
// Arithmetic is that of recur.cu, entry by entry in the same order, so the blocks are the same
// bits; the 1D moments differ by the order of the dot products' partial sums.
#include <tuple>

#include "internal.cuh"

namespace linqt {

namespace {

constexpr int kClMax = 16;          // CTAs of a cluster at most (above 8: opt-in)
constexpr int kClThreads = 1024;    // threads of a CTA at most
constexpr size_t kClSmem = 227 * 1024;  // dynamic shared memory of a CTA at most
constexpr int kClItems = 128;       // values of a block per CTA at least (32 and 256 measure the same)

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory"); }
__device__ __forceinline__ unsigned cluster_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(r));
  return r;
}
// shared::cluster address of this CTA's shared address `a` in the CTA `rank`
__device__ __forceinline__ unsigned map_rank(unsigned a, unsigned rank) {
  unsigned r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}
// volatile: stays between the cluster barriers; no memory clobber, so that the addresses and values
// of a row's next entries load meanwhile (what is read was written before the last barrier).  This
// CTA's own rows are read the same way: choosing ld.shared for them by predicate makes the two
// loads of one register wait for each other.
__device__ __forceinline__ void ld_cluster(unsigned a, double2 &v) {
  asm volatile("ld.shared::cluster.v2.f64 {%0, %1}, [%2];\n" : "=d"(v.x), "=d"(v.y) : "r"(a));
}
__device__ __forceinline__ void ld_cluster(unsigned a, float2 &v) {
  asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];\n" : "=f"(v.x), "=f"(v.y) : "r"(a));
}

// An operator's rows of one CTA in shared memory: values, the shared::cluster address of every
// column's row in the first vector block, and row starts.
struct ClRows {
  const double2 *val;
  const unsigned *adr;
  const int *rp;
};

// rows [r0, r1) of a CSR operator; `per` rows a CTA, rows of `rowbytes` bytes in the block at `vec`
__device__ ClRows load_rows(const int *__restrict__ rp, const int *__restrict__ ci, const double2 *__restrict__ v,
                            int r0, int r1, int per, unsigned vec, unsigned rowbytes, unsigned char *&dst) {
  const int k0 = rp[r0], nnz = rp[r1] - k0, nr = r1 - r0;
  double2 *sv = reinterpret_cast<double2 *>(dst);
  unsigned *sa = reinterpret_cast<unsigned *>(sv + nnz);
  int *sr = reinterpret_cast<int *>(sa + nnz);
  for (int k = threadIdx.x; k < nnz; k += blockDim.x) {
    const int j = ci[k0 + k], owner = j / per;
    sv[k] = v[k0 + k];
    sa[k] = map_rank(vec, owner) + (unsigned)(j - owner * per) * rowbytes;
  }
  for (int i = threadIdx.x; i <= nr; i += blockDim.x) sr[i] = rp[r0 + i] - k0;
  dst += ((size_t)nnz * 20 + (size_t)(nr + 1) * 4 + 15) & ~(size_t)15;
  return ClRows{sv, sa, sr};
}

// sum over a row: acc += h x, columns' rows at adr + off
template <class C>
__device__ __forceinline__ double2 gather_row(const ClRows &op, int row, unsigned off) {
  double2 acc = make_double2(0.0, 0.0);
  const int e = op.rp[row + 1];
#pragma unroll 4
  for (int k = op.rp[row]; k < e; ++k) {
    C x;
    ld_cluster(op.adr[k] + off, x);
    acc = cfma(op.val[k], x, acc);
  }
  return acc;
}

// sums of 4 values over a warp, value i valid in lane 8 i: the halves exchange two values, the
// quarters one, so 3 + 3 shuffles of a double instead of 20
__device__ __forceinline__ double warp_sum4(double a, double b, double c, double d) {
  const unsigned all = 0xffffffffu;
  const bool hi = threadIdx.x & 16, hq = threadIdx.x & 8;
  const double s0 = hi ? a : c, s1 = hi ? b : d;
  double u = (hi ? c : a) + __shfl_xor_sync(all, s0, 16), v = (hi ? d : b) + __shfl_xor_sync(all, s1, 16);
  const double t = hq ? u : v;
  double r = (hq ? v : u) + __shfl_xor_sync(all, t, 8);
  r += __shfl_xor_sync(all, r, 4);
  r += __shfl_xor_sync(all, r, 2);
  r += __shfl_xor_sync(all, r, 1);
  return r;
}

// 1D moments (k_recur_1d of recur.cu): modes, x0 and steps as there.  partials: [steps][warps of
// the cluster][2].
template <class T>
__global__ void __launch_bounds__(kClThreads, 1)
    k_cluster_1d(int n, int rshift, int per, const int *__restrict__ rp, const int *__restrict__ ci,
                 const double2 *__restrict__ hv, const typename cplx_t<T>::type *__restrict__ phi,
                 const typename cplx_t<T>::type *__restrict__ x0, int steps, int M, int mode,
                 double2 *__restrict__ partials) {
  using C = typename cplx_t<T>::type;
  extern __shared__ __align__(16) unsigned char smem[];
  const size_t len = (size_t)per << rshift;
  C *const vec = reinterpret_cast<C *>(smem);
  const unsigned rank = cluster_rank();
  const int r0 = min(n, (int)rank * per), r1 = min(n, r0 + per), items = (r1 - r0) << rshift;
  const unsigned base = (unsigned)__cvta_generic_to_shared(smem), rowbytes = sizeof(C) << rshift;
  const unsigned second = (unsigned)len * sizeof(C);
  unsigned char *dst = smem + 2 * (size_t)second;
  const ClRows H = load_rows(rp, ci, hv, r0, r1, per, base, rowbytes, dst);
  const size_t g0 = (size_t)r0 << rshift;
  for (int it = threadIdx.x; it < items; it += blockDim.x) vec[it] = x0[g0 + it];
  __syncwarp();
  cluster_arrive();
  cluster_wait();
  const int cmask = (1 << rshift) - 1;
  const int nb = gridDim.x * (blockDim.x >> 5), wid = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  int cur = 0;
  for (int s = 0; s < steps; ++s) {
    const bool need_y = mode == 2 ? (2 * s + 1 < M) : (s + 1 < M);
    double2 d0 = make_double2(0.0, 0.0), d1 = d0;
    const unsigned off = cur ? second : 0u;
    const C *const vc = vec + (cur ? len : 0);
    C *const vp = vec + (cur ? 0 : len);
    for (int it = threadIdx.x; it < items; it += blockDim.x) {
      const C xc = vc[it];
      double2 y = make_double2(0.0, 0.0);
      if (mode == 2 || need_y) {
        y = gather_row<C>(H, it >> rshift, off + (unsigned)(it & cmask) * sizeof(C));
        if (s) {
          const double2 p = to_d2(vp[it]);
          y.x = 2 * y.x - p.x;
          y.y = 2 * y.y - p.y;
        }
      }
      const C yc = from_d2<C>(y);
      if (need_y) vp[it] = yc;
      const double2 xi = to_d2(xc);
      if (mode == 1) {
        d0 = cfma_conj(to_d2(phi[g0 + it]), xi, d0);
      } else {
        d0 = cfma_conj(xi, xi, d0);
        d1 = cfma_conj(to_d2(yc), xi, d1);
      }
    }
    __syncwarp();
    if (need_y) cluster_arrive();
    const double v = warp_sum4(d0.x, d0.y, d1.x, d1.y);
    if ((threadIdx.x & 7) == 0)
      reinterpret_cast<double *>(partials + ((size_t)s * nb + wid) * 2)[(threadIdx.x & 31) >> 3] = v;
    __syncwarp();
    if (!need_y) break;
    cluster_wait();
    cur ^= 1;
  }
  __syncwarp();
  cluster_arrive();  // nobody leaves while another may still read its shared memory
  cluster_wait();
}

// L and R recursions (k_recur_lr of recur.cu): the same stores.
template <class T, bool HAS_V>
__global__ void __launch_bounds__(kClThreads, 1)
    k_cluster_lr(int n, int rshift, int per, const int *__restrict__ rp, const int *__restrict__ ci,
                 const double2 *__restrict__ hv, const int *__restrict__ vrp, const int *__restrict__ vci,
                 const double2 *__restrict__ vv, typename cplx_t<T>::type *__restrict__ Lst,
                 typename cplx_t<T>::type *__restrict__ Rst, const typename cplx_t<T>::type *__restrict__ phi, int M,
                 size_t blk) {
  using C = typename cplx_t<T>::type;
  extern __shared__ __align__(16) unsigned char smem[];
  const size_t len = (size_t)per << rshift;
  C *const vec = reinterpret_cast<C *>(smem);  // L, L, T, T
  const unsigned rank = cluster_rank();
  const int r0 = min(n, (int)rank * per), r1 = min(n, r0 + per), items = (r1 - r0) << rshift;
  const unsigned base = (unsigned)__cvta_generic_to_shared(smem), rowbytes = sizeof(C) << rshift;
  const unsigned second = (unsigned)len * sizeof(C);
  unsigned char *dst = smem + 4 * (size_t)second;
  const ClRows H = load_rows(rp, ci, hv, r0, r1, per, base, rowbytes, dst);
  ClRows V{};
  if (HAS_V) V = load_rows(vrp, vci, vv, r0, r1, per, base, rowbytes, dst);
  const size_t g0 = (size_t)r0 << rshift;
  for (int it = threadIdx.x; it < items; it += blockDim.x) {
    vec[it] = Lst[g0 + it];
    vec[2 * len + it] = HAS_V ? phi[g0 + it] : Rst[g0 + it];
  }
  __syncwarp();
  cluster_arrive();
  cluster_wait();
  const int cmask = (1 << rshift) - 1;
  int cur = 0;
  for (int m = 0; m < M; ++m) {
    const bool more = m + 1 < M;
    const unsigned off = cur ? second : 0u;
    C *const Lp = vec + (cur ? 0 : len), *const Xp = Lp + 2 * len;  // T_{m-1}, then T_{m+1}
    for (int it = threadIdx.x; it < items; it += blockDim.x) {
      const int row = it >> rshift;
      const unsigned lo = off + (unsigned)(it & cmask) * sizeof(C), xo = lo + 2 * second;
      if (more) {
        double2 aL = make_double2(0.0, 0.0), aX = aL;
        const int e = H.rp[row + 1];
#pragma unroll 4
        for (int k = H.rp[row]; k < e; ++k) {
          const unsigned a = H.adr[k];
          const double2 h = H.val[k];
          C l, x;
          ld_cluster(a + lo, l);
          ld_cluster(a + xo, x);
          aL = cfma(h, l, aL);
          aX = cfma(h, x, aX);
        }
        if (m) {
          const double2 pl = to_d2(Lp[it]), px = to_d2(Xp[it]);
          aL = make_double2(2 * aL.x - pl.x, 2 * aL.y - pl.y);
          aX = make_double2(2 * aX.x - px.x, 2 * aX.y - px.y);
        }
        const C ol = from_d2<C>(aL), ox = from_d2<C>(aX);
        Lp[it] = ol;
        Xp[it] = ox;
        Lst[(size_t)(m + 1) * blk + g0 + it] = ol;
        if (!HAS_V) Rst[(size_t)(m + 1) * blk + g0 + it] = ox;
      }
      if (HAS_V) Rst[(size_t)m * blk + g0 + it] = from_d2<C>(gather_row<C>(V, row, xo));
    }
    if (!more) break;
    __syncwarp();
    cluster_arrive();
    cluster_wait();
    cur ^= 1;
  }
  __syncwarp();
  cluster_arrive();
  cluster_wait();
}

// Chebyshev series (k_cheb_series of recur.cu): X <- sum_{s < K} coef[s] T_s(H) X
__global__ void __launch_bounds__(kClThreads, 1)
    k_cluster_series(int n, int rshift, int per, const int *__restrict__ rp, const int *__restrict__ ci,
                     const double2 *__restrict__ hv, double2 *__restrict__ X, const double2 *__restrict__ coef, int K) {
  extern __shared__ __align__(16) unsigned char smem[];
  const size_t len = (size_t)per << rshift;
  double2 *const vec = reinterpret_cast<double2 *>(smem);
  double2 *const sum = vec + 2 * len;
  const unsigned rank = cluster_rank();
  const int r0 = min(n, (int)rank * per), r1 = min(n, r0 + per), items = (r1 - r0) << rshift;
  const unsigned base = (unsigned)__cvta_generic_to_shared(smem), rowbytes = sizeof(double2) << rshift;
  const unsigned second = (unsigned)len * sizeof(double2);
  unsigned char *dst = smem + 3 * (size_t)second;
  const ClRows H = load_rows(rp, ci, hv, r0, r1, per, base, rowbytes, dst);
  const size_t g0 = (size_t)r0 << rshift;
  const double2 c0 = coef[0];
  for (int it = threadIdx.x; it < items; it += blockDim.x) {
    const double2 x = X[g0 + it];
    vec[it] = x;
    sum[it] = cmul(c0, x);
  }
  const int cmask = (1 << rshift) - 1;
  int cur = 0;
  for (int s = 1; s < K; ++s) {
    __syncwarp();
    cluster_arrive();
    const double2 cs = coef[s];
    cluster_wait();
    const unsigned off = cur ? second : 0u;
    double2 *const vp = vec + (cur ? 0 : len);
    for (int it = threadIdx.x; it < items; it += blockDim.x) {
      double2 y = gather_row<double2>(H, it >> rshift, off + (unsigned)(it & cmask) * sizeof(double2));
      if (s > 1) {
        const double2 p = vp[it];
        y.x = 2 * y.x - p.x;
        y.y = 2 * y.y - p.y;
      }
      vp[it] = y;
      sum[it] = cadd(sum[it], cmul(cs, y));
    }
    cur ^= 1;
  }
  for (int it = threadIdx.x; it < items; it += blockDim.x) X[g0 + it] = sum[it];
  __syncwarp();
  cluster_arrive();
  cluster_wait();
}

// Cluster geometry for N x R blocks: CTAs, rows per CTA, threads, shared memory (ctas == 0: the
// grid kernels take it).
struct ClGeom {
  int ctas = 0, per = 0, threads = 0, rshift = 0;
  size_t smem = 0;
};

size_t op_slice_bytes(const DeviceOp &A, int r0, int r1) {
  return ((size_t)(A.rowptr[r1] - A.rowptr[r0]) * 20 + (size_t)(r1 - r0 + 1) * 4 + 15) & ~(size_t)15;
}

// Where the line lies: reads of other SMs' shared memory run at about a fifth of L1's rate, so a step
// grows with the gathers (values read per step) while the grid's does not until its passes do.
// Measured, us per step here / on the grid: 1D, square 961 sites, 1 vector (5k gathers) 1.8 / 3.1, 16
// vectors (77k) 2.7 / 3.4, 32 (154k) 3.9 / 3.4; square 4096 x 4 (82k) 2.6 / 3.2, x 8 3.7 / 3.3;
// honeycomb 8192 x 2 (66k) 3.1 / 3.1, x 4 4.1 / 3.2; Kane-Mele 1024 x 4 (53k) 2.6 / 4.0.  L/R,
// honeycomb 800 x 16 (141k) 2.9 / 3.6, x 32 4.4 / 3.6; Kane-Mele 4096 x 1 (135k) 3.1 / 7.6,
// honeycomb 8192 x 1 (90k) 2.8 / 3.4, x 2 3.8 / 3.5.
// k_recur_1d_regs, rows of up to kRegsRow entries, is a faster grid kernel: square 12100 x 1 (60k)
// 1.70 / 1.91, 14400 x 1 (72k) 2.03 / 1.93; cubic 8000 x 1 (56k) 1.86 / 2.15, 10648 x 1 (75k) 2.26 / 2.15.
constexpr long kClGathers1d = 80000, kClGathersRegs = 65000, kClGathersLr = 140000;

// Whether the device can hold one cluster of `ctas` CTAs of func at the largest shared memory and thread
// count that cluster_geometry gives (a device with fewer SMs a GPC, or a part of one, may not).  Asked
// once per device, kernel and size.
bool cluster_fits(int device, const void *func, int ctas) {
  static std::mutex m;
  static std::map<std::tuple<int, const void *, int>, bool> known;
  std::lock_guard<std::mutex> g(m);
  const auto key = std::make_tuple(device, func, ctas);
  auto it = known.find(key);
  if (it != known.end()) return it->second;
  raise_smem_limit(func, kClSmem);
  bool ok = cudaFuncSetAttribute(func, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ctas);
  cfg.blockDim = dim3(kClThreads);
  cfg.dynamicSmemBytes = kClSmem;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = ctas;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  int n = 0;
  ok = ok && cudaOccupancyMaxActiveClusters(&n, func, &cfg) == cudaSuccess && n > 0;
  if (!ok) cudaGetLastError();
  return known[key] = ok;
}

ClGeom cluster_geometry(Session *s, const void *func, const DeviceOp &H, const DeviceOp *V, int R, size_t esz,
                        int blocks) {
  ClGeom g;
  // tests of the bounded grid barrier need the grid kernels
  if (s->inject_extra || s->inject_limit) return g;
  const long items = (long)H.n * R;
  const long line = blocks == 4 ? kClGathersLr : blocks == 2 && H.max_row <= kRegsRow ? kClGathersRegs : kClGathers1d;
  if ((blocks == 4 ? 2 * H.nnz + (V ? V->nnz : 0) : H.nnz) * R > line) return g;
  while ((1 << g.rshift) < R) ++g.rshift;
  const int want = (int)std::min<long>(kClMax, std::max<long>(1, (items + kClItems - 1) / kClItems));
  int c = 1;
  while (c < want) c <<= 1;
  for (; c <= kClMax; c <<= 1) {
    const int per = (H.n + c - 1) / c;
    size_t worst = 0;
    for (int b = 0; b < c; ++b) {
      const int r0 = std::min(H.n, b * per), r1 = std::min(H.n, r0 + per);
      worst = std::max(worst, op_slice_bytes(H, r0, r1) + (V ? op_slice_bytes(*V, r0, r1) : 0));
    }
    const size_t bytes = worst + (size_t)blocks * esz * ((size_t)per << g.rshift);
    if (bytes > kClSmem) continue;
    if (!cluster_fits(s->device, func, c)) break;  // the grid kernels take it
    g.ctas = c;
    g.per = per;
    g.smem = bytes;
    g.threads = (int)std::min<long>(kClThreads, std::max<long>(32, (((long)per << g.rshift) + 31) / 32 * 32));
    return g;
  }
  return g;
}

template <class... P, class... A>
void cluster_launch(Session *s, void (*f)(P...), const ClGeom &g, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(g.ctas);
  cfg.blockDim = dim3(g.threads);
  cfg.dynamicSmemBytes = g.smem;
  cfg.stream = s->stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = g.ctas;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  LQ_CUDA(cudaLaunchKernelEx(&cfg, f, (P)args...));
}

template <class T>
bool run_1d(Session *s, const DeviceOp &H, const void *phi, const void *x0, int steps, int M, int mode, int R,
            double2 *dots) {
  using C = typename cplx_t<T>::type;
  const ClGeom g = cluster_geometry(s, (const void *)k_cluster_1d<T>, H, nullptr, R, sizeof(C), 2);
  if (!g.ctas) return false;
  if (!dots) return true;
  const int nb = g.ctas * (g.threads / 32);
  double2 *partials = (double2 *)s->get("rec1d_part", sizeof(double2) * 2 * (size_t)steps * nb);
  cluster_launch(s, k_cluster_1d<T>, g, H.n, g.rshift, g.per, H.d_rowptr, H.d_col, H.d_val64, (const C *)phi,
                 (const C *)x0, steps, M, mode, partials);
  reduce_step_partials(s, partials, steps, nb, 1, dots);
  return true;
}

template <class T>
bool run_lr(Session *s, const DeviceOp &H, const DeviceOp *V, void *Lst, void *Rst, const void *phi, int M, int R) {
  using C = typename cplx_t<T>::type;
  auto *f = V ? k_cluster_lr<T, true> : k_cluster_lr<T, false>;
  const ClGeom g = cluster_geometry(s, (const void *)f, H, V, R, sizeof(C), 4);
  if (!g.ctas) return false;
  if (!Lst) return true;
  cluster_launch(s, f, g, H.n, g.rshift, g.per, H.d_rowptr, H.d_col, H.d_val64, V ? V->d_rowptr : nullptr,
                 V ? V->d_col : nullptr, V ? V->d_val64 : nullptr, (C *)Lst, (C *)Rst, (const C *)phi, M,
                 (size_t)H.n * R);
  return true;
}

}  // namespace

bool cluster_recur_1d(Session *s, const DeviceOp &H, const void *phi, const void *x0, int steps, int M, int mode, int R,
                      bool fp32, double2 *dots) {
  return fp32 ? run_1d<float>(s, H, phi, x0, steps, M, mode, R, dots)
              : run_1d<double>(s, H, phi, x0, steps, M, mode, R, dots);
}

bool cluster_recur_lr(Session *s, const DeviceOp &H, const DeviceOp *V, void *Lst, void *Rst, const void *phi, int M,
                      int R, bool fp32) {
  return fp32 ? run_lr<float>(s, H, V, Lst, Rst, phi, M, R) : run_lr<double>(s, H, V, Lst, Rst, phi, M, R);
}

bool cluster_cheb_series(Session *s, const DeviceOp &H, void *X, const double2 *coef, int K, int R) {
  const ClGeom g = cluster_geometry(s, (const void *)k_cluster_series, H, nullptr, R, sizeof(double2), 3);
  if (!g.ctas) return false;
  cluster_launch(s, k_cluster_series, g, H.n, g.rshift, g.per, H.d_rowptr, H.d_col, H.d_val64, (double2 *)X, coef, K);
  return true;
}

}  // namespace linqt
