// FP64 moment contraction on the INT8 tensor cores, exact in a residue number system.
//
//   raw(m0, m1) += sum_k conj(L[m0][k]) * Rv[m1][k]     (FP64 or FP32 Chebyshev blocks)
//
// The FP64 tensor-core rate of the B200 is its FP64 FMA rate (36 TFLOP/s), a hundredth of its
// INT8 rate, so the product is taken in integers (the modular form of the Ozaki scheme:
// K. Ozaki, Y. Uchino, T. Imamura, "Ozaki Scheme II: a GEMM-oriented emulation of
// floating-point matrix multiplication using an integer modular technique", 2025):
//
//  1. Per row and K chunk, every real x becomes the integer X = rint(x 2^(53-e)), e the
//     exponent with max|x| < 2^e over the chunk.  |X| <= 2^53, so the rounding is at most
//     2^-54 of the chunk's maximum: entries within a factor 2 of it are exact.
//  2. X is reduced modulo kMods pairwise coprime moduli p whose prime factors are all 1
//     mod 4, where i has an image s with s^2 = -1: a complex integer a + bi is then the pair
//     (a + s b, a - s b) mod p and a complex product is two real products, not four (or the
//     three of Gauss' form).
//  3. The 2 kMods real products run as INT8 GEMMs with exact INT32 accumulation
//     (k_rns_gemm, tcgen05 kind::i8), each reduced mod p in its epilogue.
//  4. The Chinese remainder theorem gives the exact integer sums (|Re|, |Im| <= 2^107 K,
//     below half the product of the moduli), scaled back and added over the chunks in
//     double-double arithmetic (k_rns_crt).  The sum comes as hi + lo, so that the energy
//     reconstruction (kubo_table.cu) may use more than 53 bits of it.
//  5. The sum is accepted or not, on the device (rns_rejected in rns_accept.cuh, k_commit in mu_gemm.cu).
//
// Against the FP64 tensor-core kernel (mu_gemm.cu), whose partial sums round once per term, the
// only error is that of step 1, which averages over K: a value keeps the bits above 2^-53 of its
// row chunk's largest, not 53 of its own.  Where the sides are large on the same sites, that is
// no loss (a disordered chain, currents everywhere: random states 1.1e-17 of the table's maximum, a
// local state 1.4e-16; FP64 products 1.6e-16 and 3.5e-16).  Where one is large only where the other
// is small, the table lives on the small values: currents in two regions that the states hardly
// connect were off by 5e-11 of the maximum, or all of it (FP64 products 5e-16).  So step 1's error
// is estimated from what it did, the rows' units and norms (rns_accept.cuh), and a sum that it could
// move by more than is allowed there is dropped for the FP64 kernel's, and sigma's for the site
// transforms.  That costs one launch and the rows' sums of squares: graphene 128 x 128, 8
// vectors, 512 moments 5.75 -> 5.85 ms.
//
// Measured (contraction phase, before = the FP64 kernel): Kane-Mele 64 x 64 cells, M = 1024,
// K = 524288: 121.0 -> 30.5 ms; graphene 128 x 128, M = 512, K = 262144: 15.2 -> 5.8 ms.  The
// moments are no further from a 64-bit torch computation than before (2.3e-14 and 1.4e-15).
//
// Non-finite input: a row chunk that holds an infinity or a NaN gives NaN in its row or
// column, as products with such terms do in FP64.
#include <cooperative_groups.h>
#include <cuda.h>

#include <cstdint>

#include "dd.cuh"
#include "internal.cuh"
#include "rns_accept.cuh"
#include "tc_common.cuh"

namespace linqt {

namespace {

using namespace tc;
namespace cg = cooperative_groups;

// ---------------------------------------------------------------------------
// the moduli
// ---------------------------------------------------------------------------
typedef unsigned __int128 u128;
constexpr int kMods = 17;
// 221 = 13 * 17, 205 = 5 * 41, the others prime; their product is 2^124.17
constexpr int kP[kMods] = {241, 233, 229, 221, 205, 197, 193, 181, 173, 157, 149, 137, 113, 109, 101, 97, 89};

constexpr int mod_inverse(int a, int p) {
  a %= p;
  for (int x = 1; x < p; ++x)
    if (a * x % p == 1) return x;
  return 0;
}
// the smallest s > 0 with s^2 = -1 mod p (p / 2 at most)
constexpr int root_of_minus_one(int p) {
  for (int s = 1; s < p; ++s)
    if ((s * s + 1) % p == 0) return s;
  return 0;
}
constexpr u128 product_of_mods() {
  u128 P = 1;
  for (int j = 0; j < kMods; ++j) P *= (u128)kP[j];
  return P;
}
constexpr u128 kProd = product_of_mods();

// Constants of one modulus, as the kernels index them.
struct ModTab {
  int p[kMods], s[kMods];
  double inv[kMods];          // 1 / p
  int m21[kMods];             // rint(2^21 / p): quotients of products of residues
  int m32[kMods];             // rint(2^32 / p): quotients of the INT32 sums
  unsigned u32[kMods];        // ceil(2^32 / p): quotients below 2^17, exact
  int cre[kMods], cim[kMods]; // w / 2 and w / (2 s) mod p, w = (P / p)^-1 mod p
  float invf[kMods];
  unsigned long long whi[kMods], wlo[kMods];  // P / p
};
constexpr ModTab make_mods() {
  ModTab t{};
  for (int j = 0; j < kMods; ++j) {
    const int p = kP[j], s = root_of_minus_one(p);
    t.p[j] = p;
    t.s[j] = s;
    t.inv[j] = 1.0 / p;
    t.m21[j] = ((1 << 21) + p / 2) / p;
    t.m32[j] = (int)(((1LL << 32) + p / 2) / p);
    t.u32[j] = (unsigned)(((1LL << 32) + p - 1) / p);
    const u128 W = kProd / (u128)p;
    const int w = mod_inverse((int)(W % (u128)p), p);
    t.cre[j] = w * mod_inverse(2, p) % p;
    t.cim[j] = w * mod_inverse(2 * s, p) % p;
    t.invf[j] = 1.0f / p;
    t.whi[j] = (unsigned long long)(W >> 64);
    t.wlo[j] = (unsigned long long)W;
  }
  return t;
}
constexpr ModTab kModsHost = make_mods();
__constant__ ModTab kMod = make_mods();
constexpr unsigned long long kProdHi = (unsigned long long)(kProd >> 64), kProdLo = (unsigned long long)kProd;

constexpr int kPlanes = 2 * kMods;   // residue planes per side: (a + s b, a - s b) per modulus
constexpr int kBk = 128;             // K bytes of a GEMM block (one swizzle row)
// K chunk (complex): |sum| <= 2^107 kChunkMax = 2^122, less than a quarter of the product of
// the moduli (the reconstruction rounds S / P to the nearest integer); INT32 sums of kChunkMax products
// of residues of at most 121 stay below 2^29
constexpr int kChunkMax = 32768;
constexpr int kPart = 4096;          // K (complex) that a CTA of k_residues holds in registers
constexpr int kBadExp = 1 << 20;     // exponent mark of a chunk with a non-finite value
static_assert(kChunkMax <= kMaxParts * kPart, "parts of a chunk");

// ---------------------------------------------------------------------------
// residues
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t low_bytes(int a, int b, int c, int d) {
  return __byte_perm(__byte_perm(a, b, 0x0040), __byte_perm(c, d, 0x0040), 0x5410);
}

// Residue planes of both sides: z = 2 chunk + side (0 the L side, 1 the R side).  Planes are
// stored in the blocks the GEMM loads, [chunk][plane][K block of 128][row][128 bytes], so a
// 128-row operand tile is one contiguous piece of 16 KB.  Grid (parts, rows, 2 nchunk) in
// clusters of `parts` CTAs, one (row, chunk) each: every CTA loads 4096 complex into registers
// once, the cluster exchanges the maxima of their exponents through distributed shared memory,
// and the residues are formed and written from the registers, so the FP64 blocks are read
// from HBM once.
//
// Bound by its integer arithmetic (3.7 TB/s of the 16 bytes read and 34 written per complex
// value, 67 % of issue slots).  Arithmetic per real and
// modulus: one FP64 FMA with 1.5 * 2^52, whose low word is the integer quotient q =
// rint(X / p) (off by at most one unit of 1/p of r, |r| <= p/2 + 1), and one 32-bit
// multiply-add r = X - p q on the low words; per complex and modulus two small reductions
// of r_a + s r_b and r_a - s r_b (below 2^14: a 21-bit reciprocal is enough for
// |residue| <= p/2 + 1).
template <class Tc>
__global__ void __launch_bounds__(256, 2)
    k_residues(const Tc *__restrict__ srcA, const Tc *__restrict__ srcB, long ld, long K, int kc, int rows_a,
               int rows_b, int nkb, int8_t *__restrict__ plA, int8_t *__restrict__ plB, int *__restrict__ expA,
               int *__restrict__ expB, int nchunk, RnsSide *__restrict__ side) {
  __shared__ unsigned red[8];
  __shared__ unsigned part_max;
  __shared__ double part_sq[8];
  cg::cluster_group cl = cg::this_cluster();
  const bool b_side = blockIdx.z & 1;
  const int c = blockIdx.z >> 1, row = blockIdx.y;
  const int rows = b_side ? rows_b : rows_a;
  if (row >= rows) return;  // the whole cluster leaves (grid.y covers the longer side)
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long k0 = (long)c * kc;
  const int len = (int)min((long)kc, K - k0);  // complex values of this chunk
  const Tc *x = (b_side ? srcB : srcA) + (size_t)row * ld + k0;
  const int base = blockIdx.x * kPart;
  double2 v[4][4];
  unsigned mx = 0;
#pragma unroll
  for (int g = 0; g < 4; ++g) {
    const int k = base + (g * 8 + warp) * kBk + lane * 4;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      v[g][q] = k + q < len ? to_d2(__ldg(x + k + q)) : make_double2(0.0, 0.0);
      mx = max(mx, max((unsigned)__double2hiint(v[g][q].x) & 0x7fffffffu,
                       (unsigned)__double2hiint(v[g][q].y) & 0x7fffffffu));
    }
  }
  for (int o = 16; o > 0; o >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if (lane == 0) red[warp] = mx;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned m = 0;
    for (int w = 0; w < 8; ++w) m = max(m, red[w]);
    part_max = m;
  }
  cl.sync();  // every part's maximum is written
  const int parts = (int)cl.num_blocks();
  mx = 0;
  for (int r = 0; r < parts; ++r) mx = max(mx, *cl.map_shared_rank(&part_max, r));
  cl.sync();  // no CTA leaves while another may still read its maximum
  const bool bad = mx >= 0x7ff00000u;
  // |x| < 2^e; below 2^-900 the scale stays at 2^953 (its unit is then 2^-953)
  const int e = max((int)(mx >> 20) - 1022, -900);
  if (threadIdx.x == 0 && blockIdx.x == 0) (b_side ? expB : expA)[(size_t)row * nchunk + c] = bad ? kBadExp : e;
  const double scale = bad ? 0.0 : __hiloint2double((1023 + 53 - e) << 20, 0);
  const size_t plane = (size_t)nkb * rows * kBk;
  int8_t *out = (b_side ? plB : plA) + (size_t)c * kPlanes * plane + (size_t)row * kBk + lane * 4;
  constexpr double kMagic = 6755399441055744.0;  // 1.5 * 2^52
  double sq = 0.0;  // sum of squares, in units of 2^(2 (e - 53))
#pragma unroll 1
  for (int g = 0; g < 4; ++g) {
    const int kb = (base >> 7) + g * 8 + warp;
    if (kb * kBk >= len) break;  // blocks past the chunk's end are not read
    double xr[4], xi[4];
    int lr[4], li[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      // a bad chunk holds infinities: 0 * inf would be NaN, whose conversion is unspecified
      const double a = bad ? 0.0 : v[0][q].x * scale, b = bad ? 0.0 : v[0][q].y * scale;
      const long long ia = __double2ll_rn(a), ib = __double2ll_rn(b);
      xr[q] = (double)ia;
      xi[q] = (double)ib;
      lr[q] = (int)ia;
      li[q] = (int)ib;
      sq = fma(xr[q], xr[q], fma(xi[q], xi[q], sq));
    }
#pragma unroll
    for (int h = 0; h < 3; ++h)  // rotate: v[0] is the next group
#pragma unroll
      for (int q = 0; q < 4; ++q) v[h][q] = v[h + 1][q];
    int8_t *o = out + (size_t)kb * rows * kBk;
#pragma unroll
    for (int j = 0; j < kMods; ++j) {
      constexpr ModTab T = kModsHost;
      const int p = T.p[j], s = T.s[j], m21 = T.m21[j];
      const double inv = T.inv[j];
      int u[4], w[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int ra = lr[q] - p * __double2loint(fma(xr[q], inv, kMagic));
        const int rb = li[q] - p * __double2loint(fma(xi[q], inv, kMagic));
        const int a = ra + s * rb, b = ra - s * rb;
        u[q] = a - p * ((a * m21 + (1 << 20)) >> 21);
        w[q] = b - p * ((b * m21 + (1 << 20)) >> 21);
      }
      *reinterpret_cast<uint32_t *>(o + (size_t)(2 * j) * plane) = low_bytes(u[0], u[1], u[2], u[3]);
      *reinterpret_cast<uint32_t *>(o + (size_t)(2 * j + 1) * plane) = low_bytes(w[0], w[1], w[2], w[3]);
    }
  }
  for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
  if (lane == 0) part_sq[warp] = sq;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < 8; ++w) t += part_sq[w];
    RnsSide &sd = side[blockIdx.z];
    const double unit = bad ? INFINITY : __hiloint2double((1023 - 53 + e) << 20, 0);
    if (blockIdx.x == 0) raise_to(&sd.unit, unit);
    raise_to(&sd.sq[blockIdx.x], bad ? INFINITY : t * unit * unit);
  }
}

// ---------------------------------------------------------------------------
// the INT8 GEMMs
// ---------------------------------------------------------------------------
// One 256 x 256 tile of one plane and K chunk per CTA pair (cta_group::2: an M = 256, N = 256,
// K = 32 MMA spans the two SMs of the pair, each holding 128 rows of A and 128 rows of B, so
// that an operand byte loaded from L2 serves 256 multiply-adds), persistent over the
// (chunk, plane, tile) jobs.  Per CTA: warp 0 issues the TMA loads of its own halves, warp 1
// of the leading CTA issues the MMAs, warps 2-5 reduce the finished accumulators mod p; two
// accumulators of 256 TMEM columns let the next tile's MMAs run meanwhile.  Barriers:
//   full[s]       in the leading CTA: both CTAs' loads of stage s have landed
//   empty[s]      in both: the MMAs that read stage s are done (multicast commit)
//   acc_full[a]   in both: accumulator a is complete
//   acc_empty[a]  in the leading CTA: the 8 epilogue warps of the pair have read it
// Measured 2.4-2.5 POPS at M = 1024 (tensor pipe 71-80 % of active cycles, the SM clock down to
// 1.54 GHz under the load).  Every wait is bounded: on expiry the error flag is raised, the CTA stops issuing, and it
// waits for its own copies before it meets its peer and leaves.
constexpr int kRnsTile = 256;
constexpr int kRnsStages = 6;
constexpr int kRnsHalf = 128 * kBk;          // bytes of 128 operand rows
constexpr int kRnsStage = 2 * kRnsHalf;      // per CTA: A half and B half
constexpr int kRnsThreads = 192;

struct RnsShared {
  alignas(1024) uint8_t stage[kRnsStages][kRnsStage];
  alignas(8) unsigned long long full[kRnsStages], empty[kRnsStages], acc_full[2], acc_empty[2];
  uint32_t tmem_base;
  int abort;
};

// D S32, A and B signed 8-bit, both K-major, N = 256, M = 256
constexpr uint32_t kIdescRns = (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kRnsTile >> 3) << 17) |
                               ((uint32_t)(kRnsTile >> 4) << 24);

__device__ __forceinline__ uint32_t mapa(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
// bounded wait on a barrier that the peer CTA may arrive on
__device__ __forceinline__ bool mbar_wait_cluster(unsigned long long *b, uint32_t parity, int *err) {
  for (long i = 0; i < kTcWaitLimit; ++i) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(smem_u32(b)), "r"(parity)
        : "memory");
    if (done) return true;
  }
  atomicExch(err, 1);
  return false;
}
__device__ __forceinline__ void mbar_arrive_remote(uint32_t addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];\n" ::"r"(addr) : "memory");
}
// Load a tile into this CTA's shared memory, completing on a barrier of the pair's leading CTA.
__device__ __forceinline__ void tma_load_pair(void *dst, const CUtensorMap *map, int x, int y, int z, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%3, %4, %5}], [%2];\n" ::"r"(smem_u32(dst)),
      "l"(map), "r"(bar), "r"(x), "r"(y), "r"(z)
      : "memory");
}
__device__ __forceinline__ void umma_pair(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::2.kind::i8 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(kIdescRns), "r"(accumulate));
}
// arrive on the barrier at this offset in both CTAs once the MMAs issued so far are done
__device__ __forceinline__ void commit_pair(unsigned long long *bar) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n" ::"r"(
          smem_u32(bar)),
      "h"((uint16_t)3)
      : "memory");
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kRnsThreads, 1)
    k_rns_gemm(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, int MA, int MB,
               long K, int kc, int nkb, int nchunk, uint8_t *__restrict__ res, int pitch, int *err) {
  extern __shared__ uint8_t smem_raw[];
  RnsShared &sm = *reinterpret_cast<RnsShared *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  cg::cluster_group cl = cg::this_cluster();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cl.block_rank();
  const int mt = (MA + kRnsTile - 1) / kRnsTile, nt = (MB + kRnsTile - 1) / kRnsTile;
  const int ntiles = mt * nt * kPlanes * nchunk;
  const int pair = blockIdx.x >> 1, npairs = gridDim.x >> 1;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kRnsStages; ++s) {
      mbar_init(&sm.full[s], 1);
      mbar_init(&sm.empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&sm.acc_full[a], 1);
      mbar_init(&sm.acc_empty[a], 8);
    }
    sm.abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&sm.tmem_base)),
                 "r"(512));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;\n" ::);
  }
  tc_fence_before();
  cl.sync();  // barriers of both CTAs are initialised, TMEM is allocated
  tc_fence_after();
  const uint32_t tmem = sm.tmem_base;
  // jobs of this pair: (tile n fastest, tile m, plane, chunk)
  struct Job {
    int m0, n0, plane, chunk, blocks;
  };
  auto job_of = [&](int t) {
    Job j;
    j.n0 = (t % nt) * kRnsTile;
    t /= nt;
    j.m0 = (t % mt) * kRnsTile;
    t /= mt;
    j.plane = t % kPlanes;
    j.chunk = t / kPlanes;
    j.blocks = (int)((min((long)kc, K - (long)j.chunk * kc) + kBk - 1) / kBk);
    return j;
  };

  if (warp == 0) {
    // ---------------- TMA producer
    if (lane == 0) {
      int it = 0;
      bool go = true;
      for (int t = pair; t < ntiles && go; t += npairs) {
        const Job j = job_of(t);
        // conj(a) b: the image of conj(a) under i -> s is that of a under i -> -s
        const int za = (j.chunk * kPlanes + (j.plane ^ 1)) * nkb, zb = (j.chunk * kPlanes + j.plane) * nkb;
        for (int kb = 0; kb < j.blocks; ++kb, ++it) {
          const int s = it % kRnsStages;
          if (*(volatile int *)&sm.abort ||
              (it >= kRnsStages && !mbar_wait_cluster(&sm.empty[s], ((it / kRnsStages) & 1) ^ 1, err))) {
            sm.abort = 1;
            go = false;
            break;
          }
          if (rank == 0) mbar_arrive_expect_tx(&sm.full[s], 2 * kRnsStage);
          const uint32_t bar = mapa(smem_u32(&sm.full[s]), 0);
          tma_load_pair(sm.stage[s], &tmA, 0, j.m0 + 128 * (int)rank, za + kb, bar);
          tma_load_pair(sm.stage[s] + kRnsHalf, &tmB, 0, j.n0 + 128 * (int)rank, zb + kb, bar);
        }
      }
      // the last use of every stage: its loads have landed and its MMAs are done, so nothing
      // arrives on this CTA's barriers or shared memory after it leaves
      for (int i = max(0, it - kRnsStages); i < it; ++i)
        (void)mbar_wait_cluster(&sm.empty[i % kRnsStages], (i / kRnsStages) & 1, err);
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer (leading CTA)
    if (rank == 0 && lane == 0) {
      int it = 0, n = 0;
      bool go = true;
      for (int t = pair; t < ntiles && go; t += npairs, ++n) {
        const Job j = job_of(t);
        const int a = n & 1;
        if (n >= 2 && !mbar_wait_cluster(&sm.acc_empty[a], ((n >> 1) & 1) ^ 1, err)) {
          sm.abort = 1;
          break;
        }
        tc_fence_after();
        for (int kb = 0; kb < j.blocks; ++kb, ++it) {
          const int s = it % kRnsStages;
          if (*(volatile int *)&sm.abort || !mbar_wait_cluster(&sm.full[s], (it / kRnsStages) & 1, err)) {
            sm.abort = 1;
            go = false;
            break;
          }
          tc_fence_after();
          const uint8_t *st = sm.stage[s];
#pragma unroll
          for (int kk = 0; kk < kBk / 32; ++kk)
            umma_pair(tmem + a * kRnsTile, smem_desc_sw128(st + kk * 32), smem_desc_sw128(st + kRnsHalf + kk * 32),
                      (kb | kk) ? 1u : 0u);
          commit_pair(&sm.empty[s]);
        }
        commit_pair(&sm.acc_full[a]);
      }
    }
  } else {
    // ---------------- epilogue (warps 2-5): INT32 sums mod p -> bytes
    const int q = warp & 3;  // TMEM lane quarter this warp may access
    int n = 0;
    for (int t = pair; t < ntiles; t += npairs, ++n) {
      const Job j = job_of(t);
      const int a = n & 1;
      if (!mbar_wait_cluster(&sm.acc_full[a], (n >> 1) & 1, err)) {
        sm.abort = 1;
        break;
      }
      tc_fence_after();
      const int p = kMod.p[j.plane >> 1], m32 = kMod.m32[j.plane >> 1];
      const int r = j.m0 + 128 * (int)rank + 32 * q + lane;
      uint8_t *o = res + ((size_t)(j.chunk * kPlanes + j.plane) * MA + r) * pitch + j.n0;
      const uint32_t src = tmem + a * kRnsTile + ((uint32_t)(32 * q) << 16);
#pragma unroll 1
      for (int cb = 0; cb < kRnsTile && j.n0 + cb < MB; cb += 16) {
        uint32_t v[16];
        tmem_ld16_u32(src + cb, v);
        uint32_t w[4];
#pragma unroll
        for (int i = 0; i < 16; i += 4) {
          int b[4];
#pragma unroll
          for (int h = 0; h < 4; ++h) {
            // |sum| < 2^29: the quotient is within 1/16 of the true one before the floor
            const int x = (int)v[i + h];
            int y = x - p * __mulhi(x, m32);
            y += y < 0 ? p : 0;
            b[h] = y >= p ? y - p : y;
          }
          w[i / 4] = low_bytes(b[0], b[1], b[2], b[3]);
        }
        if (r < MA) *reinterpret_cast<uint4 *>(o + cb) = make_uint4(w[0], w[1], w[2], w[3]);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_remote(mapa(smem_u32(&sm.acc_empty[a]), 0));
    }
  }
  __syncwarp();
  tc_fence_before();
  cl.sync();  // the pair is done with each other's barriers, shared memory and TMEM
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(512));
  }
}

// ---------------------------------------------------------------------------
// Chinese remainders
// ---------------------------------------------------------------------------
// X 2^ex in double-double: three pieces of at most 48 bits, each exact in FP64
__device__ __forceinline__ double2 dd_from_i128(__int128 X, int ex) {
  const unsigned long long mask = (1ull << 48) - 1;
  const double a = (double)(long long)(X >> 96), b = (double)((unsigned long long)(X >> 48) & mask),
               c = (double)((unsigned long long)X & mask);
  double2 v;
  two_sum(a * 79228162514264337593543950336.0, b * 281474976710656.0, v.x, v.y);
  v = dd_add(v, make_double2(c, 0.0));
  return make_double2(ldexp(v.x, ex), ldexp(v.y, ex));
}

// sum(i, j) (+)= sum over chunks of 2^(ea + eb - 106) X, X the integer with the residues of the
// planes; one thread per entry, chunks in order, all in double-double.  The last slab of chunks
// also leaves the sum's largest value.
__global__ void __launch_bounds__(256)
    k_rns_crt(const uint8_t *__restrict__ res, int pitch, int MA, int MB, int nchunk, const int *__restrict__ expA,
              const int *__restrict__ expB, bool first, bool last, RnsStats *__restrict__ stats,
              double2 *__restrict__ sum_hi, double2 *__restrict__ sum_lo) {
  const u128 P = ((u128)kProdHi << 64) | kProdLo;
  const size_t plane = (size_t)MA * pitch;
  unsigned long long top = 0;
  for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < (long)MA * MB; t += (long)gridDim.x * blockDim.x) {
    const int i = (int)(t / MB), j = (int)(t % MB);
    double2 re = make_double2(0.0, 0.0), im = re;
    if (!first) {
      const double2 hi = sum_hi[t], lo = sum_lo[t];
      re = make_double2(hi.x, lo.x);
      im = make_double2(hi.y, lo.y);
    }
    for (int c = 0; c < nchunk; ++c) {
      const int ea = expA[(size_t)i * nchunk + c], eb = expB[(size_t)j * nchunk + c];
      if (ea == kBadExp || eb == kBadExp) {
        re.x = im.x = __longlong_as_double(0x7ff8000000000000ll);
        continue;
      }
      const uint8_t *r = res + (size_t)c * kPlanes * plane + (size_t)i * pitch + j;
      u128 sr = 0, si = 0;
      float fr = 0.f, fi = 0.f;
#pragma unroll
      for (int m = 0; m < kMods; ++m) {
        const int u = r[(size_t)(2 * m) * plane], v = r[(size_t)(2 * m + 1) * plane];
        const unsigned p = kMod.p[m];
        unsigned a = (unsigned)(u + v) * kMod.cre[m], b = (unsigned)(u - v + (int)p) * kMod.cim[m];
        a -= p * __umulhi(a, kMod.u32[m]);
        b -= p * __umulhi(b, kMod.u32[m]);
        const u128 w = ((u128)kMod.whi[m] << 64) | kMod.wlo[m];
        sr += w * (u128)a;
        si += w * (u128)b;
        fr = fmaf((float)a, kMod.invf[m], fr);
        fi = fmaf((float)b, kMod.invf[m], fi);
      }
      // S = X + k P with |X| < P / 4 (modulo 2^128: X itself fits)
      const __int128 xr = (__int128)(sr - P * (u128)(unsigned)__float2int_rn(fr));
      const __int128 xi = (__int128)(si - P * (u128)(unsigned)__float2int_rn(fi));
      re = dd_add(re, dd_from_i128(xr, ea + eb - 106));
      im = dd_add(im, dd_from_i128(xi, ea + eb - 106));
    }
    sum_hi[t] = make_double2(re.x, im.x);
    sum_lo[t] = make_double2(re.y, im.y);
    top = max(top, max((unsigned long long)__double_as_longlong(fabs(re.x)),
                       (unsigned long long)__double_as_longlong(fabs(im.x))));
  }
  if (!last) return;
  __shared__ unsigned long long top_s;
  if (threadIdx.x == 0) top_s = 0;
  for (int o = 16; o > 0; o >>= 1) top = max(top, __shfl_xor_sync(0xffffffffu, top, o));
  __syncthreads();
  if ((threadIdx.x & 31) == 0) atomicMax(&top_s, top);
  __syncthreads();
  if (threadIdx.x == 0 && top_s > __ldcg(&stats->top)) atomicMax(&stats->top, top_s);
}

// [blocks][rows][128 bytes], box 128 bytes x 128 rows; rows past the end read as zero
CUtensorMap make_map_rns(const void *base, int rows, long blocks) {
  CUtensorMap m;
  const cuuint64_t dims[3] = {(cuuint64_t)kBk, (cuuint64_t)rows, (cuuint64_t)blocks};
  const cuuint64_t strides[2] = {(cuuint64_t)kBk, (cuuint64_t)kBk * rows};
  const cuuint32_t box[3] = {(cuuint32_t)kBk, 128, 1};
  const cuuint32_t estr[3] = {1, 1, 1};
  const CUresult r = encode_fn()(&m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<void *>(base), dims, strides, box,
                                 estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                                 CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) fail(LINQT_ERR_CUDA, "cuTensorMapEncodeTiled failed: " + std::to_string((int)r));
  return m;
}

}  // namespace

// Which kernel contracts an MA x MB x K product.
// The line, from both sides measured on one B200 (contraction phase, this kernel / mu_gemm.cu, us):
//   M = 1024, K = 65536: 3840 / 15165;  512, 65536: 1463 / 3832;  256, 65536: 680 / 870;
//   160, 65536: 434 / 514;  128, 65536: 365 / 274;  64, 65536: 248 / 152: below 160 rows the
//   256 x 256 tiles are mostly padding, and long products go to the FP64 kernel;
//   100, 8192: 70 / 81;  100, 2048: 36 / 77: but short ones are bound by the launches here and
//   by the serial K loop there;
//   1024, 512: 171 / 147;  768, 512: 113 / 83;  512, 512: 63 / 79: K < M is bound by the
//   residue tables (34 bytes per entry and chunk).
bool rns_faster(int MA, int MB, long K) {
  const int m = std::min(MA, MB);
  return m >= 160 ? K >= std::max(192, std::max(MA, MB)) : m >= 8 && K >= 192 && K <= 8192;
}

// Time of the contraction here, us: 30 of launches, 13.5 ps an entry for the residues, the GEMMs of
// the padded tiles at 2.4 POPS (fits the times above within 20 % at K >= 2048).
double rns_us(int M, long K) {
  const double tiles = (M + kRnsTile - 1) / kRnsTile, pad = tiles * kRnsTile;
  return 30 + 2.0 * M * K * 13.5e-6 + kPlanes * pad * pad * K * 2 / 2.4e9;
}

namespace {
// The split of K, from the sizes alone: kc values a chunk, the rows' exponents are of a chunk, so no
// bit of a result depends on how many chunks' planes fit at a time.
constexpr size_t kPlaneMax = 8ull << 30;  // one chunk's planes, at most
struct RnsPlan {
  int kc;
  long chunks;
  size_t planes, res, exps;  // bytes of one chunk
  size_t chunk_bytes() const { return planes + res + exps; }
};
RnsPlan rns_plan(int MA, int MB, long K) {
  const size_t per_k = (size_t)kPlanes * (MA + MB);
  const long cap = std::max<long>(kBk, std::min<long>(kChunkMax, (long)(kPlaneMax / per_k) / kBk * kBk));
  const long total = (K + cap - 1) / cap;
  RnsPlan p;
  p.kc = (int)(((K + total - 1) / total + kBk - 1) / kBk * kBk);
  p.chunks = (K + p.kc - 1) / p.kc;
  p.planes = per_k * p.kc;
  p.res = (size_t)kPlanes * MA * ((MB + 15) / 16 * 16);
  p.exps = sizeof(int) * (size_t)(MA + MB);
  return p;
}
long slab_of(const RnsPlan &p, size_t budget) {
  return std::max(1L, std::min(p.chunks, (long)(budget / p.planes)));
}
size_t held_bytes(const Session *s, const char *name) {
  auto it = s->ws.find(name);
  return it == s->ws.end() ? 0 : it->second.second;
}
}  // namespace

// Bytes of a contraction here with planes of about `budget` bytes (one chunk's at least).
size_t rns_footprint(int MA, int MB, long K, size_t budget) {
  const RnsPlan p = rns_plan(MA, MB, K);
  return slab_of(p, budget) * p.chunk_bytes() + sizeof(double2) * 2 * (size_t)MA * MB +
         sizeof(RnsSide) * 2 * (size_t)p.chunks;
}

// Chunks of K at a time whose buffers the session holds from here on: all of them or none
// (0: use the FP64 kernel).  What is held is used; where that is less than the budget allows, up to
// half of the free memory is taken (or one chunk's), and less when that fails.  Only this call is
// the worse for memory that is short now.  A served request that runs beside others fails instead, and runs
// again alone (server.cu): its result must not depend on them.
int rns_reserve(Session *s, int MA, int MB, long K) {
  if (!s->rns_budget) return 0;
  const RnsPlan p = rns_plan(MA, MB, K);
  const size_t sum = sizeof(double2) * 2 * (size_t)MA * MB, sides = sizeof(RnsSide) * 2 * (size_t)p.chunks;
  long want = slab_of(p, s->rns_budget);
  long held = std::min({(long)(held_bytes(s, "rns_planes") / p.planes), (long)(held_bytes(s, "rns_res") / p.res),
                        (long)(held_bytes(s, "rns_exp") / p.exps)});
  if (held_bytes(s, "rns_sum") < sum || held_bytes(s, "mu_sides_counter") < sides || !held_bytes(s, "mu_stats_counter") ||
      !held_bytes(s, "mu_tc_err_barrier"))
    held = 0;
  if (held >= want || s->capturing) return (int)std::min(held, want);
  if (!s->hbm_budget) {
    size_t room = free_pool_bytes(s->device);
    for (const char *name : {"rns_planes", "rns_res", "rns_exp"}) room += held_bytes(s, name);
    if (room < p.chunk_bytes()) return (int)held;
    want = std::max(1L, std::min(want, (long)(room / 2 / p.chunk_bytes())));
    if (want < 2 * held) return (int)held;  // not worth new buffers
  }
  for (; want; want /= 2) {
    try {
      s->get("rns_sum", sum);
      s->get("mu_stats_counter", sizeof(RnsStats));  // "counter", "barrier": zeroed when allocated
      s->get("mu_sides_counter", sides);
      s->get("mu_tc_err_barrier", sizeof(int) * 4);
      s->get("rns_exp", p.exps * want);
      s->get("rns_res", p.res * want);
      s->get("rns_planes", p.planes * want);
      return (int)want;
    } catch (const Error &e) {
      if (e.code != LINQT_ERR_NOMEM || s->strict_memory) throw;
      s->release("rns_");
    }
  }
  return 0;
}

// sum (hi + lo, MA x MB) = sum_k conj(A[i][k]) B[j][k], k < K (complex FP64 or FP32 rows of K), `slab`
// chunks at a time (rns_reserve), and what it is to be checked by.
RnsSum zgemm_cn_rns(Session *s, const void *A, int MA, const void *B, int MB, long K, bool fp32_inputs, int slab) {
  const RnsPlan p = rns_plan(MA, MB, K);
  const int kc = p.kc, nkb = kc / kBk, pitch = (MB + 15) / 16 * 16;
  double2 *sum_hi = (double2 *)s->get("rns_sum", sizeof(double2) * 2 * (size_t)MA * MB);
  double2 *sum_lo = sum_hi + (size_t)MA * MB;
  int8_t *plA = (int8_t *)s->get("rns_planes", p.planes * slab);
  int8_t *plB = plA + (size_t)kPlanes * MA * kc * slab;
  uint8_t *res = (uint8_t *)s->get("rns_res", p.res * slab);
  int *eA = (int *)s->get("rns_exp", p.exps * slab);
  int *eB = eA + (size_t)MA * slab;
  RnsStats *stats = (RnsStats *)s->get("mu_stats_counter", sizeof(RnsStats));
  RnsSide *side = (RnsSide *)s->get("mu_sides_counter", sizeof(RnsSide) * 2 * (size_t)p.chunks);
  int *err = (int *)s->get("mu_tc_err_barrier", sizeof(int) * 4);  // read by mu_tc_check_error
  s->barrier_used = true;
  const CUtensorMap ta = make_map_rns(plA, MA, (long)nkb * kPlanes * slab),
                    tb = make_map_rns(plB, MB, (long)nkb * kPlanes * slab);
  const int parts = (kc + kPart - 1) / kPart;  // 8 at most
  const size_t smem = sizeof(RnsShared) + 1024;
  raise_smem_limit((const void *)k_rns_gemm, smem);
  for (long c0 = 0; c0 < p.chunks; c0 += slab) {
    const int nc = (int)std::min<long>(slab, p.chunks - c0);
    const long k0 = c0 * kc, len = std::min(K - k0, (long)nc * kc);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(parts, std::max(MA, MB), 2 * nc);
    cfg.blockDim = dim3(256);
    cfg.stream = s->stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = parts;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    if (fp32_inputs)
      LQ_CUDA(cudaLaunchKernelEx(&cfg, k_residues<float2>, (const float2 *)A + k0, (const float2 *)B + k0, K, len, kc,
                                 MA, MB, nkb, plA, plB, eA, eB, nc, side + 2 * c0));
    else
      LQ_CUDA(cudaLaunchKernelEx(&cfg, k_residues<double2>, (const double2 *)A + k0, (const double2 *)B + k0, K, len,
                                 kc, MA, MB, nkb, plA, plB, eA, eB, nc, side + 2 * c0));
    const long tiles = (long)((MA + kRnsTile - 1) / kRnsTile) * ((MB + kRnsTile - 1) / kRnsTile) * kPlanes * nc;
    const int pairs = (int)std::max(1L, std::min(tiles, (long)s->sm_count / 2));
    k_rns_gemm<<<2 * pairs, kRnsThreads, smem, s->stream>>>(ta, tb, MA, MB, len, kc, nkb, nc, res, pitch, err);
    LQ_LAUNCHED();
    const int g = (int)std::max(1L, std::min(((long)MA * MB + 255) / 256, (long)s->sm_count * 8));
    k_rns_crt<<<g, 256, 0, s->stream>>>(res, pitch, MA, MB, nc, eA, eB, c0 == 0, c0 + nc == p.chunks,
                                        stats, sum_hi, sum_lo);
    LQ_LAUNCHED();
  }
  return {sum_hi, sum_lo, stats, side, (int)p.chunks};
}

// After a wait that expired: the statistics of the contractions so far are void.
void rns_clear_stats(Session *s) {
  for (const char *name : {"mu_stats_counter", "mu_sides_counter", "mu_tiles_counter"}) {
    auto it = s->ws.find(name);
    if (it != s->ws.end()) LQ_CUDA(cudaMemsetAsync(it->second.first, 0, it->second.second, s->stream));
  }
}

}  // namespace linqt
