// FP64 products on the int8 tensor cores (tcgen05 kind::i8) by error-free splitting.
//
// Every FP64 operand row is scaled by a power of two and written as kOzS signed 8-bit digits
// (Ootomo, Ozaki and Yokota, "DGEMM on integer matrix multiplication unit", 2024; Ozaki et
// al., "Error-free transformations of matrix multiplication", 2012):
//   x = 2^e sum_{i=1..S} d_i 2^-(8i - 1),   d_i in [-128, 127]
// (55 bits below the row's power of two for S = 7).  The products d_i d_j with i + j = D
// share one weight, so ND accumulators per output hold all pairs with i + j <= ND + 1,
//   acc_D = sum_{i + j = D} sum_k a_i[m][k] b_j[n][k]      (exact in int32),
// and the FP64 result is sum_D acc_D 2^(2 - 8D), times the two row scales.  With ND = 7 (28
// pairs) the dropped pairs add an error of about 2^-56 sqrt(K) (row scale) x (column
// scale): below an FP64 chain's rounding where the sums are as large as their terms.  ND = 8
// (34 pairs, 2^-63) serves the propagation, whose operands are near the identity: the row
// scale is that of the diagonal, the results are 20 times smaller (measured over a
// substep at 128 and 384 orbitals: ND = 7 3.0e-15 and 4.9e-15 of W, the FP64 pipe 6.4e-16
// and 1.1e-15).
//
// Layout and tile.  TMEM holds 512 columns of 32-bit accumulators, so 7 or 8 accumulators
// allow a 128 x 64 output tile.  The seven B slices of a tile sit one after
// the other in shared memory (64 rows each), so the products of A slice i with B slices
// 1 .. S + 1 - i are ONE matrix product of N = 64 (S + 1 - i) columns whose accumulators
// are consecutive in TMEM, starting at accumulator i: ten tcgen05.mma per 32 bytes of K
// instead of 28 (ND = 7), and each A slice is read from shared memory once or twice.
// What bounds it: per tile, the MMAs and then the drain, since one tile's accumulators fill
// TMEM and no MMA runs while they are read.  Counters (chunks of the exchange at 384 orbitals, 32
// vectors x 64 walkers of 48 electrons, 17.2K clocks a tile of six slabs): tensor pipe active 55%
// of the elapsed clocks, its shared-memory reads 47% of the peak (per 32 bytes of K the ten MMAs
// read 97 KB and the ring is filled with 43 KB, 1093 clocks at 128 bytes a clock against 896 of
// the tensor pipe), issue slots 16%; the chain's products at 384 orbitals (12 slabs, 34 pairs) 57%
// and 47%.  768 x 12288 x 384 real, row-major FP64 results: 78 us, 2.6e15 digit operations a second
// (the FP64 pipe's 37e12 a second would take 196 us for the same 7.2 GFLOP).
//
// One persistent CTA per SM: warp 8 copies slabs (bulk copies) into a two-stage ring, one thread of
// warp 9 issues the MMAs, and warps 0-7 turn the accumulators into FP64 results in
// registers (releasing TMEM to the next tile) and then run the epilogue functor while that
// tile's MMAs proceed.  Waits are bounded as in tc_gemm.cuh.
#pragma once
#include "tc_gemm.cuh"

namespace oz {

constexpr int kS = 7;                 // 8-bit digits per operand
constexpr int kBM = 128, kBN = 64;    // output tile
constexpr int kSlab = 64;             // bytes (= digits) of K per ring stage
constexpr int kStages = 2;
constexpr uint32_t kABytes = kS * kBM * kSlab, kBBytes = kS * kBN * kSlab;
constexpr uint32_t kStageBytes = kABytes + kBBytes;
constexpr int kEpi = 256, kThreads = kEpi + 64;
constexpr size_t kSmem = 1024 + kStages * kStageBytes + 8 * (2 * kStages + 3) + 16;
// int32 accumulators: at most S pairs of digits of magnitude 128 per K entry
constexpr int kMaxK = 16384;
static_assert((long long)kS * 128 * 128 * kMaxK < (1LL << 31), "int32 accumulation");
// acc_5 2^24 + acc_6 2^16 + acc_7 2^8 + acc_8 (4, 5, 6 and 7 pairs) below 2^51 for K <= 1024
static_assert((4LL * (1 << 24) + 5 * (1 << 16) + 6 * (1 << 8) + 7) * 128 * 128 * 1024 < (1LL << 51),
              "one integer for the four low accumulators");
static_assert((kS + 1) * kBN <= 512 && kSmem <= 227 * 1024, "TMEM / shared memory");

// Digit slices of a batch of rows, stored as the shared-memory images the MMAs read: for
// each batch, tile of R rows (R = 128 for an A operand, 64 for a B operand) and K slab, the
// kS slices' R x 64-byte blocks one after the other, 16-byte pieces swizzled as SWIZZLE_64B
// (piece index ^ (row / 2) mod 4).  A ring stage of an operand is then one contiguous bulk
// copy.  K is zero padded to whole slabs; rows past the last one hold any digits (their
// products are never stored).  scale [batch][rows] = 2^e of each row (0 for a zero row, NaN
// for a row with a non-finite entry or a maximum outside [2^-900, 2^900), which makes every
// output of the row NaN).
//
// What the digits hold is relative to a row's largest entry: an output's error is about
// 2^-56 sqrt(K) (A row's scale) (B row's scale), however small the output is.  So each B row
// (a column of results) is marked ok once one of its outputs reaches kFloor x (largest A
// scale) x (its own scale); the error is then below 2^-50 sqrt(K) of the column's largest
// entry, as FP64 sums of K terms are to a few bits.  A column that no output marks (entries
// of its operands spread so far apart that the large ones meet only zeros, or not finite)
// leaves the call to the FP64 pipe.  top [batch] and ok [batch][rows] where the operand's
// product is checked here.
constexpr double kFloor = 0x1p-6;
struct Slices {
  int8_t* d = nullptr;
  double* scale = nullptr;
  double* top = nullptr;          // A operand: largest scale of the batch
  unsigned char* ok = nullptr;    // B operand
  int rows = 0, batch = 0, tile = 0, nslab = 0;
  // source rows per batch, each giving one or two operand rows
  AFQ_HD int per_batch(bool two) const { return two ? rows / 2 : rows; }
  AFQ_HD int tiles() const { return (rows + tile - 1) / tile; }
  AFQ_HD long long stage() const { return (long long)kS * tile * kSlab; }
  size_t bytes() const { return (size_t)batch * tiles() * nslab * stage(); }
};
// Offset of digit (row r of the batch, K entry k, slice 0); the slices are tile x kSlab
// bytes apart.
AFQ_HD long long slice_offset(const Slices& s, int batch, int r, int k) {
  const int rt = r / s.tile, rr = r - rt * s.tile, ks = k / kSlab, kb = k % kSlab;
  return (((long long)batch * s.tiles() + rt) * s.nslab + ks) * s.stage() + rr * kSlab +
         (((kb >> 4) ^ (rr >> 1)) & 3) * 16 + (kb & 15);
}

struct Job {
  const int8_t *a, *b;
  const double *sa, *sb;            // row scales [batch][rows]
  const double* top;                // largest A scale per A batch (0 batches: one)
  unsigned char* ok;                // marks of the B rows, or null
  int a_rows, b_rows, a_tiles, b_tiles;   // rows and row tiles per batch (0: not batched)
  tc::TileSched sched;
  int M, N;                         // output rows and columns per batch
  int m_tile, n_tile;               // first row tile of A and of B of the launch
  int nslab, slab_split;            // K slabs, and slabs per z when split along K (else 0)
  const int* cplx;                  // non-null: *cplx == 0 (real A operand, found on the
  int nslab_real;                   // device) means nslab_real slabs instead
};

AFQ_D void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
          "r"(tc::smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(tc::smem_u32(bar))
      : "memory");
}
AFQ_D void umma_i8(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(acc));
}
// int32 accumulator, signed 8-bit A and B, both K-major
constexpr uint32_t idesc_i8(int M, int N) {
  return (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) |
         ((uint32_t)(M >> 4) << 24);
}
// 8 consecutive TMEM columns of this thread's lane (no wait)
AFQ_D void tmem_ld8(uint32_t taddr, int* r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]),
                 "=r"(r[6]), "=r"(r[7])
               : "r"(taddr));
}
// 32-byte store (32-byte aligned)
AFQ_D void store4(double* p, double a, double b, double c, double d) {
  asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(a), "d"(b), "d"(c), "d"(d)
               : "memory");
}
AFQ_D void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// sum_D acc_D 2^(2 - 8D), D = 2 .. 8, times 2^30: integer sums of consecutive accumulators,
// exact below 2^51, formed on top of the bits of 1.5 x 2^52 by 32 x 32 + 64-bit multiply-adds
// (subtracting that constant converts them without a conversion instruction).  SHORT (K of
// at most 1024): the four low accumulators fit one sum; otherwise the last stays apart.
// The drain is issue bound: 7 integer and 3 to 5 FP64 instructions per output.
constexpr long long kMagicBits = 0x4338000000000000LL;   // 1.5 x 2^52
constexpr int kShortSlabs = 1024 / kSlab;
AFQ_D long long mad_wide(int a, int b, long long c) {
  long long d;
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(d) : "r"(a), "r"(b), "l"(c));
  return d;
}
// The low part of the 8-accumulator form is acc_8 2^8 + acc_9.
template <int ND, bool SHORT>
AFQ_D double combine(const int (&a)[ND]) {
  constexpr double kMagic = 6755399441055744.0;
  const double hi = __longlong_as_double(mad_wide(
                        a[2], 1, mad_wide(a[1], 1 << 8, mad_wide(a[0], 1 << 16, kMagicBits)))) -
                    kMagic;
  if constexpr (SHORT) {
    static_assert(ND == 7, "one low sum: seven accumulators");
    const double lo = __longlong_as_double(mad_wide(
                          a[6], 1, mad_wide(a[5], 1 << 8, mad_wide(a[4], 1 << 16,
                                   mad_wide(a[3], 1 << 24, kMagicBits))))) -
                      kMagic;
    return fma(lo, 0x1p-32, hi);
  }
  const double mid = __longlong_as_double(mad_wide(
                         a[5], 1, mad_wide(a[4], 1 << 8, mad_wide(a[3], 1 << 16, kMagicBits)))) -
                     kMagic;
  if constexpr (ND == 7) {
    const double lo = __longlong_as_double(mad_wide(a[6], 1, kMagicBits)) - kMagic;
    return fma(fma(lo, 0x1p-8, mid), 0x1p-24, hi);
  } else {
    const double lo =
        __longlong_as_double(mad_wide(a[7], 1, mad_wide(a[6], 1 << 8, kMagicBits))) - kMagic;
    return fma(fma(lo, 0x1p-16, mid), 0x1p-24, hi);
  }
}

// The 32 columns of this thread's lane at trow (accumulators kBN columns apart).
template <int ND, bool SHORT>
AFQ_D void drain(uint32_t trow, double (&v)[32]) {
#pragma unroll
  for (int c = 0; c < 32; c += 8) {
    int r[ND][8];
#pragma unroll
    for (int d = 0; d < ND; d++) tmem_ld8(trow + d * kBN + c, r[d]);
    tmem_wait_ld();
#pragma unroll
    for (int q = 0; q < 8; q++) {
      int a[ND];
#pragma unroll
      for (int d = 0; d < ND; d++) a[d] = r[d][q];
      v[c + q] = combine<ND, SHORT>(a);
    }
  }
}

// The MMAs of 32 bytes of K: A slice i times B slices 0 .. min(S, ND - i) - 1, whose
// accumulators are i, i + 1, ...  FIRST starts the accumulators (slice 0 the first S, the
// last pair of slice 1 the eighth).
template <int ND, bool FIRST>
AFQ_D void mma_step(uint32_t tmem, uint64_t ad, uint64_t bd) {
#pragma unroll
  for (int i = 0; i < kS; i++) {
    const uint64_t ai = ad + (uint64_t)((i * kBM * kSlab) >> 4);
    const int nj = kS < ND - i ? kS : ND - i;
    constexpr bool kApart = FIRST && ND > kS;
#pragma unroll
    for (int j = 0; j < nj; j += 4) {
      int w = nj - j < 4 ? nj - j : 4;
      const bool tail = kApart && i == 1 && j + w == kS;   // its last column starts acc 7
      if (tail) w--;
      const uint64_t bj = bd + (uint64_t)((j * kBN * kSlab) >> 4);
      umma_i8(tmem + (i + j) * kBN, ai, bj, idesc_i8(kBM, w * kBN), FIRST ? i != 0 : 1);
      if (tail)
        umma_i8(tmem + (i + j + w) * kBN, ai, bj + (uint64_t)((w * kBN * kSlab) >> 4),
                idesc_i8(kBM, kBN), 0);
    }
  }
}

// Epilogue functor: epi(z, m, n, v) with v[32] the results of row m, columns n .. n + 31 of
// the launch (rows >= M and columns >= N included: the functor checks).
template <int ND, class Epi>
__global__ void __launch_bounds__(kThreads, 1)
oz_gemm_kernel(const __grid_constant__ Job job, const __grid_constant__ Epi epi, int* err) {
  extern __shared__ __align__(1024) uint8_t oz_smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(
      (reinterpret_cast<uintptr_t>(oz_smem_raw) + 1023) & ~uintptr_t(1023));
  auto stA = [&](int s) { return smem + s * kStageBytes; };
  auto stB = [&](int s) { return smem + s * kStageBytes + kABytes; };
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + kStages * kStageBytes);
  uint64_t* empty = full + kStages;
  uint64_t* accf = empty + kStages;
  uint64_t* acce = accf + 1;
  uint64_t* fin = acce + 1;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(fin + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int WPROD = kEpi / 32, WMMA = WPROD + 1;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; s++) {
      tc::mbar_init(&full[s], 1);
      tc::mbar_init(&empty[s], 1);
    }
    tc::mbar_init(accf, 1);
    tc::mbar_init(acce, kEpi);
    tc::mbar_init(fin, 1);
    tc::fence_barrier_init();
  }
  if (warp == 0) {
    tc::tmem_alloc(tmem_slot, 512);
    tc::tmem_relinquish();
  }
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  pdl_trigger();
  pdl_wait();
  const int total = job.sched.total();
  const int nslab = job.cplx && *job.cplx == 0 ? job.nslab_real : job.nslab;
  auto slabs = [&](int z, int& s0) {
    s0 = job.slab_split ? z * job.slab_split : 0;
    return job.slab_split ? min(job.slab_split, nslab - s0) : nslab;
  };

  if (warp == WPROD && lane == 0) {
    // ---- producer: one bulk copy per operand and stage (all slices)
    int g = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < total && ok; t += gridDim.x) {
      int z, mt, nt, s0;
      job.sched.decode(t, z, mt, nt);
      const int ns = slabs(z, s0);
      const int8_t* pa =
          job.a + ((long long)(z * job.a_tiles + job.m_tile + mt) * nslab + s0) * kABytes;
      const int8_t* pb =
          job.b + ((long long)(z * job.b_tiles + job.n_tile + nt) * nslab + s0) * kBBytes;
      for (int k = 0; k < ns; k++, g++) {
        const int s = g % kStages;
        if (!tc::mbar_wait(&empty[s], ((g / kStages) & 1) ^ 1)) {
          atomicOr(err, tc::ERR_TIMEOUT_PRODUCER);
          ok = false;
          break;
        }
        tc::mbar_expect_tx(&full[s], kStageBytes);
        bulk_load(stA(s), pa + (long long)k * kABytes, kABytes, &full[s]);
        bulk_load(stB(s), pb + (long long)k * kBBytes, kBBytes, &full[s]);
      }
    }
    for (int q = max(0, g - kStages); q < g; q++)
      tc::mbar_wait_drain(&full[q % kStages], (q / kStages) & 1);
  } else if (warp == WMMA && lane == 0) {
    // ---- MMA issuer
    int g = 0, li = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < total && ok; t += gridDim.x, li++) {
      int z, mt, nt, s0;
      job.sched.decode(t, z, mt, nt);
      const int ns = slabs(z, s0);
      if (!tc::mbar_wait(acce, (li & 1) ^ 1)) {
        atomicOr(err, tc::ERR_TIMEOUT_MMA);
        break;
      }
      tc::tc_fence_after();
      for (int k = 0; k < ns; k++, g++) {
        const int s = g % kStages;
        if (!tc::mbar_wait(&full[s], (g / kStages) & 1)) {
          atomicOr(err, tc::ERR_TIMEOUT_MMA);
          ok = false;
          break;
        }
        tc::tc_fence_after();
        const uint64_t ad = tc::sdesc_k<kSlab>(tc::smem_u32(stA(s)));
        const uint64_t bd = tc::sdesc_k<kSlab>(tc::smem_u32(stB(s)));
        if (k == 0)
          mma_step<ND, true>(tmem, ad, bd);
        else
          mma_step<ND, false>(tmem, ad, bd);
#pragma unroll
        for (int u = 1; u < kSlab / 32; u++) mma_step<ND, false>(tmem, ad + 2 * u, bd + 2 * u);
        tc::umma_commit(&empty[s]);
      }
      if (!ok) break;
      tc::umma_commit(accf);
    }
    tc::umma_commit(fin);
    tc::mbar_wait_drain(fin, 0);
  }
  if (warp < WPROD) {
    // ---- accumulators -> FP64 -> functor: warpgroup wg takes 32 of the 64 columns
    const int wg = warp >> 2, wq = warp & 3;
    const int row = wq * 32 + lane;
    const uint32_t trow = tmem + ((uint32_t)(wq * 32) << 16) + wg * 32;
    int li = 0;
    long long marked = -1;
    for (int t = blockIdx.x; t < total; t += gridDim.x, li++) {
      int z, mt, nt;
      job.sched.decode(t, z, mt, nt);
      const int m = mt * kBM + row, n0 = nt * kBN + wg * 32;
      const long long ra = (long long)z * job.a_rows + job.m_tile * kBM;
      const long long rb = (long long)z * job.b_rows + job.n_tile * kBN;
      const double sa = m < job.M ? job.sa[ra + m] : 0.0;
      const double sb = n0 + lane < job.N ? job.sb[rb + n0 + lane] : 0.0;   // lane's column
      // the warp goes on as one (the TMEM loads and shuffles below are warp-wide)
      if (!__all_sync(0xffffffffu, tc::mbar_wait(accf, li & 1))) {
        if (lane == 0) atomicOr(err, tc::ERR_TIMEOUT_EPILOGUE);
        break;
      }
      tc::tc_fence_after();
      double v[32];
      if (ND == 7 && (job.slab_split ? job.slab_split : nslab) <= kShortSlabs)
        drain<ND, ND == 7>(trow, v);
      else
        drain<ND, false>(trow, v);
      tc::tc_fence_before();
      tc::mbar_arrive(acce);
      const double sa30 = sa * 0x1p-30;   // (v sa) sb: no product of scales leaves the range
      // the columns this warp marked last need no second look (all CTAs share their line)
      const long long col = rb + n0 + lane;
      if (job.ok && !__all_sync(0xffffffffu, col == marked || n0 + lane >= job.N)) {
        // magnitudes by their high words (a bound rounded up); a NaN limit (a NaN scale of A,
        // the only source of NaN here) lets none pass
        const double lim = kFloor * job.top[job.a_rows ? z : 0];
        const unsigned lw = lim == lim ? (unsigned)__double2hiint(lim) + (lim > 0.0) : 0xffffffffu;
        unsigned any = 0;
#pragma unroll
        for (int c = 0; c < 32; c++) {
          v[c] *= sa30;
          any |= (((unsigned)__double2hiint(v[c]) & 0x7fffffffu) >= lw ? 1u : 0u) << c;
          v[c] *= __shfl_sync(0xffffffffu, sb, c);
        }
        any = __reduce_or_sync(0xffffffffu, any);
        if ((any >> lane & 1) && n0 + lane < job.N && sb == sb && col != marked) {
          job.ok[col] = 1;
          marked = col;
        }
      } else {
#pragma unroll
        for (int c = 0; c < 32; c++) v[c] = v[c] * sa30 * __shfl_sync(0xffffffffu, sb, c);
      }
      epi(z, m, n0, v);
    }
  }
  tc::tc_fence_before();
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(tmem, 512);
}

// ------------------------------------------------------------------ host side
// C[z][m][n] = sum_k A[z][m0 + m][k] B[z][n0 + n][k], m < M, n < N, with m0 = 128 m_tile and
// n0 = 64 n_tile.  An operand of batch 1 is shared by all batches.  slab_split > 0: z counts
// K ranges of slab_split slabs of an unbatched product instead of batches.
struct Gemm {
  const Slices *a, *b;
  int M, N, nbatch;
  int m_tile = 0, n_tile = 0;
  int slab_split = 0;
  bool m_fast = true;
  bool mark = true;            // marks of B rows, where the operands carry them
  const int* cplx = nullptr;   // as Job::cplx, Job::nslab_real
  int nslab_real = 0;
};

// ND: accumulators (7, or 8 for the digit pairs one step further down).
template <int ND, class Epi>
cudaError_t launch(const Gemm& g, const Epi& epi, int* err, cudaStream_t st) {
  if (g.M <= 0 || g.N <= 0 || g.nbatch <= 0) return cudaSuccess;
  if (g.a->tile != kBM || g.b->tile != kBN || g.a->nslab != g.b->nslab) return cudaErrorInvalidValue;
  auto kern = oz_gemm_kernel<ND, Epi>;
  static DeviceAttr attr;
  cudaError_t e = attr.ensure(kSmem, [kern](size_t b) {
    return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)b);
  });
  if (e != cudaSuccess) return e;
  Job j;
  j.a = g.a->d;
  j.b = g.b->d;
  j.sa = g.a->scale;
  j.sb = g.b->scale;
  j.top = g.a->top;
  j.ok = g.slab_split || !g.mark || !g.a->top ? nullptr : g.b->ok;   // K splits: checked summed
  const bool ab = !g.slab_split && g.a->batch > 1, bb = !g.slab_split && g.b->batch > 1;
  j.a_rows = ab ? g.a->rows : 0;
  j.b_rows = bb ? g.b->rows : 0;
  j.a_tiles = ab ? g.a->tiles() : 0;
  j.b_tiles = bb ? g.b->tiles() : 0;
  j.sched = tc::TileSched{(g.M + kBM - 1) / kBM, (g.N + kBN - 1) / kBN, g.nbatch,
                          g.m_fast ? 1 : 0, 0};
  j.M = g.M;
  j.N = g.N;
  j.m_tile = g.m_tile;
  j.n_tile = g.n_tile;
  j.nslab = g.a->nslab;
  j.slab_split = g.slab_split;
  j.cplx = g.cplx;
  j.nslab_real = g.nslab_real;
  const int total = j.sched.total();
  const int grid = total < tc::sm_count() ? total : tc::sm_count();
  return pdl_launch(kern, grid, kThreads, kSmem, st, j, epi, err);
}

}  // namespace oz
