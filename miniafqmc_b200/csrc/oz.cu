// FP64 contraction stages on the int8 tensor cores: operand splitting, the products of
// oz_gemm.cuh and the kernels around them.
#include <cooperative_groups.h>
#include <algorithm>
#include <cmath>
#include <vector>

#include "afq_kernels.h"
#include "afq_oz.h"
#include "oz_gemm.cuh"

namespace afq {

using oz::kS;
using oz::Slices;

struct OzState {
  OzInit in{};
  std::vector<void*> allocs;
  char* block = nullptr;    // rest of the last shared block
  size_t block_left = 0;
  size_t budget = 0;        // device memory that further groups of products may take
  int* err = nullptr;
  // per product (OzProduct) the walkers whose result the digits did not hold; per walker
  // whether the last exchange's did not, and whether the propagation's did not on the way
  unsigned long long* redone = nullptr;
  int *ex_gate = nullptr, *prop_bad = nullptr;
  // exchange: rows (c, a) of Lh per spin, columns (w, b, re | im) of G, T = Lh_c Gc_w^T of a
  // chunk of Cholesky vectors and walkers
  bool lreal = false;
  Slices lx[2], gx;
  double* T = nullptr;
  double* norms = nullptr;  // half of |T|^2 per partial sum
  double *sa2 = nullptr, *sb = nullptr;   // exchange_holds: of lx, of gx per spin
  int ex_w = 0, ex_c = 0;   // walkers and Cholesky vectors per chunk
  bool exchange = false;
  // products with G: static operand rows, G rows (w, re | im) shared by the sites, partial
  // products of the K splits
  struct GSite {
    bool on = false;
    Slices a;
    int rows = 0, splits = 1, slab_split = 0;
  } gs[OZ_NG];
  bool greal = false;
  Slices gb;
  double* part = nullptr;
  long long part_ld = 0;
  // vHS: Spvn rows ik, X rows (w, re | im)
  bool vhs = false, sreal = false;
  Slices sp, xb;
  // propagation: Propg1, vHS and the walker columns (j, re | im) for either
  bool prop = false, preal = false;
  Slices pa, va, pb, tb;
};

namespace {

// Device memory of the state: small buffers share blocks (a cudaMalloc costs 0.1 to 0.2 ms,
// most of a small system's set-up).
constexpr size_t kBlock = 32u << 20;
template <class T>
cudaError_t oz_alloc(OzState* o, T** p, size_t count) {
  const size_t bytes = (sizeof(T) * (count ? count : 1) + 255) / 256 * 256;
  if (bytes <= o->block_left) {
    *p = reinterpret_cast<T*>(o->block);
    o->block += bytes;
    o->block_left -= bytes;
    return cudaSuccess;
  }
  void* q = nullptr;
  const bool shared = bytes <= kBlock / 2;
  const cudaError_t e = cudaMalloc(&q, shared ? kBlock : bytes);
  if (e != cudaSuccess) return e;
  o->allocs.push_back(q);
  *p = static_cast<T*>(q);
  if (shared) {
    o->block = static_cast<char*>(q) + bytes;
    o->block_left = kBlock - bytes;
  }
  return e;
}

// Slices of `batch` x `rows` rows of K digits-worth of entries, in tiles of `tile` rows;
// checked (Slices::top, Slices::ok) when `st` is given.
struct Checked {
  cudaStream_t st;
};
constexpr size_t ok_bytes(size_t rows) { return (rows + 15) / 16 * 16; }
cudaError_t alloc_slices(OzState* o, Slices* s, int tile, int rows, int batch, int K,
                         const Checked* checked = nullptr) {
  s->tile = tile;
  s->rows = rows;
  s->batch = batch;
  s->nslab = (K + oz::kSlab - 1) / oz::kSlab;
  cudaError_t e = oz_alloc(o, &s->d, s->bytes());
  if (e == cudaSuccess) e = oz_alloc(o, &s->scale, (size_t)rows * batch);
  if (!checked || e != cudaSuccess) return e;
  if (tile == oz::kBM) {
    e = oz_alloc(o, &s->top, batch);
    if (e == cudaSuccess) e = cudaMemsetAsync(s->top, 0, sizeof(double) * batch, checked->st);
  } else {
    const size_t bytes = ok_bytes((size_t)rows * batch);
    e = oz_alloc(o, &s->ok, bytes);
    if (e == cudaSuccess) e = cudaMemsetAsync(s->ok, 1, bytes, checked->st);
  }
  return e;
}

// ------------------------------------------------------------ operand splitting
// Row r of the source starts at src + (r / per) hi + (r % per) lo (in elements).
struct RowSrc {
  const z_t* p;
  int per;
  long long hi, lo;
  AFQ_D const z_t* row(int r) const { return p + (r / per) * hi + (r % per) * lo; }
};
// How complex source rows become operand rows: kReal: one row of real parts; kPairs: one
// row of (re, im) pairs (a complex A operand); kSplitRe: rows 2r = re, 2r + 1 = im (B of a
// real A); kSplitCx: rows 2r = (re, -im) pairs, 2r + 1 = (im, re) pairs (B of a complex A).
// kDouble: rows of real doubles (RowSrc strides in doubles).
enum { kReal, kPairs, kSplitRe, kSplitCx, kDouble };

struct RowScale {
  double s1, s2, scale;   // q = rn(x s1 s2) = rn(x 2^(55 - e)), scale = 2^e
};
AFQ_D RowScale row_scale(unsigned long long maxbits) {
  RowScale r{0.0, 0.0, 0.0};
  if (maxbits == 0) return r;
  const double mx = __longlong_as_double((long long)maxbits);
  int e;
  // inf, nan, or a scale whose products could leave the range (2^900, 2^-900)
  if (maxbits >= 0x7830000000000000ull || maxbits < 0x07B0000000000000ull) {
    r.scale = __longlong_as_double(0x7ff8000000000000LL);
    return r;
  }
  const double f = frexp(mx, &e);
  if (f > 0.99) e++;   // the leading digit stays below 128 after carries
  const int h = (55 - e) / 2;
  r.s1 = ldexp(1.0, h);
  r.s2 = ldexp(1.0, 55 - e - h);
  r.scale = ldexp(1.0, e);
  return r;
}
// Digits of four entries, four packed bytes per slice.
AFQ_D void digits4(const double (&x)[4], const RowScale& s, unsigned (&out)[kS]) {
#pragma unroll
  for (int i = 0; i < kS; i++) out[i] = 0;
#pragma unroll
  for (int e = 0; e < 4; e++) {
    long long q = __double2ll_rn(x[e] * s.s1 * s.s2);
#pragma unroll
    for (int i = kS - 1; i > 0; i--) {
      const int d = (int)(signed char)(q & 0xff);
      out[i] |= (unsigned)(d & 0xff) << (8 * e);
      q = (q - d) >> 8;
    }
    out[0] |= (unsigned)((int)q & 0xff) << (8 * e);
  }
}
AFQ_D unsigned long long absbits(double x) {
  return (unsigned long long)__double_as_longlong(x) & 0x7fffffffffffffffull;
}

// Digits of a source row from entry k0 on (K entries; KD digits stored, past the row's end
// zeros), thread t of nt, four digits per step.
template <int MODE>
AFQ_D void slice_row(const z_t* __restrict__ p, int K, const Slices& s, int rb, int r0,
                     const RowScale& s0, const RowScale& s1, int kd0, int kd1, int t, int nt) {
  const z_t zero = zmk(0, 0);
  const double* pd = reinterpret_cast<const double*>(p);
  unsigned q[kS];
  const int plane = s.tile * oz::kSlab;
  for (int k = kd0 + 4 * t; k < kd1; k += 4 * nt) {
    int8_t* o = s.d + oz::slice_offset(s, rb, r0, k);
    // rows 2r and 2r + 1 share a row pair of the swizzle: the second is 64 bytes on
    if constexpr (MODE == kDouble) {
      double x[4];
#pragma unroll
      for (int e = 0; e < 4; e++) x[e] = k + e < K ? pd[k + e] : 0.0;
      digits4(x, s0, q);
#pragma unroll
      for (int i = 0; i < kS; i++) *reinterpret_cast<unsigned*>(o + i * plane) = q[i];
    } else if constexpr (MODE == kReal || MODE == kSplitRe) {
      double x[4], y[4];
#pragma unroll
      for (int e = 0; e < 4; e++) {
        const z_t v = k + e < K ? p[k + e] : zero;
        x[e] = v.x;
        y[e] = v.y;
      }
      digits4(x, s0, q);
#pragma unroll
      for (int i = 0; i < kS; i++) *reinterpret_cast<unsigned*>(o + i * plane) = q[i];
      if constexpr (MODE == kSplitRe) {
        digits4(y, s1, q);
#pragma unroll
        for (int i = 0; i < kS; i++) *reinterpret_cast<unsigned*>(o + i * plane + oz::kSlab) = q[i];
      }
    } else {   // two complex entries
      const z_t a = k / 2 < K ? p[k / 2] : zero, b = k / 2 + 1 < K ? p[k / 2 + 1] : zero;
      const double x[4] = {a.x, MODE == kPairs ? a.y : -a.y, b.x, MODE == kPairs ? b.y : -b.y};
      digits4(x, s0, q);
#pragma unroll
      for (int i = 0; i < kS; i++) *reinterpret_cast<unsigned*>(o + i * plane) = q[i];
      if constexpr (MODE == kSplitCx) {
        const double y[4] = {a.y, a.x, b.y, b.x};
        digits4(y, s0, q);
#pragma unroll
        for (int i = 0; i < kS; i++) *reinterpret_cast<unsigned*>(o + i * plane + oz::kSlab) = q[i];
      }
    }
  }
}
// Largest magnitudes (as bits) of the real (m0) and imaginary (m1) parts of entries
// [k0, k1), thread t of nt.
template <int MODE>
AFQ_D void row_max(const z_t* __restrict__ p, int k0, int k1, int t, int nt,
                   unsigned long long& m0, unsigned long long& m1) {
  m0 = m1 = 0;
  const double* pd = reinterpret_cast<const double*>(p);
  for (int k = k0 + t; k < k1; k += nt) {
    if constexpr (MODE == kDouble) {
      m0 = max(m0, absbits(pd[k]));
    } else {
      const z_t v = p[k];
      m0 = max(m0, absbits(v.x));
      m1 = max(m1, absbits(v.y));
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    m0 = max(m0, __shfl_xor_sync(0xffffffffu, m0, o));
    m1 = max(m1, __shfl_xor_sync(0xffffffffu, m1, o));
  }
}
// The check of a product whose result columns are sliced as the next one's operand (rows of
// `per` a batch): column r, whose largest entry is factor^-1 times the product's, against
// kFloor x (largest A scale) x (its own B scale old[2r], old[2r + 1]); bad [batch].
struct RowCheck {
  const double* top = nullptr;
  int batched = 0, per = 1;
  const double* old = nullptr;
  double factor = 1.0;
  int* bad = nullptr;
};
AFQ_D void check_row(const RowCheck& c, int r, unsigned long long maxbits) {
  if (!c.top) return;
  const int z = r / c.per;
  const double lim = oz::kFloor * c.top[c.batched ? z : 0] * fmax(c.old[2 * r], c.old[2 * r + 1]);
  if (!(c.factor * __longlong_as_double((long long)maxbits) >= lim)) c.bad[z] = 1;   // NaN: bad
}
// The row's scale and its mark: a zero row is ok as it is.
AFQ_D void put_scale(const Slices& s, long long i, double scale) {
  if (s.ok) {
    s.ok[i] = scale == 0.0;
  }
  s.scale[i] = scale;
}
template <int MODE>
AFQ_D void put_scales(const Slices& s, int rb, int r0, const RowScale& s0, const RowScale& s1) {
  const long long i = (long long)rb * s.rows + r0;
  put_scale(s, i, s0.scale);
  if constexpr (MODE == kSplitRe || MODE == kSplitCx) put_scale(s, i + 1, s1.scale);
  if (s.top)   // non-negative scales (and NaN above them) order like their bits
    atomicMax(reinterpret_cast<unsigned long long*>(s.top + rb),
              (unsigned long long)__double_as_longlong(s0.scale));
}
AFQ_D const z_t* src_row(const RowSrc& src, int r, bool dbl) {
  if (!dbl) return src.row(r);
  return reinterpret_cast<const z_t*>(reinterpret_cast<const double*>(src.p) +
                                      (r / src.per) * src.hi + (r % src.per) * src.lo);
}

// One warp per source row: the row's maximum, then its digits (the second read hits L1 or
// L2).  Memory bound: 16 bytes read per complex entry, 14 (28 for kSplitCx) written.
template <int MODE>
__global__ void __launch_bounds__(256)
slice_kernel(RowSrc src, int nrows, int K, Slices s, RowCheck chk) {
  pdl_trigger();
  pdl_wait();
  constexpr bool TWO = MODE == kSplitRe || MODE == kSplitCx;
  const int lane = threadIdx.x & 31, r = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (r >= nrows) return;
  const z_t* p = src_row(src, r, MODE == kDouble);
  unsigned long long m0, m1;
  row_max<MODE>(p, 0, K, lane, 32, m0, m1);
  if (lane == 0) check_row(chk, r, max(m0, m1));
  if constexpr (MODE == kPairs || MODE == kSplitCx) m0 = m1 = max(m0, m1);
  const RowScale s0 = row_scale(m0), s1 = row_scale(m1);
  const int rb = r / s.per_batch(TWO), r0 = (r - rb * s.per_batch(TWO)) * (TWO ? 2 : 1);
  if (lane == 0) put_scales<MODE>(s, rb, r0, s0, s1);
  slice_row<MODE>(p, K, s, rb, r0, s0, s1, 0, s.nslab * oz::kSlab, lane, 32);
}
// One cluster of 8 CTAs per source row (long rows: the 2nN entries of a walker's density
// matrix, 590 KB at 384 orbitals): each CTA takes an eighth of the row and reads the others'
// maxima from their shared memory.
constexpr int kSliceCluster = 8;
template <int MODE>
__global__ void __cluster_dims__(kSliceCluster, 1, 1) __launch_bounds__(256)
slice_cluster_kernel(RowSrc src, int K, Slices s, RowCheck chk) {
  pdl_trigger();
  pdl_wait();
  constexpr bool TWO = MODE == kSplitRe || MODE == kSplitCx;
  constexpr bool PAIR = MODE == kPairs || MODE == kSplitCx;   // two digits per entry
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  __shared__ unsigned long long red[2][8], mx[2];
  const int r = blockIdx.x / kSliceCluster, part = blockIdx.x % kSliceCluster;
  const z_t* p = src_row(src, r, MODE == kDouble);
  const int Kp = s.nslab * oz::kSlab;
  const int per = (s.nslab + kSliceCluster - 1) / kSliceCluster * oz::kSlab;
  const int kd0 = min(Kp, part * per), kd1 = min(Kp, kd0 + per);
  unsigned long long m0, m1;
  row_max<MODE>(p, PAIR ? kd0 / 2 : kd0, min(K, PAIR ? kd1 / 2 : kd1), threadIdx.x, 256, m0, m1);
  if ((threadIdx.x & 31) == 0) {
    red[0][threadIdx.x >> 5] = m0;
    red[1][threadIdx.x >> 5] = m1;
  }
  __syncthreads();
  if (threadIdx.x < 2) {
    unsigned long long m = 0;
    for (int i = 0; i < 8; i++) m = max(m, red[threadIdx.x][i]);
    mx[threadIdx.x] = m;
  }
  cl.sync();
  m0 = m1 = 0;
#pragma unroll
  for (int q = 0; q < kSliceCluster; q++) {
    const unsigned long long* o = cl.map_shared_rank(mx, q);
    m0 = max(m0, o[0]);
    m1 = max(m1, o[1]);
  }
  cl.sync();   // every CTA's shared memory stays until all have read it
  if (part == 0 && threadIdx.x == 0) check_row(chk, r, max(m0, m1));
  if constexpr (PAIR) m0 = m1 = max(m0, m1);
  const RowScale s0 = row_scale(m0), s1 = row_scale(m1);
  const int rb = r / s.per_batch(TWO), r0 = (r - rb * s.per_batch(TWO)) * (TWO ? 2 : 1);
  if (part == 0 && threadIdx.x == 0) put_scales<MODE>(s, rb, r0, s0, s1);
  slice_row<MODE>(p, K, s, rb, r0, s0, s1, kd0, kd1, threadIdx.x, 256);
}

// Slices nrows source rows of K entries into `s` (its first rows).  Rows above 1024 entries
// get a cluster each (16 rows of 2048 entries at one warp a row would fill two SMs).
template <int MODE>
cudaError_t slice_rows(const RowSrc& src, int nrows, int K, const Slices& s, cudaStream_t st,
                       const RowCheck& chk = RowCheck()) {
  if (nrows <= 0) return cudaSuccess;
  if (K > 1024)
    return pdl_launch(slice_cluster_kernel<MODE>, nrows * kSliceCluster, 256, 0, st, src, K, s, chk);
  return pdl_launch(slice_kernel<MODE>, (nrows + 7) / 8, 256, 0, st, src, nrows, K, s, chk);
}

// Rows of an A operand (TWO = false: one row of reals, or of pairs) or of a B operand (re and
// im rows, or pair rows) as found on the device: *cplx == 0 means a real A operand.  `s`
// describes the complex form; the real one has nslab_real slabs in the same buffers.
template <bool TWO>
__global__ void __launch_bounds__(256)
slice_found_kernel(RowSrc src, int nrows, int K, Slices s, const int* __restrict__ cplx,
                   int nslab_real) {
  pdl_trigger();
  pdl_wait();
  const int lane = threadIdx.x & 31, r = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (r >= nrows) return;
  const z_t* p = src.row(r);
  const bool cx = *cplx != 0;
  if (!cx) s.nslab = nslab_real;
  unsigned long long m0, m1;
  row_max<kPairs>(p, 0, K, lane, 32, m0, m1);
  if (cx) m0 = m1 = max(m0, m1);
  const RowScale s0 = row_scale(m0), s1 = row_scale(m1);
  constexpr int REAL = TWO ? kSplitRe : kReal, CPLX = TWO ? kSplitCx : kPairs;
  const int r0 = TWO ? 2 * r : r, Kp = s.nslab * oz::kSlab;
  if (lane == 0) put_scales<REAL>(s, 0, r0, s0, s1);
  if (cx)
    slice_row<CPLX>(p, K, s, 0, r0, s0, s1, 0, Kp, lane, 32);
  else
    slice_row<REAL>(p, K, s, 0, r0, s0, s1, 0, Kp, lane, 32);
}

// X [nchol][nw] -> rows (w, re | im): a cluster of 8 CTAs per 32 walkers, lanes on walkers
// (coalesced reads of X's rows), 16 digits per thread and store.
template <bool REALA>
__global__ void __cluster_dims__(kSliceCluster, 1, 1) __launch_bounds__(256)
slice_x_kernel(const z_t* __restrict__ X, int nc, int nw, Slices s) {
  pdl_trigger();
  pdl_wait();
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  __shared__ unsigned long long red[2][8][32], mx[2][32];
  const int lane = threadIdx.x & 31, wy = threadIdx.x >> 5;
  const int w = blockIdx.x / kSliceCluster * 32 + lane, part = blockIdx.x % kSliceCluster;
  unsigned long long m0 = 0, m1 = 0;
  if (w < nw)
    for (int c = part * 8 + wy; c < nc; c += 8 * kSliceCluster) {
      const z_t v = X[(long long)c * nw + w];
      m0 = max(m0, absbits(v.x));
      m1 = max(m1, absbits(v.y));
    }
  red[0][wy][lane] = m0;
  red[1][wy][lane] = m1;
  __syncthreads();
  if (wy < 2) {
    unsigned long long m = 0;
    for (int i = 0; i < 8; i++) m = max(m, red[wy][i][lane]);
    mx[wy][lane] = m;
  }
  cl.sync();
  m0 = m1 = 0;
#pragma unroll
  for (int q = 0; q < kSliceCluster; q++) {
    const unsigned long long* o = cl.map_shared_rank(&mx[0][0], q);
    m0 = max(m0, o[lane]);
    m1 = max(m1, o[32 + lane]);
  }
  cl.sync();   // every CTA's shared memory stays until all have read it
  if (w >= nw) return;
  if (!REALA) m0 = m1 = max(m0, m1);
  const RowScale s0 = row_scale(m0), s1 = row_scale(m1);
  if (part == 0 && wy == 0) {
    put_scale(s, 2 * w, s0.scale);
    put_scale(s, 2 * w + 1, s1.scale);
  }
  const int plane = s.tile * oz::kSlab, Kp = s.nslab * oz::kSlab;
  constexpr int NE = REALA ? 16 : 8;   // source entries per 16 digits
  for (int k = 16 * (part * 8 + wy); k < Kp; k += 16 * 8 * kSliceCluster) {
    z_t v[NE];
#pragma unroll
    for (int e = 0; e < NE; e++) {
      const int c = (REALA ? k : k / 2) + e;
      v[e] = c < nc ? X[(long long)c * nw + w] : zmk(0, 0);
    }
    int8_t* o = s.d + oz::slice_offset(s, 0, 2 * w, k);
#pragma unroll
    for (int row = 0; row < 2; row++) {
      unsigned q[4][kS];
#pragma unroll
      for (int g = 0; g < 4; g++) {
        double x[4];
#pragma unroll
        for (int e = 0; e < 4; e++) {
          if (REALA) {
            x[e] = row ? v[4 * g + e].y : v[4 * g + e].x;
          } else {   // row 0: (re, -im) pairs, row 1: (im, re) pairs
            const z_t z = v[2 * g + e / 2];
            x[e] = row ? (e & 1 ? z.x : z.y) : (e & 1 ? -z.y : z.x);
          }
        }
        digits4(x, row ? s1 : s0, q[g]);
      }
#pragma unroll
      for (int i = 0; i < kS; i++)
        *reinterpret_cast<uint4*>(o + i * plane + row * oz::kSlab) =
            make_uint4(q[0][i], q[1][i], q[2][i], q[3][i]);
    }
  }
}

// W [nw][N][n2] -> Wt [nw][n2][N]; clears top [nw] and bad [nw].
__global__ void __launch_bounds__(256)
transpose_kernel(const z_t* __restrict__ W, int N, int n2, z_t* __restrict__ Wt, double* top,
                 int* bad) {
  pdl_trigger();
  pdl_wait();
  if (threadIdx.x == 0 && blockIdx.x == 0 && blockIdx.y == 0) {
    top[blockIdx.z] = 0.0;
    bad[blockIdx.z] = 0;
  }
  __shared__ z_t t[32][33];
  const int w = blockIdx.z, k0 = blockIdx.x * 32, j0 = blockIdx.y * 32;
  const z_t* src = W + (long long)w * N * n2;
  z_t* dst = Wt + (long long)w * N * n2;
  const int x = threadIdx.x & 31, y = threadIdx.x >> 5;
  for (int i = y; i < 32; i += 8)
    if (k0 + i < N && j0 + x < n2) t[i][x] = src[(long long)(k0 + i) * n2 + j0 + x];
  __syncthreads();
  for (int i = y; i < 32; i += 8)
    if (j0 + i < n2 && k0 + x < N) dst[(long long)(j0 + i) * N + k0 + x] = t[x][i];
}

__global__ void oz_check_imag_kernel(const z_t* __restrict__ src, long long count, int* flag) {
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < count;
       e += (long long)gridDim.x * blockDim.x)
    if (src[e].y != 0.0) *flag = 1;
}
// Which of the operands are real (synchronises the stream; null operands count as real).
struct RealCheck {
  const z_t* p;
  long long count;
  bool real;
};
cudaError_t check_real(OzState* o, RealCheck* c, int n, cudaStream_t st) {
  int* flags = nullptr;
  int host[8] = {};
  cudaError_t e = oz_alloc(o, &flags, 8);
  if (e == cudaSuccess) e = cudaMemsetAsync(flags, 0, 8 * sizeof(int), st);
  for (int i = 0; i < n && e == cudaSuccess; i++)
    if (c[i].p) {
      oz_check_imag_kernel<<<148 * 8, 256, 0, st>>>(c[i].p, c[i].count, flags + i);
      e = cudaGetLastError();
    }
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(host, flags, n * sizeof(int), cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  for (int i = 0; i < n; i++) c[i].real = host[i] == 0;
  return e;
}

// ------------------------------------------------------------ exchange
// Row-major FP64 output C[m][n] in 32-byte stores (ld a multiple of 4 and C 32-byte aligned;
// the columns from N up to ld take the zeros of columns outside the operand).  A lane owns a
// row, so a store touches 32 rows: whole 32-byte sectors halve the write transactions of
// 16-byte stores, which outlasted the next tile's MMAs (768 x 12288 x 384: 86.5 us with
// 16-byte stores, 62.3 us without any).
struct EpiRows {
  double* C;
  long long ld;
  int M;
  AFQ_D void operator()(int, int m, int n0, const double* v) const {
    if (m >= M) return;
    double* p = C + (long long)m * ld + n0;
#pragma unroll
    for (int i = 0; i < 32; i += 4)
      if (n0 + i < ld) oz::store4(p + i, v[i], v[i + 1], v[i + 2], v[i + 3]);
  }
};

// Partial products of a K split: part[z][m][n] (ld a multiple of 4).
struct EpiPart {
  double* C;
  long long ld, sz;
  int M;
  AFQ_D void operator()(int z, int m, int n0, const double* v) const {
    EpiRows{C + z * sz, ld, M}(0, m, n0, v);
  }
};
// vHS: row m = ik, columns (w, re | im); lanes on consecutive ik.
struct EpiV {
  z_t* V;
  long long N2;
  int nw;
  AFQ_D void operator()(int, int m, int n0, const double* v) const {
    if (m >= N2) return;
    const int w0 = n0 / 2;
#pragma unroll
    for (int i = 0; i < 16; i++)
      if (w0 + i < nw) V[(w0 + i) * N2 + m] = zmk(v[2 * i], v[2 * i + 1]);
  }
};
// Propagation, columns (j, re | im) of walker z, S and T [nw][2n][N] (lanes on consecutive
// rows).  k = 0: S = v.  k > 0: T = (i / k) v, S += T, T stored unless last.
struct EpiChain {
  z_t *S, *T;
  int N, n2, k, last;
  AFQ_D void operator()(int z, int m, int n0, const double* v) const {
    if (m >= N) return;
    const int j0 = n0 / 2;
    const long long o = ((long long)z * n2 + j0) * N + m;
    if (k == 0) {
#pragma unroll
      for (int i = 0; i < 16; i++)
        if (j0 + i < n2) S[o + (long long)i * N] = zmk(v[2 * i], v[2 * i + 1]);
      return;
    }
    const double f = 1.0 / (double)k;
#pragma unroll
    for (int i = 0; i < 16; i++) {
      if (j0 + i >= n2) break;
      const z_t t = zmk(-f * v[2 * i + 1], f * v[2 * i]);
      z_t* s = S + o + (long long)i * N;
      *s = zadd(*s, t);
      if (!last) T[o + (long long)i * N] = t;
    }
  }
};
// W[z][m][j]: a lane owns an orbital row (32-byte stores; 2n is even).
struct EpiW {
  z_t* W;
  int N, n2;
  AFQ_D void operator()(int z, int m, int n0, const double* v) const {
    if (m >= N) return;
    const int j0 = n0 / 2;
    double* p = reinterpret_cast<double*>(W + ((long long)z * N + m) * n2 + j0);
#pragma unroll
    for (int i = 0; i < 32; i += 4)
      if (j0 + i / 2 < n2) oz::store4(p + i, v[i], v[i + 1], v[i + 2], v[i + 3]);
  }
};
// out[r][w] = sum over the K splits of the partial products, in order; marks of B's rows
// (w, re | im) as in oz_gemm_kernel.  `lanes` (a power of two up to 32) walkers by 256 / lanes
// rows per CTA and pass, so that a thread keeps its walker and a CTA writes each mark once: all
// CTAs write the same few lines, and one store per element made 1536 x 128 sums take 165 us
// longer.
__global__ void __launch_bounds__(256)
part_sum_kernel(const double* __restrict__ part, long long ld, long long sz, int splits, int rows,
                int nw, int lanes, z_t* __restrict__ out, const double* __restrict__ top,
                Slices b) {
  pdl_trigger();
  pdl_wait();
  __shared__ unsigned char mark[64];
  if (threadIdx.x < 64) mark[threadIdx.x] = 0;
  __syncthreads();
  const int wl = threadIdx.x % lanes, w0 = blockIdx.y * lanes, w = w0 + wl, rpb = 256 / lanes;
  if (w < nw) {
    const double lim = oz::kFloor * *top;
    const double lre = lim * b.scale[2 * w], lim_im = lim * b.scale[2 * w + 1];
    bool re = false, im = false;   // NaN marks nothing
    for (int r = blockIdx.x * rpb + threadIdx.x / lanes; r < rows; r += gridDim.x * rpb) {
      const z_t* p = reinterpret_cast<const z_t*>(part + r * ld) + w;
      z_t t = p[0];
      for (int q = 1; q < splits; q++) t = zadd(t, p[q * (sz / 2)]);
      out[(long long)r * nw + w] = t;
      re |= fabs(t.x) >= lre;
      im |= fabs(t.y) >= lim_im;
    }
    if (re) mark[2 * wl] = 1;
    if (im) mark[2 * wl + 1] = 1;
  }
  __syncthreads();
  const int i = threadIdx.x;
  if (i < 2 * lanes && mark[i] && 2 * w0 + i < 2 * nw) b.ok[2 * w0 + i] = 1;
}

// W_w <- P (sum_k (i V_w)^k / k!) P W_w on the FP64 pipe for the walkers whose columns miss a
// mark (ok [nw][2 n2], of the last product; bad: of those before) or when a wait timed out: a CTA per (walker, eight columns), a row per thread and pass, terms and sum in
// the scratch S, T [nw][n2][N] (columns contiguous), from Wt, the walkers as they were.  Sums
// over k in order.  All but always it reads 2 n2 marks and returns.
constexpr int kRedoCols = 8;
__global__ void __launch_bounds__(256)
prop_redo_kernel(const z_t* __restrict__ P, const z_t* __restrict__ V, const z_t* __restrict__ Wt,
                 z_t* S, z_t* T, z_t* __restrict__ W, int N, int n2, int order,
                 const unsigned char* __restrict__ ok, const int* __restrict__ bad,
                 const int* __restrict__ err, unsigned long long* redone) {
  pdl_trigger();
  pdl_wait();
  const int w = blockIdx.y, tid = threadIdx.x, j0 = blockIdx.x * kRedoCols;
  bool redo = *err != 0 || bad[w];
  for (int i = tid; i < 2 * n2; i += 256) redo |= !ok[(long long)w * 2 * n2 + i];
  if (!__syncthreads_or(redo)) return;
  if (tid == 0 && blockIdx.x == 0) atomicAdd(redone, 1ull);
  const int cols = min(kRedoCols, n2 - j0);
  const long long c0 = ((long long)w * n2 + j0) * N;
  z_t *s = S + c0, *t = T + c0;
  // rows i, i + 256, ... of M times the columns B (visible to the CTA), handed to put(i, j, v)
  auto product = [&](const z_t* M, const z_t* B, auto put) {
    for (int i = tid; i < N; i += 256) {
      z_t acc[kRedoCols];
#pragma unroll
      for (int j = 0; j < kRedoCols; j++) acc[j] = zmk(0, 0);
      const z_t* m = M + (long long)i * N;
      for (int k = 0; k < N; k++)
#pragma unroll
        for (int j = 0; j < kRedoCols; j++)
          if (j < cols) zfma(acc[j], m[k], B[(long long)j * N + k]);
#pragma unroll
      for (int j = 0; j < kRedoCols; j++)
        if (j < cols) put(i, j, acc[j]);
    }
    __syncthreads();
  };
  const z_t* Vw = V + (long long)w * N * N;
  product(P, Wt + c0, [&](int i, int j, z_t v) { s[(long long)j * N + i] = v; });
  // a term replaces the last one once every row is formed: until then it waits in W's columns
  z_t* Ww = W + (long long)w * N * n2 + j0;
  for (int k = 1; k <= order; k++) {
    const z_t f = zmk(0.0, 1.0 / (double)k);
    product(Vw, k == 1 ? s : t, [&](int i, int j, z_t v) { Ww[(long long)i * n2 + j] = zmul(f, v); });
    for (int i = tid; i < N; i += 256)
      for (int j = 0; j < cols; j++) {
        const z_t v = Ww[(long long)i * n2 + j];
        const long long o = (long long)j * N + i;
        t[o] = v;
        s[o] = zadd(s[o], v);
      }
    __syncthreads();
  }
  product(P, s, [&](int i, int j, z_t v) { Ww[(long long)i * n2 + j] = v; });
}

// Kpart[w][s][c] = tr(T T), T the n x n block of (c, w) in the chunk's product (rows
// row0 + c n + a, columns w n + b).  One CTA per block, which passes through shared memory
// by asynchronous copies: few registers and 16 n (n + 1) bytes a CTA keep several CTAs per
// SM, whose copies overlap the others' sums (the block is fresh in L2).
// norms[w][s][c] = half of |T|^2: the real parts of even columns and the imaginary parts of odd
// ones (one multiply-add an entry beside the trace's four; all of it and the scales' norms in
// this kernel took 4% of the exchange of 32 electrons at 128 orbitals).  What bounds the kernel:
// the blocks' latency at five CTAs an SM for n = 48 (counters: issue slots 41%, L1 40%, waiting
// for loads first).
constexpr int kTraceThreads = 128;
__global__ void __launch_bounds__(kTraceThreads)
trace_kernel(const z_t* __restrict__ T, int n, long long ld, int row0, int c_first,
             z_t* __restrict__ Kpart, int nblk, int w_first, int s, double* __restrict__ norms) {
  pdl_trigger();
  pdl_wait();
  extern __shared__ __align__(16) unsigned char tr_smem[];
  z_t* t = reinterpret_cast<z_t*>(tr_smem);   // [n][n + 1]
  static_assert(kTraceThreads == 128, "four partial sums");
  __shared__ double red[4][3];
  const int c = blockIdx.x, w = blockIdx.y, tid = threadIdx.x;
  const z_t* src = T + (row0 + (long long)c * n) * ld + (long long)w * n;
  // entry (a, b), stepping kTraceThreads entries at a time
  const int da = kTraceThreads / n, db = kTraceThreads - da * n;
  const int a0 = tid / n, b0 = tid - a0 * n;
  for (int a = a0, b = b0; a < n;) {
    cp_async16(t + a * (n + 1) + b, src + (long long)a * ld + b, 16);
    a += da;
    if ((b += db) >= n) {
      b -= n;
      a++;
    }
  }
  cp_async_commit();
  const int lane = tid & 31, warp = tid >> 5;
  cp_async_wait<0>();
  __syncthreads();
  z_t sum = zmk(0, 0);
  double f2 = 0.0;
  for (int a = a0, b = b0; a < n;) {
    const z_t x = t[a * (n + 1) + b];
    zfma(sum, x, t[b * (n + 1) + a]);
    const double h = b & 1 ? x.y : x.x;
    f2 = fma(h, h, f2);
    a += da;
    if ((b += db) >= n) {
      b -= n;
      a++;
    }
  }
  sum = warp_zsum(sum);
  f2 = warp_sum(f2);
  if (lane == 0) {
    red[warp][0] = sum.x;
    red[warp][1] = sum.y;
    red[warp][2] = f2;
  }
  __syncthreads();
  if (tid < 3) {
    const double r = (red[0][tid] + red[2][tid]) + (red[1][tid] + red[3][tid]);
    const long long o = ((long long)(w_first + w) * 2 + s) * nblk + c_first + c;
    if (tid < 2)
      reinterpret_cast<double*>(Kpart + o)[tid] = r;
    else
      norms[o] = r;
  }
}

// Whether the digits hold a walker's exchange energy (one CTA of 128 threads): the error of an
// entry of T is about 2^-56 sqrt(K) of its row's times its column's scale, so where the walker's
// sum of |T|^2 (norms [2 nchol], halves) reaches kFloor^2 of the sum of those products squared,
// the energy has 2^-49 sqrt(K) of the former.  sa2 [2]: sum of the squares of all row scales;
// sb + s stride: the walker's 2n column scales, per spin.
AFQ_D bool exchange_holds(const double* __restrict__ norms, int count, const double* sa2,
                          const double* __restrict__ sb, long long stride, int n, z_t* red) {
  z_t q = zmk(0, 0);
  for (int i = threadIdx.x; i < count; i += 128) q.x += norms[i];
  for (int i = threadIdx.x; i < 4 * n; i += 128) {
    const int s = i >= 2 * n;
    const double b = sb[s * stride + i - s * 2 * n];
    q.y = fma(b * b, sa2[s], q.y);
  }
  q = block_zsum(q, red);
  return 2.0 * q.x >= oz::kFloor * oz::kFloor * q.y;   // false for NaN
}
__global__ void __launch_bounds__(128)
exchange_verdict_kernel(const double* __restrict__ norms, int count, const double* sa2,
                        const double* __restrict__ sb, long long stride, int n,
                        const int* __restrict__ err, int* __restrict__ gate,
                        unsigned long long* redone) {
  pdl_trigger();
  pdl_wait();
  __shared__ z_t red[4];
  const int w = blockIdx.x;
  const bool ok = exchange_holds(norms + (long long)w * count, count, sa2, sb + 2LL * w * n, stride,
                                 n, red) && *err == 0;
  if (threadIdx.x == 0) {
    gate[w] = !ok;
    if (!ok) atomicAdd(redone, 1ull);
  }
}
// sa2[s] += sum of the squares of `count` scales of spin s (blockIdx.x, one CTA each).
__global__ void __launch_bounds__(1024)
scale_norm_kernel(const double* __restrict__ s0, const double* __restrict__ s1, int count,
                  double* sa2) {
  pdl_trigger();
  pdl_wait();
  __shared__ z_t red[32];
  const double* p = blockIdx.x ? s1 : s0;
  z_t q = zmk(0, 0);
  for (int i = threadIdx.x; i < count; i += 1024) q.x = fma(p[i], p[i], q.x);
  q = block_zsum(q, red);
  if (threadIdx.x == 0) sa2[blockIdx.x] += q.x;
}

}  // namespace

namespace {

// Whether the next group of allocations fits what is left of the budget: a sixth of the device
// memory free at set-up for all digits and workspaces together, so that other handles find
// nearly the room they did without them (C4 with 128 walkers takes 3.6 GB).
constexpr size_t kMemoryShare = 6;
bool fits(OzState* o, cudaError_t e, size_t need) {
  if (e != cudaSuccess || need > o->budget) return false;
  o->budget -= need;
  return true;
}
size_t slice_bytes(long long rows, long long K) { return (size_t)kS * (rows + 128) * (K + 64); }

// Which exchange products take the digits: blocks of n^2 N >= 3100 at 32 orbitals and more (a
// shorter K leaves the drain and T's way through memory), where a block's multiply-adds on the
// FP64 pipe take longer than its trace.  Energies of 256 walkers without and with, us: 10
// electrons at 32 orbitals, 128 vectors 238 > 183; 16 at 48, 192 vectors 661 > 412; 8 at 64, 256
// vectors 357 > 264; 6 at 128, 512 vectors 664 > 444; 8 at 32, 128 vectors 142 < 160.
// Smaller blocks: the digits take about 32 us and 1.2 ns a block, the FP64 kernel's waves 0.4 us
// an orbital and 0.3 us for each of a warp's turns at the traces of its 96 / n by 96 / n blocks
// (1 electron at 55 orbitals, 120 vectors, 213 walkers 339 > 123; 2 at 64, 128 vectors 256 / 512
// walkers 131 > 125 / 134 < 197; 4 at 64, 256 vectors 16 / 256 walkers 97 > 64 / 151 < 206).
bool exchange_pays(int N, int n, int nc, int nw) {
  if (N >= 32 && (double)n * n * N >= 3100.0) return true;
  const int g = 96 / n;
  const double blocks = 2.0 * nc * nw;
  const double ctas = 2.0 * ((nc + g - 1) / g) * ((nw + g - 1) / g);
  const double wave = 0.3 * g * ((g + 7) / 8) * ((n * n + 31) / 32) + 0.4 * N + 4.0;
  return (double)n * n * N < 3100.0 &&
         32.0 + 1.2e-3 * blocks < wave * std::ceil(ctas / (2.0 * tc::sm_count()));
}
cudaError_t create_exchange(OzState* o, cudaStream_t st) {
  const OzInit& in = o->in;
  const int N = in.N, n = in.n, nc = in.nchol, nw = in.nw;
  const long long NAK = 2LL * n * N;
  cudaError_t e = cudaSuccess;
  const int K = o->lreal ? N : 2 * N;
  if (K > oz::kMaxK || !exchange_pays(N, n, nc, nw)) return e;
  // chunk of T: walkers first (in whole 64-column tiles, up to 32 MB per 128 rows), then
  // Cholesky vectors, up to 64 MB (half of L2)
  const long long cap = 64LL << 20;
  o->ex_w = (int)std::min<long long>(nw, std::max(32LL, (32LL << 20) / (16LL * 128 * n) / 32 * 32));
  const long long per_c = 16LL * (o->ex_w + 1) * n * n;
  o->ex_c = (int)std::max(1LL, std::min<long long>(nc, cap / per_c));
  int whole = oz::kBM;   // Cholesky vectors that fill whole row tiles, within 1.25 caps
  while (whole > 1 && (whole / 2 * n) % oz::kBM == 0) whole /= 2;
  if (o->ex_c < nc && whole * per_c <= cap + cap / 4)
    o->ex_c = (int)((cap + cap / 4) / per_c / whole) * whole;
  const size_t tb = per_c * o->ex_c + 256LL * 16 * (o->ex_w + 1) * n;   // whole row tiles
  const size_t norms = (size_t)nw * 2 * nc;
  if (!fits(o, e, 2 * slice_bytes((long long)nc * n, K) + slice_bytes(2LL * nw * n, K) + tb +
                      sizeof(double) * (norms + 4LL * nw * n)))
    return e;
  for (int s = 0; s < 2 && e == cudaSuccess; s++) {
    e = alloc_slices(o, &o->lx[s], oz::kBM, nc * n, 1, K);
    if (e != cudaSuccess) break;
    const RowSrc src{in.Lh + (long long)s * n * N, n, NAK, N};
    e = o->lreal ? slice_rows<kReal>(src, nc * n, N, o->lx[s], st)
                 : slice_rows<kPairs>(src, nc * n, N, o->lx[s], st);
  }
  if (e == cudaSuccess) e = alloc_slices(o, &o->gx, oz::kBN, 2 * nw * n, 1, K);
  if (e == cudaSuccess) e = oz_alloc(o, &o->T, tb / sizeof(double));
  if (e == cudaSuccess) e = oz_alloc(o, &o->norms, norms);
  if (e == cudaSuccess) e = oz_alloc(o, &o->ex_gate, nw);
  if (e == cudaSuccess) e = oz_alloc(o, &o->sb, 4LL * nw * n);
  if (e == cudaSuccess) e = oz_alloc(o, &o->sa2, 2);
  if (e == cudaSuccess) e = cudaMemsetAsync(o->sa2, 0, 2 * sizeof(double), st);
  if (e == cudaSuccess)
    e = pdl_launch(scale_norm_kernel, 2, 1024, 0, st, o->lx[0].scale, o->lx[1].scale, nc * n, o->sa2);
  o->exchange = e == cudaSuccess;
  return e;
}

// Products with G.  K splits fill the SMs when the output tiles do not (and bound a split's
// K for the int32 accumulators), at least two slabs each.  From a K of 2nN = 256 on, where the
// FP64 pipe's serial sums take longer than four launches (vbias of 256 vectors, 16 walkers: K =
// 128 14.8 < 18.2 us, 192 19.0 < 20.3, 256 24.6 > 19.9, 512 41.5 > 22.1, 2048 150 > 22), and from
// 96 nonzeros a row and 64 walkers, where the CSR product does (K = 2048: 43 nonzeros, 16 walkers
// 18.9 < 22.2; 102 nonzeros 30.9 > 22.1, 64 walkers 66 > 26).
cudaError_t create_gsites(OzState* o, cudaStream_t st) {
  const OzInit& in = o->in;
  const int nw = in.nw;
  const long long NAK = 2LL * in.n * in.N;
  const long long rows[OZ_NG] = {in.nchol, in.nchol, NAK};
  const long long nnz[OZ_NG] = {in.SpvnT_nnz, in.nchol * NAK, in.Vakbl_nnz};
  const z_t* src[OZ_NG] = {in.SpvnT, in.Lh, in.Vakbl};
  for (int i = 0; i < OZ_NG; i++)
    if (NAK < 256 || nnz[i] * ((nw + 63) / 64) < 96 * rows[i]) src[i] = nullptr;
  cudaError_t e = cudaSuccess;
  size_t need = 0;
  for (int i = 0; i < OZ_NG; i++)
    if (src[i]) need += slice_bytes(rows[i], NAK);
  const int K = (int)(o->greal ? NAK : 2 * NAK);
  if (!o->greal) need *= 2;
  o->part_ld = (2LL * nw + 3) / 4 * 4;
  size_t pmax = 0;
  for (int i = 0; i < OZ_NG; i++) {
    if (!src[i]) continue;
    OzState::GSite& g = o->gs[i];
    g.rows = (int)rows[i];
    const int nslab = (K + oz::kSlab - 1) / oz::kSlab;
    const int tiles = ((g.rows + oz::kBM - 1) / oz::kBM) * ((2 * nw + oz::kBN - 1) / oz::kBN);
    const int least = (K + oz::kMaxK - 1) / oz::kMaxK;
    const int sp = std::max(least, std::min(std::max(1, tc::sm_count() / tiles), nslab / 2));
    g.slab_split = (nslab + sp - 1) / sp;
    g.splits = (nslab + g.slab_split - 1) / g.slab_split;
    pmax = std::max(pmax, (size_t)(g.splits * rows[i] * o->part_ld));
  }
  if (!pmax || !fits(o, e, need + slice_bytes(2 * nw, K) + 8 * pmax)) return e;
  const Checked ck{st};
  if (e == cudaSuccess) e = alloc_slices(o, &o->gb, oz::kBN, 2 * nw, 1, K, &ck);
  if (e == cudaSuccess) e = oz_alloc(o, &o->part, pmax);
  for (int i = 0; i < OZ_NG && e == cudaSuccess; i++) {
    if (!src[i]) continue;
    OzState::GSite& g = o->gs[i];
    e = alloc_slices(o, &g.a, oz::kBM, g.rows, 1, K, &ck);
    const RowSrc rs{src[i], 1, NAK, 0};
    if (e == cudaSuccess)
      e = o->greal ? slice_rows<kReal>(rs, g.rows, (int)NAK, g.a, st)
                   : slice_rows<kPairs>(rs, g.rows, (int)NAK, g.a, st);
    g.on = e == cudaSuccess;
  }
  return e;
}

// vHS as a dense product.  The CSR kernel does nnz x nw real (complex) multiply-adds at about
// 2.9e12 (1.4e12) a second (C4's 45.3 M nonzeros x 128 walkers: 3.89 ms; 0.42 M x 256: 90
// us), a tile slab here takes about 1.0 us of one SM under load plus 2 us per tile and 15 us
// of launches (C4 x 128 walkers: 32 tiles of 24 slabs per SM, 0.93 ms): the smaller of the
// two estimates.
cudaError_t create_vhs(OzState* o, cudaStream_t st) {
  const OzInit& in = o->in;
  const long long N2 = (long long)in.N * in.N;
  cudaError_t e = cudaSuccess;
  o->sreal = in.Spvn_r != nullptr;
  if ((!in.Spvn_r && !in.Spvn) || N2 > (1LL << 30)) return e;
  const int K = o->sreal ? in.nchol : 2 * in.nchol;
  if (K > oz::kMaxK) return e;
  const double csr = (double)in.spvn_nnz * in.nw / (o->sreal ? 2.9e12 : 1.45e12);
  const long long tiles = (N2 + oz::kBM - 1) / oz::kBM * ((2LL * in.nw + oz::kBN - 1) / oz::kBN);
  const int sms = tc::sm_count();
  const double dense = 15e-6 + (double)((tiles + sms - 1) / sms) *
                                   (2e-6 + 1.0e-6 * ((K + oz::kSlab - 1) / oz::kSlab));
  if (dense >= csr) return e;
  if (!fits(o, e, slice_bytes(N2, K) + slice_bytes(2LL * in.nw, K))) return e;
  const Checked ck{st};
  e = alloc_slices(o, &o->sp, oz::kBM, (int)N2, 1, K, &ck);
  if (e == cudaSuccess) e = alloc_slices(o, &o->xb, oz::kBN, 2 * in.nw, 1, K, &ck);
  if (e == cudaSuccess)
    e = o->sreal ? slice_rows<kDouble>(
                       RowSrc{reinterpret_cast<const z_t*>(in.Spvn_r), 1, in.nchol, 0}, (int)N2,
                       in.nchol, o->sp, st)
                 : slice_rows<kPairs>(RowSrc{in.Spvn, 1, in.nchol, 0}, (int)N2, in.nchol, o->sp, st);
  o->vhs = e == cudaSuccess;
  return e;
}

// Propagation: where the chain's estimate is below 0.97 of the FP64 pipe's (prop_zgemm_us), us:
// 110 for the launches of splitting, products and checks, the busiest SM's tiles (2.74 and 1.42 a
// slab each), 2.6e-6 a digit split and 1.5e-3 a row; within 8% (rms) of 190 measured chains of 50 to
// 330 orbitals, 3e8 to 2e10 operations a product.  Not for chains that run in one launch.  FP64
// pipe and digits, us: 64 orbitals, 1431 walkers of 16+16 electrons 626 < 1439; 96, 318 of 32+32 638
// < 815; 105, 3000 of 24+24 8825 > 6140; 121, 986 of 2+2 1521 > 745; 128, 119 of 32+32 492 > 365; 136, 113
// of 30+30 558 < 617; 160, 25 of 48+48 261 < 311, 76 662 > 630; 200, 20 of 40+40 312 > 277; 384, 4 of 48+48
// 248 < 264, 9 548 > 344.
double prop_digits_us(int N, int n2, int nw, int order, bool preal) {
  auto slabs = [](int K) { return (K + oz::kSlab - 1) / oz::kSlab; };
  const int sms = tc::sm_count();
  const double tiles = (double)((N + oz::kBM - 1) / oz::kBM) *
                       ((2 * n2 + oz::kBN - 1) / oz::kBN) * nw;
  const double busiest = std::ceil(tiles / sms), kp = oz::kSlab * slabs(2 * N);
  const double rows = (double)nw * (N + (order + 1.0) * n2);
  return 110.0 + busiest * (order * (2.74 + 1.42 * slabs(2 * N)) +
                            2.0 * (2.74 + 1.42 * slabs(preal ? N : 2 * N))) +
         2.6e-6 * kp * nw * (N + (order + 1.0) * 2 * n2) + 1.5e-3 * rows;
}
cudaError_t create_propagate(OzState* o, cudaStream_t st) {
  const OzInit& in = o->in;
  const int N = in.N, n2 = 2 * in.n, nw = in.nw;
  cudaError_t e = cudaSuccess;
  if (2 * N > oz::kMaxK || nw > 65535 || prop_small_fits(N, n2, nw, in.order) ||
      prop_digits_us(N, n2, nw, in.order, o->preal) >= 0.97 * prop_zgemm_us(N, n2, nw, in.order))
    return e;
  const int Kp = o->preal ? N : 2 * N;
  if (!fits(o, e, slice_bytes(N, Kp) + (size_t)nw * (slice_bytes(N, 2 * N) + slice_bytes(2 * n2, Kp) +
                                                  slice_bytes(2 * n2, 2 * N))))
    return e;
  const Checked ck{st};
  if (e == cudaSuccess) e = alloc_slices(o, &o->pa, oz::kBM, N, 1, Kp, &ck);
  if (e == cudaSuccess) e = alloc_slices(o, &o->va, oz::kBM, N, nw, 2 * N, &ck);
  if (e == cudaSuccess) e = alloc_slices(o, &o->pb, oz::kBN, 2 * n2, nw, Kp, &ck);
  if (e == cudaSuccess) e = alloc_slices(o, &o->tb, oz::kBN, 2 * n2, nw, 2 * N);
  if (e == cudaSuccess) e = oz_alloc(o, &o->prop_bad, nw);
  if (e == cudaSuccess)
    e = o->preal ? slice_rows<kReal>(RowSrc{in.P, 1, N, 0}, N, N, o->pa, st)
                 : slice_rows<kPairs>(RowSrc{in.P, 1, N, 0}, N, N, o->pa, st);
  o->prop = e == cudaSuccess;
  return e;
}

// The trace kernel's shared memory for n x n blocks.
cudaError_t trace_attr(int n, size_t* smem) {
  *smem = sizeof(z_t) * n * (n + 1);
  static DeviceAttr attr;
  return attr.ensure(*smem, [](size_t b) {
    cudaError_t r = cudaFuncSetAttribute(trace_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)b);
    if (r == cudaSuccess)
      r = cudaFuncSetAttribute(trace_kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                               (int)cudaSharedmemCarveoutMaxShared);
    return r;
  });
}

// ek[w] = 1/2 sum of the walker's partial sums in a fixed order; gate[w]: the digits do not
// hold it or a wait timed out.
__global__ void __launch_bounds__(128)
ek_sum_kernel(const z_t* __restrict__ part, const double* __restrict__ norms, int count,
              const double* sa2, const double* __restrict__ sb, long long stride, int n,
              const int* __restrict__ err, int* __restrict__ gate, z_t* __restrict__ ek) {
  pdl_trigger();
  pdl_wait();
  __shared__ z_t red[4];
  const int w = blockIdx.x;
  z_t s = zmk(0, 0);
  for (int q = threadIdx.x; q < count; q += 128) s = zadd(s, part[(long long)w * count + q]);
  s = block_zsum(s, red);
  const bool ok = exchange_holds(norms + (long long)w * count, count, sa2, sb + 2LL * w * n, stride,
                                 n, red) && *err == 0;
  if (threadIdx.x == 0) {
    ek[w] = zscale(s, 0.5);
    gate[w] = !ok;
  }
}

// Chunks of oz_exchange_buffers: w walkers and c Cholesky vectors at a time; false when even
// one walker and one vector exceed the scratch.
bool buffers_plan(const OzBuffers& b, int N, int n, int nc, int nw, int* w, int* c) {
  const long long Kp = (2LL * N + oz::kSlab - 1) / oz::kSlab * oz::kSlab;
  if (2 * N > oz::kMaxK || n > 96) return false;
  const long long grows = std::min<long long>(b.g_bytes / (kS * Kp), b.g_rows) / oz::kBN * oz::kBN;
  const long long arows = std::min<long long>(b.a_bytes / (kS * Kp), b.a_rows) / oz::kBM * oz::kBM;
  long long cw = std::min<long long>(nw, grows / (2 * n));
  cw = std::min<long long>(cw, b.parts / (2LL * nc));
  if (cw < 1 || arows < n) return false;
  cw = (nw + (nw + cw - 1) / cw - 1) / ((nw + cw - 1) / cw);   // chunks of even size
  // Cholesky vectors: as many row tiles as T and A hold, of these the count whose tiles fill
  // the last wave of SMs best
  const long long ld = (2 * cw * n + 3) / 4 * 4, nt = (2 * cw * n + oz::kBN - 1) / oz::kBN;
  const long long most = std::min<long long>(arows, b.t_bytes / (8 * ld)) / oz::kBM;
  long long best = 0;
  double eff = -1.0;
  for (long long m = 1; m <= most; m++) {
    const long long t = m * nt, sms = tc::sm_count();
    const double f = (double)t / (double)((t + sms - 1) / sms * sms + sms / 4);
    if (f > eff) {
      eff = f;
      best = m;
    }
  }
  const long long cc = best * oz::kBM / n;
  if (cc < 1) return false;
  *w = (int)cw;
  *c = (int)std::min<long long>(cc, nc);
  return true;
}

}  // namespace

// As exchange_pays, and n walkers times electrons >= 200 for the splitting of Lh, which every
// call repeats (16 electrons at 200 orbitals: 8 walkers 336 < 378 us, 33 walkers 984 > 475; at 384,
// 2 walkers 588 < 1228), from 1.5e9 real operations (two waves of tiles).
bool oz_exchange_buffers_fit(const OzBuffers& b, int N, int n, int nc, int nw) {
  int w, c;
  return n >= 4 && N >= 40 && (double)n * n * N >= 5000.0 && (double)n * nw >= 200.0 &&
         16.0 * nc * n * (double)n * N * nw >= 1.5e9 && buffers_plan(b, N, n, nc, nw, &w, &c);
}

cudaError_t oz_exchange_buffers(const OzBuffers& b, const z_t* Lh, const z_t* Gc, int N, int n,
                                int nc, int nw, z_t* ek, cudaStream_t st) {
  int cw = 0, cc = 0;
  if (!buffers_plan(b, N, n, nc, nw, &cw, &cc)) return cudaErrorInvalidValue;
  const long long NAK = 2LL * n * N;
  size_t smem = 0;
  cudaError_t e = trace_attr(n, &smem);
  if (e == cudaSuccess) e = cudaMemsetAsync(b.flags, 0, 2 * sizeof(int), st);
  if (e == cudaSuccess) e = cudaMemsetAsync(b.sa2, 0, 2 * sizeof(double), st);
  if (e != cudaSuccess) return e;
  int *err = b.flags, *cplx = b.flags + 1;
  oz_check_imag_kernel<<<148 * 8, 256, 0, st>>>(Lh, nc * NAK, cplx);
  Slices a, g;
  a.d = b.a;
  a.scale = b.a_scale;
  a.tile = oz::kBM;
  a.batch = 1;
  g = a;
  g.d = b.g;
  g.scale = b.g_scale;
  g.tile = oz::kBN;
  a.nslab = g.nslab = (2 * N + oz::kSlab - 1) / oz::kSlab;
  const int nslab_real = (N + oz::kSlab - 1) / oz::kSlab;
  for (int w0 = 0; w0 < nw; w0 += cw) {
    const int w = std::min(cw, nw - w0);
    g.rows = 2 * w * n;
    const long long ld = (2LL * w * n + 3) / 4 * 4;
    for (int s = 0; s < 2; s++) {
      g.scale = b.g_scale + (long long)s * b.g_rows;
      const RowSrc gs{Gc + w0 * NAK + (long long)s * n * N, n, NAK, N};
      pdl_launch(slice_found_kernel<true>, (w * n + 7) / 8, 256, 0, st, gs, w * n, N, g, cplx,
                 nslab_real);
      for (int c0 = 0; c0 < nc; c0 += cc) {
        const int c = std::min(cc, nc - c0);
        a.rows = c * n;
        const RowSrc as{Lh + c0 * NAK + (long long)s * n * N, n, NAK, N};
        pdl_launch(slice_found_kernel<false>, (c * n + 7) / 8, 256, 0, st, as, c * n, N, a, cplx,
                   nslab_real);
        if (w0 == 0)
          pdl_launch(scale_norm_kernel, 1, 1024, 0, st, a.scale, nullptr, c * n, b.sa2 + s);
        oz::Gemm gm{&a, &g, c * n, 2 * w * n, 1};
        gm.cplx = cplx;
        gm.nslab_real = nslab_real;
        if ((e = oz::launch<7>(gm, EpiRows{b.T, ld, c * n}, err, st)) != cudaSuccess) return e;
        pdl_launch(trace_kernel, dim3(c, w), kTraceThreads, smem, st,
                   reinterpret_cast<const z_t*>(b.T), n, ld / 2, 0, c0, b.part, nc, 0, s, b.norms);
      }
    }
    pdl_launch(ek_sum_kernel, w, 128, 0, st, b.part, b.norms, 2 * nc, b.sa2, b.g_scale, b.g_rows,
               n, err, b.gate + w0, ek + w0);
  }
  return cudaGetLastError();
}

cudaError_t oz_create(const OzInit& in, OzState** out, cudaStream_t st) {
  *out = nullptr;
  OzState* o = new OzState();
  o->in = in;
  size_t total_b = 0;
  cudaError_t e = cudaMemGetInfo(&o->budget, &total_b);
  o->budget /= kMemoryShare;
  if (e == cudaSuccess) e = oz_alloc(o, &o->err, 1);
  if (e == cudaSuccess) e = cudaMemsetAsync(o->err, 0, sizeof(int), st);
  if (e == cudaSuccess) e = oz_alloc(o, &o->redone, OZ_NPRODUCTS);
  if (e == cudaSuccess)
    e = cudaMemsetAsync(o->redone, 0, OZ_NPRODUCTS * sizeof(unsigned long long), st);
  const long long NAK = 2LL * in.n * in.N;
  RealCheck rc[4] = {{in.Lh, in.nchol * NAK, true},
                     {in.SpvnT, in.nchol * NAK, true},
                     {in.Vakbl, NAK * NAK, true},
                     {in.P, (long long)in.N * in.N, true}};
  if (e == cudaSuccess) e = check_real(o, rc, 4, st);
  o->lreal = rc[0].real;
  o->greal = rc[0].real && rc[1].real && rc[2].real;   // one format of G for its three products
  o->preal = rc[3].real;
  if (e == cudaSuccess && in.Lh && in.n <= 64) e = create_exchange(o, st);
  if (e == cudaSuccess) e = create_gsites(o, st);
  if (e == cudaSuccess) e = create_vhs(o, st);
  if (e == cudaSuccess) e = create_propagate(o, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e == cudaErrorMemoryAllocation) {   // the FP64 pipe's kernels need none of this
    cudaGetLastError();
    oz_destroy(o);
    return cudaSuccess;
  }
  if (e != cudaSuccess) {
    oz_destroy(o);
    return e;
  }
  *out = o;
  return cudaSuccess;
}

void oz_destroy(OzState* o) {
  if (!o) return;
  for (void* p : o->allocs) cudaFree(p);
  delete o;
}

OzGate oz_gate(const OzState* o, int product) {
  const Slices& b = product == OZ_VHS ? o->xb : o->gb;
  OzGate g;
  g.ok = reinterpret_cast<const uint4*>(b.ok);
  g.n16 = (int)(ok_bytes(b.rows) / 16);
  g.err = o->err;
  g.redone = o->redone + product;
  g.walkers = o->in.nw;
  return g;
}
const int* oz_exchange_gate(const OzState* o) { return o->ex_gate; }

cudaError_t oz_redone(const OzState* o, unsigned long long* redone) {
  return cudaMemcpy(redone, o->redone, OZ_NPRODUCTS * sizeof(unsigned long long),
                    cudaMemcpyDeviceToHost);
}

bool oz_has_gsite(const OzState* o, int site) { return o && o->gs[site].on; }
int oz_gsite_launches() { return 3; }

cudaError_t oz_gsite(OzState* o, int site, const z_t* Gc, z_t* out, cudaStream_t st) {
  const OzState::GSite& g = o->gs[site];
  const int nw = o->in.nw, NAK = 2 * o->in.n * o->in.N;
  const RowSrc src{Gc, 1, NAK, 0};
  cudaError_t e = o->greal ? slice_rows<kSplitRe>(src, nw, NAK, o->gb, st)
                           : slice_rows<kSplitCx>(src, nw, NAK, o->gb, st);
  if (e != cudaSuccess) return e;
  const long long sz = g.rows * o->part_ld;
  oz::Gemm gm{&g.a, &o->gb, g.rows, 2 * nw, g.splits, 0, 0, g.slab_split};
  e = oz::launch<7>(gm, EpiPart{o->part, o->part_ld, sz, g.rows}, o->err, st);
  if (e != cudaSuccess) return e;
  int lanes = 1;
  while (lanes < 32 && lanes < nw) lanes *= 2;
  const int ny = (nw + lanes - 1) / lanes, rpb = 256 / lanes;
  const int nx = std::min((g.rows + rpb - 1) / rpb, std::max(1, tc::sm_count() * 16 / ny));
  return pdl_launch(part_sum_kernel, dim3(nx, ny), 256, 0, st, o->part, o->part_ld, sz, g.splits,
                    g.rows, nw, lanes, out, g.a.top, o->gb);
}

bool oz_has_vhs(const OzState* o) { return o && o->vhs; }

cudaError_t oz_vhs(OzState* o, const z_t* X, z_t* vHS, cudaStream_t st) {
  const int nw = o->in.nw, nc = o->in.nchol;
  const int grid = (nw + 31) / 32 * kSliceCluster;
  if (o->sreal)
    pdl_launch(slice_x_kernel<true>, grid, 256, 0, st, X, nc, nw, o->xb);
  else
    pdl_launch(slice_x_kernel<false>, grid, 256, 0, st, X, nc, nw, o->xb);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  const long long N2 = (long long)o->in.N * o->in.N;
  oz::Gemm g{&o->sp, &o->xb, (int)N2, 2 * nw, 1};
  g.m_fast = false;   // the CTAs that share an Spvn tile run together
  return oz::launch<7>(g, EpiV{vHS, N2, nw}, o->err, st);
}

bool oz_has_propagate(const OzState* o) { return o && o->prop; }
int oz_propagate_launches(const OzState* o) { return 3 + 2 * (2 + o->in.order); }

cudaError_t oz_propagate(OzState* o, const z_t* P, z_t* W, const z_t* vHS, z_t* S, z_t* T,
                         z_t* Wt, cudaStream_t st) {
  const int N = o->in.N, n2 = 2 * o->in.n, nw = o->in.nw, order = o->in.order;
  pdl_launch(transpose_kernel, dim3((N + 31) / 32, (n2 + 31) / 32, nw), 256, 0, st, W, N, n2, Wt,
             o->va.top, o->prop_bad);
  cudaError_t e = cudaGetLastError();
  auto pslice = [&](const z_t* src, const RowCheck& chk) {   // walker columns as Propg1's B operand
    const RowSrc rs{src, 1, N, 0};
    return o->preal ? slice_rows<kSplitRe>(rs, nw * n2, N, o->pb, st, chk)
                    : slice_rows<kSplitCx>(rs, nw * n2, N, o->pb, st, chk);
  };
  // each product is checked where its result is sliced (the last term with the sum it went
  // into, the last product by its marks)
  RowCheck chk;
  chk.per = n2;
  chk.bad = o->prop_bad;
  if (e == cudaSuccess) e = pslice(Wt, RowCheck());
  oz::Gemm g{&o->pa, &o->pb, N, 2 * n2, nw};
  g.mark = false;
  if (e == cudaSuccess) e = oz::launch<8>(g, EpiChain{S, T, N, n2, 0, 0}, o->err, st);
  chk.top = o->pa.top;
  chk.old = o->pb.scale;
  if (e == cudaSuccess && order > 0)
    e = slice_rows<kPairs>(RowSrc{vHS, 1, N, 0}, nw * N, N, o->va, st);
  oz::Gemm gv{&o->va, &o->tb, N, 2 * n2, nw};
  for (int k = 1; k <= order && e == cudaSuccess; k++) {
    e = slice_rows<kSplitCx>(RowSrc{k == 1 ? S : T, 1, N, 0}, nw * n2, N, o->tb, st, chk);
    if (e == cudaSuccess)
      e = oz::launch<8>(gv, EpiChain{S, T, N, n2, k, k == order}, o->err, st);
    chk.top = o->va.top;
    chk.batched = 1;
    chk.old = o->tb.scale;
    chk.factor = k;   // T_k = (i / k) V T_{k-1}
  }
  if (e == cudaSuccess) e = pslice(S, chk);
  g.mark = true;
  if (e == cudaSuccess) e = oz::launch<8>(g, EpiW{W, N, n2}, o->err, st);
  if (e != cudaSuccess) return e;
  return pdl_launch(prop_redo_kernel, dim3((n2 + kRedoCols - 1) / kRedoCols, nw), 256, 0, st, P,
                    vHS, Wt, S, T, W, N, n2, order, o->pb.ok, o->prop_bad, o->err,
                    o->redone + OZ_PROPAGATE);
}

bool oz_has_exchange(const OzState* o, int nwalk) { return o && o->exchange && nwalk <= o->in.nw; }

int oz_exchange_launches(const OzState* o, int nwalk) {
  const int cw = (nwalk + o->ex_w - 1) / o->ex_w;
  const int cc = (o->in.nchol + o->ex_c - 1) / o->ex_c;
  return 3 + 4 * cw * cc;
}

cudaError_t oz_exchange(OzState* o, const z_t* Gc, int nwalk, z_t* Kpart, int nblk,
                        cudaStream_t st) {
  const int N = o->in.N, n = o->in.n, nc = o->in.nchol;
  const long long NAK = 2LL * n * N;
  size_t smem = 0;
  cudaError_t e = trace_attr(n, &smem);
  for (int s = 0; s < 2 && e == cudaSuccess; s++) {
    const RowSrc src{Gc + (long long)s * n * N, n, NAK, N};
    Slices gx = o->gx;
    gx.scale = o->sb + 2LL * s * o->in.nw * n;
    e = o->lreal ? slice_rows<kSplitRe>(src, nwalk * n, N, gx, st)
                 : slice_rows<kSplitCx>(src, nwalk * n, N, gx, st);
    for (int w0 = 0; w0 < nwalk && e == cudaSuccess; w0 += o->ex_w) {
      const int w = std::min(o->ex_w, nwalk - w0);
      for (int c0 = 0; c0 < nc && e == cudaSuccess; c0 += o->ex_c) {
        const int c = std::min(o->ex_c, nc - c0);
        // the row tiles that hold the chunk's rows [c0 n, (c0 + c) n)
        const int t0 = c0 * n / oz::kBM, row0 = c0 * n - t0 * oz::kBM;
        oz::Gemm g{&o->lx[s], &gx, row0 + c * n, 2 * w * n, 1, t0, 2 * w0 * n / oz::kBN};
        const long long ld = (2LL * w * n + 3) / 4 * 4;
        EpiRows epi{o->T, ld, row0 + c * n};
        if ((e = oz::launch<7>(g, epi, o->err, st)) != cudaSuccess) break;
        e = pdl_launch(trace_kernel, dim3(c, w), kTraceThreads, smem, st,
                       reinterpret_cast<const z_t*>(o->T), n, ld / 2, row0, c0, Kpart, nblk, w0, s,
                       o->norms);
      }
    }
  }
  if (e != cudaSuccess) return e;
  return pdl_launch(exchange_verdict_kernel, nwalk, 128, 0, st, o->norms, 2 * nblk, o->sa2, o->sb,
                    2LL * o->in.nw * n, n, o->err, o->ex_gate, o->redone + OZ_EXCHANGE);
}

cudaError_t oz_error(OzState* o, int* flags, cudaStream_t st) {
  cudaError_t e = cudaMemcpyAsync(flags, o->err, sizeof(int), cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e == cudaSuccess && *flags) e = cudaMemsetAsync(o->err, 0, sizeof(int), st);
  return e;
}

cudaError_t oz_set_wait_clocks(long long clocks) { return tc::set_wait_clocks(clocks); }

}  // namespace afq
