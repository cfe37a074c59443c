// FP64 contraction stages on the int8 tensor cores: operand splitting, the products of
// oz_gemm.cuh and the kernels around them.
#include <algorithm>
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
  int* err = nullptr;
  // exchange: rows (c, a) of Lh per spin, columns (w, b, re | im) of G, T = Lh_c Gc_w^T of a
  // chunk of Cholesky vectors and walkers
  bool lreal = false;
  Slices lx[2], gx;
  double* T = nullptr;
  int ex_w = 0, ex_c = 0;   // walkers and Cholesky vectors per chunk
  bool exchange = false;
};

namespace {

template <class T>
cudaError_t oz_alloc(OzState* o, T** p, size_t count) {
  void* q = nullptr;
  const cudaError_t e = cudaMalloc(&q, sizeof(T) * (count ? count : 1));
  if (e == cudaSuccess) {
    o->allocs.push_back(q);
    *p = static_cast<T*>(q);
  }
  return e;
}

// Slices of `batch` x `rows` rows of K digits-worth of entries, in tiles of `tile` rows.
cudaError_t alloc_slices(OzState* o, Slices* s, int tile, int rows, int batch, int K) {
  s->tile = tile;
  s->rows = rows;
  s->batch = batch;
  s->nslab = (K + oz::kSlab - 1) / oz::kSlab;
  cudaError_t e = oz_alloc(o, &s->d, s->bytes());
  if (e == cudaSuccess) e = oz_alloc(o, &s->scale, (size_t)rows * batch);
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
enum { kReal, kPairs, kSplitRe, kSplitCx };

struct RowScale {
  double s1, s2, scale;   // q = rn(x s1 s2) = rn(x 2^(55 - e)), scale = 2^e
};
AFQ_D RowScale row_scale(unsigned long long maxbits) {
  RowScale r{0.0, 0.0, 0.0};
  if (maxbits == 0) return r;
  const double mx = __longlong_as_double((long long)maxbits);
  int e;
  if (maxbits >= 0x7FE0000000000000ull) {   // inf, nan, or 2^e beyond the range
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

// One warp (WIDE = false) or one CTA (WIDE) per source row: the row's maximum, then its
// digits, four K entries per thread and step.  Memory bound: 16 bytes read per complex
// entry and up to 14 (28 for kSplitCx) written; the second read of the row hits L1 / L2.
template <int MODE, bool WIDE>
__global__ void __launch_bounds__(256)
slice_kernel(RowSrc src, int nrows, int K, Slices s) {
  __shared__ unsigned long long red[2][8];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int r = WIDE ? blockIdx.x : blockIdx.x * 8 + warp;
  if (r >= nrows) return;   // whole warps (WIDE: never)
  const int t = WIDE ? threadIdx.x : lane, nt = WIDE ? 256 : 32;
  const z_t* p = src.row(r);
  unsigned long long m0 = 0, m1 = 0;   // of the real and of the imaginary parts
  for (int k = t; k < K; k += nt) {
    const z_t v = p[k];
    m0 = max(m0, absbits(v.x));
    m1 = max(m1, absbits(v.y));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    m0 = max(m0, __shfl_xor_sync(0xffffffffu, m0, o));
    m1 = max(m1, __shfl_xor_sync(0xffffffffu, m1, o));
  }
  if constexpr (WIDE) {
    if (lane == 0) {
      red[0][warp] = m0;
      red[1][warp] = m1;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 8; i++) {
      m0 = max(m0, red[0][i]);
      m1 = max(m1, red[1][i]);
    }
  }
  if constexpr (MODE == kPairs || MODE == kSplitCx) m0 = m1 = max(m0, m1);
  const RowScale s0 = row_scale(m0), s1 = row_scale(m1);
  constexpr bool TWO = MODE == kSplitRe || MODE == kSplitCx;
  const int rb = r / s.per_batch(TWO), r0 = (r - rb * s.per_batch(TWO)) * (TWO ? 2 : 1);
  if (t == 0) {
    double* sc = s.scale + (long long)rb * s.rows + r0;
    sc[0] = s0.scale;
    if constexpr (TWO) sc[1] = s1.scale;
  }
  const z_t zero = zmk(0, 0);
  unsigned q[kS];
  const int Kp = s.nslab * oz::kSlab, plane = s.tile * oz::kSlab;
  for (int k = 4 * t; k < Kp; k += 4 * nt) {
    int8_t* o = s.d + oz::slice_offset(s, rb, r0, k);
    // rows 2r and 2r + 1 share a row pair of the swizzle: the second is 64 bytes on
    if constexpr (MODE == kReal || MODE == kSplitRe) {
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

// Slices nrows source rows of K complex entries into `s` (its first rows).
template <int MODE>
cudaError_t slice_rows(const RowSrc& src, int nrows, int K, const Slices& s, cudaStream_t st) {
  if (nrows <= 0) return cudaSuccess;
  if (K > 2048)
    slice_kernel<MODE, true><<<nrows, 256, 0, st>>>(src, nrows, K, s);
  else
    slice_kernel<MODE, false><<<(nrows + 7) / 8, 256, 0, st>>>(src, nrows, K, s);
  return cudaGetLastError();
}

__global__ void oz_check_imag_kernel(const z_t* __restrict__ src, long long count, int* flag) {
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < count;
       e += (long long)gridDim.x * blockDim.x)
    if (src[e].y != 0.0) *flag = 1;
}
// every value real?  (synchronises the stream)
cudaError_t is_real(OzState* o, const z_t* p, long long count, bool* real, cudaStream_t st) {
  int flag = 1;
  cudaError_t e = cudaMemsetAsync(o->err, 0, sizeof(int), st);
  if (e != cudaSuccess) return e;
  oz_check_imag_kernel<<<148 * 8, 256, 0, st>>>(p, count, o->err);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  e = cudaMemcpyAsync(&flag, o->err, sizeof(int), cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e == cudaSuccess) e = cudaMemsetAsync(o->err, 0, sizeof(int), st);
  *real = flag == 0;
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

// Kpart[w][s][c] = tr(T T), T the n x n block of (c, w) in the chunk's product (rows
// row0 + c n + a, columns w n + b).  One CTA per block, which passes through shared memory
// by asynchronous copies: few registers and 16 n (n + 1) bytes a CTA keep several CTAs per
// SM, whose copies overlap the others' sums (the block is fresh in L2).
constexpr int kTraceThreads = 128;
__global__ void __launch_bounds__(kTraceThreads)
trace_kernel(const z_t* __restrict__ T, int n, long long ld, int row0, int c_first,
             z_t* __restrict__ Kpart, int nblk, int w_first, int s) {
  extern __shared__ __align__(16) unsigned char tr_smem[];
  z_t* t = reinterpret_cast<z_t*>(tr_smem);   // [n][n + 1]
  __shared__ z_t red[kTraceThreads / 32];
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
  cp_async_wait<0>();
  __syncthreads();
  z_t sum = zmk(0, 0);
  for (int a = a0, b = b0; a < n;) {
    zfma(sum, t[a * (n + 1) + b], t[b * (n + 1) + a]);
    a += da;
    if ((b += db) >= n) {
      b -= n;
      a++;
    }
  }
  sum = block_zsum(sum, red);
  if (tid == 0) Kpart[((long long)(w_first + w) * 2 + s) * nblk + c_first + c] = sum;
}

}  // namespace

cudaError_t oz_create(const OzInit& in, OzState** out, cudaStream_t st) {
  *out = nullptr;
  const int N = in.N, n = in.n, nc = in.nchol, nw = in.nw;
  const long long NAK = 2LL * n * N;
  OzState* o = new OzState();
  o->in = in;
  cudaError_t e = oz_alloc(o, &o->err, 1);
  if (e == cudaSuccess) e = cudaMemsetAsync(o->err, 0, sizeof(int), st);
  if (e == cudaSuccess && in.Lh && n <= 64) {
    e = is_real(o, in.Lh, (long long)nc * NAK, &o->lreal, st);
    const int K = o->lreal ? N : 2 * N;
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
    size_t free_b = 0, total_b = 0;
    if (e == cudaSuccess) e = cudaMemGetInfo(&free_b, &total_b);
    const size_t need = 2 * (size_t)kS * (nc * n + 128) * (K + 64) +
                        (size_t)kS * (2 * nw * n + 64) * (K + 64) + tb;
    if (e == cudaSuccess && need < free_b / 2) {
      for (int s = 0; s < 2 && e == cudaSuccess; s++) {
        e = alloc_slices(o, &o->lx[s], oz::kBM, nc * n, 1, K);
        if (e != cudaSuccess) break;
        const RowSrc src{in.Lh + (long long)s * n * N, n, NAK, N};
        e = o->lreal ? slice_rows<kReal>(src, nc * n, N, o->lx[s], st)
                     : slice_rows<kPairs>(src, nc * n, N, o->lx[s], st);
      }
      if (e == cudaSuccess) e = alloc_slices(o, &o->gx, oz::kBN, 2 * nw * n, 1, K);
      if (e == cudaSuccess) e = oz_alloc(o, &o->T, tb / sizeof(double));
      if (e == cudaSuccess) o->exchange = true;
    }
  }
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e == cudaErrorMemoryAllocation) {   // the FP64 pipe's kernels need none of this
    cudaGetLastError();
    oz_destroy(o);
    return cudaSuccess;
  }
  if (e != cudaSuccess || !o->exchange) {
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

bool oz_has_exchange(const OzState* o, int nwalk) { return o && o->exchange && nwalk <= o->in.nw; }

int oz_exchange_launches(const OzState* o, int nwalk) {
  const int cw = (nwalk + o->ex_w - 1) / o->ex_w;
  const int cc = (o->in.nchol + o->ex_c - 1) / o->ex_c;
  return 2 + 4 * cw * cc;
}

cudaError_t oz_exchange(OzState* o, const z_t* Gc, int nwalk, z_t* Kpart, int nblk,
                        cudaStream_t st) {
  const int N = o->in.N, n = o->in.n, nc = o->in.nchol;
  const long long NAK = 2LL * n * N;
  const size_t smem = sizeof(z_t) * n * (n + 1);
  static DeviceAttr attr;
  cudaError_t e = attr.ensure(smem, [](size_t b) {
    cudaError_t r = cudaFuncSetAttribute(trace_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)b);
    if (r == cudaSuccess)
      r = cudaFuncSetAttribute(trace_kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                               (int)cudaSharedmemCarveoutMaxShared);
    return r;
  });
  for (int s = 0; s < 2 && e == cudaSuccess; s++) {
    const RowSrc src{Gc + (long long)s * n * N, n, NAK, N};
    e = o->lreal ? slice_rows<kSplitRe>(src, nwalk * n, N, o->gx, st)
                 : slice_rows<kSplitCx>(src, nwalk * n, N, o->gx, st);
    for (int w0 = 0; w0 < nwalk && e == cudaSuccess; w0 += o->ex_w) {
      const int w = std::min(o->ex_w, nwalk - w0);
      for (int c0 = 0; c0 < nc && e == cudaSuccess; c0 += o->ex_c) {
        const int c = std::min(o->ex_c, nc - c0);
        // the row tiles that hold the chunk's rows [c0 n, (c0 + c) n)
        const int t0 = c0 * n / oz::kBM, row0 = c0 * n - t0 * oz::kBM;
        oz::Gemm g{&o->lx[s], &o->gx, row0 + c * n, 2 * w * n, 1, t0, 2 * w0 * n / oz::kBN};
        const long long ld = (2LL * w * n + 3) / 4 * 4;
        EpiRows epi{o->T, ld, row0 + c * n};
        if ((e = oz::launch(g, epi, o->err, st)) != cudaSuccess) break;
        trace_kernel<<<dim3(c, w), kTraceThreads, smem, st>>>(
            reinterpret_cast<const z_t*>(o->T), n, ld / 2, row0, c0, Kpart, nblk, w0, s);
        e = cudaGetLastError();
      }
    }
  }
  return e;
}

cudaError_t oz_error(OzState* o, int* flags) {
  *flags = 0;
  cudaError_t e = cudaMemcpy(flags, o->err, sizeof(int), cudaMemcpyDeviceToHost);
  if (e == cudaSuccess && *flags) e = cudaMemset(o->err, 0, sizeof(int));
  return e;
}

cudaError_t oz_set_wait_clocks(long long clocks) { return tc::set_wait_clocks(clocks); }

}  // namespace afq
