// FP64 kernels of the walker step (the plain form): mixed density matrix and overlaps,
// sigma (Philox), CSR SpMM for vHS / vbias / Vakbl, weight update, Householder
// re-orthogonalisation and the local energy.  Internal device layouts:
//   W   [nw][N][2n]   (spin s occupies columns s*n .. s*n+n-1 of each row)
//   tw  [N][2n]       trial, same interleave
//   Gc  [nw][2][n][N] per-walker compact density matrices (linear index s*n*N + a*N + k)
//   vHS [nw][N][N], vbias / X / xraw [nchol][nw] (reference layout)
#include <cooperative_groups.h>
#include <cmath>
#include <cstdlib>

#include "afq_kernels.h"
#include "afq_common.cuh"
#include "gj.cuh"

namespace afq {

// ============================================================ mixed density matrix
// One CTA per (walker, spin).  T1 = W_s^T tw_s (n x n, mixed_density_matrix.hpp:83);
// Gauss-Jordan with partial pivoting (max |re|+|im|, as izamax; gj.cuh) gives det(T1) and
// T1^-1 (ma_operations.hpp:244-260); Gc_s = T1^-1 W_s^T (mixed_density_matrix.hpp:91).
// want_gc == 0 runs only the elimination for the determinant (Overlap, :124-138).
constexpr int DM_KC = 32;
constexpr int DM_THREADS = 256;

size_t dm_smem_bytes(int n) {
  size_t ldT = n + 1;
  size_t buf = std::max((size_t)2 * DM_KC * n, (size_t)n * 65);   // phase 1 slabs | W^T chunk
  return sizeof(z_t) * (n * ldT + buf);
}

// R = ceil(n / 16): the register blocks are R x R (a runtime bound left 16 predicated blocks of
// multiply-adds to issue for any n; 1024 walkers of 48+48 electrons at 384 orbitals 2.50 ->
// 2.28 ms, 16 of 16+16 at 64 orbitals 31 -> 23 us).
template <int R>
__global__ void __launch_bounds__(DM_THREADS, 2)
dm_kernel(const z_t* __restrict__ W, const z_t* __restrict__ tw, int N, int n,
          z_t* __restrict__ Gc, z_t* __restrict__ Wd, int* __restrict__ info, int want_gc,
          int save_old) {
  pdl_trigger();
  pdl_wait();
  extern __shared__ __align__(16) unsigned char dm_smem[];
  const int w = blockIdx.x >> 1, s = blockIdx.x & 1;
  const int ldT = n + 1;
  z_t* T = reinterpret_cast<z_t*>(dm_smem);
  z_t* buf = T + n * ldT;
  __shared__ GjState gj;
  const long long ldw = 2 * n;
  const z_t* Ws = W + (long long)w * N * ldw + s * n;
  const z_t* ts = tw + s * n;
  const int tid = threadIdx.x, nt = blockDim.x;

  // ---- phase 1: T1 = W_s^T tw_s; thread (ta, tb) of a 16 x 16 grid owns rows
  // a = ta + 16i and columns b = tb + 16j (i, j < R = ceil(n/16)), a register block that
  // reuses each shared-memory operand R times
  const int ta = tid / 16, tb = tid % 16;
  {
    z_t acc[R][R];
#pragma unroll
    for (int i = 0; i < R; i++)
#pragma unroll
      for (int j = 0; j < R; j++) acc[i][j] = zmk(0, 0);
    for (int k0 = 0; k0 < N; k0 += DM_KC) {
      const int kc = min(DM_KC, N - k0);
      for (int e = tid; e < kc * n; e += nt) {
        int kk = e / n, a = e % n;
        buf[kk * n + a] = Ws[(long long)(k0 + kk) * ldw + a];
        buf[DM_KC * n + kk * n + a] = ts[(long long)(k0 + kk) * ldw + a];
      }
      __syncthreads();
      for (int kk = 0; kk < kc; kk++) {
        z_t av[R], bv[R];
#pragma unroll
        for (int i = 0; i < R; i++) {
          const int a = ta + 16 * i, b = tb + 16 * i;
          av[i] = (a < n) ? buf[kk * n + a] : zmk(0, 0);
          bv[i] = (b < n) ? buf[DM_KC * n + kk * n + b] : zmk(0, 0);
        }
#pragma unroll
        for (int i = 0; i < R; i++)
#pragma unroll
          for (int j = 0; j < R; j++)
            zfma(acc[i][j], av[i], bv[j]);
      }
      __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < R; i++)
#pragma unroll
      for (int j = 0; j < R; j++) {
        const int a = ta + 16 * i, b = tb + 16 * j;
        if (a < n && b < n) T[a * ldT + b] = acc[i][j];
      }
  }

  // ---- phase 2: pivoted elimination
  gj_run<(R > 2 ? 2 : 1), DM_THREADS / 32>(T, ldT, n, want_gc, 0, gj);
  const int sing = gj.sing;
  const z_t det = gj.det;

  // ---- phase 3: Gc_s = T1^-1 W_s^T, T1^-1[a][b] = T[pivrow[a]][invp[b]]
  if (want_gc) {
    z_t* Gout = Gc + ((long long)w * 2 + s) * n * N;
    const z_t* Ta[R];
#pragma unroll
    for (int i = 0; i < R; i++) {
      const int a = ta + 16 * i;
      Ta[i] = T + ((!sing && a < n) ? gj.pivrow[a] * ldT : 0);
    }
    // Gc[a][k] = sum_b Tinv[a][b] W[k][b] over 64-row chunks of W: thread (ta, tk) owns
    // rows a = ta + 16i (i < R) and chunk columns k = tk + 16j (j < 4)
    constexpr int KC3 = 64;
    const int tk = tb;
    for (int k0 = 0; k0 < N; k0 += KC3) {
      const int kc = min(KC3, N - k0);
      for (int e = tid; e < kc * n; e += nt) {
        int kk = e / n, b = e % n;
        buf[b * (KC3 + 1) + kk] = Ws[(long long)(k0 + kk) * ldw + b];
      }
      __syncthreads();
      z_t acc[R][4];
#pragma unroll
      for (int i = 0; i < R; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = zmk(0, 0);
      if (!sing)
        for (int b = 0; b < n; b++) {
          z_t tv[R], wv[4];
          const int ib = gj.invp[b];
#pragma unroll
          for (int i = 0; i < R; i++) tv[i] = ta + 16 * i < n ? Ta[i][ib] : zmk(0, 0);
#pragma unroll
          for (int j = 0; j < 4; j++) wv[j] = buf[b * (KC3 + 1) + tk + 16 * j];
#pragma unroll
          for (int i = 0; i < R; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) zfma(acc[i][j], tv[i], wv[j]);
        }
#pragma unroll
      for (int i = 0; i < R; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) {
          const int a = ta + 16 * i, kk = tk + 16 * j;
          if (a < n && kk < kc) Gout[(long long)a * N + k0 + kk] = acc[i][j];
        }
      __syncthreads();
    }
  }
  if (tid == 0) {
    z_t* d = Wd + (long long)w * 8;
    if (save_old) {
      if (s == 0) d[5] = d[4];
      d[6 + s] = d[2 + s];
    }
    d[2 + s] = det;
    info[w * 2 + s] = sing;
  }
}

template <int R>
cudaError_t launch_dm_r(const z_t* W, const z_t* tw, int N, int n, int nw, z_t* Gc, z_t* Wd,
                          int* info, int want_gc, int save_old, cudaStream_t st) {
  size_t smem = dm_smem_bytes(n);
  static DeviceAttr attr;
  cudaError_t e = attr.ensure(smem, [](size_t b) {
    cudaError_t r = cudaFuncSetAttribute(dm_kernel<R>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)b);
    if (r == cudaSuccess)   // several CTAs per SM need the full shared-memory carveout
      r = cudaFuncSetAttribute(dm_kernel<R>, cudaFuncAttributePreferredSharedMemoryCarveout,
                               (int)cudaSharedmemCarveoutMaxShared);
    return r;
  });
  if (e != cudaSuccess) return e;
  pdl_launch(dm_kernel<R>, 2 * nw, DM_THREADS, smem, st, W, tw, N, n, Gc, Wd, info, want_gc, save_old);
  return cudaGetLastError();
}

cudaError_t launch_dm(const z_t* W, const z_t* tw, int N, int n, int nw, z_t* Gc, z_t* Wd,
                      int* info, int want_gc, int save_old, cudaStream_t st) {
  switch ((n + 15) / 16) {
    case 1: return launch_dm_r<1>(W, tw, N, n, nw, Gc, Wd, info, want_gc, save_old, st);
    case 2: return launch_dm_r<2>(W, tw, N, n, nw, Gc, Wd, info, want_gc, save_old, st);
    case 3: return launch_dm_r<3>(W, tw, N, n, nw, Gc, Wd, info, want_gc, save_old, st);
    case 4: return launch_dm_r<4>(W, tw, N, n, nw, Gc, Wd, info, want_gc, save_old, st);
  }
  return cudaErrorInvalidValue;   // the register blocks cover n <= 64
}

// ============================================================ sigma
// X = x + i vbias, hybridW[w] = -sum_c i vb (x + i/2 vb)  (miniafqmc_base.cpp:281-289).
// A cluster of up to 8 CTAs per 32 walkers (lanes), a CTA's 32 warps and the cluster's CTAs on
// Cholesky rows; the groups' sums meet in the first CTA in a fixed order.  The field's normals
// cost two FP64 logarithm / sine evaluations' latency per row and warp: one CTA per 32
// walkers took 20 us at 256 rows and 90 us at 1536.  A CTA per 32 rows, per 64 where the clusters
// would fill half the SMs: two turns of a warp cost less than many clusters' start (256 rows, 32
// / 512 walkers 10.0 / 14.1 us with 8 CTAs, 12.0 / 12.1 with 4; 16 rows, 1024 walkers 7.5 with
// one, 14.5 with 8).
constexpr int kSigmaCluster = 8;
__global__ void __launch_bounds__(1024)
sigma_kernel(const z_t* __restrict__ vbias, z_t* __restrict__ X, double* __restrict__ xraw,
             z_t* __restrict__ hybridW, int nchol, int nw, const DevScalars* __restrict__ sc,
             int use_xraw) {
  pdl_trigger();
  pdl_wait();
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  __shared__ z_t red[32][33];
  __shared__ z_t part[32];
  const int ctas = cl.num_blocks();
  const int lane = threadIdx.x, g = threadIdx.y, rank = blockIdx.x % ctas;
  const int w = blockIdx.x / ctas * 32 + lane;
  const unsigned long long seed = sc->seed, step = sc->step;
  const long long nwg = sc->nwalk_global > 0 ? sc->nwalk_global : nw;
  const long long woff = sc->walker_offset;
  z_t hw = zmk(0, 0);
  if (w < nw) {
    for (int c = rank * 32 + g; c < nchol; c += 32 * ctas) {
      long long e = (long long)c * nw + w;
      double x;
      if (use_xraw) {
        x = xraw[e];
      } else {
        // the stream is indexed by the global walker so shards reproduce one ensemble
        long long eg = (long long)c * nwg + woff + w;
        double x0, x1;
        normal_pair(seed, step, (unsigned long long)eg >> 1, &x0, &x1);
        x = (eg & 1) ? x1 : x0;
        xraw[e] = x;
      }
      z_t vb = vbias[e];
      z_t ivb = zmk(-vb.y, vb.x);                      // i vb
      z_t t = zmk(x - 0.5 * vb.y, 0.5 * vb.x);         // x + (i/2) vb
      hw = zsub(hw, zmul(ivb, t));
      X[e] = zmk(x - vb.y, vb.x);                      // x + i vb
    }
  }
  red[g][lane] = hw;
  __syncthreads();
  if (g == 0) {
    z_t s = zmk(0, 0);
    for (int q = 0; q < 32; q++) s = zadd(s, red[q][lane]);
    if (ctas == 1) {   // uniform
      if (w < nw) hybridW[w] = s;
    }
    part[lane] = s;
  }
  if (ctas == 1) return;
  cl.sync();
  if (rank == 0 && g == 0 && w < nw) {
    z_t s = zmk(0, 0);
    for (int q = 0; q < ctas; q++) s = zadd(s, cl.map_shared_rank(part, q)[lane]);
    hybridW[w] = s;
  }
  cl.sync();   // every CTA's sums stay until the first has read them
}

cudaError_t launch_sigma(const z_t* vbias, z_t* X, double* xraw, z_t* hybridW, int nchol,
                         int nw, const DevScalars* sc, int use_xraw, cudaStream_t st) {
  const unsigned groups = (nw + 31) / 32;
  unsigned ctas = 1;
  while (ctas < kSigmaCluster && 32 * (int)ctas < nchol) ctas *= 2;
  while (ctas > 1 && groups * ctas > 74 && nchol < 64 * (int)ctas) ctas /= 2;
  return pdl_launch_cluster(sigma_kernel, ctas, groups * ctas, dim3(32, 32), 0, st, vbias, X,
                            xraw, hybridW, nchol, nw, sc, use_xraw);
}

// ============================================================ CSR x dense (walker-fast B)
// out[w][r] = sum_p A[p] B[col(p)][w] for the rows r of a CSR, B [ncols][nw] walker
// fastest (vHS = Spvn X, vHS.hpp:47-56).  A warp owns a row; its lanes own walkers;
// the nonzeros of a row are fetched 32 at a time and broadcast with shuffles.  The CTA
// stages its [rows x walkers] results in shared memory and writes them walker-major.
// ROWS warps (rows) per CTA, WPL walkers per lane (CTA covers 32 WPL walkers); the set-up
// tuner picks the shape (every shape sums each output in CSR order: same results).
// GATED: the form after a digit product, a few CTAs that loop over the rows (one CTA per row
// group took 50 us to return at once at 384 orbitals; the loop costs the plain form 7 of 91 us
// at 128 orbitals, 256 walkers).
template <bool REALV, int ROWS, int WPL, bool GATED>
__global__ void __launch_bounds__(ROWS * 32)
csr_walker_kernel(const int* __restrict__ rowIndex, const int* __restrict__ cols,
                  const z_t* __restrict__ zvals, const double* __restrict__ rvals,
                  const z_t* __restrict__ B, int nrows, int nw, z_t* __restrict__ out,
                  long long out_ld, OzGate gate) {
  pdl_trigger();
  pdl_wait();
  if (GATED && !oz_gate_open(gate)) return;
  constexpr int WALK = 32 * WPL;
  __shared__ z_t tile[ROWS][WALK + 1];
  const int lane = threadIdx.x & 31, wy = threadIdx.x >> 5;
  const int w0 = blockIdx.y * WALK;
  for (int r0 = blockIdx.x * ROWS; r0 < nrows; r0 += gridDim.x * ROWS) {
    const int r = r0 + wy;
    z_t acc[WPL];
#pragma unroll
    for (int j = 0; j < WPL; j++) acc[j] = zmk(0, 0);
    if (r < nrows) {
      const int beg = rowIndex[r], end = rowIndex[r + 1];
      for (int p0 = beg; p0 < end; p0 += 32) {
        const int cnt = min(32, end - p0);
        int myc = 0;
        z_t myv = zmk(0, 0);
        double myr = 0.0;
        if (lane < cnt) {
          myc = cols[p0 + lane];
          if (REALV) myr = rvals[p0 + lane];
          else myv = zvals[p0 + lane];
        }
        for (int q = 0; q < cnt; q++) {
          const int c = __shfl_sync(0xffffffffu, myc, q);
          const z_t* br = B + (long long)c * nw;
          if (REALV) {
            const double v = __shfl_sync(0xffffffffu, myr, q);
#pragma unroll
            for (int j = 0; j < WPL; j++) {
              const int w = w0 + 32 * j + lane;
              if (w < nw) zfma_r(acc[j], v, br[w]);
            }
          } else {
            z_t v;
            v.x = __shfl_sync(0xffffffffu, myv.x, q);
            v.y = __shfl_sync(0xffffffffu, myv.y, q);
#pragma unroll
            for (int j = 0; j < WPL; j++) {
              const int w = w0 + 32 * j + lane;
              if (w < nw) zfma(acc[j], v, br[w]);
            }
          }
        }
      }
    }
#pragma unroll
    for (int j = 0; j < WPL; j++) tile[wy][32 * j + lane] = acc[j];
    __syncthreads();
    for (int e = threadIdx.x; e < ROWS * WALK; e += ROWS * 32) {
      const int wl = e / ROWS, rr = e % ROWS;
      const int w = w0 + wl, rw = r0 + rr;
      if (w < nw && rw < nrows) out[(long long)w * out_ld + rw] = tile[rr][wl];
    }
    if constexpr (!GATED) break;
    __syncthreads();   // the next rows reuse the tile
  }
}

template <int ROWS, int WPL>
cudaError_t csr_walker_launch(const int* rowIndex, const int* cols, const z_t* zvals,
                              const double* rvals, const z_t* B, int nrows, int nw, z_t* out,
                              long long out_ld, cudaStream_t st, const OzGate& gate) {
  dim3 grid((nrows + ROWS - 1) / ROWS, (nw + 32 * WPL - 1) / (32 * WPL));
  if (gate.ok) {
    grid.x = std::min(grid.x, 8u * device_sms());
    return rvals ? pdl_launch(csr_walker_kernel<true, ROWS, WPL, true>, grid, ROWS * 32, 0, st,
                              rowIndex, cols, nullptr, rvals, B, nrows, nw, out, out_ld, gate)
                 : pdl_launch(csr_walker_kernel<false, ROWS, WPL, true>, grid, ROWS * 32, 0, st,
                              rowIndex, cols, zvals, nullptr, B, nrows, nw, out, out_ld, gate);
  }
  return rvals ? pdl_launch(csr_walker_kernel<true, ROWS, WPL, false>, grid, ROWS * 32, 0, st,
                            rowIndex, cols, nullptr, rvals, B, nrows, nw, out, out_ld, gate)
               : pdl_launch(csr_walker_kernel<false, ROWS, WPL, false>, grid, ROWS * 32, 0, st,
                            rowIndex, cols, zvals, nullptr, B, nrows, nw, out, out_ld, gate);
}

const char* csr_walker_cfg_name(int cfg) {
  static const char* names[kCsrWalkerCfgs + 1] = {"16x2", "16x2", "8x2", "4x2",
                                                  "16x1", "8x4",  "4x4", "32x1"};
  return cfg >= 0 && cfg <= kCsrWalkerCfgs ? names[cfg] : "?";
}

// cfg: 0 built-in (16 rows x 2 walkers per lane), 1..kCsrWalkerCfgs the shapes above
cudaError_t launch_csr_walker(const int* rowIndex, const int* cols, const z_t* zvals,
                              const double* rvals, const z_t* B, int nrows, int nw, z_t* out,
                              long long out_ld, cudaStream_t st, int cfg, const OzGate& gate) {
  switch (cfg) {
    case 2: return csr_walker_launch<8, 2>(rowIndex, cols, zvals, rvals, B, nrows, nw, out, out_ld, st, gate);
    case 3: return csr_walker_launch<4, 2>(rowIndex, cols, zvals, rvals, B, nrows, nw, out, out_ld, st, gate);
    case 4: return csr_walker_launch<16, 1>(rowIndex, cols, zvals, rvals, B, nrows, nw, out, out_ld, st, gate);
    case 5: return csr_walker_launch<8, 4>(rowIndex, cols, zvals, rvals, B, nrows, nw, out, out_ld, st, gate);
    case 6: return csr_walker_launch<4, 4>(rowIndex, cols, zvals, rvals, B, nrows, nw, out, out_ld, st, gate);
    case 7: return csr_walker_launch<32, 1>(rowIndex, cols, zvals, rvals, B, nrows, nw, out, out_ld, st, gate);
    default: return csr_walker_launch<16, 2>(rowIndex, cols, zvals, rvals, B, nrows, nw, out, out_ld, st, gate);
  }
}

// ============================================================ CSR x walker-major G
// out[r][w] = sum_p A[p] G[w][col(p)] (vbias = SpvnT Gc when SpvnT is sparse,
// vbias.hpp:63; Gcloc = Vakbl Gc, energy.hpp:89).  Warp per row, lanes over walkers.
__global__ void __launch_bounds__(256)
csr_gather_kernel(const int* __restrict__ rowIndex, const int* __restrict__ cols,
                  const z_t* __restrict__ vals, const z_t* __restrict__ G, long long ldg,
                  int nrows, int nw, z_t* __restrict__ out, OzGate gate) {
  pdl_trigger();
  pdl_wait();
  if (!oz_gate_open(gate)) return;
  const int lane = threadIdx.x & 31;
  const int r = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (r >= nrows) return;
  const int beg = rowIndex[r], end = rowIndex[r + 1];
  for (int w0 = 0; w0 < nw; w0 += 32) {
    const int w = w0 + lane;
    z_t acc = zmk(0, 0);
    for (int p0 = beg; p0 < end; p0 += 32) {
      const int cnt = min(32, end - p0);
      int myc = 0;
      z_t myv = zmk(0, 0);
      if (lane < cnt) { myc = cols[p0 + lane]; myv = vals[p0 + lane]; }
      for (int q = 0; q < cnt; q++) {
        const int c = __shfl_sync(0xffffffffu, myc, q);
        z_t v;
        v.x = __shfl_sync(0xffffffffu, myv.x, q);
        v.y = __shfl_sync(0xffffffffu, myv.y, q);
        if (w < nw) zfma(acc, v, G[(long long)w * ldg + c]);
      }
    }
    if (w < nw) out[(long long)r * nw + w] = acc;
  }
}

cudaError_t launch_csr_gather(const int* rowIndex, const int* cols, const z_t* vals, const z_t* G,
                              long long ldg, int nrows, int nw, z_t* out, cudaStream_t st,
                              const OzGate& gate) {
  if (gate.ok)
    return pdl_launch(csr_gather_kernel, (nrows + 7) / 8, 256, 0, st, rowIndex, cols, vals, G, ldg,
                      nrows, nw, out, gate);
  csr_gather_kernel<<<(nrows + 7) / 8, 256, 0, st>>>(rowIndex, cols, vals, G, ldg, nrows, nw, out,
                                                     gate);
  return cudaGetLastError();
}

// ============================================================ weights
// miniafqmc_base.cpp:316-327; one CTA, fixed-order reduction of sum Re e4.
__global__ void __launch_bounds__(1024)
weights_kernel(z_t* __restrict__ Wd, const z_t* __restrict__ hybridW, int nw, double dt,
               DevScalars* __restrict__ sc, int update_eshift) {
  pdl_trigger();
  pdl_wait();
  __shared__ z_t red[32];
  const double eshift = sc->eshift;
  double sum = 0.0;
  for (int w = threadIdx.x; w < nw; w += blockDim.x) {
    z_t* d = Wd + (long long)w * 8;
    z_t ratio = zdiv(zmul(d[2], d[3]), zmul(d[6], d[7]));
    double ang = atan2(ratio.y, ratio.x);
    double scale = fmax(0.0, cos(ang));
    z_t lr = zmk(log(hypot(ratio.x, ratio.y)), ang);
    z_t hw = hybridW[w];
    z_t e4 = zmk(-(hw.x + lr.x) / dt, -(hw.y + lr.y) / dt);
    double f = scale * exp(-dt * (0.5 * (e4.x + d[5].x) - eshift));
    d[4] = e4;
    d[1] = zmk(d[1].x * f, d[1].y * f);
    sum += e4.x;
  }
  z_t t = block_zsum(zmk(sum, 0.0), red);
  if (threadIdx.x == 0) {
    sc->e4sum = t.x;
    if (update_eshift) sc->eshift = t.x / nw;
    sc->step += 1;
  }
}

cudaError_t launch_weights(z_t* Wd, const z_t* hybridW, int nw, double dt, DevScalars* sc,
                           int update_eshift, cudaStream_t st) {
  pdl_launch(weights_kernel, 1, 1024, 0, st, Wd, hybridW, nw, dt, sc, update_eshift);
  return cudaGetLastError();
}

// Sharded substeps: the last weight update's local sum of Re W_data[:,4] into a device
// double, and Eshift = (the ensemble's sum, all-reduced in place by the caller) / walkers
// of the whole ensemble (miniafqmc_base.cpp:327).
__global__ void e4sum_out_kernel(const DevScalars* __restrict__ sc, double* __restrict__ out) {
  *out = sc->e4sum;
}
__global__ void eshift_from_kernel(DevScalars* __restrict__ sc, const double* __restrict__ total,
                                   int nw) {
  const long long ng = sc->nwalk_global > 0 ? sc->nwalk_global : nw;
  sc->eshift = *total / (double)ng;
}
cudaError_t launch_e4sum_out(const DevScalars* sc, double* out, cudaStream_t st) {
  e4sum_out_kernel<<<1, 1, 0, st>>>(sc, out);
  return cudaGetLastError();
}
cudaError_t launch_eshift_from(DevScalars* sc, const double* total, int nw, cudaStream_t st) {
  eshift_from_kernel<<<1, 1, 0, st>>>(sc, total, nw);
  return cudaGetLastError();
}

__global__ void set_scalars_kernel(DevScalars* sc, unsigned long long seed,
                                   unsigned long long step, int set_eshift, double eshift,
                                   int walker_offset, long long nwalk_global) {
  sc->seed = seed;
  sc->step = step;
  if (set_eshift) sc->eshift = eshift;
  if (nwalk_global > 0) {
    sc->walker_offset = walker_offset;
    sc->nwalk_global = nwalk_global;
  }
}

cudaError_t launch_set_scalars(DevScalars* sc, unsigned long long seed, unsigned long long step,
                               int set_eshift, double eshift, cudaStream_t st,
                               int walker_offset, long long nwalk_global) {
  set_scalars_kernel<<<1, 1, 0, st>>>(sc, seed, step, set_eshift, eshift, walker_offset,
                                      nwalk_global);
  return cudaGetLastError();
}

// ============================================================ orthogonalisation
// LQ of W_s seen column-major (zgelqf + zunglq, afqmc_sys.hpp:200-204) is the QR of
// B = conj(W_s) (N x n): Householder reflectors with zlarfg's conventions (real beta
// of sign -sign(Re alpha); tau = (beta - alpha)/beta; v = x/(alpha - beta)), each
// H^H = I - conj(tau) v v^H applied from the left (zgeqr2), then Q = H(1)..H(n) formed
// by backward accumulation (zung2r) and W_s = conj(Q).  One CTA per (walker, spin)
// works in place on the walker buffer (L2 resident); threads are laid out as
// (column, row-group) so row segments are read contiguously.
constexpr int QR_THREADS = 256;

__global__ void __launch_bounds__(QR_THREADS)
ortho_kernel(z_t* __restrict__ W, int N, int n) {
  pdl_trigger();
  pdl_wait();
  __shared__ z_t tau_s[64];
  __shared__ z_t sdot[4][65];
  __shared__ z_t red[QR_THREADS / 32];
  __shared__ z_t s_ctau, s_scal;
  __shared__ double s_beta;
  __shared__ int s_skip;
  const int w = blockIdx.x >> 1, s = blockIdx.x & 1;
  const long long ld = 2 * n;
  z_t* B = W + (long long)w * N * ld + s * n;
  const int tid = threadIdx.x;
  const int lc = tid % 64, rg = tid / 64;   // column lane, row group (4 groups)

  for (long long e = tid; e < (long long)N * n; e += QR_THREADS) {
    long long i = e / n, c = e % n;
    z_t v = B[i * ld + c];
    B[i * ld + c] = zconj(v);
  }
  __syncthreads();

  for (int j = 0; j < n; j++) {
    // xnorm^2 over rows j+1..N-1 of column j
    double part = 0.0;
    for (int i = j + 1 + tid; i < N; i += QR_THREADS) {
      z_t v = B[(long long)i * ld + j];
      part += v.x * v.x + v.y * v.y;
    }
    z_t tot = block_zsum(zmk(part, 0.0), red);
    if (tid == 0) {
      z_t alpha = B[(long long)j * ld + j];
      double xn2 = tot.x;
      if (xn2 == 0.0 && alpha.y == 0.0) {
        s_skip = 1;
        tau_s[j] = zmk(0, 0);
      } else {
        double nrm = sqrt(alpha.x * alpha.x + alpha.y * alpha.y + xn2);
        double beta = -copysign(nrm, alpha.x);
        z_t tau = zmk((beta - alpha.x) / beta, -alpha.y / beta);
        tau_s[j] = tau;
        s_ctau = zconj(tau);
        s_scal = zrecip(zmk(alpha.x - beta, alpha.y));
        s_beta = beta;
        s_skip = 0;
      }
    }
    __syncthreads();
    if (s_skip) continue;
    const z_t scal = s_scal;
    for (int i = j + 1 + tid; i < N; i += QR_THREADS) {
      long long o = (long long)i * ld + j;
      B[o] = zmul(B[o], scal);
    }
    __syncthreads();
    if (tid == 0) B[(long long)j * ld + j] = zmk(s_beta, 0.0);
    // s_l = v^H B[j:, l] for l > j (v_j = 1)
    const int l = j + 1 + lc;
    z_t acc = zmk(0, 0);
    if (l < n) {
      if (rg == 0) acc = B[(long long)j * ld + l];
      for (int i = j + 1 + rg; i < N; i += 4)
        zfma_conj(acc, B[(long long)i * ld + j], B[(long long)i * ld + l]);
    }
    sdot[rg][lc] = acc;
    __syncthreads();
    if (rg == 0 && l < n)
      sdot[0][lc] = zadd(zadd(sdot[0][lc], sdot[1][lc]), zadd(sdot[2][lc], sdot[3][lc]));
    __syncthreads();
    if (l < n) {
      const z_t f = zmul(s_ctau, sdot[0][lc]);
      if (rg == 0) {
        long long o = (long long)j * ld + l;
        B[o] = zsub(B[o], f);
      }
      for (int i = j + 1 + rg; i < N; i += 4) {
        long long o = (long long)i * ld + l;
        B[o] = zsub(B[o], zmul(B[(long long)i * ld + j], f));
      }
    }
    __syncthreads();
  }

  // Q = H(1) ... H(n) applied to the first n columns of the identity (zung2r)
  for (int i = n - 1; i >= 0; i--) {
    const z_t tau = tau_s[i];
    if (i < n - 1) {
      const int l = i + 1 + lc;
      z_t acc = zmk(0, 0);
      if (l < n) {
        if (rg == 0) acc = B[(long long)i * ld + l];   // v_i = 1
        for (int r = i + 1 + rg; r < N; r += 4)
          zfma_conj(acc, B[(long long)r * ld + i], B[(long long)r * ld + l]);
      }
      sdot[rg][lc] = acc;
      __syncthreads();
      if (rg == 0 && l < n)
        sdot[0][lc] = zadd(zadd(sdot[0][lc], sdot[1][lc]), zadd(sdot[2][lc], sdot[3][lc]));
      __syncthreads();
      if (l < n) {
        const z_t f = zmul(tau, sdot[0][lc]);
        if (rg == 0) {
          long long o = (long long)i * ld + l;
          B[o] = zsub(B[o], f);
        }
        for (int r = i + 1 + rg; r < N; r += 4) {
          long long o = (long long)r * ld + l;
          B[o] = zsub(B[o], zmul(B[(long long)r * ld + i], f));
        }
      }
      __syncthreads();
    }
    const z_t mt = zmk(-tau.x, -tau.y);
    for (int r = i + 1 + tid; r < N; r += QR_THREADS) {
      long long o = (long long)r * ld + i;
      B[o] = zmul(B[o], mt);
    }
    if (tid == 0) B[(long long)i * ld + i] = zmk(1.0 - tau.x, -tau.y);
    for (int r = tid; r < i; r += QR_THREADS) B[(long long)r * ld + i] = zmk(0, 0);
    __syncthreads();
  }

  for (long long e = tid; e < (long long)N * n; e += QR_THREADS) {
    long long i = e / n, c = e % n;
    z_t v = B[i * ld + c];
    B[i * ld + c] = zconj(v);
  }
}

// The same reflectors with the walker's N x n block in shared memory (row stride odd: columns
// are read without bank conflicts), CL column lanes x 256 / CL row groups, four barriers per
// reflector.  The kernel above pays L2 latency for every dependent step: 16 walkers of 16+16
// electrons at 64 orbitals 82 -> 48 us, 256 of 32+32 at 128 orbitals 673 -> 340 us.
constexpr size_t kOrthoSmem = 200 << 10;
size_t ortho_smem_bytes(int N, int n) { return sizeof(z_t) * (size_t)N * (n | 1); }

template <int CL>
__global__ void __launch_bounds__(QR_THREADS)
ortho_smem_kernel(z_t* __restrict__ W, int N, int n) {
  pdl_trigger();
  pdl_wait();
  constexpr int G = QR_THREADS / CL;
  extern __shared__ __align__(16) unsigned char qr_smem[];
  z_t* B = reinterpret_cast<z_t*>(qr_smem);   // conj(W_s) [N][ld]
  __shared__ z_t tau_s[64];
  __shared__ z_t sdot[G][CL + 1];
  __shared__ double red[2][QR_THREADS / 32];
  const int w = blockIdx.x >> 1, sp = blockIdx.x & 1, ld = n | 1;
  const long long ldw = 2 * n;
  z_t* Ws = W + (long long)w * N * ldw + sp * n;
  const int tid = threadIdx.x, lc = tid % CL, rg = tid / CL, lane = tid & 31, warp = tid >> 5;
  for (int i = rg; i < N; i += G)
    if (lc < n) B[i * ld + lc] = zconj(Ws[i * ldw + lc]);
  __syncthreads();

  // sum over the row groups of column lane lc's partial products, in order
  auto total = [&](z_t part) {
    sdot[rg][lc] = part;
    __syncthreads();
    z_t t = sdot[0][lc];
#pragma unroll
    for (int q = 1; q < G; q++) t = zadd(t, sdot[q][lc]);
    return t;
  };
  for (int j = 0; j < n; j++) {
    double part = 0.0;   // |x|^2 of rows j + 1 ... of column j
    for (int i = j + 1 + tid; i < N; i += QR_THREADS) {
      const z_t v = B[i * ld + j];
      part += v.x * v.x + v.y * v.y;
    }
    part = warp_sum(part);
    if (lane == 0) red[j & 1][warp] = part;
    __syncthreads();
    double xn2 = 0.0;
#pragma unroll
    for (int q = 0; q < QR_THREADS / 32; q++) xn2 += red[j & 1][q];
    const z_t alpha = B[j * ld + j];
    if (xn2 == 0.0 && alpha.y == 0.0) {   // uniform: H is the identity
      if (tid == 0) tau_s[j] = zmk(0, 0);
      continue;
    }
    const double beta = -copysign(sqrt(alpha.x * alpha.x + alpha.y * alpha.y + xn2), alpha.x);
    const z_t tau = zmk((beta - alpha.x) / beta, -alpha.y / beta);
    const z_t scal = zrecip(zmk(alpha.x - beta, alpha.y));
    __syncthreads();   // alpha is read
    for (int i = j + 1 + tid; i < N; i += QR_THREADS) B[i * ld + j] = zmul(B[i * ld + j], scal);
    if (tid == 0) {
      tau_s[j] = tau;
      B[j * ld + j] = zmk(beta, 0.0);
    }
    __syncthreads();
    const int l = j + 1 + lc;   // s_l = v^H B[j:, l], v_j = 1
    z_t acc = zmk(0, 0);
    if (l < n) {
      if (rg == 0) acc = B[j * ld + l];
      for (int i = j + 1 + rg; i < N; i += G) zfma_conj(acc, B[i * ld + j], B[i * ld + l]);
    }
    const z_t f = zmul(zconj(tau), total(acc));
    if (l < n) {
      if (rg == 0) B[j * ld + l] = zsub(B[j * ld + l], f);
      for (int i = j + 1 + rg; i < N; i += G)
        B[i * ld + l] = zsub(B[i * ld + l], zmul(B[i * ld + j], f));
    }
    __syncthreads();
  }
  __syncthreads();   // an identity reflector leaves its turn early: tau_s[n - 1] may just be written

  // Q = H(1) ... H(n) applied to the first n columns of the identity (zung2r)
  for (int i = n - 1; i >= 0; i--) {
    const z_t tau = tau_s[i];
    const int l = i + 1 + lc;
    z_t acc = zmk(0, 0);
    if (l < n) {
      if (rg == 0) acc = B[i * ld + l];   // v_i = 1
      for (int r = i + 1 + rg; r < N; r += G) zfma_conj(acc, B[r * ld + i], B[r * ld + l]);
    }
    const z_t f = zmul(tau, total(acc));
    if (l < n) {
      if (rg == 0) B[i * ld + l] = zsub(B[i * ld + l], f);
      for (int r = i + 1 + rg; r < N; r += G)
        B[r * ld + l] = zsub(B[r * ld + l], zmul(B[r * ld + i], f));
    }
    __syncthreads();
    const z_t mt = zmk(-tau.x, -tau.y);
    for (int r = tid; r < N; r += QR_THREADS)
      B[r * ld + i] = r < i ? zmk(0, 0) : r == i ? zmk(1.0 - tau.x, -tau.y) : zmul(B[r * ld + i], mt);
    __syncthreads();
  }
  for (int i = rg; i < N; i += G)
    if (lc < n) Ws[i * ldw + lc] = zconj(B[i * ld + lc]);
}

template <int CL>
cudaError_t launch_ortho_smem(z_t* W, int N, int n, int nw, cudaStream_t st) {
  const size_t smem = ortho_smem_bytes(N, n);
  static DeviceAttr attr;
  const cudaError_t e = attr.ensure(smem, [](size_t b) {
    cudaError_t r = cudaFuncSetAttribute(ortho_smem_kernel<CL>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)b);
    if (r == cudaSuccess)
      r = cudaFuncSetAttribute(ortho_smem_kernel<CL>, cudaFuncAttributePreferredSharedMemoryCarveout,
                               (int)cudaSharedmemCarveoutMaxShared);
    return r;
  });
  if (e != cudaSuccess) return e;
  return pdl_launch(ortho_smem_kernel<CL>, 2 * nw, QR_THREADS, smem, st, W, N, n);
}

cudaError_t launch_ortho(z_t* W, int N, int n, int nw, cudaStream_t st) {
  if (ortho_smem_bytes(N, n) <= kOrthoSmem && n <= 64)
    return n <= 16   ? launch_ortho_smem<16>(W, N, n, nw, st)
           : n <= 32 ? launch_ortho_smem<32>(W, N, n, nw, st)
                     : launch_ortho_smem<64>(W, N, n, nw, st);
  pdl_launch(ortho_kernel, 2 * nw, QR_THREADS, 0, st, W, N, n);
  return cudaGetLastError();
}

// CholeskyQR2 re-orthogonalisation (FP64): G = W_s^H W_s, G = R^H R (R upper, positive
// real diagonal), W_s <- W_s R^-1, done twice.  The columns span the same space as the
// Householder result and differ from it by a diagonal of +-1, so G, overlap ratios,
// weights and energies are unchanged; only raw overlaps may change sign.  One CTA per
// (walker, spin); the n x n factors live in shared memory, W streams through it in
// 32-row chunks.  A walker whose Gram matrix is not positive definite is left as is
// and flagged in info.
// One pass leaves W R^-1 orthonormal to about n eps kappa(W)^2; the second pass is
// skipped when kappa_F = |R|_F |R^-1|_F (>= the 2-norm condition number) is at most 4n,
// i.e. orthonormal to ~1e-11 or better.  Walkers re-orthogonalised every few steps meet
// that bound; a run may force both passes with two_pass = 1.
constexpr int CQ_KC = 32;

size_t cholqr_smem_bytes(int n) {
  return sizeof(z_t) * ((size_t)2 * n * (n + 1) + (size_t)CQ_KC * (n + 1));
}

template <int R>   // ceil(n / 16): the register blocks in use
__global__ void __launch_bounds__(256)
ortho_cholqr_kernel(z_t* __restrict__ W, int N, int n, int* __restrict__ info, int two_pass) {
  pdl_trigger();
  pdl_wait();
  extern __shared__ __align__(16) unsigned char cq_smem[];
  const int w = blockIdx.x >> 1, s = blockIdx.x & 1;
  const int ld = n + 1;
  z_t* G = reinterpret_cast<z_t*>(cq_smem);     // Gram matrix, then R
  z_t* Ri = G + n * ld;                          // R^-1
  z_t* buf = Ri + n * ld;                        // W chunk [KC][n+1]
  __shared__ int s_bad;
  __shared__ z_t s_red[32];
  const long long ldw = 2 * n;
  z_t* B = W + (long long)w * N * ldw + s * n;
  const int tid = threadIdx.x, nt = blockDim.x;
  const int ta = tid / 16, tb = tid % 16;   // n <= 64, 256 threads
  if (tid == 0) s_bad = 0;
  for (int pass = 0; pass < 2; pass++) {
    // ---- Gram matrix G[a][b] = sum_k conj(B[k][a]) B[k][b]; thread (ta, tb) of a 16 x 16
    // grid owns a = ta + 16i, b = tb + 16j (i, j < R = ceil(n/16)): R^2 products per 2R
    // shared-memory reads
    {
      z_t acc[R][R];
#pragma unroll
      for (int i = 0; i < R; i++)
#pragma unroll
        for (int j = 0; j < R; j++) acc[i][j] = zmk(0, 0);
      for (int k0 = 0; k0 < N; k0 += CQ_KC) {
        const int kc = min(CQ_KC, N - k0);
        for (int e = tid; e < kc * n; e += nt) {
          int kk = e / n, a = e % n;
          buf[kk * ld + a] = B[(long long)(k0 + kk) * ldw + a];
        }
        __syncthreads();
        for (int kk = 0; kk < kc; kk++) {
          z_t av[R], bv[R];
#pragma unroll
          for (int i = 0; i < R; i++) {
            const int a = ta + 16 * i, b = tb + 16 * i;
            av[i] = (a < n) ? buf[kk * ld + a] : zmk(0, 0);
            bv[i] = (b < n) ? buf[kk * ld + b] : zmk(0, 0);
          }
          // blocks i > j hold only a > b: the lower triangle, which nothing reads
#pragma unroll
          for (int i = 0; i < R; i++)
#pragma unroll
            for (int j = i; j < R; j++)
              zfma_conj(acc[i][j], av[i], bv[j]);
        }
        __syncthreads();
      }
#pragma unroll
      for (int i = 0; i < R; i++)
#pragma unroll
        for (int j = i; j < R; j++) {
          const int a = ta + 16 * i, b = tb + 16 * j;
          if (a < n && b < n) G[a * ld + b] = acc[i][j];
        }
    }
    __syncthreads();
    // ---- Cholesky G = R^H R in place (upper triangle)
    for (int j = 0; j < n; j++) {
      const double dj = G[j * ld + j].x;
      if (!(dj > 0.0)) {
        if (tid == 0) s_bad = 1;
        break;
      }
      const double d = sqrt(dj), inv = 1.0 / d;
      __syncthreads();
      for (int l = j + tid; l < n; l += nt)
        G[j * ld + l] = (l == j) ? zmk(d, 0.0) : zscale(G[j * ld + l], inv);
      __syncthreads();
      const int m = n - j - 1;
      for (int e = tid; e < m * m; e += nt) {
        int a = j + 1 + e / m, b = j + 1 + e % m;
        if (b < a) continue;   // upper triangle only
        z_t t = G[a * ld + b];
        zfma(t, zmk(-G[j * ld + a].x, G[j * ld + a].y), G[j * ld + b]);   // -= conj(R_ja) R_jb
        G[a * ld + b] = t;
      }
      __syncthreads();
    }
    __syncthreads();
    if (s_bad) break;
    // ---- R^-1 (upper) by back substitution, one column per thread
    for (int j = tid; j < n; j += nt) {
      for (int i = n - 1; i >= 0; i--) {
        z_t t = (i == j) ? zmk(1.0, 0.0) : zmk(0.0, 0.0);
        if (i <= j) {
          for (int l = i + 1; l <= j; l++) t = zsub(t, zmul(G[i * ld + l], Ri[l * ld + j]));
          t = zscale(t, 1.0 / G[i * ld + i].x);
        }
        Ri[i * ld + j] = t;
      }
    }
    __syncthreads();
    bool last = pass == 1;
    if (pass == 0 && !two_pass) {   // |R|_F^2 and |R^-1|_F^2 over the upper triangles
      double r2 = 0.0, q2 = 0.0;
      for (int e = tid; e < n * n; e += nt) {
        const int a = e / n, b = e % n;
        if (b < a) continue;
        const z_t g = G[a * ld + b], q = Ri[a * ld + b];
        r2 += g.x * g.x + g.y * g.y;
        q2 += q.x * q.x + q.y * q.y;
      }
      const z_t t = block_zsum(zmk(r2, q2), s_red);
      last = t.x * t.y <= 16.0 * n * n;
    }
    // ---- B <- B R^-1 in 32-row chunks: thread (tk, tb) owns rows k = tk + 16i (i < 2)
    // and columns b = tb + 16j (j < R); R^-1 is upper triangular (zeros below)
    for (int k0 = 0; k0 < N; k0 += CQ_KC) {
      const int kc = min(CQ_KC, N - k0);
      for (int e = tid; e < kc * n; e += nt) {
        int kk = e / n, a = e % n;
        buf[kk * ld + a] = B[(long long)(k0 + kk) * ldw + a];
      }
      __syncthreads();
      z_t acc[2][R];
#pragma unroll
      for (int i = 0; i < 2; i++)
#pragma unroll
        for (int j = 0; j < R; j++) acc[i][j] = zmk(0, 0);
      // R^-1 is upper triangular: rows a in [16r, 16r + 16) reach columns b = tb + 16j
      // only for j >= r
#pragma unroll
      for (int r = 0; r < R; r++) {
        const int a1 = min(16 * r + 16, n);
        for (int a = 16 * r; a < a1; a++) {
          z_t bv[2], rv[R];
#pragma unroll
          for (int i = 0; i < 2; i++) bv[i] = buf[(ta + 16 * i) * ld + a];
#pragma unroll
          for (int j = r; j < R; j++) {
            const int b = tb + 16 * j;
            rv[j] = (b < n) ? Ri[a * ld + b] : zmk(0, 0);
          }
#pragma unroll
          for (int i = 0; i < 2; i++)
#pragma unroll
            for (int j = r; j < R; j++)
              zfma(acc[i][j], bv[i], rv[j]);
        }
      }
#pragma unroll
      for (int i = 0; i < 2; i++)
#pragma unroll
        for (int j = 0; j < R; j++) {
          const int kk = ta + 16 * i, b = tb + 16 * j;
          if (kk < kc && b < n) B[(long long)(k0 + kk) * ldw + b] = acc[i][j];
        }
      __syncthreads();
    }
    if (last) break;
  }
  if (tid == 0) info[w * 2 + s] |= s_bad ? 2 : 0;
}

template <int R>
cudaError_t launch_cholqr_r(z_t* W, int N, int n, int nw, int* info, cudaStream_t st) {
  size_t smem = cholqr_smem_bytes(n);
  static DeviceAttr attr;
  cudaError_t e = attr.ensure(smem, [](size_t b) {
    cudaError_t r = cudaFuncSetAttribute(ortho_cholqr_kernel<R>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)b);
    if (r == cudaSuccess)
      r = cudaFuncSetAttribute(ortho_cholqr_kernel<R>, cudaFuncAttributePreferredSharedMemoryCarveout,
                               (int)cudaSharedmemCarveoutMaxShared);
    return r;
  });
  if (e != cudaSuccess) return e;
  static const int two_pass = [] {
    const char* e = getenv("AFQ_CHOLQR_PASSES");
    return e && atoi(e) == 2 ? 1 : 0;
  }();
  pdl_launch(ortho_cholqr_kernel<R>, 2 * nw, 256, smem, st, W, N, n, info, two_pass);
  return cudaGetLastError();
}

cudaError_t launch_ortho_cholqr(z_t* W, int N, int n, int nw, int* info, cudaStream_t st) {
  switch ((n + 15) / 16) {
    case 1: return launch_cholqr_r<1>(W, N, n, nw, info, st);
    case 2: return launch_cholqr_r<2>(W, N, n, nw, info, st);
    case 3: return launch_cholqr_r<3>(W, N, n, nw, info, st);
    case 4: return launch_cholqr_r<4>(W, N, n, nw, info, st);
  }
  return cudaErrorInvalidValue;   // the register tiles cover n <= 64
}

// ============================================================ small propagation chain
// W_w <- P exp(i V_w) P W_w for a small orbital count in ONE launch: a CTA per (walker, eight
// columns) keeps P, then V, then P in shared memory, the Taylor terms' columns beside it and
// their sum in registers.  The eight products as launches of their own cost 8.5 us each at 64
// orbitals and 16 walkers (latency: 64-step K chains on a few SMs); sums run over k in the
// same order, so the walkers are the same bit for bit.  512 threads: 64 rows x 8 columns (one
// warp issues an FP64 multiply-add only every ten clocks, so four warps per scheduler), rows
// i and i + 64 in one pass.
constexpr int PS_COLS = 8, PS_THREADS = 512, PS_ROWS = PS_THREADS / PS_COLS;
constexpr int kPropSmallMaxN = 112;

size_t prop_small_smem(int N) { return sizeof(z_t) * ((size_t)N * (N + 1) + 2 * (size_t)N * PS_COLS); }

__global__ void __launch_bounds__(PS_THREADS)
prop_small_kernel(const z_t* __restrict__ P, const z_t* __restrict__ V, z_t* __restrict__ W,
                  int N, int n2, int order) {
  pdl_trigger();
  pdl_wait();
  extern __shared__ __align__(16) unsigned char ps_smem[];
  z_t* M = reinterpret_cast<z_t*>(ps_smem);   // [N][N + 1]
  z_t* T = M + N * (N + 1);                   // [N][8], two buffers
  z_t* U = T + N * PS_COLS;
  const int tid = threadIdx.x, jl = tid % PS_COLS, i0 = tid / PS_COLS;
  const int j = blockIdx.x * PS_COLS + jl;
  z_t* Ww = W + (long long)blockIdx.y * N * n2;
  const z_t* Vw = V + (long long)blockIdx.y * N * N;
  auto load = [&](const z_t* src) {
    const int dr = PS_THREADS / N, dc = PS_THREADS - dr * N;
    for (int r = tid / N, c = tid - tid / N * N; r < N;) {
      cp_async16(M + r * (N + 1) + c, src + r * N + c, 16);
      r += dr;
      if ((c += dc) >= N) {
        c -= N;
        r++;
      }
    }
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();
  };
  const bool two = i0 + PS_ROWS < N, one = i0 < N;
  const z_t* M0 = M + (one ? i0 : 0) * (N + 1);
  const z_t* M1 = M + (two ? i0 + PS_ROWS : 0) * (N + 1);
  z_t acc[2], S[2];
  auto product = [&](const z_t* B) {
    acc[0] = acc[1] = zmk(0, 0);
    if (N <= PS_ROWS) {
#pragma unroll 8
      for (int k = 0; k < N; k++) zfma(acc[0], M0[k], B[k * PS_COLS + jl]);
    } else {
#pragma unroll 4
      for (int k = 0; k < N; k++) {
        const z_t b = B[k * PS_COLS + jl];
        zfma(acc[0], M0[k], b);
        zfma(acc[1], M1[k], b);
      }
    }
  };
  auto put = [&](z_t* B, const z_t (&v)[2]) {
    if (one) B[i0 * PS_COLS + jl] = v[0];
    if (two) B[(i0 + PS_ROWS) * PS_COLS + jl] = v[1];
  };
  const z_t zero = zmk(0, 0);
  {
    const z_t w0[2] = {one && j < n2 ? Ww[(long long)i0 * n2 + j] : zero,
                       two && j < n2 ? Ww[(long long)(i0 + PS_ROWS) * n2 + j] : zero};
    put(T, w0);
  }
  load(P);
  product(T);
  S[0] = acc[0];
  S[1] = acc[1];
  put(U, S);
  if (order > 0) {
    __syncthreads();   // every row of P is read
    load(Vw);
  }
  z_t *cur = U, *nxt = T;
  for (int k = 1; k <= order; k++) {   // T = (i / k) V T; S += T
    product(cur);
    const z_t f = zmk(0.0, 1.0 / (double)k);
    const z_t t[2] = {zmul(f, acc[0]), zmul(f, acc[1])};
    S[0] = zadd(S[0], t[0]);
    S[1] = zadd(S[1], t[1]);
    if (k < order)
      put(nxt, t);
    else
      put(nxt, S);
    __syncthreads();
    z_t* x = cur;
    cur = nxt;
    nxt = x;
  }
  if (order > 0)
    load(P);
  else
    __syncthreads();
  product(cur);
  if (j < n2) {
    if (one) Ww[(long long)i0 * n2 + j] = acc[0];
    if (two) Ww[(long long)(i0 + PS_ROWS) * n2 + j] = acc[1];
  }
}

// The chain of order + 2 separate products (ZGEMM), us: per product 4.5 for the launch, then the
// longer of a serial sum over k (0.076 an orbital) and the tiles of the busiest SM (0.3 each and
// 21 TFLOP/s of the whole chip, padding included), for the best of zgemm's tile shapes.  Within
// 8% (rms) of 330 measured chains of 6 to 330 orbitals, 1e5 to 2e10 operations a product.
double prop_zgemm_us(int N, int n2, int nw, int order) {
  static const int shape[][2] = {{64, 32}, {64, 64}, {64, 96}, {32, 64}, {32, 96}, {128, 64}, {32, 32}};
  const int sms = device_sms();
  double best = 1e30;
  for (const auto& s : shape) {
    const double tiles = (double)((N + s[0] - 1) / s[0]) * ((n2 + s[1] - 1) / s[1]) * nw;
    const double busiest = std::ceil(tiles / sms);
    best = std::min(best, std::max(0.076 * N, busiest * (0.3 + N * 8.0 * s[0] * s[1] * sms / 21e6)));
  }
  return (order + 2) * (4.5 + best);
}
// Up to 1.2e8 real operations per product and where its own estimate is below 0.8 of the separate
// products': per wave of CTAs one start a product, then a multiply-add chain (0.052 us an orbital)
// or the multiply-adds of the CTAs that share an SM (0.038 us an orbital, CTA and row pass); within
// 11% of 110 chains.  Separate and in one launch, us: 64 orbitals, 16 walkers of 16+16 electrons
// 70 > 36, 100 orbitals, 20 walkers of 30+30 150 > 127; 30 orbitals, 332 walkers of 14+14 85 < 125,
// 16 orbitals, 875 walkers of 7+7 84 < 95, 11 orbitals, 721 walkers of 5+5 66 > 52.
bool prop_small_fits(int N, int n2, int nw, int order) {
  if (N > kPropSmallMaxN || nw > 65535 || 8.0 * N * N * (double)n2 * nw > 1.2e8) return false;
  const int sms = device_sms();
  const int occ = std::max(1, std::min(4, (int)((227 << 10) / (prop_small_smem(N) + 1024))));
  const double ctas = std::ceil((double)((n2 + PS_COLS - 1) / PS_COLS) * nw / sms);
  const double waves = std::floor(ctas / occ), rest = ctas - waves * occ;
  auto wave = [&](double share) {
    const int passes = N <= PS_ROWS ? 1 : 2;
    return (order + 2) * (1.0 + std::max(0.052 * N, 0.038 * share * N * passes));
  };
  const double us = waves * wave(occ) + (rest > 0 ? wave(rest) : 0.0);
  return us < 0.8 * prop_zgemm_us(N, n2, nw, order);
}

cudaError_t launch_prop_small(const z_t* P, const z_t* V, z_t* W, int N, int n2, int nw, int order,
                              cudaStream_t st) {
  const size_t smem = prop_small_smem(N);
  static DeviceAttr attr;
  cudaError_t e = attr.ensure(smem, [](size_t b) {
    cudaError_t r = cudaFuncSetAttribute(prop_small_kernel,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)b);
    if (r == cudaSuccess)
      r = cudaFuncSetAttribute(prop_small_kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                               (int)cudaSharedmemCarveoutMaxShared);
    return r;
  });
  if (e != cudaSuccess) return e;
  pdl_launch(prop_small_kernel, dim3((n2 + PS_COLS - 1) / PS_COLS, nw), PS_THREADS, smem, st, P, V,
             W, N, n2, order);
  return cudaGetLastError();
}

// ============================================================ walker layout
// Both layouts hold runs of n entries (orbital row i, spin s): one warp per device row,
// 16-byte entries, coalesced on both sides.
__global__ void __launch_bounds__(256)
walker_layout_kernel(const z_t* __restrict__ src, z_t* __restrict__ dst, int N, int n,
                     long long rows, int to_ref) {
  const long long r = blockIdx.x * 8LL + (threadIdx.x >> 5);   // w N + i
  if (r >= rows) return;
  const long long w = r / N, i = r - w * N;
  for (int j = threadIdx.x & 31; j < 2 * n; j += 32) {
    const int s = j >= n;
    const long long dev = r * 2 * n + j, ref = ((w * 2 + s) * N + i) * n + (j - s * n);
    if (to_ref)
      dst[ref] = src[dev];
    else
      dst[dev] = src[ref];
  }
}

cudaError_t launch_walker_layout(const z_t* src, z_t* dst, int N, int n, int nw, int to_ref,
                                 cudaStream_t st) {
  const long long rows = (long long)nw * N;
  walker_layout_kernel<<<(unsigned)((rows + 7) / 8), 256, 0, st>>>(src, dst, N, n, rows, to_ref);
  return cudaGetLastError();
}

// ============================================================ exchange energy
// K_w = 1/2 sum_{s,c} tr(T T), T = Lh_s[c] Gc_s^T (n x n), for Gn Cholesky vectors x Gw
// walkers per CTA: a (Gn*n) x (Gw*n) complex tile over K = N, then the trace of each
// n x n block squared from shared memory.  Partial sums per (walker, spin, c-block).
constexpr int EX_T = 96, EX_BK = 16, EX_TM = 6, EX_TN = 6, EX_THREADS = 256;

size_t exch_smem_bytes() {
  size_t main = sizeof(z_t) * 2 * EX_BK * 2 * (EX_T + 1);
  size_t epi = sizeof(z_t) * EX_T * (EX_T + 1);
  return std::max(main, epi);
}

__global__ void __launch_bounds__(EX_THREADS)
exchange_kernel(const z_t* __restrict__ Lh, const z_t* __restrict__ Gc, int N, int n, int nchol,
                int nw, int Gn, int Gw, z_t* __restrict__ Kpart, int nblk,
                const int* __restrict__ gate) {
  pdl_trigger();
  pdl_wait();
  extern __shared__ __align__(16) unsigned char ex_smem[];
  z_t* As = reinterpret_cast<z_t*>(ex_smem);          // [2][BK][T+1]
  z_t* Bs = As + 2 * EX_BK * (EX_T + 1);
  const int s = blockIdx.z;
  const int c0 = blockIdx.x * Gn;
  const long long NAK = 2LL * n * N;
  const int Mr = Gn * n, Nc = Gw * n;
  const int tid = threadIdx.x, tx = tid % 16, ty = tid / 16;

  for (int w0 = blockIdx.y * Gw; w0 < nw; w0 += gridDim.y * Gw) {
    if (gate) {   // uniform
      bool any = false;
      for (int w = w0; w < min(nw, w0 + Gw); w++) any |= gate[w] != 0;
      if (!any) continue;
    }
    auto load = [&](int stage, int k0) {
      z_t* as = As + stage * EX_BK * (EX_T + 1);
      z_t* bs = Bs + stage * EX_BK * (EX_T + 1);
      for (int e = tid; e < EX_T * EX_BK; e += EX_THREADS) {
        int m = e / EX_BK, k = e % EX_BK, gk = k0 + k;
        int cv = m / n, a = m % n;
        const z_t* src = Lh;
        int bytes = 0;
        if (m < Mr && c0 + cv < nchol && gk < N) {
          src = Lh + (long long)(c0 + cv) * NAK + (long long)s * n * N + (long long)a * N + gk;
          bytes = 16;
        }
        cp_async16(as + k * (EX_T + 1) + m, src, bytes);
        const z_t* srcb = Gc;
        int bb = 0;
        if (m < Nc && w0 + m / n < nw && gk < N) {
          int wl = m / n, b = m % n;
          srcb = Gc + (long long)(w0 + wl) * NAK + (long long)s * n * N + (long long)b * N + gk;
          bb = 16;
        }
        cp_async16(bs + k * (EX_T + 1) + m, srcb, bb);
      }
      cp_async_commit();
    };

    z_t acc[EX_TM][EX_TN];
#pragma unroll
    for (int i = 0; i < EX_TM; i++)
#pragma unroll
      for (int j = 0; j < EX_TN; j++) acc[i][j] = zmk(0, 0);
    const int nk = (N + EX_BK - 1) / EX_BK;
    load(0, 0);
    for (int kt = 0; kt < nk; kt++) {
      if (kt + 1 < nk) {
        load((kt + 1) & 1, (kt + 1) * EX_BK);
        cp_async_wait<1>();
      } else {
        cp_async_wait<0>();
      }
      __syncthreads();
      const z_t* as = As + (kt & 1) * EX_BK * (EX_T + 1);
      const z_t* bs = Bs + (kt & 1) * EX_BK * (EX_T + 1);
#pragma unroll 4
      for (int kk = 0; kk < EX_BK; kk++) {
        z_t a[EX_TM], b[EX_TN];
#pragma unroll
        for (int i = 0; i < EX_TM; i++) a[i] = as[kk * (EX_T + 1) + ty + 16 * i];
#pragma unroll
        for (int j = 0; j < EX_TN; j++) b[j] = bs[kk * (EX_T + 1) + tx + 16 * j];
#pragma unroll
        for (int i = 0; i < EX_TM; i++)
#pragma unroll
          for (int j = 0; j < EX_TN; j++) zfma(acc[i][j], a[i], b[j]);
      }
      __syncthreads();
    }
    z_t* Ts = reinterpret_cast<z_t*>(ex_smem);             // [T][T+1], reuses the slabs
#pragma unroll
    for (int i = 0; i < EX_TM; i++)
#pragma unroll
      for (int j = 0; j < EX_TN; j++) Ts[(ty + 16 * i) * (EX_T + 1) + tx + 16 * j] = acc[i][j];
    __syncthreads();
    const int lane = tid & 31, warp = tid >> 5;
    for (int wl = warp; wl < Gw; wl += EX_THREADS / 32) {
      z_t sum = zmk(0, 0);
      for (int cv = 0; cv < Gn; cv++)
        for (int t = lane; t < n * n; t += 32) {
          int a = t / n, b = t % n;
          zfma(sum, Ts[(cv * n + a) * (EX_T + 1) + wl * n + b], Ts[(cv * n + b) * (EX_T + 1) + wl * n + a]);
        }
      sum = warp_zsum(sum);
      if (w0 + wl < nw && (!gate || gate[w0 + wl])) {   // zeros past the Cholesky blocks, where nblk is a finer blocking's
        z_t* k = Kpart + ((long long)(w0 + wl) * 2 + s) * nblk;
        for (int q = blockIdx.x + lane * gridDim.x; q < nblk; q += 32 * gridDim.x)
          k[q] = lane == 0 && q == blockIdx.x ? sum : zmk(0, 0);
      }
    }
    __syncthreads();   // the next walkers' slabs reuse the tile
  }
}

cudaError_t launch_exchange(const z_t* Lh, const z_t* Gc, int N, int n, int nchol, int nw,
                            z_t* Kpart, int* nblk_out, cudaStream_t st, const int* gate,
                            int stride) {
  if (n > EX_T) return cudaErrorInvalidValue;
  const int Gn = EX_T / n, Gw = EX_T / n;
  const int nblk = (nchol + Gn - 1) / Gn;
  *nblk_out = nblk;
  if (!Kpart) return cudaSuccess;
  size_t smem = exch_smem_bytes();
  static DeviceAttr attr;
  cudaError_t e = attr.ensure(smem, [](size_t b) {
    return cudaFuncSetAttribute(exchange_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)b);
  });
  if (e != cudaSuccess) return e;
  // a gated launch mostly does nothing: few CTAs, each looping over the walker groups
  dim3 grid(nblk, std::min((nw + Gw - 1) / Gw, gate ? 4 : 65535), 2);
  if (gate)
    return pdl_launch(exchange_kernel, grid, EX_THREADS, smem, st, Lh, Gc, N, n, nchol, nw, Gn, Gw,
                      Kpart, stride ? stride : nblk, gate);
  exchange_kernel<<<grid, EX_THREADS, smem, st>>>(Lh, Gc, N, n, nchol, nw, Gn, Gw, Kpart,
                                                  stride ? stride : nblk, gate);
  return cudaGetLastError();
}

// ============================================================ energy reductions
// Per walker: E1 = sum Gc.haj (energy.hpp:100); mode 0 (Vakbl): E2 = 1/2 sum Gc.Gcloc
// (energy.hpp:93-97); mode 1 (Cholesky): EJ = 1/2 sum_c cv^2, EK = 1/2 sum Kpart.
__global__ void __launch_bounds__(256)
energy_reduce_kernel(const z_t* __restrict__ Gc, const z_t* __restrict__ haj, int nak,
                     const z_t* __restrict__ Gcloc, const z_t* __restrict__ cv, int nchol,
                     const z_t* __restrict__ Kpart, int nblk, int nw, int mode,
                     z_t* __restrict__ Wd, double* __restrict__ parts) {
  pdl_trigger();
  pdl_wait();
  __shared__ z_t red[8];
  const int w = blockIdx.x;
  const z_t* g = Gc + (long long)w * nak;
  z_t e1 = zmk(0, 0), e2 = zmk(0, 0);
  for (int i = threadIdx.x; i < nak; i += blockDim.x) {
    z_t gi = g[i];
    zfma(e1, gi, haj[i]);
    if (mode == 0) zfma(e2, gi, Gcloc[(long long)i * nw + w]);
  }
  e1 = block_zsum(e1, red);
  z_t ej = zmk(0, 0), ek = zmk(0, 0);
  if (mode == 0) {
    e2 = block_zsum(e2, red);
  } else {
    for (int c = threadIdx.x; c < nchol; c += blockDim.x) {
      z_t v = cv[(long long)c * nw + w];
      zfma(ej, v, v);
    }
    for (int q = threadIdx.x; q < 2 * nblk; q += blockDim.x)
      ek = zadd(ek, Kpart[(long long)w * 2 * nblk + q]);
    ej = block_zsum(ej, red);
    ek = block_zsum(ek, red);
  }
  if (threadIdx.x == 0) {
    z_t e;
    if (mode == 0) {
      e = zadd(zscale(e2, 0.5), e1);
    } else {
      ej = zscale(ej, 0.5);
      ek = zscale(ek, 0.5);
      e = zsub(zadd(e1, ej), ek);
      if (parts) {
        parts[3 * w] = e1.x; parts[3 * w + 1] = ej.x; parts[3 * w + 2] = ek.x;
      }
    }
    Wd[(long long)w * 8] = e;
  }
}

cudaError_t launch_energy_reduce(const z_t* Gc, const z_t* haj, int nak, const z_t* Gcloc,
                                 const z_t* cv, int nchol, const z_t* Kpart, int nblk, int nw,
                                 int mode, z_t* Wd, double* parts, cudaStream_t st) {
  pdl_launch(energy_reduce_kernel, nw, 256, 0, st, Gc, haj, nak, Gcloc, cv, nchol, Kpart, nblk, nw,
             mode, Wd, parts);
  return cudaGetLastError();
}

// sum Re(eloc) Re(w) and sum Re(w) (afqmc_sys.hpp:127-132), fixed-order reduction.
__global__ void __launch_bounds__(1024)
eav_kernel(const z_t* __restrict__ Wd, int nw, DevScalars* __restrict__ sc) {
  pdl_trigger();
  pdl_wait();
  __shared__ z_t red[32];
  double a = 0.0, b = 0.0;
  for (int w = threadIdx.x; w < nw; w += blockDim.x) {
    const z_t* d = Wd + (long long)w * 8;
    a += d[0].x * d[1].x;
    b += d[1].x;
  }
  z_t t = block_zsum(zmk(a, b), red);
  if (threadIdx.x == 0) {
    sc->esum[0] = t.x;
    sc->esum[1] = t.y;
  }
}

cudaError_t launch_eav(const z_t* Wd, int nw, DevScalars* sc, cudaStream_t st) {
  pdl_launch(eav_kernel, 1, 1024, 0, st, Wd, nw, sc);
  return cudaGetLastError();
}

}  // namespace afq
