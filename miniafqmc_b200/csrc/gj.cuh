// Gauss-Jordan inverse and determinant of an n x n complex FP64 matrix (n <= 64) in shared
// memory by one CTA: in-place exchange steps with implicit partial pivoting (largest
// |re| + |im| of the column over the unused rows, the first on ties, as izamax), in panels of
// eight pivots.
//
// One warp runs a panel's eight exchange steps on the panel's columns alone, a row per lane
// and register (no barrier inside); afterwards those columns hold the matrix M that the
// eight steps apply to the panel's pivot rows, so every other column takes one rank-8 update
//   A[i][c] <- (i a pivot row of the panel ? 0 : A[i][c]) + sum_q M[i][q] A[p_q][c].
// What bounds it: an exchange step at a time read and wrote the whole matrix in shared memory
// per pivot (74 KB, 576 clocks at n = 48) and crossed two barriers; the panels read and write
// it once per eight pivots with three barriers.  What remains is the panel's serial chain: one
// warp issues a DFMA about every ten clocks, 1240 clocks a pivot.  2048 matrices of 48 x 48 in
// the mixed form 0.56 -> 0.43 ms, of 64 x 64 1.31 -> 0.79 ms.
#pragma once
#include "afq_common.cuh"

namespace afq {

constexpr int kGjPanel = 8;

struct GjState {        // in shared memory
  int pivrow[64];       // row of pivot j; afterwards T1^-1[a][b] = T[pivrow[a]][invp[b]]
  int invp[64];
  unsigned long long used;
  z_t det;
  int sing;
};

// 1 / a = conj(a) / |a|^2, a scaled by a power of two so that |a|^2 lies in [1, 8): its
// reciprocal by two Newton-Raphson steps from the single-precision one (24 -> 48 -> 53 bits;
// a third of the latency of two FP64 divisions).  Magnitudes near the ends of the range:
// Smith's form.
AFQ_D z_t gj_recip(z_t a) {
  const double m = fmax(fabs(a.x), fabs(a.y));
  const int e = (int)(((unsigned long long)__double_as_longlong(m) >> 52) & 0x7ff);
  if (e < 64 || e > 1982) return zrecip(a);
  const double s = __longlong_as_double((long long)(2046 - e) << 52);   // 2^(1023 - e)
  const double x = a.x * s, y = a.y * s, d = fma(x, x, y * y);
  double r = (double)(1.0f / (float)d);
  r = fma(r, fma(-d, r, 1.0), r);
  r = fma(r, fma(-d, r, 1.0), r);
  r *= s;
  return zmk(x * r, -y * r);
}

// The pivot of a column (entry v[r] of row lane + 32 r): largest |re| + |im| by its bits
// (non-negative doubles order like them), then the lowest row.  nan_singular: a column
// without a comparable entry (all NaN) counts as singular; otherwise the first unused row
// serves and the NaN spreads.  Returns the row; *sing on a singular column (the row is then
// an arbitrary one).
template <int RPL>
AFQ_D int gj_pivot(const z_t (&v)[RPL], int n, unsigned long long used, int nan_singular, int* sing) {
  const int lane = threadIdx.x & 31;
  unsigned long long best = 0;
  int row = 64, any = 64;
#pragma unroll
  for (int r = RPL - 1; r >= 0; r--) {
    const int i = lane + 32 * r;
    const bool free_row = i < n && !((used >> i) & 1);
    const double m = zabs1(v[r]);
    const unsigned long long k = (unsigned long long)__double_as_longlong(m);
    if (free_row) any = i;
    if (free_row && m == m && k >= best) {
      best = k;
      row = i;
    }
  }
  const unsigned hi = __reduce_max_sync(0xffffffffu, (unsigned)(best >> 32));
  const bool th = row < 64 && (unsigned)(best >> 32) == hi;
  const unsigned lo = __reduce_max_sync(0xffffffffu, th ? (unsigned)best : 0u);
  int p = (int)__reduce_min_sync(0xffffffffu, th && (unsigned)best == lo ? (unsigned)row : 64u);
  if (p < 64) {
    if ((hi | lo) == 0) *sing = 1;
  } else {   // no comparable entry
    if (nan_singular) *sing = 1;
    p = (int)__reduce_min_sync(0xffffffffu, (unsigned)any) & 63;
  }
  return p;
}

// One panel on one warp: columns j0 .. j0 + kb - 1 of T, RPL rows per lane.  The chain from one
// pivot to the next is its reciprocal, the row factors and the next column alone; the other
// columns' updates fill its latency.
template <int RPL>
AFQ_D void gj_panel(z_t* T, int ld, int n, int j0, int kb, int nan_singular, GjState& s) {
  const int lane = threadIdx.x & 31;
  z_t a[kGjPanel][RPL];   // [column][row]
#pragma unroll
  for (int r = 0; r < RPL; r++)
#pragma unroll
    for (int c = 0; c < kGjPanel; c++) {
      const int i = lane + 32 * r;
      a[c][r] = (i < n && c < kb) ? T[i * ld + j0 + c] : zmk(0, 0);
    }
  unsigned long long used = s.used;
  z_t det = s.det;
  int sing = 0;
  auto bcast = [&](const z_t (&v)[RPL], int p) {   // the pivot row's entry of a column
    const z_t t = (RPL > 1 && p >= 32) ? v[RPL - 1] : v[0];
    z_t o;
    o.x = __shfl_sync(0xffffffffu, t.x, p & 31);
    o.y = __shfl_sync(0xffffffffu, t.y, p & 31);
    return o;
  };
  int p = gj_pivot<RPL>(a[0], n, used, nan_singular, &sing);
  z_t pv = bcast(a[0], p);
  z_t inv = gj_recip(pv);
#pragma unroll
  for (int q = 0; q < kGjPanel; q++) {
    if (q >= kb) break;   // uniform
    used |= 1ull << p;
    det = zmul(det, pv);
    if (lane == 0) s.pivrow[j0 + q] = p;
    z_t pr[kGjPanel];
#pragma unroll
    for (int c = 0; c < kGjPanel; c++)
      if (c != q) pr[c] = bcast(a[c], p);
    // row i: A[i][c] - A[i][q] inv A[p][c], and -A[i][q] inv at c = q; the pivot row itself
    // inv A[p][c], and inv at c = q: one factor per row
    z_t g[RPL];
    bool mine[RPL];
#pragma unroll
    for (int r = 0; r < RPL; r++) {
      mine[r] = lane + 32 * r == p;
      g[r] = mine[r] ? inv : zmul(zmk(-a[q][r].x, -a[q][r].y), inv);
      a[q][r] = g[r];
    }
    auto update = [&](int c) {
#pragma unroll
      for (int r = 0; r < RPL; r++) {
        z_t t = mine[r] ? zmk(0, 0) : a[c][r];
        zfma(t, g[r], pr[c]);
        a[c][r] = t;
      }
    };
    if (q + 1 < kGjPanel) {
      update(q + 1);
      if (q + 1 < kb) {
        p = gj_pivot<RPL>(a[q + 1], n, used, nan_singular, &sing);
        pv = bcast(a[q + 1], p);
        inv = gj_recip(pv);
      }
    }
#pragma unroll
    for (int c = 0; c < kGjPanel; c++)
      if (c != q && c != q + 1) update(c);
  }
#pragma unroll
  for (int r = 0; r < RPL; r++)
#pragma unroll
    for (int c = 0; c < kGjPanel; c++) {
      const int i = lane + 32 * r;
      if (i < n && c < kb) T[i * ld + j0 + c] = a[c][r];
    }
  if (lane == 0) {
    s.used = used;
    s.det = det;
    s.sing = sing;
  }
}

// T (row stride ld) in place by all NW warps of the CTA; want_inv = 0: the determinant only
// (rows already used and columns already done are left alone).  s.det = 0 and s.sing = 1 for a
// singular matrix.  Starts and ends with a barrier.
template <int RPL, int NW>
AFQ_D void gj_run(z_t* T, int ld, int n, int want_inv, int nan_singular, GjState& s) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    s.used = 0;
    s.det = zmk(1.0, 0.0);
    s.sing = 0;
  }
  __syncthreads();
  for (int j0 = 0; j0 < n; j0 += kGjPanel) {
    const int kb = min(kGjPanel, n - j0);
    if (warp == 0) gj_panel<RPL>(T, ld, n, j0, kb, nan_singular, s);
    __syncthreads();
    if (s.sing) break;   // uniform
    unsigned long long P = 0;
    z_t R[kGjPanel][RPL];   // the pivot rows at this lane's columns
#pragma unroll
    for (int q = 0; q < kGjPanel; q++) {
      const int p = q < kb ? s.pivrow[j0 + q] : 0;
      if (q < kb) P |= 1ull << p;
#pragma unroll
      for (int r = 0; r < RPL; r++) {
        const int c = lane + 32 * r;
        R[q][r] = (q < kb && c < n) ? T[p * ld + c] : zmk(0, 0);
      }
    }
    const unsigned long long skip = want_inv ? 0 : s.used;
    __syncthreads();
    bool on[RPL];
#pragma unroll
    for (int r = 0; r < RPL; r++) {
      const int c = lane + 32 * r;
      on[r] = c < n && (c < j0 ? want_inv != 0 : c >= j0 + kb);
    }
#pragma unroll 4
    for (int i = warp; i < n; i += NW) {
      if ((skip >> i) & 1) continue;
      z_t* Ti = T + i * ld;
      // the two products of each part in sums of their own: half the dependent chain
      z_t acc[RPL], sub[RPL];
#pragma unroll
      for (int r = 0; r < RPL; r++) {
        acc[r] = on[r] && !((P >> i) & 1) ? Ti[lane + 32 * r] : zmk(0, 0);
        sub[r] = zmk(0, 0);
      }
#pragma unroll
      for (int q = 0; q < kGjPanel; q++) {
        const z_t m = q < kb ? Ti[j0 + q] : zmk(0, 0);   // no branch: loads of all rows in flight
#pragma unroll
        for (int r = 0; r < RPL; r++) {
          acc[r].x = fma(m.x, R[q][r].x, acc[r].x);
          sub[r].x = fma(m.y, R[q][r].y, sub[r].x);
          acc[r].y = fma(m.x, R[q][r].y, acc[r].y);
          sub[r].y = fma(m.y, R[q][r].x, sub[r].y);
        }
      }
#pragma unroll
      for (int r = 0; r < RPL; r++) acc[r] = zmk(acc[r].x - sub[r].x, acc[r].y + sub[r].y);
#pragma unroll
      for (int r = 0; r < RPL; r++)
        if (on[r]) Ti[lane + 32 * r] = acc[r];
    }
    __syncthreads();
  }
  if (warp == 0) {   // inverse permutation and the determinant's sign
    int inv_cnt = 0;
    if (!s.sing)
      for (int a = lane; a < n; a += 32) {
        const int pa = s.pivrow[a];
        s.invp[pa] = a;
        for (int b = a + 1; b < n; b++) inv_cnt += pa > s.pivrow[b];
      }
    inv_cnt = __reduce_add_sync(0xffffffffu, inv_cnt);
    if (lane == 0) {
      if (s.sing)
        s.det = zmk(0, 0);
      else if (inv_cnt & 1)
        s.det = zmk(-s.det.x, -s.det.y);
    }
  }
  __syncthreads();
}

}  // namespace afq
