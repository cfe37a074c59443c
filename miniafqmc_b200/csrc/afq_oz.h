// FP64 form on the int8 tensor cores (oz_gemm.cuh): the contraction stages whose operands
// are written as signed 8-bit digits.  Results agree with an FP64 product to FP64 rounding
// (the digits keep 55 bits below each row's power of two).
#pragma once
#include "afq_common.cuh"

namespace afq {

struct OzState;

struct OzInit {
  int N, n, nchol, nw;
  const z_t* Lh;   // [nchol][2][n][N] half-rotated factors (null: no exchange)
};

// Slices the static operands of the products that take this path (rules in oz.cu) and
// allocates their workspaces; *out stays null when none does or memory is short.
cudaError_t oz_create(const OzInit& in, OzState** out, cudaStream_t st);
void oz_destroy(OzState* o);
bool oz_has_exchange(const OzState* o, int nwalk);
int oz_exchange_launches(const OzState* o, int nwalk);
// Exchange partial sums of nwalk walkers, one per Cholesky vector: Kpart[nwalk][2][nblk] with
// nblk = nchol.
cudaError_t oz_exchange(OzState* o, const z_t* Gc, int nwalk, z_t* Kpart, int nblk,
                        cudaStream_t st);
// Timeout flags raised by the kernels (0 when clean), and the bound of their waits.
cudaError_t oz_error(OzState* o, int* flags);
cudaError_t oz_set_wait_clocks(long long clocks);

}  // namespace afq
