// FP64 form on the int8 tensor cores (oz_gemm.cuh): the contraction stages whose operands
// are written as signed 8-bit digits, 55 bits below each row's power of two.  Each walker's
// result (an orbital's column of the propagation, a walker's exchange energy) agrees with an
// FP64 product's in its norm; where the digits do not hold that (rows whose large entries
// meet only zeros of the other operand, infinities) or a wait times out, the product's gate
// opens on the device, and the caller's next launch, the FP64 pipe's form of the product, runs
// instead of returning at once.
#pragma once
#include <stdint.h>
#include "afq_common.cuh"

namespace afq {

struct OzState;

struct OzInit {
  int N, n, nchol, nw, order;
  const z_t* Lh;         // [nchol][2][n][N] half-rotated factors (null: no Cholesky energy)
  const z_t* SpvnT;      // dense [nchol][2nN] (null: vbias stays on the CSR path)
  const z_t* Vakbl;      // dense [2nN][2nN] or null
  const z_t* Spvn;       // dense [N^2][nchol] of complex values, or null
  const double* Spvn_r;  // dense [N^2][nchol] of real values, or null
  long long spvn_nnz, SpvnT_nnz, Vakbl_nnz;
  const z_t* P;          // Propg1 [N][N]
};

// Slices the static operands of the products that take this path (rules in oz.cu) and
// allocates their workspaces; *out stays null when none does or memory is short.
cudaError_t oz_create(const OzInit& in, OzState** out, cudaStream_t st);
void oz_destroy(OzState* o);
// Products of G [nw][2nN] with a static operand, out [rows][nw]: vbias (SpvnT), the Coulomb
// vector (Lh), Vakbl G; then the other products.
enum OzProduct { OZ_VBIAS, OZ_COULOMB, OZ_VAKBL, OZ_NG, OZ_VHS = OZ_NG, OZ_PROPAGATE, OZ_EXCHANGE,
                 OZ_NPRODUCTS };
// The gate of the last call of a product with G or of vHS; that of the exchange, per walker;
// and per product the walkers whose result was left to the FP64 pipe (waits for the device).
OzGate oz_gate(const OzState* o, int product);
const int* oz_exchange_gate(const OzState* o);
cudaError_t oz_redone(const OzState* o, unsigned long long* redone);
bool oz_has_gsite(const OzState* o, int site);
int oz_gsite_launches();
cudaError_t oz_gsite(OzState* o, int site, const z_t* Gc, z_t* out, cudaStream_t st);
// vHS [nw][N][N] from X [nchol][nw].
bool oz_has_vhs(const OzState* o);
cudaError_t oz_vhs(OzState* o, const z_t* X, z_t* vHS, cudaStream_t st);
// W [nw][N][2n] <- P (sum_k (i vHS)^k / k!) P W, on the FP64 pipe for walkers the digits do not
// hold; S, T, Wt scratch [nw][2n][N].
bool oz_has_propagate(const OzState* o);
int oz_propagate_launches(const OzState* o);
cudaError_t oz_propagate(OzState* o, const z_t* P, z_t* W, const z_t* vHS, z_t* S, z_t* T,
                         z_t* Wt, cudaStream_t st);
bool oz_has_exchange(const OzState* o, int nwalk);
int oz_exchange_launches(const OzState* o, int nwalk);
// Exchange partial sums of nwalk walkers, one per Cholesky vector: Kpart[nwalk][2][nblk] with
// nblk = nchol.
cudaError_t oz_exchange(OzState* o, const z_t* Gc, int nwalk, z_t* Kpart, int nblk,
                        cudaStream_t st);
// Exchange energies of caller-owned device buffers through a fixed scratch (no allocation, no
// synchronisation): ek[nwalk].  Whether Lh is real is found on the device.
struct OzBuffers {
  int8_t *a, *g;              // digits of a chunk of Lh rows and of G rows
  size_t a_bytes, g_bytes;
  double *a_scale, *g_scale;  // a_rows, 2 g_rows (per spin) row scales
  int a_rows, g_rows;
  double* T;
  size_t t_bytes;
  z_t* part;                  // partial sums
  double* norms;              // their norms (parts)
  long long parts;
  int* flags;                 // timeout flags, Lh complex
  double* sa2;                // [2] squares of the Lh row scales
  int* gate;                  // [nwalk], as oz_exchange_gate
};
bool oz_exchange_buffers_fit(const OzBuffers& b, int N, int n, int nc, int nw);
cudaError_t oz_exchange_buffers(const OzBuffers& b, const z_t* Lh, const z_t* Gc, int N, int n,
                                int nc, int nw, z_t* ek, cudaStream_t st);
// Timeout flags raised by the kernels (0 when clean), read into pinned memory on the handle's
// stream (a copy on the legacy stream would wait for the work of the caller's blocking streams),
// and the bound of their waits.
cudaError_t oz_error(OzState* o, int* flags, cudaStream_t st);
cudaError_t oz_set_wait_clocks(long long clocks);

}  // namespace afq
