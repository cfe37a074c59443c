// Exchange energy of a walker batch with no device allocation at all.
//
// Some callers cannot call cudaMalloc: code that records its work into a CUDA graph
// under stream capture (an allocation there breaks the capture), and host frameworks
// that hand every byte of device memory to their own pool and forbid allocations after
// start-up.  This entry point serves them: the caller passes device inputs and outputs,
// and what the exchange needs besides (partial sums, operand digits, a chunk of the products)
// lives in fixed file-scope device arrays instead of per-handle buffers.
#include <cstdint>
#include <mutex>

#include "../../include/afqmc_b200.h"
#include "afq_kernels.h"
#include "afq_oz.h"

namespace {

// Partial sums of the exchange contraction: one complex value per (walker, spin,
// Cholesky block); 2^18 of them = 4 MiB, held by every device that loads the library.
constexpr long long kMaxExchangePartials = 1LL << 18;
static __device__ __align__(256) z_t g_exchange_scratch[kMaxExchangePartials];

// Chunks of the digit products (oz.cu): 48 MiB of T (five waves of 64 KB output tiles), 24
// MiB of G digits and 6 MiB of Lh digits with their row scales and norms, loaded with this file's
// kernels by the first call on a device.  With 40 and 20 MiB, 96 walkers at 200 orbitals
// split into two uneven chunks: 10.8 against 7.0 ms (28.0 ms on the FP64 pipe).
constexpr size_t kTBytes = 48u << 20, kGBytes = 24u << 20, kABytes = 6u << 20;
constexpr int kGRows = 16384, kARows = 4096;
struct Scratch {
  double T[kTBytes / 8];
  int8_t g[kGBytes], a[kABytes];
  double g_scale[2 * kGRows], a_scale[kARows];
  int flags[8];
  double norms[kMaxExchangePartials], sa2[2];
  int gate[kMaxExchangePartials / 2];
};
static __device__ __align__(256) Scratch g_oz_scratch;

constexpr int kMaxDevices = 64;
std::mutex g_scratch_mu;
z_t* g_scratch_addr[kMaxDevices] = {};
Scratch* g_oz_addr[kMaxDevices] = {};

// EK[w] = 1/2 sum over spins and Cholesky blocks of the partials, in a fixed order.
__global__ void __launch_bounds__(128)
exchange_finish_kernel(const z_t* __restrict__ part, int nblk, z_t* __restrict__ ek,
                       const int* __restrict__ gate) {
  const int w = blockIdx.x;
  if (gate && gate[w] == 0) return;
  __shared__ z_t red[4];
  z_t s = zmk(0, 0);
  for (int q = threadIdx.x; q < 2 * nblk; q += blockDim.x)
    s = zadd(s, part[(long long)w * 2 * nblk + q]);
  s = block_zsum(s, red);
  if (threadIdx.x == 0) ek[w] = zscale(s, 0.5);
}

}  // namespace

extern "C" afq_status afq_exchange_energy_noalloc(const double* Lh, const double* Gc, int nmo,
                                                  int naea, int nchol, int nwalk, double* ek,
                                                  void* stream) {
  if (!Lh || !Gc || !ek || nmo <= 0 || naea <= 0 || nchol <= 0 || nwalk <= 0)
    return AFQ_ERR_ARG;
  // the exchange kernel reads Lh and Gc with 16-byte asynchronous copies and the finish
  // kernel stores whole complex values: a buffer that is only 8-byte aligned (a view at an
  // odd double offset) would fault on the device, so it is refused here
  if ((reinterpret_cast<uintptr_t>(Lh) | reinterpret_cast<uintptr_t>(Gc) |
       reinterpret_cast<uintptr_t>(ek)) & 15u)
    return AFQ_ERR_ARG;
  if (naea > 96 || naea > nmo) return AFQ_ERR_UNSUPPORTED;
  int nblk = 0;
  afq::launch_exchange(nullptr, nullptr, nmo, naea, nchol, nwalk, nullptr, &nblk, nullptr);
  const long long used = 2LL * nwalk * nblk;
  if (used > kMaxExchangePartials) return AFQ_ERR_UNSUPPORTED;   // batch too large for scratch
  // one CTA row per group of 96 / naea walkers: the grid's y extent is at most 65535
  if ((nwalk + 96 / naea - 1) / (96 / naea) > 65535) return AFQ_ERR_UNSUPPORTED;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return AFQ_ERR_CUDA;
  z_t* scratch = nullptr;
  Scratch* oz = nullptr;
  {
    // set-up, once per device with that device current: the host-side symbol is only a
    // stand-in, the kernels need the device address of the array
    std::lock_guard<std::mutex> lock(g_scratch_mu);
    if (!g_scratch_addr[dev]) {
      void* p = nullptr;
      if (cudaGetSymbolAddress(&p, g_exchange_scratch) != cudaSuccess || !p) return AFQ_ERR_CUDA;
      void* q = nullptr;
      if (cudaGetSymbolAddress(&q, g_oz_scratch) != cudaSuccess || !q) return AFQ_ERR_CUDA;
      g_oz_addr[dev] = static_cast<Scratch*>(q);
      g_scratch_addr[dev] = static_cast<z_t*>(p);
    }
    scratch = g_scratch_addr[dev];
    oz = g_oz_addr[dev];
  }
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const afq::OzBuffers b{oz->a, oz->g, kABytes, kGBytes, oz->a_scale, oz->g_scale, kARows, kGRows,
                         oz->T, kTBytes, scratch, oz->norms, kMaxExchangePartials, oz->flags,
                         oz->sa2, oz->gate};
  const int* gate = nullptr;   // after the digit products: only what they leave to the FP64 pipe
  if (afq::oz_exchange_buffers_fit(b, nmo, naea, nchol, nwalk)) {
    if (afq::oz_exchange_buffers(b, reinterpret_cast<const z_t*>(Lh),
                                 reinterpret_cast<const z_t*>(Gc), nmo, naea, nchol, nwalk,
                                 reinterpret_cast<z_t*>(ek), st) != cudaSuccess)
      return AFQ_ERR_CUDA;
    gate = oz->gate;
  } else if (cudaMemsetAsync(scratch, 0, sizeof(z_t) * used, st) != cudaSuccess) {
    return AFQ_ERR_CUDA;   // the array keeps the previous call's contents
  }
  int nb = 0;
  if (afq::launch_exchange(reinterpret_cast<const z_t*>(Lh), reinterpret_cast<const z_t*>(Gc), nmo,
                           naea, nchol, nwalk, scratch, &nb, st, gate) != cudaSuccess)
    return AFQ_ERR_CUDA;
  exchange_finish_kernel<<<nwalk, 128, 0, st>>>(scratch, nb, reinterpret_cast<z_t*>(ek), gate);
  return cudaGetLastError() == cudaSuccess ? AFQ_OK : AFQ_ERR_CUDA;
}
