// binning_noalloc.cu -- the random-shift binning of irbc_bin_particles
// without any memory allocation, for callers that cannot allocate device
// memory while they run: code inside an allocator callback or a memory
// pool's reservation path, host threads that must not take the driver's
// allocation lock, and embedders whose device memory is budgeted up front.
//
// Its scratch (the scan's partial sums; start holds the counters) lives in one
// file-scope __device__ array of fixed size, present on every GPU that loads
// the library until the process exits.  The caller passes the particle
// positions and the three output arrays, all in device memory.
#include <cstdint>
#include <mutex>

#include "irbc.h"
#include "sim.h"

namespace irbc {

// limits of the static scratch
constexpr int64_t kNoAllocMaxCells = 1 << 20;                      // 1,048,576 cells
constexpr int64_t kNoAllocScanBlocks = (kNoAllocMaxCells + 1024) / 1024 + 1;  // scan tiles of 1024
constexpr int64_t kNoAllocInts = 3 * kNoAllocScanBlocks;
static_assert(kNoAllocScanBlocks <= kScanLook, "no room for the sums of groups");

// 3 ints per scan tile
static __device__ __align__(256) int g_bin_scratch[kNoAllocInts];

namespace {
// Device address of g_bin_scratch per device ordinal.  The host symbol is a
// stand-in and must not be handed to a kernel, so the address is looked up
// once per device with cudaGetSymbolAddress while that device is current,
// and kept for the life of the process.  A cudaDeviceReset unloads the
// module and can move the array, leaving the kept address stale: this entry
// point must not be used on a device after it has been reset.
std::mutex g_scratch_mu;
int* g_scratch_dev[256] = {nullptr};

int scratch_for_current_device(int** out) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 256) return IRBC_ERR_CUDA;
  std::lock_guard<std::mutex> lock(g_scratch_mu);
  if (!g_scratch_dev[dev]) {
    void* ptr = nullptr;
    if (cudaGetSymbolAddress(&ptr, g_bin_scratch) != cudaSuccess || !ptr) return IRBC_ERR_CUDA;
    g_scratch_dev[dev] = static_cast<int*>(ptr);
  }
  *out = g_scratch_dev[dev];
  return 0;
}
}  // namespace

}  // namespace irbc

using namespace irbc;

extern "C" int irbc_bin_particles_noalloc(const irbc_params* p, const double* x, const double* y,
                                          const double* z, int64_t n, double rx, double ry, double rz,
                                          int32_t* cell, int32_t* start, int32_t* order) {
  if (!p || n < 0 || (n > 0 && (!x || !y || !z || !cell || !order)) || !start) return IRBC_ERR_ARG;
  if (p->a != 1.0 || p->Lx <= 0 || p->Ly <= 0 || p->Lz <= 0 || n >= (1LL << 31)) return IRBC_ERR_ARG;
  if (!(rx >= 0 && rx < 1 && ry >= 0 && ry < 1 && rz >= 0 && rz < 1)) return IRBC_ERR_ARG;
  DevParams d{};  // the grid fields the binning reads
  d.a = p->a; d.Lx = p->Lx; d.Ly = p->Ly; d.Lz = p->Lz;
  d.nx = (int)(p->Lx / p->a);
  d.ny = (int)(p->Ly / p->a);
  d.nz = (int)(p->Lz / p->a) + 1;
  d.ncell = (int64_t)d.nx * d.ny * d.nz;
  if (d.ncell > kNoAllocMaxCells) return IRBC_ERR_CAPACITY;  // box beyond the static scratch
  int* base = nullptr;
  int rc = scratch_for_current_device(&base);
  if (rc) return rc;
  const cudaStream_t st = 0;
  bin_particles(d, x, y, z, n, rx, ry, rz, cell, start, order, base, st);
  if (cudaGetLastError() != cudaSuccess) return IRBC_ERR_CUDA;
  return cudaStreamSynchronize(st) == cudaSuccess ? 0 : IRBC_ERR_CUDA;
}
