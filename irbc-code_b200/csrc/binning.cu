// binning.cu -- standalone random-shift cell binning (counting sort) for
// callers that hold particle positions in device memory.
//
// Follows the binning of CollisionStep (Src/solfuncs.cpp:139-147): cell of a
// particle in the grid shifted by (rx, ry, rz) is cindex[floor(bbound(x-rx))]
// [floor(bbound(y-ry))][floor(z-rz+1)], then Cells[c].sol lists the
// particles of each cell in ascending index.  Here that list is the counting
// sort: start[C+1] (exclusive scan of the counts) and order[n] (particle
// indices grouped by cell, ascending within each cell).
#include <cstdint>
#include "irbc.h"
#include "sim.h"

namespace irbc {

// the run of equal cells in consecutive lanes that this lane is in: its first
// lane and, there, its length (all 32 lanes call; cell < 0: none)
__device__ __forceinline__ int cell_run(int c, int lane, int& len) {
  const int before = __shfl_up_sync(0xffffffffu, c, 1);
  const unsigned heads = __ballot_sync(0xffffffffu, lane == 0 || before != c);
  const int first = 31 - __clz(heads & (0xffffffffu >> (31 - lane)));
  const unsigned after = first == 31 ? 0u : heads & (0xffffffffu << (first + 1));
  len = (after ? __ffs(after) - 1 : 32) - first;
  return first;
}

// start itself holds the counters, so that the sort needs no memory of its own:
// the count of cell c is made in start[c + 1], whose exclusive scan is c's first
// place; the places are then handed out by adding to it, which leaves the first
// place of c + 1.
__global__ void __launch_bounds__(256) k_bin_count(DevParams p, const double* x, const double* y, const double* z,
                                                   int64_t n, double rx, double ry, double rz, int* cell, int* count) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int lane = threadIdx.x & 31;
  int c = -1, len;
  if (i < n) {
    const int fx = (int)floor(bbound(x[i] - rx, p.Lx));
    const int fy = (int)floor(bbound(y[i] - ry, p.Ly));
    const int fz = (int)floor(z[i] - rz + 1.0);
    c = cell_of(p, fx, fy, fz);
    cell[i] = c;
  }
  const int first = cell_run(c, lane, len);
  if (c >= 0 && first == lane) atomicAdd(&count[c], len);
}
__global__ void __launch_bounds__(256) k_bin_place(const int* cell, int64_t n, int* next, int* order) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int lane = threadIdx.x & 31;
  const int c = i < n ? cell[i] : -1;
  int len, at = 0;
  const int first = cell_run(c, lane, len);
  if (c >= 0 && first == lane) at = atomicAdd(&next[c], len);
  at = __shfl_sync(0xffffffffu, at, first) + lane - first;
  if (c >= 0) order[at] = (int)i;
}

__device__ __forceinline__ void insertion_sort(int* a, int m) {
  for (int q = 1; q < m; ++q) {
    const int v = a[q];
    int r = q;
    while (r > 0 && a[r - 1] > v) { a[r] = a[r - 1]; --r; }
    a[r] = v;
  }
}
// Ascending particle index within each cell, by sixteen lanes: each holds up to
// kSortPer of the cell's entries and counts the smaller ones.  Fuller cells are
// sorted by insertion by one lane.  5.2 M particles, ten a cell: 55 us; with the
// insertion for every cell and four allocations the whole call took 2.05 ms,
// now 0.19.
constexpr int kSortLanes = 16, kSortPer = 4;
__global__ void __launch_bounds__(256) k_bin_segsort(const int* start, int64_t ncell, int* order) {
  const int64_t c = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / kSortLanes;
  const int lane = threadIdx.x & (kSortLanes - 1);
  const unsigned half = (threadIdx.x & 16) ? 0xffff0000u : 0x0000ffffu;
  if (c >= ncell) return;  // (a whole half-warp)
  const int s0 = start[c], m = start[c + 1] - s0;
  if (m < 2) return;
  int* a = order + s0;
  if (m <= kSortLanes) {  // 97 of 100 cells of ten particles on average
    const int v = lane < m ? a[lane] : 0x7fffffff;
    int r = 0;
#pragma unroll
    for (int u = 0; u < kSortLanes; ++u) r += __shfl_sync(half, v, u, kSortLanes) < v ? 1 : 0;
    __syncwarp(half);
    if (lane < m) a[r] = v;
    return;
  }
  if (m <= kSortLanes * kSortPer) {
    int v[kSortPer], r[kSortPer];
#pragma unroll
    for (int q = 0; q < kSortPer; ++q) {
      v[q] = q * kSortLanes + lane < m ? a[q * kSortLanes + lane] : 0x7fffffff;
      r[q] = 0;
    }
#pragma unroll
    for (int q = 0; q < kSortPer; ++q) {
      if (q * kSortLanes >= m) break;
      for (int u = 0; u < kSortLanes; ++u) {
        const int w = __shfl_sync(half, v[q], u, kSortLanes);
#pragma unroll
        for (int k = 0; k < kSortPer; ++k) r[k] += w < v[k] ? 1 : 0;
      }
    }
    __syncwarp(half);
#pragma unroll
    for (int q = 0; q < kSortPer; ++q)
      if (q * kSortLanes + lane < m) a[r[q]] = v[q];
    return;
  }
  if (lane == 0) insertion_sort(a, m);
}
// The same by a thread per cell, for cells with few entries, where most of sixteen
// lanes have none.  The whole call, sixteen lanes and this: 134 M cells with 2 M
// particles 5.9 and 1.3 ms, 0.5 M cells with 1, 2 and 4 a cell 81 and 59, 97 and
// 69, 120 and 94 us; 65,000 cells with 4 and 8 a cell 54 and 55, 60 and 66.  More a
// cell depends on their order (5.2 M particles, ten a cell: in cell order 164 and
// 194 us, in no order 199 and 181).
__global__ void __launch_bounds__(256) k_bin_segsort_sparse(const int* start, int64_t ncell, int* order) {
  const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= ncell) return;
  const int s0 = start[c];
  insertion_sort(order + s0, start[c + 1] - s0);
}
constexpr int kSparse = 4;  // particles a cell

// The full sort; part: scan_part_ints(C) of scratch, which may be order.
void bin_particles(const DevParams& p, const double* x, const double* y, const double* z, int64_t n,
                   double rx, double ry, double rz, int* cell, int* start, int* order, int* part, cudaStream_t st) {
  const unsigned nb = (unsigned)((n + 255) / 256);
  cudaMemsetAsync(start, 0, sizeof(int) * (p.ncell + 1), st);
  if (n == 0) return;
  if (p.ncell == 0) {  // a side shorter than a cell: no cell to be in
    cudaMemsetAsync(cell, 0, sizeof(int) * n, st);
    return;
  }
  k_bin_count<<<nb, 256, 0, st>>>(p, x, y, z, n, rx, ry, rz, cell, start + 1);
  launch_scan3(start + 1, nullptr, nullptr, start + 1, nullptr, nullptr, nullptr, p.ncell, part, st);
  k_bin_place<<<nb, 256, 0, st>>>(cell, n, start + 1, order);
  if (n < kSparse * p.ncell)
    k_bin_segsort_sparse<<<(unsigned)((p.ncell + 255) / 256), 256, 0, st>>>(start, p.ncell, order);
  else
    k_bin_segsort<<<(unsigned)((p.ncell * kSortLanes + 255) / 256), 256, 0, st>>>(start, p.ncell, order);
}

}  // namespace irbc
