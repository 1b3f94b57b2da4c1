// fp32.cuh -- (part of fast.cu) the FP32-bulk solvent: positions and velocities stored as
// float4 (x, y, z, inside-flag bits) and (vx, vy, vz, reference-index bits),
// 32 bytes per particle.  Free flight, walls, wrap, binning and the SRD
// rotation run in float; the per-cell momentum and relative-energy sums are
// accumulated in double; particles near the membrane are promoted to double
// for reflectionFed and its cubic root solve; the membrane itself stays FP64.
#include <cstdio>
#include "fast.h"
#include "fp32.h"
#include "cells_tile.cuh"

namespace irbc {

static inline unsigned nbf(int64_t n, int t) { return (unsigned)((n + t - 1) / t); }

// ---- conversions between the FP64 arrays (set-up, state exchange) and FP32
__global__ void k_to_f32(Solvent s, SolventF f) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= s.n) return;
  f.pos[i] = make_float4((float)s.x[i], (float)s.y[i], (float)s.z[i], __int_as_float(s.indio[i]));
  const SolVel r = s.v[i];
  f.vel[i] = make_float4((float)r.vx, (float)r.vy, (float)r.vz, __int_as_float(r.id));
  f.pid[i] = s.pid[i];
}
__global__ void k_to_f64(SolventF f, Solvent s) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= s.n) return;
  float4 p = f.pos[i], v = f.vel[i];
  s.x[i] = p.x; s.y[i] = p.y; s.z[i] = p.z; s.indio[i] = __float_as_int(p.w);
  SolVel r;
  r.vx = v.x; r.vy = v.y; r.vz = v.z; r.id = __float_as_int(v.w); r.pad = 0;
  s.v[i] = r;
  s.pid[i] = f.pid[i];
}
void f32_from_f64(Solvent& s, SolventF& f, cudaStream_t st) {
  if (s.n) k_to_f32<<<nbf(s.n, 256), 256, 0, st>>>(s, f);
}
void f32_to_f64(SolventF& f, Solvent& s, cudaStream_t st) {
  if (s.n) k_to_f64<<<nbf(s.n, 256), 256, 0, st>>>(f, s);
}

// ---- collision --------------------------------------------------------------
__device__ __forceinline__ int shifted_cell_f(const DevParams& p, float4 q, const double r[3]) {
  int fx = (int)floor(bbound((double)q.x - r[0], p.Lx));
  int fy = (int)floor(bbound((double)q.y - r[1], p.Ly));
  int fz = (int)floor((double)q.z - r[2] + 1.0);
  return cell_of(p, fx, fy, fz);
}

// block `bid` of the count: kCountPer particles per thread
__device__ __forceinline__ void count_f_block(const DevParams& p, const SolventF& f, int* cnt, int* slot,
                                              uint64_t eoff, int64_t bid) {
  const uint64_t epoch = epoch_of(p, eoff);
  // the grid shift, drawn once per block
  __shared__ double sr[3];
  if (threadIdx.x == 0) grid_shift(p, epoch, sr);
  __syncthreads();
  const double r[3] = {sr[0], sr[1], sr[2]};
  const int64_t i0 = bid * blockDim.x * kCountPer + threadIdx.x;
  int c[kCountPer];
#pragma unroll
  for (int u = 0; u < kCountPer; ++u) {
    const int64_t i = i0 + (int64_t)u * blockDim.x;
    c[u] = i < f.n ? shifted_cell_f(p, f.pos[i], r) : -1;
  }
  int sl[kCountPer];
  claim_slots<kCountPer>(cnt, c, i0, blockDim.x, f.n, sl);
#pragma unroll
  for (int u = 0; u < kCountPer; ++u) {
    const int64_t i = i0 + (int64_t)u * blockDim.x;
    if (i < f.n) {
      f.pid[i] = c[u];  // the cell of this collision
      slot[i] = sl[u];
    }
  }
}
__global__ void __launch_bounds__(256) k_count_f(DevParams p, SolventF f, int* cnt, int* slot, uint64_t eoff) {
  count_f_block(p, f, cnt, slot, eoff, blockIdx.x);
}

__device__ __forceinline__ void perm_f_item(const int* __restrict__ key, const int* __restrict__ slot,
                                            const int* __restrict__ start, int64_t n, int* __restrict__ perm,
                                            int64_t i) {
  if (i >= n) return;
  perm[(int64_t)start[key[i]] + slot[i]] = (int)i;
}
__global__ void k_perm_f(const int* __restrict__ key, const int* __restrict__ slot, const int* __restrict__ start,
                         int64_t n, int* __restrict__ perm) {
  perm_f_item(key, slot, start, n, perm, (int64_t)blockIdx.x * blockDim.x + threadIdx.x);
}

// physical re-sort by collision cell every kResortEvery collisions
__device__ __forceinline__ void gather_f_item(const SolventF& f, const int* __restrict__ perm, int64_t j) {
  if (j >= f.n) return;
  const int i = perm[j];
  f.pos2[j] = f.pos[i];
  f.vel2[j] = f.vel[i];
  f.pid2[j] = f.pid[i];
}
__device__ __forceinline__ void copy_back_f_item(const SolventF& f, int64_t j) {
  if (j >= f.n) return;
  f.pos[j] = f.pos2[j];
  f.vel[j] = f.vel2[j];
  f.pid[j] = f.pid2[j];
}
__global__ void k_gather_f(SolventF f, const int* __restrict__ perm) {
  gather_f_item(f, perm, (int64_t)blockIdx.x * blockDim.x + threadIdx.x);
}
__global__ void k_copy_back_f(SolventF f) { copy_back_f_item(f, (int64_t)blockIdx.x * blockDim.x + threadIdx.x); }

void launch_collide_count_f(const DevParams& p, SolventF& f, Solvent& s, Cells& c, uint64_t epoch,
                            cudaStream_t st) {
  cudaMemsetAsync(c.cnt, 0, sizeof(int) * c.n, st);
  if (f.n) k_count_f<<<nbf(f.n, 256 * kCountPer), 256, 0, st>>>(p, f, c.cnt, s.slot, epoch);
}

// per-cell statistics (sums in double, reference particle order) and the
// float rotation: k_cells_tile<true> (cells_tile.cuh)
int launch_collide_finish_f(const DevParams& p, SolventF& f, Solvent& s, Cells& c, Membrane& m, uint64_t epoch,
                            cudaStream_t st, bool resort) {
  const int scans = launch_collide_scan(p, c, m, st);
  if (f.n) k_perm_f<<<nbf(f.n, 256), 256, 0, st>>>(f.pid, s.slot, c.start, f.n, s.perm);
  k_cells_tile<true><<<cells_tile_blocks(c.n), 32 * kTileWarps, 0, st>>>(p, s, f, c, m, epoch);
  if (resort) launch_resort_f(f, s, st);
  return scans + 1 + (f.n ? (resort ? 3 : 1) : 0);
}

void launch_resort_f(SolventF& f, Solvent& s, cudaStream_t st) {
  if (f.n) {
    k_gather_f<<<nbf(f.n, 256), 256, 0, st>>>(f, s.perm);
    k_copy_back_f<<<nbf(f.n, 256), 256, 0, st>>>(f);
  }
}

}  // namespace irbc
