// multi.cuh -- (part of fast.cu) one launch per phase over a cohort of FP32
// simulations (multi.h): the fused kernels of the streaming, the membrane
// chain and the collision's particle phases.  Each block reads its member
// and its block index within that member from the phase's block table
// (KM_MEMBER) and runs the single-simulation kernel's device code.
#include "multi.h"

namespace irbc {

// ---- streaming -------------------------------------------------------------
__global__ void __launch_bounds__(256, 6) km_stream_bulk(Member* __restrict__ mem, const int2* __restrict__ tab, int H,
                                                        int par) {
  KM_MEMBER;
  // copies: the descriptor is not reloaded after the stores below
  const DevParams p = M.p;
  const SolventArrays s = arrays_of(M.s, M.f);
  const NearQueue h = queue_of(M.fb, par);
  const unsigned char* __restrict__ cflag = M.c.flag;
  const int64_t n = M.f.n;
  // the queue of the next stretch starts empty
  if (b == 0 && threadIdx.x == 0) M.fb.qn[par ^ 1] = M.fb.qn[4 + (par ^ 1)] = 0;
  for (int pass = 0; pass < kMultiStreamPasses; ++pass) {
    const int64_t i = ((int64_t)b * kMultiStreamPasses + pass) * blockDim.x + threadIdx.x;
    if (i >= n) break;
    bulk_f_item<false>(p, s, cflag, h, H, i, s.pos[i], s.vel[i]);
  }
}

// a block's copy of what the near-membrane kernel reads of its member
struct NearMember {
  DevParams p;
  SolventArrays s;
  NearArgs A;
};
template <int G, int KEEP, bool ONE>
__global__ void __launch_bounds__(kNearT, kNearMinBlocks)
    km_near(const Member* __restrict__ mem, const int2* __restrict__ tab, int H, int par) {
  __shared__ __align__(16) unsigned char raw[sizeof(NearMember)];
  __shared__ unsigned short kept[kNearT / G][KEEP];
  NearMember& N = *reinterpret_cast<NearMember*>(raw);
  const int2 e = __ldg(tab + blockIdx.x);
  const Member& M = mem[e.x];
  if (threadIdx.x == 0) {
    N.s = arrays_of(M.s, M.f);
    N.A = near_of(M.p, M.c, M.fb, par, 0, 0);
  }
  for (int i = threadIdx.x; i < (int)sizeof(DevParams) / 4; i += blockDim.x) ((int*)&N.p)[i] = ((const int*)&M.p)[i];
  __syncthreads();
  near_groups<float, G, KEEP, ONE>(N.p, N.s, N.A, H, kept[threadIdx.x / G], e.y, kNearBlocksMember);
}

int multi_stream(const MultiPlan& P, int H, int par, cudaStream_t st, cudaEvent_t snap) {
  km_stream_bulk<<<P.blocks[MP_STREAM], 256, 0, st>>>(P.mem, P.table(MP_STREAM), H, par);
  if (snap) cudaStreamWaitEvent(st, snap, 0);
  const int n0 = P.blocks[MP_NEAR_SHORT], n1 = P.blocks[MP_NEAR_LONG];
  const auto few = H == 1 ? km_near<kShortGOne, kShortKeep, true> : km_near<kShortGMember, kShortKeep, false>;
  if (n0 > 0) few<<<n0, kNearT, 0, st>>>(P.mem, P.table(MP_NEAR_SHORT), H, par);
  if (n1 > 0) km_near<kLongG, kLongKeep, false><<<n1, kNearT, 0, st>>>(P.mem, P.table(MP_NEAR_LONG), H, par);
  return 1 + (n0 > 0) + (n1 > 0);
}

// ---- membrane ----------------------------------------------------------------
// a cluster per member; the descriptor's parts are copied to shared memory,
// so that they are not read again from global memory after the kernel's stores
struct SegMember {
  DevParams p;
  Membrane m;
  FastBufs f;
};
__device__ __forceinline__ void seg_member(const Member& M, SegMember& S) {
  auto copy = [](void* d, const void* s, int bytes) {
    for (int i = threadIdx.x; i < bytes / 4; i += blockDim.x) ((int*)d)[i] = ((const int*)s)[i];
  };
  copy(&S.p, &M.p, sizeof(DevParams));
  copy(&S.m, &M.m, sizeof(Membrane));
  copy(&S.f, &M.fb, sizeof(FastBufs));
  __syncthreads();
}
#define KM_SEG_MEMBER                                            \
  __shared__ __align__(16) unsigned char raw[sizeof(SegMember)]; \
  SegMember& S = *reinterpret_cast<SegMember*>(raw);             \
  const int2 e = __ldg(tab + blockIdx.x);                        \
  seg_member(mem[e.x], S)
__global__ void __launch_bounds__(kSegT) km_membrane(const Member* __restrict__ mem, const int2* __restrict__ tab,
                                                     uint64_t eoff, int H) {
  extern __shared__ __align__(16) unsigned char seg_sh[];
  KM_SEG_MEMBER;
  membrane_segment(S.p, S.m, S.f, epoch_of(S.p, eoff), H, SEG_WHOLE, seg_sh);
}
__global__ void __launch_bounds__(kWideT) km_wide_first(const Member* __restrict__ mem, const int2* __restrict__ tab) {
  KM_SEG_MEMBER;
  wide_first_block(S.p, S.m, S.f, SEG_WHOLE, e.y);
}
__global__ void __launch_bounds__(kWideT) km_wide_tri(const Member* __restrict__ mem, const int2* __restrict__ tab) {
  KM_SEG_MEMBER;
  wide_tri_block(S.p, S.m, S.f, e.y);
}
__global__ void __launch_bounds__(kSegT) km_wide_terms(const Member* __restrict__ mem, const int2* __restrict__ tab) {
  extern __shared__ __align__(16) unsigned char seg_sh[];
  KM_SEG_MEMBER;
  wide_terms_block(S.p, S.m, S.f, SEG_WHOLE, e.y, seg_sh);
}
__global__ void __launch_bounds__(kWideT) km_wide_gather(const Member* __restrict__ mem, const int2* __restrict__ tab,
                                                         uint64_t eoff, int s, int more) {
  __shared__ TailSmem tail;
  KM_SEG_MEMBER;
  wide_gather_block(S.p, S.m, S.f, epoch_of(S.p, eoff), s, SEG_WHOLE, more, e.y, tail);
}
__global__ void __launch_bounds__(kRecordT) km_tri_records(const Member* __restrict__ mem, const int2* __restrict__ tab,
                                                           int H) {
  __shared__ RecordSmem S;
  const int2 e = __ldg(tab + blockIdx.x);
  const Member& M = mem[e.x];
  records_block(M.p, M.fb, 0, H, 0, e.y, S);
}

int multi_membrane(const MultiPlan& P, uint64_t eoff, int H, cudaStream_t st) {
  const int2* tab = P.table(MP_MEMBRANE);
  for (const MultiPlan::Seg& s : P.seg) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(s.members * s.nc);
    cfg.blockDim = dim3(kSegT);
    cfg.dynamicSmemBytes = s.smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = s.nc;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, km_membrane, (const Member*)P.mem, tab, eoff, H);
    tab += s.members * s.nc;
  }
  const int wide = P.blocks[MP_WIDE_FIRST] > 0 ? H : 0;
  if (wide) km_wide_first<<<P.blocks[MP_WIDE_FIRST], kWideT, 0, st>>>(P.mem, P.table(MP_WIDE_FIRST));
  for (int s = 0; s < wide; ++s) {
    km_wide_tri<<<P.blocks[MP_WIDE_TRI], kWideT, 0, st>>>(P.mem, P.table(MP_WIDE_TRI));
    km_wide_terms<<<P.blocks[MP_WIDE_TERMS], kSegT, P.wide_smem, st>>>(P.mem, P.table(MP_WIDE_TERMS));
    km_wide_gather<<<P.blocks[MP_WIDE_GATHER], kWideT, 0, st>>>(P.mem, P.table(MP_WIDE_GATHER), eoff, s, s + 1 < H);
  }
  km_tri_records<<<P.blocks[MP_RECORDS], kRecordT, 0, st>>>(P.mem, P.table(MP_RECORDS), H);
  return (int)P.seg.size() + (wide ? 1 + 3 * wide : 0) + 1;
}

// ---- collision: particle phases ---------------------------------------------------
__global__ void __launch_bounds__(256) km_count(Member* __restrict__ mem, const int2* __restrict__ tab,
                                                uint64_t eoff) {
  KM_MEMBER;
  count_f_block(M.p, M.f, M.c.cnt, M.s.slot, eoff, b);
}
__global__ void __launch_bounds__(256) km_perm(Member* __restrict__ mem, const int2* __restrict__ tab) {
  KM_MEMBER;
  perm_f_item(M.f.pid, M.s.slot, M.c.start, M.f.n, M.s.perm, (int64_t)b * blockDim.x + threadIdx.x);
}
__global__ void __launch_bounds__(32 * kTileWarps) km_tile(Member* __restrict__ mem, const int2* __restrict__ tab,
                                                           uint64_t eoff) {
  KM_MEMBER;
  // copies: the descriptor is not reloaded after the tile's stores
  const DevParams p = M.p;
  Solvent s = M.s;
  SolventF f = M.f;
  const Cells c = M.c;
  const Membrane m = M.m;
  cells_tile_block<true>(p, s, f, c, m, eoff, b);
}
__global__ void __launch_bounds__(256) km_move(Member* __restrict__ mem, const int2* __restrict__ tab, int back) {
  KM_MEMBER;
  const int64_t j = (int64_t)b * blockDim.x + threadIdx.x;
  if (back) copy_back_f_item(M.f, j);
  else gather_f_item(M.f, M.s.perm, j);
}

int multi_collide_count(const MultiPlan& P, uint64_t eoff, cudaStream_t st) {
  km_count<<<P.blocks[MP_COUNT], 256, 0, st>>>(P.mem, P.table(MP_COUNT), eoff);
  return 1;
}

int multi_collide_back(const MultiPlan& P, uint64_t eoff, bool resort, cudaStream_t st) {
  km_perm<<<P.blocks[MP_PERM], 256, 0, st>>>(P.mem, P.table(MP_PERM));
  km_tile<<<P.blocks[MP_TILE], 32 * kTileWarps, 0, st>>>(P.mem, P.table(MP_TILE), eoff);
  if (!resort) return 2;
  km_move<<<P.blocks[MP_MOVE], 256, 0, st>>>(P.mem, P.table(MP_MOVE), 0);
  km_move<<<P.blocks[MP_MOVE], 256, 0, st>>>(P.mem, P.table(MP_MOVE), 1);
  return 4;
}

// ---- kernel limits (host) ---------------------------------------------------------------
// Every kernel's dynamic shared-memory limit on the current device, set
// before any launch: irbc_create calls this for each new simulation, so a
// launch issued by one host thread never races another thread's first-
// launch attribute call (the request server sets new simulations up on
// threads of their own while others step).
void set_kernel_limits() {
  const auto dyn = cudaFuncAttributeMaxDynamicSharedMemorySize;
  cudaFuncSetAttribute(k_membrane, dyn, kSegSmemMax);
  cudaFuncSetAttribute(km_membrane, dyn, kSegSmemMax);
  cudaFuncSetAttribute(k_wide_terms, dyn, kSegSmemMax);
  cudaFuncSetAttribute(km_wide_terms, dyn, kSegSmemMax);
  // clusters of sixteen blocks (the discocyte's)
  cudaFuncSetAttribute(k_membrane, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  cudaFuncSetAttribute(km_membrane, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  set_collide_kernel_limits();
}

// ---- the tables' sizes (host) -------------------------------------------------------
void multi_blocks(const Member& M, int out[MP_NPHASE]) {
  const int64_t ns = M.f.n, nc = M.c.n;
  out[MP_STREAM] = (int)nbf(ns, 256 * kMultiStreamPasses);
  out[MP_NEAR_SHORT] = short_lists(M.fb.lmax) ? kNearBlocksMember : 0;
  out[MP_NEAR_LONG] = short_lists(M.fb.lmax) ? 0 : kNearBlocksMember;
  const bool wide = wide_membrane(M.fb);
  out[MP_MEMBRANE] = wide ? 0 : segment_blocks(M.fb);
  out[MP_WIDE_FIRST] = wide ? wide_first_blocks(M.p) : 0;
  out[MP_WIDE_TRI] = wide ? wide_tri_blocks(M.p) : 0;
  out[MP_WIDE_TERMS] = wide ? wide_terms_blocks(M.p, SEG_WHOLE) : 0;
  out[MP_WIDE_GATHER] = wide ? wide_gather_blocks(M.p) : 0;
  out[MP_RECORDS] = (int)nb(M.p.nt, kRecordTris);
  out[MP_ZERO] = (int)nb(nc, 256);
  out[MP_VBIN] = (int)nb(M.p.nv, 32);
  out[MP_COUNT] = (int)nbf(ns, 256 * kCountPer);
  out[MP_SCAN] = (int)scan_part_blocks(nc);
  out[MP_SCAN_SUMS] = (int)scan_groups(nc);
  out[MP_PERM] = (int)nbf(ns, 256);
  out[MP_TILE] = (int)cells_tile_blocks(nc);
  out[MP_MOVE] = (int)nbf(ns, 256);
}

int multi_vbin_smem(const Member& M) {
  return (int)sizeof(uint64_t) * M.p.nv;
}

int multi_segment(const Member& M, int* smem) {
  if (wide_membrane(M.fb)) {
    *smem = (int)wide_smem(M.p);
    return 0;
  }
  const int nc = segment_blocks(M.fb);
  *smem = (int)seg_smem(M.p, M.fb, nc);
  return nc;
}

}  // namespace irbc
