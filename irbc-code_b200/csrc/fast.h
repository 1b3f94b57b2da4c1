// fast.h -- buffers and launchers of the production step (fast.cu).
#pragma once
#include "cull.h"
#include "sim.h"

namespace irbc {

// vertex positions/velocities as seen by the streaming of one step of a
// stretch (the arrays hold kSegMax steps, nv entries each)
struct Snap {
  double *x, *y, *z, *vx, *vy, *vz;
  const int *t1, *t2, *t3;
};
// the most steps a stretch has: a stretch lies between two collisions (10 to
// 12 steps apart at the configured dtcd / dtmd); longer ones are cut, for the
// room that the snapshots take (kSegMax x 96 bytes per triangle)
constexpr int kSegMax = 16;
constexpr int kSegT = 512;  // threads per block of the membrane kernel
// triangles whose area and volume terms the summing blocks of the membrane
// kernel stage in shared memory (what is left of 227 KB); more stay in global
// memory.  seg_terms(nt): the doubles staged for nt triangles, the warp tree's
// padding included
constexpr int kSegTerms = 20000;
__host__ __device__ constexpr int seg_terms(int nt) { return (nt + 32 + 15) / 16 * 16; }

// near-membrane streaming: lanes per particle and room for kept entries, for
// lists of up to kShortList entries and for longer ones; threads per block,
// blocks per SM, blocks per simulation alone and per member of a cohort.  A
// simulation alone has few particles near the membrane (some 10 000), so more
// lanes each finish sooner: 8 lanes 93 us a stretch, 1 and 2 lanes 199 and 154
// (600 vertices); 32 lanes 242 us, 16 and 8 lanes 316 and 534 (2562).  Sixteen
// members fill the GPU, where idle lanes cost: 4 lanes 911 us, 8 lanes 1063.
// Stretches of one step take short lists as they are, 4 lanes a particle
// (kShortGOne): eight FP64 members of 600 vertices 287 us a step, with the cull
// and the queue's counter 319; 8 lanes 295.
constexpr int kShortList = 128, kShortG = 8, kShortGMember = 4, kShortGOne = 4, kShortKeep = 64;
constexpr int kLongG = 32, kLongKeep = 512;
constexpr int kNearT = 128, kNearMinBlocks = 4, kNearBlocks = 148 * kNearMinBlocks, kNearBlocksMember = 148;
inline bool short_lists(int lmax) { return lmax <= kShortList; }
// the side-wall bands (3a) that a triangle's corners lie in: tri_record
enum : int { BAND_LX = 1, BAND_HX = 2, BAND_LY = 4, BAND_HY = 8 };

// A mesh split into one patch of vertices per block of the membrane's cluster
// (build_patches in api.cu; segment.cuh): where block b's tables lie.
struct PatchHdr {
  int no, nl, ntri, ned, ndih, nsend;  // own vertices, vertices touched, items, coordinates sent
  int base;                            // first own vertex in the snapshots
  int own, tri, edge, dih, ent, eend, send;  // offsets of the tables in the block's part of the blob
  int blob, bytes;                     // that part
  int ne, nt, nd;                      // edge, triangle and bending entries of its vertices
  int o_tab, o_e, o_d, o_t, o_s;       // shared memory: tables, entries, vertex state
};
struct PatchPlan {
  PatchHdr* hdr = nullptr;
  unsigned char* blob = nullptr;
  int nc = 0;                          // blocks; 0: no patches (the state stays in global memory)
  int sw = 0;                          // summing warps of blocks 0 and 1
  int nl = 0;                          // the most vertices a block touches
  int o_misc = 0, o_c = 0, o_terms = 0, o_sum = 0, o_tail = 0, smem = 0;  // shared memory
};
constexpr unsigned short kNoEntry = 0xffff;
struct PatchTri {
  unsigned short v[3], d[3];  // corners; where their entries go (kNoEntry: another block's vertex)
  int g;                      // >= 0: the triangle whose area and volume terms this block writes
  double tarea;
};
struct PatchEdge {
  unsigned short v[2], pad[2];
  double l0, kp;
};
struct PatchDih {
  unsigned short v[4], d[4];  // l1, l4, l2, l3
};
struct PatchSend {
  unsigned short own, slot, cta, pad;
};
// whether the device runs a cluster of nc membrane blocks with smem bytes each
bool cluster_fits(int nc, int smem);
// where everything lies in the blocks' shared memory (host)
void patch_layout(PatchPlan& P, PatchHdr* hdr, int nt);
// the most shared memory the membrane kernel takes, its most vertices per block
constexpr int kSegSmemMax = 224 * 1024, kPatchOwn = 256;

struct FastBufs {
  PatchPlan patch;
  int* pidx = nullptr;      // place of each vertex in the snapshots
  int *st1 = nullptr, *st2 = nullptr, *st3 = nullptr;  // the triangles' corners by that place
  Snap snap{};
  TriPre* pre = nullptr;  // kSegMax x nt
  unsigned char* bands = nullptr;  // kSegMax x nt: BAND_* of each record's corners
  float4* cull = nullptr; // 2 x 3 x nt: what no step of a stretch's part needs to test (TriCull)
  int* queue = nullptr;   // particles near the membrane (capacity Ns)
  unsigned char* qk = nullptr;  // the step of the stretch from which on
  int* qn = nullptr;      // [par] their number, [4 + par] those taken, in the second part [2 + par] (two parities: cohorts)
  bool one_block = false; // the membrane kernel as one block (meshes that fit, one_block_fits)
  bool cluster = false;   // ... as a cluster of eight blocks whatever the mesh
  int lmax = 0;           // (host) longest list
  double* slot = nullptr; // force terms: 3 doubles per slot, 4E + 9T + 4E slots
  double* a4 = nullptr;   // 4 x area of each triangle
  double* fac = nullptr;  // factors of the global area and volume forces
  double *ux = nullptr, *uy = nullptr;  // unwrapped vertex coordinates
  int* gstart = nullptr;  // per vertex: where its edge, triangle and bending entries of gidx start
  int* gidx = nullptr;    // its slots in the reference's order
  int* vd = nullptr;      // bond draws per vertex this step, VF_* flags
  double* vX = nullptr;   // the parasite's WCA force on it (3 per vertex)
  double* vS = nullptr;   // its bond spring's force (3 per vertex)
};

__host__ __device__ inline Snap snap_of(const FastBufs& f, int step, int nv) {
  Snap s = f.snap;
  const int64_t o = (int64_t)step * nv;
  s.x += o; s.y += o; s.z += o; s.vx += o; s.vy += o; s.vz += o;
  return s;
}
// snapshot of the membrane as it is, as step 0
void fast_snap_prep(const DevParams& p, Membrane& m, FastBufs& f, cudaStream_t st);
// the streaming of a stretch of H steps; sf: the FP32-bulk solvent, or null.
// ev0/ev1 (optional) are recorded around the bulk kernel.  The bulk kernel
// reads no membrane data; the triangle records and the near-membrane kernel
// read the snapshots and first wait for `snap` (optional: their producer).
// first > 0: they run in two parts, the first `first` steps after snap1 and the
// others after snap.  recorded: the triangle records are made already
// (launch_records, before snap).  Returns the number of kernels it launched.
struct SolventF;
int fast_stream(const DevParams& p, const Solvent& s, const SolventF* sf, const Cells& c, FastBufs& f, int H,
                cudaStream_t st, cudaEvent_t ev0 = nullptr, cudaEvent_t ev1 = nullptr, cudaEvent_t snap = nullptr,
                int first = 0, cudaEvent_t snap1 = nullptr, bool recorded = false);
// the triangle records of the steps [s0, s1), part `part` of a stretch
void launch_records(const DevParams& p, const FastBufs& f, int s0, int s1, int part, cudaStream_t st);
bool is_membrane_kernel(const void* fn);
// the membrane of the H steps from step s0 of a stretch (s0 + H <= kSegMax) in
// one launch (segment.cuh); eoff: the stretch's; parts: SEG_FIRST | SEG_SECOND,
// or one of them with H = 1.  Returns the number of kernels launched.
enum : int { SEG_FIRST = 1, SEG_SECOND = 2, SEG_WHOLE = 3 };
int launch_membrane(const DevParams& p, Membrane& m, const FastBufs& fb, uint64_t eoff, int s0, int H, int parts,
                    cudaStream_t st);
// whether a mesh suits the one-block membrane step
bool one_block_fits(const DevParams& p);
// every kernel's dynamic shared-memory limit on the current device (before
// any launch; irbc_create calls it)
void set_kernel_limits();

}  // namespace irbc
