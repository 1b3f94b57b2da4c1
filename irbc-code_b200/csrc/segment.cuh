// segment.cuh -- (part of fast.cu) the membrane of a stretch of timesteps in
// one launch.
//
// Between two collisions the solvent does not act on the membrane: vertex
// kicks, drift, forces and bonds (maincode.cpp:487-496, 566-744) of several
// steps depend only on one another.  So one launch of a thread-block cluster
// advances the membrane through a whole stretch (up to kSegMax steps) and
// leaves for every step what the streaming reads, the half-kicked vertices
// (snap; k_tri_records makes the per-triangle records of them).  Its phases are separated by
// cluster barriers (barrier.cluster arrive.release / wait.acquire); three per
// step:
//   A  per triangle: area and volume terms (to the summing blocks' shared
//      memory) and every force term up to the factors that need Sarea and
//      Volume
//   B  blocks 0 and 1: the ordered sums Sarea and Volume (TotalVA); the
//      others: edge and bending terms, beside them the bond preparation
//   C  per vertex component: the gather of its force terms in the reference's
//      order, external forces, second half-kick, and the next step's first
//      half-kick, snapshot and drift; the last block: bond events and the
//      parasite
// A step's chain of eight dependent launches (at least 2 us apart from the
// host, each cold) took 67 us on the 600-vertex mesh and 128 us on the
// 2562-vertex discocyte.  A step inside a launch takes 12 and 21 us, and with some
// 20 us for a launch's start and end, two launches to 12 steps, 14 and 31 (FP32
// 15 and 22, whose sums take less).  What is left is latency, in cycles of a step
// of 24 000 (600 vertices) and 43 000 (2562): the triangles 3 000 and
// 4 700, the ordered sums 10 000 and 19 000 (the other blocks' terms and bonds
// end before them), phase C 8 000 and 11 000, the three barriers with what they
// wait for of stores to other blocks some 5 000.  A quarter of the vertices a
// block hardly changes them.
#include <cooperative_groups.h>
#include "div.h"

namespace irbc {

// ---- the ordered sums ------------------------------------------------------------
// a[0] + a[1] + ... added left to right in double, bit for bit, by G warps
// instead of one thread.  One thread needs 11.4 cycles per addition (8.15 for
// the FP64 addition itself): 30 us for 5120 triangles.  Here the terms are
// kSumRuns runs, and run u is added three times:
//   1. in any order, for an estimate g of the sum before the run;
//   2. left to right from g (one lane per run); the increments, whose rounding
//      is then in them, give a better estimate h, mostly within 8 units in the
//      last place (ulp) of the true sum;
//   3. left to right from sixteen neighbouring doubles, lane k of sixteen from
//      h + (k - 8) ulp.  A lane whose end is one of the next run's starts
//      stores which; the true sum, which starts as lane 8 of run 0, then hops
//      from run to run through these maps (10 cycles a run).
// A run's end to end cost hardly depends on its length below 40 terms, so short
// sums take half as many runs (sum_runs).  Where the map leads nowhere (the sum passes near zero, where an ulp is small:
// about two of 32 runs of the discocyte's volume, none of the trophozoite's)
// the run is added again from the true value, so the result never depends on
// the estimates.  More runs of fewer lanes miss more often; 16 runs of 32 lanes
// miss half as often but take twice the shared-memory reads, which bound
// step 3.
constexpr int kSumRuns = 32, kSumTry = 16;
__device__ __forceinline__ int sum_runs(int n) { return n <= 2048 ? kSumRuns / 2 : kSumRuns; }
struct SumScratch {
  double g[kSumRuns], h[kSumRuns], ulp[kSumRuns];
  double en[kSumRuns][kSumTry];
  unsigned long long map[kSumRuns];  // 4 bits a lane: the next run's lane, 15 none
};

__device__ __forceinline__ void bar_named(int id, int threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// t + a[0] + ... + a[n-1], left to right; the next 8 terms are loaded while
// the current 8 are added
__device__ __forceinline__ double add_run(double t, const double* a, int n) {
  int i = 0;
  if (n >= 16) {
    double cur[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) cur[k] = a[k];
    for (; i + 16 <= n; i += 8) {
      double nxt[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) nxt[k] = a[i + 8 + k];
#pragma unroll
      for (int k = 0; k < 8; ++k) t += cur[k];
#pragma unroll
      for (int k = 0; k < 8; ++k) cur[k] = nxt[k];
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) t += cur[k];
    i += 8;
  }
  for (; i < n; ++i) t += a[i];
  return t;
}

__device__ __forceinline__ double ulp_of(double x) {
  return fabs(__longlong_as_double(__double_as_longlong(x) + 1) - x);
}
// which of the starts h + (k - 8) u, k < 15, is t; 15: none
__device__ __forceinline__ int sum_lane(double t, double h, double u) {
  const double q = rint((t - h) / u);
  if (!(q >= -8.0 && q <= 6.0)) return 15;
  return __double_as_longlong(h + q * u) == __double_as_longlong(t) ? (int)q + 8 : 15;
}

// by G warps (threads tid in [0, 32 G), G <= 16), which meet at named barrier
// `bar`; the result in warp 0.  Runs are an odd number of terms long, so that
// lanes that read one run each use different banks.
__device__ __forceinline__ double ordered_sum(const double* a, int n, SumScratch& S, int tid, int G, int bar) {
  const int lane = tid & 31, w = tid >> 5, k = lane & 15;
  const int R = sum_runs(n), L = ((n + R - 1) / R) | 1;
  for (int u = 2 * w + (lane >> 4); u < R; u += 2 * G) {
    const int b = min(u * L, n), m = min(b + L, n) - b;
    double x = 0.0;
#pragma unroll 4
    for (int i = k; i < m; i += kSumTry) x += a[b + i];
    for (int o = 8; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    if (k == 0) S.g[u] = x;
  }
  bar_named(bar, 32 * G);
  if (w == 0) {
    const int b = min(lane * L, n), m = lane < R ? min(b + L, n) - b : 0;
    // the sum of S.g over the runs before this lane's
    auto before = [&]() {
      double x = 0.0;
#pragma unroll 8
      for (int u = 0; u < R; ++u) {
        const double y = S.g[u];
        x += u < lane ? y : 0.0;
      }
      return x;
    };
    const double g = before();
    const double e = add_run(g, a + b, m);
    __syncwarp();
    S.g[lane] = e - g;
    __syncwarp();
    const double h = before();
    S.h[lane] = h;
    S.ulp[lane] = ulp_of(h);
  }
  bar_named(bar, 32 * G);
  for (int u = 2 * w + (lane >> 4); u < R; u += 2 * G) {
    const int b = min(u * L, n), m = min(b + L, n) - b;
    const double e = add_run(S.h[u] + (double)(k - 8) * S.ulp[u], a + b, m);
    S.en[u][k] = e;
    const int to = u + 1 < R ? sum_lane(e, S.h[u + 1], S.ulp[u + 1]) : 0;
    const unsigned half = (lane >> 4) ? 0xffff0000u : 0x0000ffffu;
    const unsigned lo = __reduce_or_sync(half, k < 8 ? (unsigned)to << (4 * k) : 0u);
    const unsigned hi = __reduce_or_sync(half, k >= 8 ? (unsigned)to << (4 * (k - 8)) : 0u);
    if (k == 0) S.map[u] = ((unsigned long long)hi << 32) | lo;
  }
  bar_named(bar, 32 * G);
  double t = 0.0;
  if (w == 0) {
    int at = 8, u = 0;  // the true sum before run u is lane `at`'s start
    while (true) {
      // four runs at a time while the maps lead on
      while (u + 4 < R) {
        const unsigned long long m0 = S.map[u], m1 = S.map[u + 1], m2 = S.map[u + 2], m3 = S.map[u + 3];
        const int a0 = (int)(m0 >> (4 * at)) & 15, a1 = (int)(m1 >> (4 * a0)) & 15;
        const int a2 = (int)(m2 >> (4 * a1)) & 15, a3 = (int)(m3 >> (4 * a2)) & 15;
        if (a0 == 15 || a1 == 15 || a2 == 15 || a3 == 15) break;
        at = a3;
        u += 4;
      }
      while (u + 1 < R) {
        const int to = (int)(S.map[u] >> (4 * at)) & 15;
        if (to == 15) break;
        at = to;
        ++u;
      }
      t = S.en[u][at];  // the true sum after run u
      if (++u == R) break;
      // no lane of run u starts from it: that run, and more if need be, again
      do {
        const int b = min(u * L, n);
        t = add_run(t, a + b, min(b + L, n) - b);
        if (++u == R) return t;
        at = sum_lane(t, S.h[u], S.ulp[u]);
      } while (at == 15);
    }
  }
  return t;
}

// the FP32-bulk build, which claims no bit parity: the same terms as a fixed
// warp tree (lane l adds its contiguous run left to right, then a butterfly).
// The terms lie at tree_at(): runs an odd number of doubles apart, so the
// lanes read different banks (packed, a 160-term run put all 32 lanes on one
// bank: 24 us against 1 us)
__device__ __forceinline__ int tree_run(int n) { return (n + 31) / 32; }
__device__ __forceinline__ int tree_at(int i, int run) { return (run & 1) ? i : i + i / run; }
__device__ __forceinline__ double tree_sum(const double* a, int n, bool padded, int lane) {
  const int run = tree_run(n), b = min(lane * run, n), m = min(b + run, n) - b;
  double t = 0.0;
  const double* q = a + (padded ? tree_at(b, run) : b);
#pragma unroll 8
  for (int i = 0; i < m; ++i) t += q[i];
  for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  return t;
}

// ---- per-item force terms ---------------------------------------------------------
// (Src/memfuncs.cpp:233-427) stored per term in slots, so that the gather can
// add them in the reference's order.  X(v): vertex v unwrapped.
#define SEG_X(v) (f.ux[v])
#define SEG_Y(v) (f.uy[v])

// WLC and POW terms of edge i
__device__ __forceinline__ void edge_item(const DevParams& p, const Membrane& m, const FastBufs& f, int i) {
  const int l1 = m.e1[i], l2 = m.e2[i];
  const double l0 = m.l0[i];
  double A[3];
  A[0] = SEG_X(l1) - SEG_X(l2); A[1] = SEG_Y(l1) - SEG_Y(l2); A[2] = m.z[l1] - m.z[l2];
  double aa = sqrt(A[0] * A[0] + A[1] * A[1] + A[2] * A[2]);
  A[0] /= aa; A[1] /= aa; A[2] /= aa;
  double xx = aa / (2.5 * l0);
  double xxx = 1.0 / (4.0 * (1.0 - xx) * (1.0 - xx));
  const double kp = m.kappap[i];
  double* S = f.slot + (int64_t)12 * i;
  for (int k = 0; k < 3; ++k) {
    S[0 + k] = (-1.0 / (p.elap)) * (xxx - 0.25 + xx) * A[k];
    S[3 + k] = kp * A[k] / (aa * aa);
    S[6 + k] = (1.0 / (p.elap)) * (xxx - 0.25 + xx) * A[k];
    S[9 + k] = -kp * A[k] / (aa * aa);
  }
}

// area and volume terms of triangle i (Areatri / Voltri, :124-157) and its
// force terms: per corner C (the global area term without its factor alpha =
// beta / (4 area)), alphad * C, and the volume term without betav and / 6
__device__ __forceinline__ void tri_item(const DevParams& p, const Membrane& m, const FastBufs& f, int i,
                                         double& area_out, double& vol_out) {
  const int l1 = m.t1[i], l2 = m.t2[i], l3 = m.t3[i];
  const double x1 = SEG_X(l1), y1 = SEG_Y(l1), z1 = m.z[l1];
  const double x2 = SEG_X(l2), y2 = SEG_Y(l2), z2 = m.z[l2];
  const double x3 = SEG_X(l3), y3 = SEG_Y(l3), z3 = m.z[l3];
  double A[3] = {x2 - x1, y2 - y1, z2 - z1}, B[3] = {x3 - x1, y3 - y1, z3 - z1}, e0[3];
  cp(A, B, e0);
  const double area = 0.5 * sqrt(e0[0] * e0[0] + e0[1] * e0[1] + e0[2] * e0[2]);
  double Cn[3];
  Cn[0] = (x1 + x2 + x3) / 3.0;
  Cn[1] = (y1 + y2 + y3) / 3.0;
  Cn[2] = (z1 + z2 + z3) / 3.0;
  area_out = area;
  vol_out = (1.0 / 6.0) * ((e0[0] * Cn[0]) + (e0[1] * Cn[1]) + (e0[2] * Cn[2]));
  const double alphad = -p.kappad * (area - m.tarea[i]) / (4.0 * m.tarea[i] * area);
  f.a4[i] = 4.0 * area;
  double A13[3] = {x1 - x3, y1 - y3, z1 - z3}, A32[3] = {x3 - x2, y3 - y2, z3 - z2}, eta[3], C[3];
  cp(A13, A, eta);
  double e3[3] = {eta[0] / 3.0, eta[1] / 3.0, eta[2] / 3.0};
  double* S = f.slot + (int64_t)12 * p.ne + (int64_t)27 * i;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const double* side = c == 0 ? A32 : (c == 1 ? A13 : A);
    cp(eta, side, C);
    for (int k = 0; k < 3; ++k) { S[6 * c + k] = C[k]; S[6 * c + 3 + k] = alphad * C[k]; }
    cp(Cn, side, C);
    for (int k = 0; k < 3; ++k) S[18 + 3 * c + k] = e3[k] + C[k];
  }
}

// bending terms of a dihedral (l1, l2, l3, l4): r[0..3] on l1, l4, l2, l3
__device__ __forceinline__ void dih_terms(const DevParams& p, double x1, double y1, double z1, double x2, double y2,
                                          double z2, double x3, double y3, double z3, double x4, double y4, double z4,
                                          double r[4][3]) {
  double a21[3] = {x2 - x1, y2 - y1, z2 - z1}, a31[3] = {x3 - x1, y3 - y1, z3 - z1};
  double a24[3] = {x2 - x4, y2 - y4, z2 - z4}, a34[3] = {x3 - x4, y3 - y4, z3 - z4};
  double a32[3] = {x3 - x2, y3 - y2, z3 - z2}, t1[3], t2[3], eta[3], zeta[3], C[3], D[3], E[3], F[3];
  t1[0] = div3(x1 + x2 + x3);
  t1[1] = div3(y1 + y2 + y3);
  t1[2] = div3(z1 + z2 + z3);
  t2[0] = div3(x4 + x2 + x3);
  t2[1] = div3(y4 + y2 + y3);
  t2[2] = div3(z4 + z2 + z3);
  cp(a21, a31, eta);
  cp(a34, a24, zeta);
  double etam = sqrt(eta[0] * eta[0] + eta[1] * eta[1] + eta[2] * eta[2]);
  double zetam = sqrt(zeta[0] * zeta[0] + zeta[1] * zeta[1] + zeta[2] * zeta[2]);
  double costh = (eta[0] * zeta[0] + eta[1] * zeta[1] + eta[2] * zeta[2]) / (etam * zetam);
  if (costh > 1.0) costh = 1.0;
  if (costh < -1.0) costh = -1.0;
  if (costh == 1.0) costh -= 0.0005;
  if (costh == -1.0) costh += 0.0005;
  double sinth = sqrt(1.0 - costh * costh);
  double tt0 = t1[0] - t2[0];
  double tt1 = t1[1] - t2[1];
  double factor = (((eta[0] - zeta[0]) * tt0) + ((eta[1] - zeta[1]) * tt1) + ((eta[2] - zeta[2]) * (t1[2] - t2[2])));
  double fact = (factor >= 0.0) ? 1.0 : -1.0;
  sinth = fact * sinth;
  double betab = p.kappab * (sinth * p.cth0 - costh * p.sth0) / sinth;
  double b11 = -(betab * costh) / (etam * etam);
  double b22 = -(betab * costh) / (zetam * zetam);
  double b12 = betab / (etam * zetam);
  cp(eta, a32, C);
  cp(zeta, a32, D);
  for (int k = 0; k < 3; ++k) { r[0][k] = b11 * C[k] + b12 * D[k]; r[1][k] = -b12 * C[k] - b22 * D[k]; }
  cp(eta, a31, C); cp(zeta, a31, D); cp(eta, a34, E); cp(zeta, a34, F);
  for (int k = 0; k < 3; ++k) r[2][k] = -b11 * C[k] + b12 * (E[k] - D[k]) + b22 * F[k];
  cp(eta, a21, C); cp(zeta, a21, D); cp(eta, a24, E); cp(zeta, a24, F);
  for (int k = 0; k < 3; ++k) r[3][k] = b11 * C[k] + b12 * (-E[k] + D[k]) - b22 * F[k];
}
__device__ __forceinline__ void dih_item(const DevParams& p, const Membrane& m, const FastBufs& f, int i) {
  int l2, l3;
  if (m.iedge[i] == -1) { l3 = m.e1[i]; l2 = m.e2[i]; } else { l2 = m.e1[i]; l3 = m.e2[i]; }
  const int l1 = m.es1[i], l4 = m.es2[i];
  double r[4][3];
  dih_terms(p, SEG_X(l1), SEG_Y(l1), m.z[l1], SEG_X(l2), SEG_Y(l2), m.z[l2], SEG_X(l3), SEG_Y(l3), m.z[l3], SEG_X(l4),
            SEG_Y(l4), m.z[l4], r);
  double* S = f.slot + (int64_t)12 * p.ne + (int64_t)27 * p.nt + (int64_t)12 * i;
  for (int c = 0; c < 4; ++c)
    for (int k = 0; k < 3; ++k) S[3 * c + k] = r[c][k];
}

// the parasite's WCA force (pfdt, Src/memfuncs.cpp:459-475) on a vertex at
// (ux, uy, z), parasite at pp, both unwrapped; false beyond its cutoff
__device__ __forceinline__ bool wca_at(const DevParams& p, const double pp[3], double ux, double uy, double z,
                                       double X[3]) {
  double cutoff = p.paraR, epsilon = 0.1, sigma = 0.890898718 * cutoff;
  double A[3];
  A[0] = pp[0] - ux;
  A[1] = pp[1] - uy;
  A[2] = pp[2] - z;
  double aa = A[0] * A[0] + A[1] * A[1] + A[2] * A[2];
  if (aa <= cutoff * cutoff) {
    double ex = (sigma * sigma * sigma * sigma * sigma * sigma) / (aa * aa * aa);
    X[0] = (24.0 * epsilon / aa) * ((2.0 * ex * ex) - ex) * A[0];
    X[1] = (24.0 * epsilon / aa) * ((2.0 * ex * ex) - ex) * A[1];
    X[2] = (24.0 * epsilon / aa) * ((2.0 * ex * ex) - ex) * A[2];
    return true;
  }
  return false;
}

// per-vertex results of the bond preparation that the gather and the tail
// read: the number of bond draws, and which of the vectors below apply
enum : int { VF_WCA = 1 << 20, VF_SPRING = 1 << 21, VF_BONDED = 1 << 22, VF_DRAWS = (1 << 20) - 1 };

// They are taken after the drift and before the step's bond events, and the
// gather adds the spring and the parasite's force from here, so that it may run
// beside the events and the parasite's move.

// a bonded vertex ii at (x, y, z), images (ix, iy): the probability pr of its
// bond to break (maincode.cpp:668-690) and the bond spring's force sp
// (:612-640) when the flags returned have VF_SPRING
__device__ __forceinline__ int bonded_prep(const DevParams& p, const Membrane& m, int ii, double x, double y, double z,
                                           int ix, int iy, double& pr, double sp[3]) {
  double A[3], B[3];
  int flags = VF_BONDED;
  int jj = m.bondl[ii];
  const double xl = m.xlig[jj], yl = m.ylig[jj];
  A[0] = (x + ix * p.Lx) - (xl + ix * p.Lx);
  A[1] = (y + iy * p.Ly) - (yl + iy * p.Ly);
  A[2] = z - 0.0;
  double xx = sqrt(A[0] * A[0] + A[1] * A[1] + A[2] * A[2]);
  if (xx > p.el0) {
    B[0] = -p.ks * (xx - p.el0) * A[0] / xx;
    B[1] = -p.ks * (xx - p.el0) * A[1] / xx;
    B[2] = -p.ks * (xx - p.el0) * A[2] / xx;
  } else {
    B[0] = B[1] = B[2] = 0.0;
  }
  double bb = sqrt(B[0] * B[0] + B[1] * B[1] + B[2] * B[2]);
  double koff = p.offrate * exp(bb / p.FD);
  pr = 1.0 - exp(-koff * p.dtmd);
  m.poff[ii] = pr;
  // the bond spring
  A[0] = x - xl;
  A[1] = y - yl;
  A[2] = z;
  A[0] -= p.Lx * round(A[0] / p.Lx);
  A[1] -= p.Ly * round(A[1] / p.Ly);
  double aa = sqrt(A[0] * A[0] + A[1] * A[1] + A[2] * A[2]);
  A[0] /= aa; A[1] /= aa; A[2] /= aa;
  if (aa > p.el0) {
    flags |= VF_SPRING;
    for (int k = 0; k < 3; ++k) sp[k] = -p.ks * (aa - p.el0) * A[k];
  }
  return flags;
}

// The candidate ligands of a free knob near the wall, by sixteen lanes (half a
// warp; both halves call together, `on`: this half has a vertex)
// (maincode.cpp:692-723): those on the list of its cell (cells below z = 2
// whose centre is within 1.5 of the ligand along x and y, after the reference's
// fabs-then-round, :138-154) within dthr, sorted by distance, then index, into
// m.pair_j; returns their number.  Ligand gx * nligy + gy lies at (0.5 gx,
// 0.5 gy), so a lane takes one ligand of the window around the vertex: at most
// nine with dthr = 0.5.  pd, pj: the half's room for kMaxPairs candidates.  (One
// thread per vertex, inserting into sorted global lists, took 18 us of a step.)
__device__ __forceinline__ int bond_pairs(const DevParams& p, const Membrane& m, bool on, int ii, double x, double y,
                                          double z, int ix, int iy, int pid, double* pd, int* pj) {
  const int lane = threadIdx.x & 15, shift = threadIdx.x & 16;
  const int ck = pid % p.nz, cj = (pid / p.nz) % p.ny, ci = pid / (p.nz * p.ny);
  on = on && -1.0 + (double)ck * p.a + p.a <= 2.0;
  const double reach = p.dthr + 1e-6;
  const int gx0 = max((int)ceil((x - reach) * 2.0), 0), gx1 = min((int)floor((x + reach) * 2.0), p.nligx - 1);
  const int gy0 = max((int)ceil((y - reach) * 2.0), 0), gy1 = min((int)floor((y + reach) * 2.0), p.nligy - 1);
  const int wy = max(gy1 - gy0 + 1, 1), W = on && gy1 >= gy0 ? max(gx1 - gx0 + 1, 0) * wy : 0;
  const double zz = z - 0.0;
  const double hx = ((double)ci * p.a + ((double)ci * p.a + p.a)) * 0.5;
  const double hy = ((double)cj * p.a + ((double)cj * p.a + p.a)) * 0.5;
  int n = 0;
  for (int c0 = 0; __any_sync(0xffffffffu, c0 < W); c0 += 16) {
    const int c = c0 + lane, gx = gx0 + c / wy, gy = gy0 + c % wy;
    const double xl = 0.5 * gx, yl = 0.5 * gy;
    const double A0 = (x + ix * p.Lx) - (xl + ix * p.Lx), A1 = (y + iy * p.Ly) - (yl + iy * p.Ly);
    const double aaa = (A0 * A0 + A1 * A1 + zz * zz);
    bool in = c < W && aaa <= p.dthr * p.dthr;
    if (in) {
      double B0 = fabs(hx - xl), B1 = fabs(hy - yl);
      B0 -= p.Lx * round(B0 / p.Lx);
      B1 -= p.Ly * round(B1 / p.Ly);
      in = (B0 < 1.5) && (B1 < 1.5);
    }
    const unsigned b = (__ballot_sync(0xffffffffu, in) >> shift) & 0xffffu;
    const int at = n + __popc(b & ((1u << lane) - 1u));
    if (in && at < kMaxPairs) { pd[at] = aaa; pj[at] = gx * p.nligy + gy; }
    n = min(n + __popc(b), kMaxPairs);
  }
  __syncwarp();
  for (int e = lane; e < n; e += 16) {
    const double d = pd[e];
    const int j = pj[e];
    int r = 0;
    for (int u = 0; u < n; ++u) r += (pd[u] < d || (pd[u] == d && pj[u] < j)) ? 1 : 0;
    m.pair_j[(int64_t)ii * kMaxPairs + r] = j;
  }
  __syncwarp();
  return n;
}

// every vertex's bond preparation, spring and parasite force by the cluster's
// `workers` threads numbered `worker` (whole warps); room: 24 kMaxPairs bytes a
// warp of the block
__device__ __forceinline__ void bond_prep_all(const DevParams& p, const Membrane& m, const FastBufs& f, int worker,
                                              int workers, unsigned char* room) {
  const int lane = threadIdx.x & 31;
  double* pd = reinterpret_cast<double*>(room) + (threadIdx.x >> 4) * kMaxPairs;
  int* pj = reinterpret_cast<int*>(room + (kSegT / 16) * kMaxPairs * sizeof(double)) + (threadIdx.x >> 4) * kMaxPairs;
  const MemScalars* sc = m.sc;
  const double pp[3] = {(sc->para[0] + sc->paradx * p.Lx), (sc->para[1] + sc->parady * p.Ly), sc->para[2]};
  for (int i0 = worker - lane; i0 < p.nv; i0 += workers) {
    const int i = i0 + lane;
    bool free = false;
    int flags = 0;
    if (i < p.nv) {
      const int bondi = m.bondi[i];
      if (bondi == 1) {
        double pr, sp[3];
        flags = 1 | bonded_prep(p, m, i, m.x[i], m.y[i], m.z[i], m.ix[i], m.iy[i], pr, sp);
        if (flags & VF_SPRING)
          for (int k = 0; k < 3; ++k) f.vS[3 * i + k] = sp[k];
      } else {
        free = (m.z[i] < p.dthr) && (bondi == 0) && (m.knob[i] == 1);
      }
      double X[3];
      if (wca_at(p, pp, (m.x[i] + m.ix[i] * p.Lx), (m.y[i] + m.iy[i] * p.Ly), m.z[i], X)) {
        flags |= VF_WCA;
        f.vX[3 * i] = X[0]; f.vX[3 * i + 1] = X[1]; f.vX[3 * i + 2] = X[2];
      }
    }
    // the free knobs near the wall, two at a time by the halves of the warp
    for (unsigned todo = __ballot_sync(0xffffffffu, free); todo;) {
      const int s0 = __ffs(todo) - 1;
      todo &= todo - 1;
      const int s1 = todo ? __ffs(todo) - 1 : -1;
      if (todo) todo &= todo - 1;
      const int src = lane < 16 ? s0 : s1, j = i0 + max(src, 0);
      const int n = bond_pairs(p, m, src >= 0, j, m.x[j], m.y[j], m.z[j], m.ix[j], m.iy[j], m.pid[j], pd, pj);
      const int n0 = __shfl_sync(0xffffffffu, n, 0), n1 = __shfl_sync(0xffffffffu, n, 16);
      if (lane == s0 || lane == s1) {
        const int mine = lane == s0 ? n0 : n1;
        flags |= mine;
        m.npair[i] = mine;
        m.pon[i] = 1.0 - exp(-p.onrate * p.dtmd);
      }
    }
    if (i < p.nv) f.vd[i] = flags;
  }
}

// per-triangle record of the streaming (reflectionFed at rstep = 0,
// Src/solfuncs.cpp:457-509) from a snapshot of the vertices: the corner A1 at
// t, A2 at t + dtmd, the normals X and Xdt there
__device__ __forceinline__ TriPre tri_record(const DevParams& p, const Snap& sn, int p1, int p2, int p3) {
  const double rstep = 0.0, dtmd = p.dtmd, Lx = p.Lx, Ly = p.Ly;
  const int z0 = 0;
  const double vx1 = sn.vx[p1], vy1 = sn.vy[p1], vz1 = sn.vz[p1];
  const double vx2 = sn.vx[p2], vy2 = sn.vy[p2], vz2 = sn.vz[p2];
  const double vx3 = sn.vx[p3], vy3 = sn.vy[p3], vz3 = sn.vz[p3];
  double v1x = (sn.x[p1] + z0 * Lx) + vx1 * rstep, v1y = (sn.y[p1] + z0 * Ly) + vy1 * rstep, v1z = sn.z[p1] + vz1 * rstep;
  double v2x = (sn.x[p2] + z0 * Lx) + vx2 * rstep, v2y = (sn.y[p2] + z0 * Ly) + vy2 * rstep, v2z = sn.z[p2] + vz2 * rstep;
  double v3x = (sn.x[p3] + z0 * Lx) + vx3 * rstep, v3y = (sn.y[p3] + z0 * Ly) + vy3 * rstep, v3z = sn.z[p3] + vz3 * rstep;
  double w1x = v1x + vx1 * (dtmd - rstep), w1y = v1y + vy1 * (dtmd - rstep), w1z = v1z + vz1 * (dtmd - rstep);
  double w2x = v2x + vx2 * (dtmd - rstep), w2y = v2y + vy2 * (dtmd - rstep), w2z = v2z + vz2 * (dtmd - rstep);
  double w3x = v3x + vx3 * (dtmd - rstep), w3y = v3y + vy3 * (dtmd - rstep), w3z = v3z + vz3 * (dtmd - rstep);
  double t0[3], t1v[3];
  TriPre q;
  t0[0] = v2x - v1x; t0[1] = v2y - v1y; t0[2] = v2z - v1z;
  t1v[0] = v3x - v1x; t1v[1] = v3y - v1y; t1v[2] = v3z - v1z;
  cp(t0, t1v, q.X);
  t0[0] = w2x - w1x; t0[1] = w2y - w1y; t0[2] = w2z - w1z;
  t1v[0] = w3x - w1x; t1v[1] = w3y - w1y; t1v[2] = w3z - w1z;
  cp(t0, t1v, q.Xdt);
  q.A1[0] = v1x; q.A1[1] = v1y; q.A1[2] = v1z;
  q.A2[0] = w1x; q.A2[1] = w1y; q.A2[2] = w1z;
  return q;
}

// ---- the tail: bond events and the parasite -----------------------------------------
// One block: exclusive scans of the per-vertex draw counts and WCA flags (each
// thread owns a contiguous run of vertices, so order is kept), the bond draws
// made in parallel and the successful ones applied in draw order by one thread
// (bond_dynamics, maincode.cpp:16-54), and pfdt's parasite sum in vertex order
// with the parasite kick (Src/memfuncs.cpp:469-482, maincode.cpp:736-744) and,
// when another step follows, its next drift (:576-598).
constexpr int kTailDraws = 4096, kWcaList = 512;
struct TailSmem {
  double wx[kWcaList * 3];
  int wd[kSegT / 32], ww[kSegT / 32];
  int evv[kTailDraws];
  short evr[kTailDraws];
};

__device__ __forceinline__ void para_drift(const DevParams& p, MemScalars* sc) {
  for (int k = 0; k < 3; ++k)
    sc->para[k] += (sc->paraV[k] * p.dtmd) + (sc->paraft[k] * p.dtmd * p.dtmd / (2.0 * p.PRmass));
  if (sc->para[0] > p.Lx) { sc->para[0] -= p.Lx; sc->paradx += 1; }
  else if (sc->para[0] < 0) { sc->para[0] += p.Lx; sc->paradx -= 1; }
  if (sc->para[1] > p.Ly) { sc->para[1] -= p.Ly; sc->parady += 1; }
  else if (sc->para[1] < 0) { sc->para[1] += p.Ly; sc->parady -= 1; }
}

// bond_dynamics (maincode.cpp:16-54) by one thread: more draws than the lists
// below hold
__device__ __noinline__ void bond_events_serial(const DevParams& p, const Membrane& m, const FastBufs& f,
                                                uint64_t epoch) {
  uint64_t k = 0;
  for (int ii = 0; ii < p.nv; ++ii) {
    const int n = f.vd[ii] & VF_DRAWS;
    if (m.bondi[ii] == 1) {
      double randoff = draw_uniform(p.seed, STREAM_BOND, epoch, k++);
      int jj = m.bondl[ii];
      if (m.poff[ii] > randoff) { m.bondi[ii] = 0; m.bondl[ii] = p.randno; m.ligi[jj] = 0; }
    } else {
      for (int r = 0; r < n; ++r) {
        int j = m.pair_j[(int64_t)ii * kMaxPairs + r];
        double pon = m.pon[ii];
        double randon = draw_uniform(p.seed, STREAM_BOND, epoch, k++);
        if ((pon > randon) && (m.ligi[j] == 0)) { m.ligi[j] = 1; m.bondi[ii] = 1; m.bondl[ii] = j; }
      }
    }
  }
}

template <int T>
__device__ __forceinline__ void tail_block(const DevParams& p, const Membrane& m, const FastBufs& f, uint64_t epoch,
                                           bool drift_next, TailSmem& S) {
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  MemScalars* sc = m.sc;
  const int chunk = (p.nv + T - 1) / T;
  const int v0 = min(tid * chunk, p.nv), v1 = min(v0 + chunk, p.nv);
  int nd = 0, nw = 0;
  for (int ii = v0; ii < v1; ++ii) {
    const int q = f.vd[ii];
    nd += q & VF_DRAWS;
    nw += (q & VF_WCA) ? 1 : 0;
  }
  int sd = nd, sw = nw;  // inclusive scans over the warp
  for (int o = 1; o < 32; o <<= 1) {
    const int a = __shfl_up_sync(0xffffffffu, sd, o), b = __shfl_up_sync(0xffffffffu, sw, o);
    if (lane >= o) { sd += a; sw += b; }
  }
  if (lane == 31) { S.wd[w] = sd; S.ww[w] = sw; }
  __syncthreads();
  int od = sd - nd, ow = sw - nw, ndt = 0, nwt = 0;
  for (int u = 0; u < T / 32; ++u) {
    const int a = S.wd[u], b = S.ww[u];
    if (u < w) { od += a; ow += b; }
    ndt += a; nwt += b;
  }
  const bool fits = ndt <= kTailDraws && nwt <= kWcaList;
  bool any = false;
  if (fits && (nd | nw)) {
    for (int ii = v0; ii < v1; ++ii) {
      const int q = f.vd[ii], n = q & VF_DRAWS;
      if (n > 0) {
        const bool bonded = m.bondi[ii] == 1;
        const double pr = bonded ? m.poff[ii] : m.pon[ii];
        for (int r = 0; r < n; ++r) {
          const bool ev = pr > draw_uniform(p.seed, STREAM_BOND, epoch, (uint64_t)(od + r));
          S.evv[od + r] = ev ? ii : -1;
          S.evr[od + r] = (short)(bonded ? -1 : r);
          any |= ev;
        }
        od += n;
      }
      if (q & VF_WCA) {
        S.wx[3 * ow] = f.vX[3 * ii]; S.wx[3 * ow + 1] = f.vX[3 * ii + 1]; S.wx[3 * ow + 2] = f.vX[3 * ii + 2];
        ++ow;
      }
    }
  }
  const int events = __syncthreads_or(any);
  if (tid == 32) {
    double fx = 0, fy = 0, fz = 0;
    if (fits) {
      for (int q = 0; q < nwt; ++q) { fx += S.wx[3 * q]; fy += S.wx[3 * q + 1]; fz += S.wx[3 * q + 2]; }
    } else {
      for (int ii = 0; ii < p.nv; ++ii)
        if (f.vd[ii] & VF_WCA) { fx += f.vX[3 * ii]; fy += f.vX[3 * ii + 1]; fz += f.vX[3 * ii + 2]; }
    }
    sc->parafdt[0] += fx; sc->parafdt[1] += fy; sc->parafdt[2] += fz;
    for (int c = 0; c < 3; ++c) sc->paraV[c] += ((sc->paraft[c] + sc->parafdt[c]) * p.dtmd / (2.0 * p.PRmass));
    for (int c = 0; c < 3; ++c) { sc->paraft[c] = sc->parafdt[c]; sc->parafdt[c] = 0.0; }
    if (drift_next) para_drift(p, sc);
  }
  if (fits && events && tid < 32) {
    for (int k0 = 0; k0 < ndt; k0 += 32) {
      const int k = k0 + tid;
      unsigned ev = __ballot_sync(0xffffffffu, k < ndt && S.evv[k] >= 0);
      if (tid == 0) {
        while (ev) {
          const int b = __ffs(ev) - 1;
          ev &= ev - 1;
          const int ii = S.evv[k0 + b], r = S.evr[k0 + b];
          if (r < 0) {
            int jj = m.bondl[ii];
            m.bondi[ii] = 0; m.bondl[ii] = p.randno; m.ligi[jj] = 0;
          } else {
            int j = m.pair_j[(int64_t)ii * kMaxPairs + r];
            if (m.ligi[j] == 0) { m.ligi[j] = 1; m.bondi[ii] = 1; m.bondl[ii] = j; }
          }
        }
      }
    }
  } else if (!fits && tid == 0) {
    bond_events_serial(p, m, f, epoch);
  }
}

// ---- the stretch ------------------------------------------------------------------------
// SEG_FIRST: first half-kick .. TotalVA; SEG_SECOND: forces .. bond events
// (the halves either side of maincode.cpp:602); a whole step has both

// component k of vertex i: first half-kick with force fk, snapshot, drift and
// wrap (maincode.cpp:487-496, 566-574); the unwrapped coordinate for the
// force terms
__device__ __forceinline__ void kick_drift(const DevParams& p, const Membrane& m, const FastBufs& f, const Snap& sn,
                                           int i, int k, double v, double fk) {
  double* X = k == 0 ? m.x : (k == 1 ? m.y : m.z);
  v += (fk * p.dtmd / (2.0 * p.pmass));
  (k == 0 ? m.vx : (k == 1 ? m.vy : m.vz))[i] = v;
  double x = X[i];
  (k == 0 ? sn.x : (k == 1 ? sn.y : sn.z))[i] = x;
  (k == 0 ? sn.vx : (k == 1 ? sn.vy : sn.vz))[i] = v;
  x += (v * p.dtmd);
  if (k < 2) {
    const double L = k == 0 ? p.Lx : p.Ly;
    int* I = k == 0 ? m.ix : m.iy;
    int im = I[i];
    const int im0 = im;
    if (x > L) { x -= L; im += 1; }
    if (x < 0) { x += L; im -= 1; }
    if (im != im0) I[i] = im;
    (k == 0 ? f.ux : f.uy)[i] = x + im * L;
  }
  X[i] = x;
}

// The phases of a step with the state in global memory, by G threads numbered g.
// The first half-kick of the first step (SEG_FIRST), or only the unwrapped
// coordinates that the force terms read
__device__ __forceinline__ void global_first(const DevParams& p, const Membrane& m, const FastBufs& f, int parts, int g,
                                             int G) {
  if (parts & SEG_FIRST) {
    const Snap sn = snap_of(f, 0, p.nv);
    for (int q = g; q < 3 * p.nv; q += G) {
      const int i = q / 3, k = q - 3 * i;
      double* F = k == 0 ? m.fx : (k == 1 ? m.fy : m.fz);
      kick_drift(p, m, f, sn, i, k, (k == 0 ? m.vx : (k == 1 ? m.vy : m.vz))[i], F[i]);
      F[i] = 0.0;
    }
    if (g == 0) para_drift(p, m.sc);
  } else {
    for (int i = g; i < p.nv; i += G) { f.ux[i] = m.x[i] + m.ix[i] * p.Lx; f.uy[i] = m.y[i] + m.iy[i] * p.Ly; }
  }
}
// A: the triangles; their area and volume terms to a_to and v_to
__device__ __forceinline__ void global_tri(const DevParams& p, const Membrane& m, const FastBufs& f, double* a_to,
                                           double* v_to, bool pad, int g, int G) {
  const int run = tree_run(p.nt);
  for (int i = g; i < p.nt; i += G) {
    double ar, vo;
    tri_item(p, m, f, i, ar, vo);
    const int at = pad ? tree_at(i, run) : i;
    a_to[at] = ar;
    v_to[at] = vo;
  }
}
// B: Sarea or Volume from its terms by sw warps (thread st of them, named
// barrier bar), and the factor of the global area or volume force
__device__ __forceinline__ void global_sum(const DevParams& p, const Membrane& m, const FastBufs& f, int parts, bool area,
                                           const double* src, bool pad, SumScratch& S, int st, int sw, int bar) {
  double* sum = area ? &m.sc->Sarea : &m.sc->Volume;
  if (parts & SEG_FIRST) {
    double r;
    if (p.tree_sums) r = tree_sum(src, p.nt, pad, st & 31);
    else r = ordered_sum(src, p.nt, S, st, sw, bar);
    if (st == 0) *sum = r;
  }
  if (st == 0) {
    if (area) f.fac[0] = -p.kappasa * (*sum - p.Sarea0) / p.Sarea0;
    else f.fac[1] = -p.kappav * (*sum - p.Volume0) / (p.Volume0);
  }
}
// ... beside them the edge and bending terms
__device__ __forceinline__ void global_terms(const DevParams& p, const Membrane& m, const FastBufs& f, int worker,
                                             int workers) {
  for (int q = worker; q < 2 * p.ne; q += workers) {
    if (q < p.ne) dih_item(p, m, f, q);
    else edge_item(p, m, f, q - p.ne);
  }
}
// C: the gather of step s and the kicks
__device__ __forceinline__ void global_gather(const DevParams& p, const Membrane& m, const FastBufs& f, int s, int parts,
                                              bool more, int g, int G) {
  const Snap sn = snap_of(f, s + 1, p.nv);
  const double beta = f.fac[0], betav = f.fac[1];
  const int base_t = 4 * p.ne;
  for (int q = g; q < 3 * p.nv; q += G) {
    const int i = q / 3, k = q - 3 * i;
    const int q0 = f.gstart[3 * i], q1 = f.gstart[3 * i + 1], q2 = f.gstart[3 * i + 2], q3 = f.gstart[3 * i + 3];
    const int vd = f.vd[i];
    const double* S = f.slot + k;
    double acc = 0.0;
#pragma unroll 8
    for (int e = q0; e < q1; ++e) acc += S[3 * (int64_t)f.gidx[e]];
#pragma unroll 2
    for (int e = q1; e < q2; e += 2) {
      // the three terms of a triangle's corner (tri_item): slots n, n + 1
      // and gidx[e + 1]
      const int n = f.gidx[e];
      acc += (beta / f.a4[(n - base_t) / 9]) * S[3 * (int64_t)n];
      acc += S[3 * (int64_t)(n + 1)];
      acc += betav * S[3 * (int64_t)f.gidx[e + 1]] / 6.0;
    }
#pragma unroll 8
    for (int e = q2; e < q3; ++e) acc += S[3 * (int64_t)f.gidx[e]];
    // the first half-kick has reset the force (:490)
    double* F = k == 0 ? m.fx : (k == 1 ? m.fy : m.fz);
    double fk = (parts & SEG_FIRST) ? 0.0 : F[i];
    if (vd & VF_WCA) fk -= f.vX[3 * i + k];  // pfdt's -X
    fk += acc;
    if (k == 2) fk += -p.Fg / (double)p.nv;
    if (vd & VF_SPRING) fk += f.vS[3 * i + k];
    if (k == 2) {
      double cc = m.z[i];
      if (cc < 0.5) fk += 300.0 * exp(-50.0 * cc);
      cc = p.Lz - m.z[i];
      if (cc < 0.5) fk -= 300.0 * exp(-50.0 * cc);
    }
    // second half-kick (maincode.cpp:727-733)
    double* V = k == 0 ? m.vx : (k == 1 ? m.vy : m.vz);
    const double v = V[i] + (fk * p.dtmd / (2.0 * p.pmass));
    raise_health(p, !isfinite(fk + v), HEALTH_MEMBRANE);
    if (more) {
      kick_drift(p, m, f, sn, i, k, v, fk);
    } else {
      V[i] = v;
      F[i] = fk;
    }
  }
}

// The membrane of H steps by a cluster of blocks that keep its state in global
// memory: the one-block and eight-block forms of irbc_set_membrane_kernels, for
// whole steps.  Bound by the load and store units: a warp's scattered 8-byte
// accesses take a cycle a line (the discocyte on eight blocks: 92 us a step).
// seg_smem() bytes of shared memory, the same layout in every block.
__device__ __forceinline__ void membrane_global(const DevParams& p, const Membrane& m, const FastBufs& f,
                                                 uint64_t epoch, int H, unsigned char* smem) {
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  const int cta = (int)cl.block_rank(), nc = (int)cl.num_blocks();
  const int T = kSegT, t = threadIdx.x;
  const int g = cta * T + t, G = nc * T;
  SumScratch& ss0 = *reinterpret_cast<SumScratch*>(smem);
  SumScratch& ss1 = *reinterpret_cast<SumScratch*>(smem + (nc == 1 ? sizeof(SumScratch) : 0));
  TailSmem& tail = *reinterpret_cast<TailSmem*>(smem + 2 * sizeof(SumScratch));
  double* terms = reinterpret_cast<double*>(smem + 2 * sizeof(SumScratch) + ((sizeof(TailSmem) + 15) & ~size_t(15)));
  // the summing warps: Sarea by the first sw warps of block 0, Volume by the
  // first sw of block 1 (of block 0's next sw when it is alone); a cluster of
  // four or more blocks gives both whole blocks, smaller ones share a block's
  // warps with the force terms.  The warp tree takes one warp each.
  const int vb = nc > 1 ? 1 : 0, voff = nc > 1 ? 0 : 1;
  const int sw = p.tree_sums ? 1 : (nc >= 4 ? T / 32 : (nc > 1 ? 8 : 4));
  const int wrp = t >> 5;
  const bool area_w = cta == 0 && wrp < sw;
  const bool vol_w = cta == vb && wrp >= voff * sw && wrp < (voff + 1) * sw;
  // the other threads, numbered through the cluster
  const int busy0 = nc > 1 ? 32 * sw : 64 * sw;  // summing threads of block 0
  const int busy1 = nc > 1 ? 32 * sw : 0;
  const int worker = cta == 0 ? t - busy0 : (cta == 1 ? (T - busy0) + t - busy1 : g - busy0 - busy1);
  const int workers = G - busy0 - busy1;
  // the area and volume terms: in the summing blocks' shared memory when they
  // fit (terms of block 0 and of block 1; one after the other in a block
  // alone), else in global memory (meshes of more triangles than a closed
  // surface of 8192 vertices has)
  const bool staged = p.nt <= kSegTerms;
  const bool pad = staged && p.tree_sums;
  double* a_to = staged ? (nc > 1 ? cl.map_shared_rank(terms, 0) : terms) : m.area;
  double* v_to = staged ? (nc > 1 ? cl.map_shared_rank(terms, 1) : terms + seg_terms(p.nt)) : m.vol;
  double* v_at = staged ? (nc > 1 ? terms : terms + seg_terms(p.nt)) : m.vol;
  const double* a_at = staged ? terms : m.area;

  global_first(p, m, f, SEG_WHOLE, g, G);
  cl.sync();
  for (int s = 0; s < H; ++s) {
    global_tri(p, m, f, a_to, v_to, pad, g, G);
    cl.sync();
    if (area_w || vol_w) {
      global_sum(p, m, f, SEG_WHOLE, area_w, area_w ? a_at : v_at, pad, area_w ? ss0 : ss1,
                 area_w ? t : t - 32 * voff * sw, sw, area_w ? 1 : 2);
    } else {
      global_terms(p, m, f, worker, workers);
      bond_prep_all(p, m, f, worker, workers, reinterpret_cast<unsigned char*>(&tail));
    }
    cl.sync();
    const bool more = s + 1 < H;
    const int gb = nc >= 4 ? nc - 1 : nc;  // blocks that gather
    if (cta < gb) global_gather(p, m, f, s, SEG_WHOLE, more, g, gb * T);
    // (a block that also gathers reads vX and vd there, which the tail only reads)
    if (cta == nc - 1) tail_block<kSegT>(p, m, f, epoch + s, more, tail);
    cl.sync();
  }
}

// The membrane of a mesh that no cluster holds in patches (from about 2600
// vertices on): a kernel a phase over the whole GPU, three dependent
// launches a step.  A cluster's few blocks lose to their scattered accesses, the
// more the larger the mesh; us a step in a 64 x 32 x 32 box with 50,000
// particles, a cluster of eight on global memory against this, FP64 and FP32:
// 2892 vertices 97, 92 and 62, 53; 4002 vertices 114, 108 and 66, 52; 7842
// vertices 209, 197 and 70, 59.  So do cohorts, a launch a phase over all their
// members: 1, 2 and 16 members of 7842 vertices 220, 231, 566 and 82, 93, 380.
constexpr int kWideT = 256;
// blocks of each phase (a block of the terms: kSegT threads, two for the sums; the
// gather's last one: the tail)
__host__ __device__ inline int wide_first_blocks(const DevParams& p) { return (3 * p.nv + kWideT - 1) / kWideT; }
__host__ __device__ inline int wide_tri_blocks(const DevParams& p) { return (p.nt + kWideT - 1) / kWideT; }
__host__ __device__ inline int wide_bond0(const DevParams& p) { return (2 * p.ne + 31) / 32 * 32; }
__host__ __device__ inline int wide_terms_blocks(const DevParams& p, int parts) {
  return 2 + ((parts & SEG_SECOND) ? (wide_bond0(p) + p.nv + kSegT - 1) / kSegT : 0);
}
__host__ __device__ inline int wide_gather_blocks(const DevParams& p) { return wide_first_blocks(p) + 1; }

__device__ __forceinline__ void wide_first_block(const DevParams& p, const Membrane& m, const FastBufs& f, int parts,
                                                 int b) {
  global_first(p, m, f, parts, b * kWideT + threadIdx.x, wide_first_blocks(p) * kWideT);
}
__device__ __forceinline__ void wide_tri_block(const DevParams& p, const Membrane& m, const FastBufs& f, int b) {
  global_tri(p, m, f, m.area, m.vol, false, b * kWideT + threadIdx.x, wide_tri_blocks(p) * kWideT);
}
// blocks 0 and 1: the sums, their terms staged in shared memory first where
// they fit; the others: a term or a vertex's bond preparation per thread
__device__ __forceinline__ void wide_terms_block(const DevParams& p, const Membrane& m, const FastBufs& f, int parts,
                                                 int b, unsigned char* smem) {
  const int t = threadIdx.x;
  if (b < 2) {
    const bool area = b == 0, staged = p.nt <= kSegTerms, pad = staged && p.tree_sums;
    const int run = tree_run(p.nt), sw = p.tree_sums ? 1 : kSegT / 32;
    const double* src = area ? m.area : m.vol;
    SumScratch& S = *reinterpret_cast<SumScratch*>(smem);
    double* terms = reinterpret_cast<double*>(smem + sizeof(SumScratch));
    if (staged && (parts & SEG_FIRST))
      for (int i = t; i < p.nt; i += kSegT) terms[pad ? tree_at(i, run) : i] = src[i];
    __syncthreads();
    if (t < 32 * sw) global_sum(p, m, f, parts, area, staged ? terms : src, pad, S, t, sw, 1);
    return;
  }
  const int worker = (b - 2) * kSegT + t, bond0 = wide_bond0(p);
  if (worker < bond0) global_terms(p, m, f, worker, bond0);
  else bond_prep_all(p, m, f, worker - bond0, 1 << 30, smem);
}
__device__ __forceinline__ void wide_gather_block(const DevParams& p, const Membrane& m, const FastBufs& f,
                                                  uint64_t epoch, int s, int parts, bool more, int b, TailSmem& tail) {
  const int n = wide_first_blocks(p);
  if (b == n) tail_block<kWideT>(p, m, f, epoch + s, more, tail);
  else global_gather(p, m, f, s, parts, more, b * kWideT + threadIdx.x, n * kWideT);
}
__global__ void __launch_bounds__(kWideT) k_wide_first(DevParams p, Membrane m, FastBufs f, int parts) {
  wide_first_block(p, m, f, parts, blockIdx.x);
}
__global__ void __launch_bounds__(kWideT) k_wide_tri(DevParams p, Membrane m, FastBufs f) {
  wide_tri_block(p, m, f, blockIdx.x);
}
__global__ void __launch_bounds__(kSegT) k_wide_terms(DevParams p, Membrane m, FastBufs f, int parts) {
  extern __shared__ __align__(16) unsigned char seg_sh[];
  wide_terms_block(p, m, f, parts, blockIdx.x, seg_sh);
}
__global__ void __launch_bounds__(kWideT) k_wide_gather(DevParams p, Membrane m, FastBufs f, uint64_t eoff, int s,
                                                        int parts, int more) {
  __shared__ TailSmem tail;
  wide_gather_block(p, m, f, epoch_of(p, eoff), s, parts, more, blockIdx.x, tail);
}

// ---- the membrane in patches ---------------------------------------------------------
// The vertices are split among the cluster's blocks into connected patches
// (host, build_patches).  A block keeps in shared memory its vertices' state
// (phase C: a component of a vertex per thread), the coordinates of its vertices
// and of those its items touch, and the force terms of its own vertices, at the
// place where the gather reads them.  Items on a seam are computed by each block
// that owns one of their vertices (every time by the same operations), so
// between the phases only coordinates of seam vertices, the area and volume
// terms and the two factors cross blocks, through distributed shared memory.
// what the tail in block 0 reads: the vertices in the parasite's reach (w) and
// those with bond draws (d), in the order they arrived, and the same as bits by
// vertex, from which each one's place in vertex order follows
constexpr int kTailWca = 768, kTailDraw = 1024, kTailEvents = 128, kTailWords = 8192 / 32;
struct PatchTail {
  double wX[3][kTailWca], dpr[kTailDraw];
  int wid[kTailWca], did[kTailDraw], dval[kTailDraw], od[kTailDraw];
  unsigned wbits[kTailWords], dbits[kTailWords];
  unsigned short wpre[kTailWords], dpre[kTailWords];  // bits before each word
  unsigned short word[kTailWca], dord[kTailDraw];     // list entries in vertex order
  int ev[kTailEvents], evv[kTailEvents], evr[kTailEvents];
  int nw, ndr, nev;
  MemScalars sc;
};
// warps of a block that do the bond preparation, half-warps of them that look
// for bond candidates
constexpr int kBondWarps = 8, kBondHalves = 2 * kBondWarps;
struct PatchMisc {
  double fac[2], para[3];
  int paradx, parady;
  int nb;                                // free knobs of the block near the wall
  int next;                              // chunk of edges or bending terms to be taken next
  unsigned short bond[kPatchOwn];
  unsigned char pn[kPatchOwn];           // their candidates
  int bpid[kPatchOwn];                   // their cells
  double pd[kBondHalves][kMaxPairs];
  int pj[kBondHalves][kMaxPairs];
};
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }

// bits before each of n words, by one warp
__device__ __forceinline__ void bit_prefix(const unsigned* bits, unsigned short* pre, int n, int lane) {
  int base = 0;
  for (int q0 = 0; q0 < n; q0 += 32) {
    const int q = q0 + lane, c = q < n ? __popc(bits[q]) : 0;
    int x = c;
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (q < n) pre[q] = (unsigned short)(base + x - c);
    base += __shfl_sync(0xffffffffu, x, 31);
  }
}
__device__ __forceinline__ int bit_rank(const unsigned* bits, const unsigned short* pre, int i) {
  return pre[i >> 5] + __popc(bits[i >> 5] & ((1u << (i & 31)) - 1u));
}

// the tail, by tn threads (tid) of block 0
__device__ __forceinline__ void patch_tail(const DevParams& p, const Membrane& m, const FastBufs& f, uint64_t epoch,
                                           PatchTail& S, int tid, int tn) {
  const int nw = S.nw, nd = S.ndr, words = (p.nv + 31) / 32;
  const bool wfits = nw <= kTailWca, dfits = nd <= kTailDraw;
  if (wfits)
    for (int e = tid; e < nw; e += tn) atomicOr(&S.wbits[S.wid[e] >> 5], 1u << (S.wid[e] & 31));
  if (dfits)
    for (int e = tid; e < nd; e += tn) atomicOr(&S.dbits[S.did[e] >> 5], 1u << (S.did[e] & 31));
  bar_named(4, tn);
  if (tid < 32) bit_prefix(S.wbits, S.wpre, words, tid);
  else if (tid < 64) bit_prefix(S.dbits, S.dpre, words, tid - 32);
  bar_named(4, tn);
  if (wfits)
    for (int e = tid; e < nw; e += tn) S.word[bit_rank(S.wbits, S.wpre, S.wid[e])] = (unsigned short)e;
  if (dfits)
    for (int e = tid; e < nd; e += tn) S.dord[bit_rank(S.dbits, S.dpre, S.did[e])] = (unsigned short)e;
  bar_named(4, tn);
  for (int q = tid; q < words; q += tn) S.wbits[q] = S.dbits[q] = 0u;
  if (tid < 32) {
    // pfdt's parasite sum in vertex order, lane c its component c
    double fc = 0.0;
    if (tid < 3) {
      if (wfits) {
        int r = 0;
        for (; r + 8 <= nw; r += 8) {
          double x[8];
#pragma unroll
          for (int k = 0; k < 8; ++k) x[k] = S.wX[tid][S.word[r + k]];
#pragma unroll
          for (int k = 0; k < 8; ++k) fc += x[k];
        }
        for (; r < nw; ++r) fc += S.wX[tid][S.word[r]];
      } else {
        for (int ii = 0; ii < p.nv; ++ii)
          if (f.vd[ii] & VF_WCA) fc += f.vX[3 * ii + tid];
      }
      MemScalars& sc = S.sc;
      sc.parafdt[tid] += fc;
      sc.paraV[tid] += ((sc.paraft[tid] + sc.parafdt[tid]) * p.dtmd / (2.0 * p.PRmass));
      sc.paraft[tid] = sc.parafdt[tid];
      sc.parafdt[tid] = 0.0;
    }
    __syncwarp();
  } else {
    // bond draws: each entry's first draw index by a scan over the entries in
    // vertex order (second warp), then the draws (every warp but the first)
    const int lane = tid & 31, on = tn - 32;
    if (dfits && tid < 64) {
      int base = 0;
      for (int r0 = 0; r0 < nd; r0 += 32) {
        const int r = r0 + lane, n = r < nd ? S.dval[S.dord[r]] & VF_DRAWS : 0;
        int x = n;
        for (int o = 1; o < 32; o <<= 1) {
          const int y = __shfl_up_sync(0xffffffffu, x, o);
          if (lane >= o) x += y;
        }
        if (r < nd) S.od[r] = base + x - n;
        base += __shfl_sync(0xffffffffu, x, 31);
      }
    }
    bar_named(5, on);
    if (dfits)
      for (int r = tid - 32; r < nd; r += on) {
        const int e = S.dord[r], n = S.dval[e] & VF_DRAWS, od = S.od[r];
        const double pr = S.dpr[e];
        for (int q = 0; q < n; ++q) {
          if (pr > draw_uniform(p.seed, STREAM_BOND, epoch, (uint64_t)(od + q))) {
            const int k = atomicAdd(&S.nev, 1);
            if (k < kTailEvents) {
              S.ev[k] = od + q;
              S.evv[k] = S.did[e];
              S.evr[k] = (S.dval[e] & VF_BONDED) ? -1 : q;
            }
          }
        }
      }
    bar_named(5, on);
    if (tid >= 64) return;
    __syncwarp();
    if (lane == 0) {
      if (dfits && S.nev <= kTailEvents) {
        // the successful draws in draw order
        for (int done = -1, k = 0; k < S.nev; ++k) {
          int at = 0, best = 0x7fffffff;
          for (int u = 0; u < S.nev; ++u)
            if (S.ev[u] > done && S.ev[u] < best) { best = S.ev[u]; at = u; }
          done = best;
          const int ii = S.evv[at], r = S.evr[at];
          if (r < 0) {
            const int jj = m.bondl[ii];
            m.bondi[ii] = 0; m.bondl[ii] = p.randno; m.ligi[jj] = 0;
          } else {
            const int j = m.pair_j[(int64_t)ii * kMaxPairs + r];
            if (m.ligi[j] == 0) { m.ligi[j] = 1; m.bondi[ii] = 1; m.bondl[ii] = j; }
          }
        }
      } else {
        bond_events_serial(p, m, f, epoch);
      }
      S.ndr = 0;
      S.nev = 0;
    }
  }
  if (tid == 0) S.nw = 0;
}

// room for a warp's entries on a list of the tail, its place taken with one
// atomic (block 0's shared memory serves them one at a time: with one per entry
// the discocyte's bond preparation took 16 000 cycles, most of it waiting);
// this lane's entry
__device__ __forceinline__ int tail_room(int* count, bool on) {
  const unsigned b = __ballot_sync(0xffffffffu, on);
  if (b == 0u) return 0;
  const int lane = threadIdx.x & 31, first = __ffs(b) - 1;
  int at = 0;
  if (lane == first) at = atomicAdd(count, __popc(b));
  return __shfl_sync(0xffffffffu, at, first) + __popc(b & ((1u << lane) - 1u));
}
// vertices' bond draws onto the tail's list, by a whole warp
__device__ __forceinline__ void patch_draws(PatchTail* T, bool on, int i, int val, double pr) {
  const int e = tail_room(&T->ndr, on);
  if (on && e < kTailDraw) { T->did[e] = i; T->dval[e] = val; T->dpr[e] = pr; }
}

// the parasite's position to every block
__device__ __forceinline__ void patch_para(cooperative_groups::cluster_group& cl, PatchMisc* misc, const MemScalars& sc,
                                           int lane, int nc) {
  for (int b = lane; b < nc; b += 32) {
    PatchMisc* q = cl.map_shared_rank(misc, b);
    q->para[0] = sc.para[0]; q->para[1] = sc.para[1]; q->para[2] = sc.para[2];
    q->paradx = sc.paradx; q->parady = sc.parady;
  }
}

__device__ __forceinline__ void membrane_patch(const DevParams& p, const Membrane& m, const FastBufs& f,
                                               uint64_t epoch, int H, int parts, unsigned char* smem) {
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  const PatchPlan& P = f.patch;
  const int cta = (int)cl.block_rank(), nc = (int)cl.num_blocks(), t = threadIdx.x;
  const PatchHdr hd = P.hdr[cta];
  // at the same place in every block (remote blocks write there): misc, the
  // coordinates, and in blocks 0 and 1 the sums' and the tail's room
  PatchMisc* misc = reinterpret_cast<PatchMisc*>(smem + P.o_misc);
  double* cx = reinterpret_cast<double*>(smem + P.o_c);  // unwrapped x, y and z: P.nl each
  double* terms = reinterpret_cast<double*>(smem + P.o_terms);
  SumScratch& ss = *reinterpret_cast<SumScratch*>(smem + P.o_sum);
  PatchTail& tail = *reinterpret_cast<PatchTail*>(smem + P.o_tail);
  // the block's own: tables, the entries of its vertices' terms, their state
  unsigned char* tab = smem + hd.o_tab;
  double* E = reinterpret_cast<double*>(smem + hd.o_e);   // 7 x ned: edges
  double* D = reinterpret_cast<double*>(smem + hd.o_d);   // 3 x nd: bending entries
  double* Y = reinterpret_cast<double*>(smem + hd.o_t);   // 8 x nt: triangle entries
  double* sx = reinterpret_cast<double*>(smem + hd.o_s);  // position, velocity: 3 each per vertex
  double* sv = sx + 3 * hd.no;
  int* sim = reinterpret_cast<int*>(sv + 3 * hd.no);      // images along x and y
  int* sfl = sim + 2 * hd.no;                             // bond draws and VF_* flags
  for (int i = t; i < hd.bytes / 16; i += kSegT)
    reinterpret_cast<int4*>(tab)[i] = reinterpret_cast<const int4*>(P.blob + hd.blob)[i];
  const int* own = reinterpret_cast<const int*>(tab + hd.own);
  const PatchTri* tri = reinterpret_cast<const PatchTri*>(tab + hd.tri);
  const PatchEdge* edge = reinterpret_cast<const PatchEdge*>(tab + hd.edge);
  const PatchDih* dih = reinterpret_cast<const PatchDih*>(tab + hd.dih);
  const unsigned short* ent = reinterpret_cast<const unsigned short*>(tab + hd.ent);
  const unsigned short* eend = reinterpret_cast<const unsigned short*>(tab + hd.eend);
  const PatchSend* send = reinterpret_cast<const PatchSend*>(tab + hd.send);
  // blocks 0 and 1 give their first sw warps to the sums (Sarea, Volume);
  // block 0's also run the tail
  const int busy = cta < 2 ? 32 * P.sw : 0;
  const int wt = t - busy, nwk = kSegT - busy, no3 = 3 * hd.no, lane = t & 31;
  const bool summing = wt < 0;
  // block 1's summing warps help with phase C (block 0's run the tail then)
  const int cw = cta == 1 ? t : wt, ncw = cta == 1 ? kSegT : nwk;
  const double pon = 1.0 - exp(-p.onrate * p.dtmd);
  PatchTail* T = cl.map_shared_rank(&tail, 0);
  const bool pad = p.tree_sums != 0;
  const int run = tree_run(p.nt);
  // f dt / (2 m) of a half-kick
  const Divisor mass2{2.0 * p.pmass, 1.0 / (2.0 * p.pmass)};
  const double grav = -p.Fg / (double)p.nv, rlap = 1.0 / (p.elap);

  // component k of own vertex v: first half-kick with force F, snapshot of step
  // s, drift and wrap (maincode.cpp:487-496, 566-574), the unwrapped coordinate
  auto kick = [&](int q, int v, int k, int s, double vel, double F) {
    vel += div_by(F * p.dtmd, mass2);
    double x = sx[q];
    const int64_t o = (int64_t)s * p.nv + hd.base + v;
    (k == 0 ? f.snap.x : (k == 1 ? f.snap.y : f.snap.z))[o] = x;
    (k == 0 ? f.snap.vx : (k == 1 ? f.snap.vy : f.snap.vz))[o] = vel;
    x += (vel * p.dtmd);
    double u = x;
    if (k < 2) {
      const double L = k == 0 ? p.Lx : p.Ly;
      int im = sim[2 * v + k];
      if (x > L) { x -= L; im += 1; }
      if (x < 0) { x += L; im -= 1; }
      sim[2 * v + k] = im;
      u = x + im * L;
    }
    sx[q] = x;
    sv[q] = vel;
    cx[k * P.nl + v] = u;
  };
  // the seam's coordinates to the blocks that read them
  auto publish = [&](int me, int n) {
    bar_named(3, n);
    for (int q = me; q < hd.nsend; q += n) {
      const PatchSend e = send[q];
      double* to = cl.map_shared_rank(cx, e.cta) + e.slot;
      to[0] = cx[e.own]; to[P.nl] = cx[P.nl + e.own]; to[2 * P.nl] = cx[2 * P.nl + e.own];
    }
  };
  __syncthreads();
  for (int q = wt; q < no3 && !summing; q += nwk) {
    const int v = q / 3, k = q - 3 * v, i = own[v];
    sx[q] = (k == 0 ? m.x : (k == 1 ? m.y : m.z))[i];
    double* F = (k == 0 ? m.fx : (k == 1 ? m.fy : m.fz)) + i;
    const double vel = (k == 0 ? m.vx : (k == 1 ? m.vy : m.vz))[i];
    if (k < 2) sim[q - v] = (k == 0 ? m.ix : m.iy)[i];
    if (parts & SEG_FIRST) {
      kick(q, v, k, 0, vel, *F);
      *F = 0.0;
    } else {
      sv[q] = vel;
      cx[k * P.nl + v] = k == 2 ? sx[q] : sx[q] + sim[q - v] * (k == 0 ? p.Lx : p.Ly);
    }
  }
  cluster_arrive();  // every block has started: its shared memory may be written
  cluster_wait();
  if (!summing) publish(wt, nwk);
  if (t == 0) misc->nb = misc->next = 0;
  if (cta == 0 && t < 32) {
    if (t == 0) {
      tail.sc = *m.sc;
      if (parts & SEG_FIRST) para_drift(p, &tail.sc);
      tail.nw = tail.ndr = tail.nev = 0;
    }
    for (int q = t; q < kTailWords; q += 32) tail.wbits[q] = tail.dbits[q] = 0u;
    __syncwarp();
    patch_para(cl, misc, tail.sc, t, nc);
  }
  cluster_arrive();
  cluster_wait();
  for (int s = 0; s < H; ++s) {
    const bool more = s + 1 < H;
    if (summing) {
      cluster_arrive();
      cluster_wait();
      double r = 0.0;
      if (parts & SEG_FIRST) {
        if (p.tree_sums) { if (t < 32) r = tree_sum(terms, p.nt, pad, t); }
        else r = ordered_sum(terms, p.nt, ss, t, P.sw, 1);
        if (t == 0) *(cta == 0 ? &m.sc->Sarea : &m.sc->Volume) = r;
      } else if (t < 32) {
        r = cta == 0 ? m.sc->Sarea : m.sc->Volume;
      }
      if (t < nc && (parts & SEG_SECOND))
        // the factor of the global area or volume force, to every block
        cl.map_shared_rank(misc, t)->fac[cta] = cta == 0 ? -p.kappasa * (r - p.Sarea0) / p.Sarea0
                                                         : -p.kappav * (r - p.Volume0) / (p.Volume0);
      cluster_arrive();
      cluster_wait();
      if (!(parts & SEG_SECOND)) break;
      // the tail beside phase C
      if (cta == 0) {
        patch_tail(p, m, f, epoch + s, tail, t, 32 * P.sw);
        if (t < 32 && more) {
          if (t == 0) para_drift(p, &tail.sc);
          __syncwarp();
          patch_para(cl, misc, tail.sc, t, nc);
        }
        cluster_arrive();
        cluster_wait();
        continue;
      }
    } else {
    // A: triangles
    for (int q = wt; q < hd.ntri; q += nwk) {
      const PatchTri e = tri[q];
      const double x1 = cx[e.v[0]], y1 = cx[P.nl + e.v[0]], z1 = cx[2 * P.nl + e.v[0]];
      const double x2 = cx[e.v[1]], y2 = cx[P.nl + e.v[1]], z2 = cx[2 * P.nl + e.v[1]];
      const double x3 = cx[e.v[2]], y3 = cx[P.nl + e.v[2]], z3 = cx[2 * P.nl + e.v[2]];
      double A[3] = {x2 - x1, y2 - y1, z2 - z1}, B[3] = {x3 - x1, y3 - y1, z3 - z1}, e0[3], Cn[3];
      cp(A, B, e0);
      const double area = 0.5 * sqrt(e0[0] * e0[0] + e0[1] * e0[1] + e0[2] * e0[2]);
      Cn[0] = div3(x1 + x2 + x3);
      Cn[1] = div3(y1 + y2 + y3);
      Cn[2] = div3(z1 + z2 + z3);
      if (e.g >= 0) {
        const int at = pad ? tree_at(e.g, run) : e.g;
        cl.map_shared_rank(terms, 0)[at] = area;
        cl.map_shared_rank(terms, 1)[at] = (1.0 / 6.0) * ((e0[0] * Cn[0]) + (e0[1] * Cn[1]) + (e0[2] * Cn[2]));
      }
      if (!(parts & SEG_SECOND)) continue;
      // per corner: C (the area terms without their factors), the volume term
      // without betav and / 6, alphad, 4 area
      const double alphad = -p.kappad * (area - e.tarea) / (4.0 * e.tarea * area);
      double A13[3] = {x1 - x3, y1 - y3, z1 - z3}, A32[3] = {x3 - x2, y3 - y2, z3 - z2}, eta[3], C[3];
      cp(A13, A, eta);
      const double e3[3] = {div3(eta[0]), div3(eta[1]), div3(eta[2])};
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        if (e.d[c] == kNoEntry) continue;
        const double* side = c == 0 ? A32 : (c == 1 ? A13 : A);
        double* to = Y + e.d[c];
        cp(eta, side, C);
        to[0] = C[0]; to[hd.nt] = C[1]; to[2 * hd.nt] = C[2];
        cp(Cn, side, C);
        to[3 * hd.nt] = e3[0] + C[0]; to[4 * hd.nt] = e3[1] + C[1]; to[5 * hd.nt] = e3[2] + C[2];
        to[6 * hd.nt] = alphad;
        to[7 * hd.nt] = 4.0 * area;
      }
    }
    cluster_arrive();
    if (parts & SEG_SECOND) {
      // B: the first warps prepare the bonds (a chain of dependent reads and few
      // operations) beside the others' edge and bending terms, then join them
      if (wt < 32 * kBondWarps) {
        for (int v0 = wt - lane; v0 < hd.no; v0 += 32 * kBondWarps) {
          const int v = v0 + lane;
          const bool on = v < hd.no;
          const int i = on ? own[v] : 0;
          int flags = 0, bondi = -1, knob = 0, pid = 0;
          double pr = 0.0, w[3];
          bool wca = false;
          if (on) {
            bondi = m.bondi[i];
            knob = m.knob[i];
            pid = m.pid[i];
            const double u[3] = {cx[v], cx[P.nl + v], cx[2 * P.nl + v]};
            const double pp[3] = {(misc->para[0] + misc->paradx * p.Lx), (misc->para[1] + misc->parady * p.Ly),
                                  misc->para[2]};
            wca = wca_at(p, pp, u[0], u[1], u[2], w);
            if (wca)
              for (int k = 0; k < 3; ++k) f.vX[3 * i + k] = w[k];
            if (bondi == 1) {
              double sp[3];
              flags = bonded_prep(p, m, i, sx[3 * v], sx[3 * v + 1], u[2], sim[2 * v], sim[2 * v + 1], pr, sp);
              if (flags & VF_SPRING)
                for (int k = 0; k < 3; ++k) f.vS[3 * i + k] = sp[k];
              flags |= 1;
            } else if ((u[2] < p.dthr) && (bondi == 0) && (knob == 1)) {
              const int at = atomicAdd(&misc->nb, 1);
              misc->bond[at] = (unsigned short)v;
              misc->bpid[at] = pid;
            }
          }
          patch_draws(T, bondi == 1, i, flags, pr);
          const int e = tail_room(&T->nw, wca);
          if (wca) {
            if (e < kTailWca) { T->wid[e] = i; T->wX[0][e] = w[0]; T->wX[1][e] = w[1]; T->wX[2][e] = w[2]; }
            flags |= VF_WCA;
          }
          if (on) f.vd[i] = sfl[v] = flags;
        }
        bar_named(6, 32 * kBondWarps);
        // free knobs near the wall, half a warp each: candidates and their order
        const int nb = misc->nb, half = wt >> 4;
        for (int e0 = half & ~1; e0 < nb; e0 += kBondHalves) {
          const int e = e0 + (half & 1);
          const bool on = e < nb;
          const int v = on ? misc->bond[e] : 0, i = on ? own[v] : 0;
          const int n = bond_pairs(p, m, on, i, sx[3 * v], sx[3 * v + 1], cx[2 * P.nl + v], sim[2 * v], sim[2 * v + 1],
                                   on ? misc->bpid[e] : 0, misc->pd[half], misc->pj[half]);
          if (on && (wt & 15) == 0) {
            m.pon[i] = pon;
            m.npair[i] = n;
            f.vd[i] = sfl[v] |= n;
            misc->pn[e] = (unsigned char)n;
          }
        }
        if (nb > 0) {
          bar_named(6, 32 * kBondWarps);
          for (int e0 = wt - lane; e0 < nb; e0 += 32 * kBondWarps) {
            const int e = e0 + lane, n = e < nb ? misc->pn[e] : 0;
            patch_draws(T, n > 0, e < nb ? own[misc->bond[e]] : 0, n, pon);
          }
        }
      }
      // chunks of 32 bending terms, then edges, each by the next free warp
      const int nd = (hd.ndih + 31) / 32, nch = nd + (hd.ned + 31) / 32;
      while (true) {
        int ch = 0;
        if (lane == 0) ch = atomicAdd(&misc->next, 1);
        ch = __shfl_sync(0xffffffffu, ch, 0);
        if (ch >= nch) break;
        if (ch < nd) {
          const int q = 32 * ch + lane;
          if (q >= hd.ndih) continue;
          const PatchDih e = dih[q];
          const double *c1 = cx + e.v[0], *c4 = cx + e.v[1], *c2 = cx + e.v[2], *c3 = cx + e.v[3];
          double r[4][3];
          dih_terms(p, c1[0], c1[P.nl], c1[2 * P.nl], c2[0], c2[P.nl], c2[2 * P.nl], c3[0], c3[P.nl], c3[2 * P.nl],
                    c4[0], c4[P.nl], c4[2 * P.nl], r);
#pragma unroll
          for (int c = 0; c < 4; ++c)
            if (e.d[c] != kNoEntry)
              for (int k = 0; k < 3; ++k) D[k * hd.nd + e.d[c]] = r[c][k];
          continue;
        }
        const int q = 32 * (ch - nd) + lane;
        if (q >= hd.ned) continue;
        const PatchEdge e = edge[q];
        double A[3];
        A[0] = cx[e.v[0]] - cx[e.v[1]];
        A[1] = cx[P.nl + e.v[0]] - cx[P.nl + e.v[1]];
        A[2] = cx[2 * P.nl + e.v[0]] - cx[2 * P.nl + e.v[1]];
        const double aa = sqrt(A[0] * A[0] + A[1] * A[1] + A[2] * A[2]);
        A[0] /= aa; A[1] /= aa; A[2] /= aa;
        const double xx = aa / (2.5 * e.l0);
        const double xxx = 1.0 / (4.0 * (1.0 - xx) * (1.0 - xx));
        // the terms on the second end (wl A, pk); those on the first are their
        // negatives
        double* to = E + q;
        to[0] = rlap * (xxx - 0.25 + xx);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          to[(1 + k) * hd.ned] = A[k];
          to[(4 + k) * hd.ned] = -e.kp * A[k] / (aa * aa);
        }
      }
    }
    cluster_wait();
    cluster_arrive();
    cluster_wait();
    if (!(parts & SEG_SECOND)) break;
    }
    // C: the triangles' factors; then each vertex component adds its terms in
    // order, external forces, kicks
    {
      const double beta = misc->fac[0], betav = misc->fac[1];
      const Divisor six{6.0, 1.0 / 6.0};
      for (int e = cw; e < hd.nt; e += ncw) {
        double* q = Y + e;
        q[7 * hd.nt] = beta / q[7 * hd.nt];
#pragma unroll
        for (int k = 3; k < 6; ++k) q[k * hd.nt] = div_by(betav * q[k * hd.nt], six);
      }
      if (cw == 0) misc->nb = misc->next = 0;
      bar_named(3, ncw);
    }
    for (int q = cw; q < no3; q += ncw) {
      const int v = q / 3, k = q - 3 * v, i = own[v];
      const unsigned short *e0 = ent + 3 * v, *e1 = e0 + 3;
      double acc = 0.0;
#pragma unroll 2
      for (int e = e0[0]; e < e1[0]; ++e) {
        const int c = eend[e];  // 2 x edge + (1: its second end)
        const double* r = E + (c >> 1);
        const double wk = r[0] * r[(1 + k) * hd.ned], pk = r[(4 + k) * hd.ned];
        acc += (c & 1) ? wk : -wk;
        acc += (c & 1) ? pk : -pk;
      }
#pragma unroll 2
      for (int e = e0[1]; e < e1[1]; ++e) {
        const double* r = Y + e;
        const double C = r[k * hd.nt];
        acc += r[7 * hd.nt] * C;
        acc += r[6 * hd.nt] * C;
        acc += r[(3 + k) * hd.nt];
      }
      const double* d = D + k * hd.nd;
#pragma unroll 4
      for (int e = e0[2]; e < e1[2]; ++e) acc += d[e];
      // the first half-kick has reset the force (:490)
      double* F = (k == 0 ? m.fx : (k == 1 ? m.fy : m.fz)) + i;
      double fk = (parts & SEG_FIRST) ? 0.0 : *F;
      const int vd = sfl[v];
      if (vd & VF_WCA) fk -= f.vX[3 * i + k];  // pfdt's -X
      fk += acc;
      if (k == 2) fk += grav;
      if (vd & VF_SPRING) fk += f.vS[3 * i + k];
      if (k == 2) {
        double cc = cx[2 * P.nl + v];
        if (cc < 0.5) fk += 300.0 * exp(-50.0 * cc);
        cc = p.Lz - cx[2 * P.nl + v];
        if (cc < 0.5) fk -= 300.0 * exp(-50.0 * cc);
      }
      // second half-kick (maincode.cpp:727-733)
      const double vel = sv[q] + div_by(fk * p.dtmd, mass2);
      raise_health(p, !isfinite(fk + vel), HEALTH_MEMBRANE);
      if (more) {
        kick(q, v, k, s + 1, vel, fk);
      } else {
        sv[q] = vel;
        *F = fk;
      }
    }
    if (more) publish(cw, ncw);
    cluster_arrive();
    cluster_wait();
  }
  if (!summing)
    for (int q = wt; q < no3; q += nwk) {
      const int v = q / 3, k = q - 3 * v, i = own[v];
      (k == 0 ? m.x : (k == 1 ? m.y : m.z))[i] = sx[q];
      (k == 0 ? m.vx : (k == 1 ? m.vy : m.vz))[i] = sv[q];
      if (k < 2) (k == 0 ? m.ix : m.iy)[i] = sim[q - v];
    }
  cluster_arrive();  // no block ends while another may write to its memory
  cluster_wait();
  if (cta == 0 && t == 0) {
    MemScalars* sc = m.sc;
    for (int k = 0; k < 3; ++k) {
      sc->para[k] = tail.sc.para[k]; sc->paraV[k] = tail.sc.paraV[k];
      sc->paraft[k] = tail.sc.paraft[k]; sc->parafdt[k] = tail.sc.parafdt[k];
    }
    sc->paradx = tail.sc.paradx; sc->parady = tail.sc.parady;
  }
}

__device__ __forceinline__ void membrane_segment(const DevParams& p, const Membrane& m, const FastBufs& f,
                                                 uint64_t epoch, int H, int parts, unsigned char* smem) {
  if (f.patch.nc > 0) membrane_patch(p, m, f, epoch, H, parts, smem);
  else membrane_global(p, m, f, epoch, H, smem);
}

__global__ void __launch_bounds__(kSegT) k_membrane(DevParams p, Membrane m, FastBufs f, uint64_t eoff, int H, int parts) {
  extern __shared__ __align__(16) unsigned char seg_sh[];
  membrane_segment(p, m, f, epoch_of(p, eoff), H, parts, seg_sh);
}

void patch_layout(PatchPlan& P, PatchHdr* hdr, int nt) {
  int o = 0;
  auto take = [&](size_t bytes) { const int at = o; o += (int)((bytes + 15) / 16 * 16); return at; };
  P.o_misc = take(sizeof(PatchMisc));
  P.o_c = take(3 * (size_t)P.nl * sizeof(double));
  const int common = o;
  P.o_terms = take((size_t)seg_terms(nt) * sizeof(double));
  P.o_sum = take(sizeof(SumScratch));
  P.o_tail = take(sizeof(PatchTail));
  const int sums = o;
  for (int b = 0; b < P.nc; ++b) {
    PatchHdr& h = hdr[b];
    o = b == 0 ? sums : (b == 1 ? P.o_tail : common);  // block 0 alone has a tail
    h.o_tab = take(h.bytes);
    h.o_e = take(7 * (size_t)h.ned * sizeof(double));
    h.o_d = take(3 * (size_t)h.nd * sizeof(double));
    h.o_t = take(8 * (size_t)h.nt * sizeof(double));
    h.o_s = take((size_t)h.no * (6 * sizeof(double) + 3 * sizeof(int)));
    P.smem = std::max(P.smem, o);
  }
}

static size_t seg_smem(const DevParams& p, const FastBufs& f, int nc) {
  if (f.patch.nc > 0) return f.patch.smem;
  const size_t fixed = 2 * sizeof(SumScratch) + ((sizeof(TailSmem) + 15) & ~size_t(15));
  return fixed + (p.nt <= kSegTerms ? (nc > 1 ? 1 : 2) * (size_t)seg_terms(p.nt) * sizeof(double) : 0);
}

// k_wide_terms: the staged terms, or the bond preparation's room
static size_t wide_smem(const DevParams& p) {
  const size_t sum = sizeof(SumScratch) + (p.nt <= kSegTerms ? (size_t)seg_terms(p.nt) * sizeof(double) : 0);
  return std::max(sum, (size_t)(kSegT / 16) * kMaxPairs * (sizeof(double) + sizeof(int)));
}

// the streaming's records of every triangle for the steps [s0, s1) of a stretch
// and what none of them needs to test (TriCull), by a lane per triangle and
// kRecordRows rows of steps.  A kernel of its own: in the membrane kernel their
// scattered loads and 96-byte stores bound the few blocks it has.  Latency
// bound: 5 to 7 us (a kernel for the records and one for the cull took 7 + 12,
// the latter a serial loop over the steps; 16 members 29 + 13 -> 21).
constexpr int kRecordTris = 32, kRecordRows = 8, kRecordT = kRecordTris * kRecordRows;
struct RecordSmem {
  double first[12][kRecordTris];
  double dX[kRecordRows][kRecordTris], dA[kRecordRows][kRecordTris];
  int bands[kRecordRows][kRecordTris];
};
__device__ __forceinline__ void records_block(const DevParams& p, const FastBufs& f, int s0, int s1, int part, int64_t bid,
                                              RecordSmem& S) {
  const int lane = threadIdx.x % kRecordTris, row = threadIdx.x / kRecordTris;
  const int64_t j = bid * kRecordTris + lane;
  const bool on = j < p.nt;
  const int c[3] = {on ? f.st1[j] : 0, on ? f.st2[j] : 0, on ? f.st3[j] : 0};
  const double rx = p.Lx - (3.0 * p.a), ry = p.Ly - (3.0 * p.a), l = 3.0 * p.a;
  CullMove mv{0.0, 0.0, 0};
  TriPre t0{};
  for (int base = s0; base < s1; base += kRecordRows) {
    const int s = base + row;
    TriPre t{};
    int b = 0;
    if (on && s < s1) {
      const Snap sn = snap_of(f, s, p.nv);
      t = tri_record(p, sn, c[0], c[1], c[2]);
      for (int k = 0; k < 3; ++k) {
        const double x = sn.x[c[k]], y = sn.y[c[k]];
        b |= (x < l ? BAND_LX : 0) | (x > rx ? BAND_HX : 0) | (y < l ? BAND_LY : 0) | (y > ry ? BAND_HY : 0);
      }
      const int64_t q = (int64_t)s * p.nt + j;
      f.pre[q] = t;
      f.bands[q] = (unsigned char)b;
    }
    if (base == s0) {
      if (row == 0)
        for (int k = 0; k < 3; ++k) {
          S.first[k][lane] = t.X[k]; S.first[3 + k][lane] = t.Xdt[k];
          S.first[6 + k][lane] = t.A1[k]; S.first[9 + k][lane] = t.A2[k];
        }
      __syncthreads();
      for (int k = 0; k < 3; ++k) {
        t0.X[k] = S.first[k][lane]; t0.Xdt[k] = S.first[3 + k][lane];
        t0.A1[k] = S.first[6 + k][lane]; t0.A2[k] = S.first[9 + k][lane];
      }
    }
    if (on && s < s1) cull_fold(mv, t0, t, b);
  }
  S.dX[row][lane] = mv.dX;
  S.dA[row][lane] = mv.dA;
  S.bands[row][lane] = mv.bands;
  __syncthreads();
  if (row != 0 || !on) return;
  for (int r = 1; r < kRecordRows; ++r) {
    mv.dX = fmax(mv.dX, S.dX[r][lane]);
    mv.dA = fmax(mv.dA, S.dA[r][lane]);
    mv.bands |= S.bands[r][lane];
  }
  cull_store(p, f.cull + 3 * ((int64_t)part * p.nt + j), t0, mv);
}
__global__ void __launch_bounds__(kRecordT) k_tri_records(DevParams p, FastBufs f, int s0, int s1, int part) {
  __shared__ RecordSmem S;
  records_block(p, f, s0, s1, part, blockIdx.x, S);
}

// whether a membrane runs as a kernel a phase
static bool wide_membrane(const FastBufs& f) { return f.patch.nc == 0 && !f.one_block && !f.cluster; }

// blocks of the membrane's cluster (not where wide_membrane)
int segment_blocks(const FastBufs& f) {
  if (f.patch.nc > 0) return f.patch.nc;
  return f.one_block ? 1 : 8;
}

bool one_block_fits(const DevParams& p) { return p.nv <= 1024 && p.nt <= 6144; }

// whether the device runs a cluster of nc blocks with smem bytes each
bool cluster_fits(int nc, int smem) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(nc);
  cfg.blockDim = dim3(kSegT);
  cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = nc;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  int n = 0;
  const bool ok = cudaOccupancyMaxActiveClusters(&n, k_membrane, &cfg) == cudaSuccess && n > 0;
  cudaGetLastError();
  return ok;
}

int launch_membrane(const DevParams& p, Membrane& m, const FastBufs& fb, uint64_t eoff, int s0, int H, int parts,
                    cudaStream_t st) {
  FastBufs f = fb;
  f.snap = snap_of(fb, s0, p.nv);
  if (wide_membrane(f)) {
    eoff += (uint64_t)s0;
    k_wide_first<<<wide_first_blocks(p), kWideT, 0, st>>>(p, m, f, parts);
    for (int s = 0; s < H; ++s) {
      k_wide_tri<<<wide_tri_blocks(p), kWideT, 0, st>>>(p, m, f);
      k_wide_terms<<<wide_terms_blocks(p, parts), kSegT, wide_smem(p), st>>>(p, m, f, parts);
      if (parts & SEG_SECOND)
        k_wide_gather<<<wide_gather_blocks(p), kWideT, 0, st>>>(p, m, f, eoff, s, parts, s + 1 < H);
    }
    return 1 + H * ((parts & SEG_SECOND) ? 3 : 2);
  }
  const int nc = segment_blocks(f);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(nc);
  cfg.blockDim = dim3(kSegT);
  cfg.dynamicSmemBytes = seg_smem(p, f, nc);
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = nc;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, k_membrane, p, m, f, eoff + (uint64_t)s0, H, parts);
  return 1;
}

}  // namespace irbc
