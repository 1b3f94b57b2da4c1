// fast.cu -- the production step, a stretch of timesteps at a time: the bulk
// streaming of every particle, the near-membrane streaming of those in cells
// with triangles, and the membrane (segment.cuh) on a side stream beside the
// bulk.
//
// Results equal the one-kernel-per-phase path (kernels.cu) bit for bit.
#include <algorithm>
#include <cstdio>
#include "fast.h"
#include "fp32.h"

namespace irbc {

static inline unsigned nb(int64_t n, int t) { return (unsigned)((n + t - 1) / t); }

#define UXm(v) (m.x[v] + m.ix[v] * p.Lx)
#define UYm(v) (m.y[v] + m.iy[v] * p.Ly)

// ================================================================ stream =====
// reflectionFed's per-triangle test and hit, reading the vertex snapshot.
// Returns true if the triangle was hit (state updated).  `q` holds the
// triangle's precomputed normals, used when the particle is outside the
// periodic stencil bands (3a from each side wall), where reflectionFed
// applies no shift.
__device__ __forceinline__ bool tri_visit(const DevParams& p, const Snap& sn, const TriPre& q, int jj,
                                          double& X_, double& Y_, double& Z_, double& VX, double& VY, double& VZ,
                                          int indio, double& fulldt, bool use_pre) {
  const double rstep = 0.0, dtmd = p.dtmd, a = p.a, Lx = p.Lx, Ly = p.Ly;
  int flg = 0;
  const double solvx = X_ + 0 * Lx, solvy = Y_ + 0 * Ly, solvz = Z_;
  double bt, bdt;
  double v1x, v1y, v1z, v2x, v2y, v2z, v3x, v3y, v3z;
  int p1, p2, p3;
  if (use_pre) {
    double PSt0 = solvx - q.A1[0], PSt1 = solvy - q.A1[1], PSt2 = solvz - q.A1[2];
    double PD0 = (solvx + VX * (dtmd - rstep)) - q.A2[0];
    double PD1 = (solvy + VY * (dtmd - rstep)) - q.A2[1];
    double PD2 = (solvz + VZ * (dtmd - rstep)) - q.A2[2];
    bt = q.X[0] * PSt0 + q.X[1] * PSt1 + q.X[2] * PSt2;
    bdt = q.Xdt[0] * PD0 + q.Xdt[1] * PD1 + q.Xdt[2] * PD2;
    if ((indio == 1) && (bt < 0)) flg = 1;
    if ((indio == 0) && (bt > 0)) flg = 1;
    if (!((bt * bdt <= 0) && (flg == 0))) return false;
    // the corners are read only for a crossing candidate
    p1 = sn.t1[jj]; p2 = sn.t2[jj]; p3 = sn.t3[jj];
    v1x = q.A1[0]; v1y = q.A1[1]; v1z = q.A1[2];
    v2x = (sn.x[p2] + 0 * Lx) + sn.vx[p2] * rstep; v2y = (sn.y[p2] + 0 * Ly) + sn.vy[p2] * rstep;
    v2z = sn.z[p2] + sn.vz[p2] * rstep;
    v3x = (sn.x[p3] + 0 * Lx) + sn.vx[p3] * rstep; v3y = (sn.y[p3] + 0 * Ly) + sn.vy[p3] * rstep;
    v3z = sn.z[p3] + sn.vz[p3] * rstep;
  } else {
    p1 = sn.t1[jj]; p2 = sn.t2[jj]; p3 = sn.t3[jj];
    v1x = (sn.x[p1] + 0 * Lx) + sn.vx[p1] * rstep; v1y = (sn.y[p1] + 0 * Ly) + sn.vy[p1] * rstep;
    v1z = sn.z[p1] + sn.vz[p1] * rstep;
    v2x = (sn.x[p2] + 0 * Lx) + sn.vx[p2] * rstep; v2y = (sn.y[p2] + 0 * Ly) + sn.vy[p2] * rstep;
    v2z = sn.z[p2] + sn.vz[p2] * rstep;
    v3x = (sn.x[p3] + 0 * Lx) + sn.vx[p3] * rstep; v3y = (sn.y[p3] + 0 * Ly) + sn.vy[p3] * rstep;
    v3z = sn.z[p3] + sn.vz[p3] * rstep;
    double rstencilx = Lx - (3.0 * a), lstencilx = 3.0 * a, rstencily = Ly - (3.0 * a), lstencily = 3.0 * a;
    if (solvx < lstencilx) {
      v1x -= (v1x > rstencilx) ? Lx : 0; v2x -= (v2x > rstencilx) ? Lx : 0; v3x -= (v3x > rstencilx) ? Lx : 0;
    } else if (solvx > rstencilx) {
      v1x += (v1x < lstencilx) ? Lx : 0; v2x += (v2x < lstencilx) ? Lx : 0; v3x += (v3x < lstencilx) ? Lx : 0;
    }
    if (solvy < lstencily) {
      v1y -= (v1y > rstencily) ? Ly : 0; v2y -= (v2y > rstencily) ? Ly : 0; v3y -= (v3y > rstencily) ? Ly : 0;
    } else if (solvy > rstencily) {
      v1y += (v1y < lstencily) ? Ly : 0; v2y += (v2y < lstencily) ? Ly : 0; v3y += (v3y < lstencily) ? Ly : 0;
    }
    double w1x = v1x + sn.vx[p1] * (dtmd - rstep), w1y = v1y + sn.vy[p1] * (dtmd - rstep), w1z = v1z + sn.vz[p1] * (dtmd - rstep);
    double w2x = v2x + sn.vx[p2] * (dtmd - rstep), w2y = v2y + sn.vy[p2] * (dtmd - rstep), w2z = v2z + sn.vz[p2] * (dtmd - rstep);
    double w3x = v3x + sn.vx[p3] * (dtmd - rstep), w3y = v3y + sn.vy[p3] * (dtmd - rstep), w3z = v3z + sn.vz[p3] * (dtmd - rstep);
    double X[3], Xdt[3], t0[3], t1v[3];
    t0[0] = v2x - v1x; t0[1] = v2y - v1y; t0[2] = v2z - v1z;
    t1v[0] = v3x - v1x; t1v[1] = v3y - v1y; t1v[2] = v3z - v1z;
    cp(t0, t1v, X);
    t0[0] = w2x - w1x; t0[1] = w2y - w1y; t0[2] = w2z - w1z;
    t1v[0] = w3x - w1x; t1v[1] = w3y - w1y; t1v[2] = w3z - w1z;
    cp(t0, t1v, Xdt);
    double PSt0 = solvx - v1x, PSt1 = solvy - v1y, PSt2 = solvz - v1z;
    double PD0 = (solvx + VX * (dtmd - rstep)) - w1x;
    double PD1 = (solvy + VY * (dtmd - rstep)) - w1y;
    double PD2 = (solvz + VZ * (dtmd - rstep)) - w1z;
    bt = X[0] * PSt0 + X[1] * PSt1 + X[2] * PSt2;
    bdt = Xdt[0] * PD0 + Xdt[1] * PD1 + Xdt[2] * PD2;
    if ((indio == 1) && (bt < 0)) flg = 1;
    if ((indio == 0) && (bt > 0)) flg = 1;
    if (!((bt * bdt <= 0) && (flg == 0))) return false;
  }
  // crossing candidate: contact time from the cubic, barycentric test (:526-594)
  const double mvx1 = sn.vx[p1], mvy1 = sn.vy[p1], mvz1 = sn.vz[p1];
  const double mvx2 = sn.vx[p2], mvy2 = sn.vy[p2], mvz2 = sn.vz[p2];
  const double mvx3 = sn.vx[p3], mvy3 = sn.vy[p3], mvz3 = sn.vz[p3];
  double a10[3], a20[3], d1[3], d2[3], a1v[3], a2v[3], b1[3], b2[3], b3[3], d11[3], d22[3];
  a10[0] = v2x - v1x; a10[1] = v2y - v1y; a10[2] = v2z - v1z;
  a20[0] = v3x - v1x; a20[1] = v3y - v1y; a20[2] = v3z - v1z;
  d1[0] = mvx2 - mvx1; d1[1] = mvy2 - mvy1; d1[2] = mvz2 - mvz1;
  d2[0] = mvx3 - mvx1; d2[1] = mvy3 - mvy1; d2[2] = mvz3 - mvz1;
  a1v[0] = solvx - v1x; a1v[1] = solvy - v1y; a1v[2] = solvz - v1z;
  a2v[0] = VX - mvx1; a2v[1] = VY - mvy1; a2v[2] = VZ - mvz1;
  cp(a10, a20, b1);
  cp(a10, d2, d11);
  cp(d1, a20, d22);
  cp(d1, d2, b3);
  for (int k = 0; k < 3; ++k) b2[k] = d11[k] + d22[k];
  double a2b3 = a2v[0] * b3[0] + a2v[1] * b3[1] + a2v[2] * b3[2];
  double a1b3 = a1v[0] * b3[0] + a1v[1] * b3[1] + a1v[2] * b3[2];
  double a2b2 = a2v[0] * b2[0] + a2v[1] * b2[1] + a2v[2] * b2[2];
  double a1b2 = a1v[0] * b2[0] + a1v[1] * b2[1] + a1v[2] * b2[2];
  double a2b1 = a2v[0] * b1[0] + a2v[1] * b1[1] + a2v[2] * b1[2];
  double a1b1 = a1v[0] * b1[0] + a1v[1] * b1[1] + a1v[2] * b1[2];
  double tt = solve_p3_tt((a1b3 + a2b2) / a2b3, (a1b2 + a2b1) / a2b3, a1b1 / a2b3, dtmd);
  double PS2[3], pd[3];
  PS2[0] = (solvx + VX * tt) - (v1x + mvx1 * tt);
  PS2[1] = (solvy + VY * tt) - (v1y + mvy1 * tt);
  PS2[2] = (solvz + VZ * tt) - (v1z + mvz1 * tt);
  pd[0] = (solvx + VX * tt); pd[1] = (solvy + VY * tt); pd[2] = (solvz + VZ * tt);
  a10[0] = (v2x + mvx2 * tt) - (v1x + mvx1 * tt);
  a10[1] = (v2y + mvy2 * tt) - (v1y + mvy1 * tt);
  a10[2] = (v2z + mvz2 * tt) - (v1z + mvz1 * tt);
  a20[0] = (v3x + mvx3 * tt) - (v1x + mvx1 * tt);
  a20[1] = (v3y + mvy3 * tt) - (v1y + mvy1 * tt);
  a20[2] = (v3z + mvz3 * tt) - (v1z + mvz1 * tt);
  double pa1 = PS2[0] * a10[0] + PS2[1] * a10[1] + PS2[2] * a10[2];
  double pa2 = PS2[0] * a20[0] + PS2[1] * a20[1] + PS2[2] * a20[2];
  double a1a2 = a10[0] * a20[0] + a10[1] * a20[1] + a10[2] * a20[2];
  double a12 = a10[0] * a10[0] + a10[1] * a10[1] + a10[2] * a10[2];
  double a22 = a20[0] * a20[0] + a20[1] * a20[1] + a20[2] * a20[2];
  double den = (a12 * a22) - (a1a2 * a1a2);
  double eta = ((pa1 * a22) - (pa2 * a1a2)) / den;
  double zeta = ((pa2 * a12) - (pa1 * a1a2)) / den;
  if ((eta >= 0) && (zeta >= 0) && (eta + zeta <= 1) && (tt < (dtmd - rstep))) {
    fulldt += tt;
    double vd0 = (1.0 - eta - zeta) * mvx1 + eta * mvx2 + zeta * mvx3;
    double vd1 = (1.0 - eta - zeta) * mvy1 + eta * mvy2 + zeta * mvy3;
    double vd2 = (1.0 - eta - zeta) * mvz1 + eta * mvz2 + zeta * mvz3;
    VX = 2.0 * vd0 - VX; VY = 2.0 * vd1 - VY; VZ = 2.0 * vd2 - VZ;
    X_ = pd[0]; Y_ = pd[1]; Z_ = pd[2];
    return true;
  }
  return false;
}

// free flight, walls and wrap after the membrane (maincode.cpp:516-560)
__device__ __forceinline__ void wall_step(const DevParams& p, double dt, double& X, double& Y, double& Z, double& VX,
                                          double& VY, double& VZ) {
  // the particle has flown dt and lies beyond a wall
  const double ul = p.Lz, ll = 0;
  double A[3], B[3];
  const double wall = Z > ul ? ul : ll;
  A[0] = X - VX * dt; A[1] = Y - VY * dt; A[2] = Z - VZ * dt;
  double sp = (wall - A[2]) / (Z - A[2]);
  B[0] = A[0] + sp * (X - A[0]); B[1] = A[1] + sp * (Y - A[1]); B[2] = A[2] + sp * (Z - A[2]);
  double dist = sqrt(((B[0] - A[0]) * (B[0] - A[0])) + ((B[1] - A[1]) * (B[1] - A[1])) + ((B[2] - A[2]) * (B[2] - A[2])));
  double dtt = dist / sqrt((VX * VX) + (VY * VY) + (VZ * VZ));
  if (Z > ul) { VX = p.wallspeed; VY = 0; VZ = 0; }
  else { VX *= -1.0; VY *= -1.0; VZ *= -1.0; }
  X = B[0] + VX * (dt - dtt);
  Y = B[1] + VY * (dt - dtt);
  Z = B[2] + VZ * (dt - dtt);
}
__device__ __forceinline__ void finish_stream(const DevParams& p, double fullts, double& X, double& Y, double& Z,
                                              double& VX, double& VY, double& VZ) {
  const double dt = p.dtmd - fullts;
  X += VX * dt;
  Y += VY * dt;
  Z += VZ * dt;
  if (Z > p.Lz || Z < 0) wall_step(p, dt, X, Y, Z, VX, VY, VZ);
  X = bbound(X, p.Lx);
  Y = bbound(Y, p.Ly);
}
// the same in float (the FP32-bulk solvent away from the membrane)
__device__ __forceinline__ void wall_step_f(float wallspeed, float Lz, float dt, float& X, float& Y, float& Z,
                                            float& VX, float& VY, float& VZ) {
  const float wall = Z > Lz ? Lz : 0.0f;
  float ax = X - VX * dt, ay = Y - VY * dt, az = Z - VZ * dt;
  float sp = (wall - az) / (Z - az);
  float bx = ax + sp * (X - ax), by = ay + sp * (Y - ay), bz = az + sp * (Z - az);
  float dist = sqrtf((bx - ax) * (bx - ax) + (by - ay) * (by - ay) + (bz - az) * (bz - az));
  float dtt = dist / sqrtf(VX * VX + VY * VY + VZ * VZ);
  if (Z > Lz) { VX = wallspeed; VY = 0.0f; VZ = 0.0f; }
  else { VX = -VX; VY = -VY; VZ = -VZ; }
  X = bx + VX * (dt - dtt); Y = by + VY * (dt - dtt); Z = bz + VZ * (dt - dtt);
}

__device__ __forceinline__ bool in_stencil(const DevParams& p, double x, double y) {
  return (x < 3.0 * p.a) || (x > p.Lx - (3.0 * p.a)) || (y < 3.0 * p.a) || (y > p.Ly - (3.0 * p.a));
}

// A particle's state through a stretch, in the arithmetic of the solvent's
// precision R: double, or float for the FP32-bulk solvent, which is promoted to
// double for reflectionFed and rounded back after every step.
template <typename R>
struct Flight {
  R X, Y, Z, VX, VY, VZ;
};
template <typename R>
__device__ __forceinline__ int cell_at(const DevParams& p, R X, R Y, R Z) {
  const int fx = (int)floor(bbound(X, (R)p.Lx));
  const int fy = (int)floor(bbound(Y, (R)p.Ly));
  const int fz = (int)floor(Z + R(1));
  return cell_of(p, fx, fy, fz);
}
// one step of free flight
__device__ __forceinline__ void free_step(const DevParams& p, Flight<double>& q) {
  finish_stream(p, 0.0, q.X, q.Y, q.Z, q.VX, q.VY, q.VZ);
}
__device__ __forceinline__ void free_step(const DevParams& p, Flight<float>& q) {
  const float Lz = (float)p.Lz, dt = (float)p.dtmd;
  q.X = q.X + q.VX * dt; q.Y = q.Y + q.VY * dt; q.Z = q.Z + q.VZ * dt;
  if (q.Z > Lz || q.Z < 0.0f) wall_step_f((float)p.wallspeed, Lz, dt, q.X, q.Y, q.Z, q.VX, q.VY, q.VZ);
  q.X = bbound(q.X, (float)p.Lx);
  q.Y = bbound(q.Y, (float)p.Ly);
}
// the step of a particle that has spent fulldt of it at the membrane
template <typename R>
__device__ __forceinline__ void end_step(const DevParams& p, double fulldt, Flight<R>& q) {
  double X = q.X, Y = q.Y, Z = q.Z, VX = q.VX, VY = q.VY, VZ = q.VZ;
  finish_stream(p, fulldt, X, Y, Z, VX, VY, VZ);
  raise_health(p, solvent_bad(p, X, Y, Z, VX, VY, VZ), HEALTH_SOLVENT);
  q.X = (R)X; q.Y = (R)Y; q.Z = (R)Z; q.VX = (R)VX; q.VY = (R)VY; q.VZ = (R)VZ;
}
// the solvent's arrays
struct SolventArrays {
  double *x, *y, *z;
  SolVel* v;
  int* indio;
  float4 *pos, *vel;
};
inline __host__ __device__ SolventArrays arrays_of(const Solvent& s, const SolventF& f) {
  return SolventArrays{s.x, s.y, s.z, s.v, s.indio, f.pos, f.vel};
}
__device__ __forceinline__ int flight_load(const SolventArrays& s, int64_t i, Flight<double>& q) {
  const SolVel r = s.v[i];
  q = {s.x[i], s.y[i], s.z[i], r.vx, r.vy, r.vz};
  return s.indio[i];
}
__device__ __forceinline__ int flight_load(const SolventArrays& s, int64_t i, Flight<float>& q) {
  const float4 a = s.pos[i], b = s.vel[i];
  q = {a.x, a.y, a.z, b.x, b.y, b.z};
  return __float_as_int(a.w);
}
__device__ __forceinline__ void flight_store(const SolventArrays& s, int64_t i, const Flight<double>& q) {
  s.x[i] = q.X; s.y[i] = q.Y; s.z[i] = q.Z;
  s.v[i].vx = q.VX; s.v[i].vy = q.VY; s.v[i].vz = q.VZ;
}
__device__ __forceinline__ void flight_store(const SolventArrays& s, int64_t i, const Flight<float>& q) {
  s.pos[i] = make_float4(q.X, q.Y, q.Z, s.pos[i].w);
  s.vel[i] = make_float4(q.VX, q.VY, q.VZ, s.vel[i].w);
}

// ---- hand-off to the near-membrane kernels -------------------------------------------
// Particle i, in a listed cell from step k of the stretch on: into the bucket of
// that cell (rank lrank among the listed cells) when the list fits the kernels'
// capacity hcap and the bucket has room, else onto the queue.
struct HandOff {
  const int* lstart;
  const int* lrank;
  int* bcnt;
  int2* bucket;
  int* queue;
  unsigned char* qk;
  int* qn;
  int hcap;
};
inline __host__ __device__ HandOff hand_off_of(const Cells& c, const FastBufs& f, int par) {
  return HandOff{c.lstart, c.lrank, f.bcnt, f.bucket, f.queue, f.qk, f.qn + par, f.hcap};
}
__device__ __forceinline__ void enqueue(const HandOff& h, int i, int k) {
  const int q = atomicAdd(h.qn, 1);
  h.queue[q] = i;
  h.qk[q] = (unsigned char)k;
}
__device__ __forceinline__ void hand_off(const HandOff& h, int pid, int i, int k) {
  if (h.lstart[pid + 1] - h.lstart[pid] <= h.hcap) {
    const int a = h.lrank[pid];
    const int slot = atomicAdd(h.bcnt + a, 1);
    if (slot < kBucket) { h.bucket[(int64_t)a * kBucket + slot] = make_int2(i, k); return; }
  }
  enqueue(h, i, k);
}

// ---- the bulk of a stretch --------------------------------------------------------------
// Between two collisions a particle away from the membrane only flies, so one
// pass takes each particle through all H steps of the stretch: its state is
// read and written once instead of H times.  The arithmetic is the steps', one
// after the other.  A particle that a step finds in a listed cell is handed over
// at that step, with its state.  `cflag` tells per cell whether it is listed
// (1), and whether a particle in it that flies less than a cell may meet a
// listed cell, a side wall or the grid's edge (2): the others need no look at
// the cells on their way.  Bound by HBM: FP64 80 bytes a particle (the 32-byte
// record carries the index), FP32 48.
template <typename R>
__device__ __forceinline__ bool flies_free(const DevParams& p, const Flight<R>& q, unsigned char cf, int H) {
  // (a moving top wall gives its speed to what it reflects)
  const R reach = fmax(fmax(fabs(q.VX), fabs(q.VY)), fmax(fabs(q.VZ), fabs((R)p.wallspeed))) * (R)(H * p.dtmd);
  return !(cf & 2) && reach < R(0.99);
}
// through steps k .. H-1; returns H, or the step that finds it in a listed cell
// (pid)
__device__ __forceinline__ void fly_free(const DevParams& p, Flight<double>& q, int H) {
  double dx = q.VX * p.dtmd, dy = q.VY * p.dtmd, dz = q.VZ * p.dtmd;
  for (int k = 0; k < H; ++k) {
    q.X += dx; q.Y += dy; q.Z += dz;
    if (q.Z > p.Lz || q.Z < 0) {
      wall_step(p, p.dtmd, q.X, q.Y, q.Z, q.VX, q.VY, q.VZ);
      dx = q.VX * p.dtmd; dy = q.VY * p.dtmd; dz = q.VZ * p.dtmd;
    }
  }
}
__device__ __forceinline__ void fly_free(const DevParams& p, Flight<float>& q, int H) {
  const float Lz = (float)p.Lz, dt = (float)p.dtmd;
  float dx = q.VX * dt, dy = q.VY * dt, dz = q.VZ * dt;
  for (int k = 0; k < H; ++k) {
    q.X += dx; q.Y += dy; q.Z += dz;
    if (q.Z > Lz || q.Z < 0.0f) {
      wall_step_f((float)p.wallspeed, Lz, dt, q.X, q.Y, q.Z, q.VX, q.VY, q.VZ);
      dx = q.VX * dt; dy = q.VY * dt; dz = q.VZ * dt;
    }
  }
}
template <typename R>
__device__ __forceinline__ int fly(const DevParams& p, Flight<R>& q, const unsigned char* __restrict__ cflag, int H,
                                   int& pid) {
  pid = cell_at(p, q.X, q.Y, q.Z);
  unsigned char cf = __ldg(cflag + pid);
  if (flies_free(p, q, cf, H)) {
    fly_free(p, q, H);
    raise_health(p, solvent_bad(p, q.X, q.Y, q.Z, q.VX, q.VY, q.VZ), HEALTH_SOLVENT);
    return H;
  }
  for (int k = 0;;) {
    if (cf & 1) return k;
    free_step(p, q);
    raise_health(p, solvent_bad(p, q.X, q.Y, q.Z, q.VX, q.VY, q.VZ), HEALTH_SOLVENT);
    if (++k == H) return H;
    pid = cell_at(p, q.X, q.Y, q.Z);
    cf = __ldg(cflag + pid);
  }
}

__global__ void __launch_bounds__(256) k_stream_bulk(DevParams p, SolventArrays s, int64_t n,
                                                     const unsigned char* __restrict__ cflag, HandOff h, int H) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double X = s.x[i], Y = s.y[i], Z = s.z[i];
  const SolVel r = s.v[i];
  Flight<double> q{X, Y, Z, r.vx, r.vy, r.vz};
  int pid;
  const int k = fly(p, q, cflag, H, pid);
  if (k > 0) {
    s.x[i] = q.X; s.y[i] = q.Y; s.z[i] = q.Z;
    if (q.VX != r.vx || q.VY != r.vy || q.VZ != r.vz || r.vx != r.vx) {
      s.v[i].vx = q.VX; s.v[i].vy = q.VY; s.v[i].vz = q.VZ;
    }
  }
  if (k < H) hand_off(h, pid, (int)i, k);
}
// one particle of the FP32-bulk solvent, loaded as (a, b)
__device__ __forceinline__ void bulk_f_item(const DevParams& p, const SolventArrays& s,
                                            const unsigned char* __restrict__ cflag, const HandOff& h, int H, int64_t i,
                                            float4 a, float4 b) {
  Flight<float> q{a.x, a.y, a.z, b.x, b.y, b.z};
  int pid;
  const int k = fly(p, q, cflag, H, pid);
  if (k > 0) {
    s.pos[i] = make_float4(q.X, q.Y, q.Z, a.w);
    if (q.VX != b.x || q.VY != b.y || q.VZ != b.z || b.x != b.x) s.vel[i] = make_float4(q.VX, q.VY, q.VZ, b.w);
  }
  if (k < H) hand_off(h, pid, (int)i, k);
}
__global__ void __launch_bounds__(256) k_stream_bulk_f(DevParams p, SolventArrays s, int64_t n,
                                                       const unsigned char* __restrict__ cflag, HandOff h, int H) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) bulk_f_item(p, s, cflag, h, H, i, s.pos[i], s.vel[i]);
}

// ---- near the membrane ---------------------------------------------------------------------
// reflectionFed's crossing test on a record's precomputed normals (the use_pre
// case of tri_visit, Src/solfuncs.cpp:461-517): whether the full test can hit.
// (X, Y, Z): the particle; (U, V, W): where it would fly in this step
__device__ __forceinline__ bool tri_crossing(const TriPre& q, double X, double Y, double Z, double U, double V, double W,
                                             int indio) {
  double PSt0 = X - q.A1[0], PSt1 = Y - q.A1[1], PSt2 = Z - q.A1[2];
  double PD0 = U - q.A2[0];
  double PD1 = V - q.A2[1];
  double PD2 = W - q.A2[2];
  const double bt = q.X[0] * PSt0 + q.X[1] * PSt1 + q.X[2] * PSt2;
  const double bdt = q.Xdt[0] * PD0 + q.Xdt[1] * PD1 + q.Xdt[2] * PD2;
  int flg = 0;
  if ((indio == 1) && (bt < 0)) flg = 1;
  if ((indio == 0) && (bt > 0)) flg = 1;
  return (bt * bdt <= 0) && (flg == 0);
}

// one TriPre record through the read-only path as six 16-byte loads (the
// records are 96 bytes from a 256-byte aligned base)
__device__ __forceinline__ TriPre ldg_tri(const TriPre* __restrict__ q) {
  const double2* r = reinterpret_cast<const double2*>(q);
  const double2 a = __ldg(r), b = __ldg(r + 1), c = __ldg(r + 2), d = __ldg(r + 3), e = __ldg(r + 4),
                g = __ldg(r + 5);
  TriPre t;
  t.X[0] = a.x; t.X[1] = a.y; t.X[2] = b.x;
  t.Xdt[0] = b.y; t.Xdt[1] = c.x; t.Xdt[2] = c.y;
  t.A1[0] = d.x; t.A1[1] = d.y; t.A1[2] = e.x;
  t.A2[0] = e.y; t.A2[1] = g.x; t.A2[2] = g.y;
  return t;
}

// Inside the periodic stencil bands (3a from each side wall) reflectionFed
// shifts a corner that lies in the opposite band by a period (:471-493).  A
// triangle without such a corner gives what its record holds.  band_of: the
// bands a particle's corners would be shifted from, as tri_bands reports them.
__device__ __forceinline__ int band_of(const DevParams& p, double x, double y) {
  const double rx = p.Lx - (3.0 * p.a), ry = p.Ly - (3.0 * p.a), l = 3.0 * p.a;
  return (x < l ? BAND_HX : (x > rx ? BAND_LX : 0)) | (y < l ? BAND_HY : (y > ry ? BAND_LY : 0));
}

// The triangle walk of reflectionFed for one particle, by a whole warp:
// lanes run the crossing test on 32 list entries at a time, and every
// crossing candidate gets the full test (contact time, barycentric test) on
// its own lane, all from the same particle state.  The reference's loop
// changes the state only at a hit, so up to and including the first hit of
// the 32 these are exactly its tests: the lowest hit is applied and the walk
// resumes after it with the updated state -- the same sequence of states as
// the sequential loop.  L: the list's triangles, len of them; pre, bands: this
// step's records.
__device__ __forceinline__ void heavy_walk(const DevParams& p, const Snap& sn, const TriPre* __restrict__ pre,
                                           const unsigned char* __restrict__ bands, const int* __restrict__ L, int len,
                                           int lane, int indio, double& X, double& Y, double& Z, double& VX, double& VY,
                                           double& VZ, double& fulldt) {
  for (int cur = 0; cur < len;) {
    const int band = band_of(p, X, Y);
    const int e = cur + lane;
    double x = X, y = Y, z = Z, vx = VX, vy = VY, vz = VZ, fd = 0.0;
    bool hit = false;
    if (e < len) {
      const int jj = __ldg(L + e);
      const TriPre t = ldg_tri(pre + jj);
      const bool plain = !(__ldg(bands + jj) & band);
      if (!plain || tri_crossing(t, X, Y, Z, X + VX * p.dtmd, Y + VY * p.dtmd, Z + VZ * p.dtmd, indio))
        hit = tri_visit(p, sn, t, jj, x, y, z, vx, vy, vz, indio, fd, plain);
    }
    const unsigned hb = __ballot_sync(0xffffffffu, hit);
    if (hb == 0u) {
      cur += 32;
      continue;
    }
    const int src = __ffs(hb) - 1;
    X = __shfl_sync(0xffffffffu, x, src);
    Y = __shfl_sync(0xffffffffu, y, src);
    Z = __shfl_sync(0xffffffffu, z, src);
    VX = __shfl_sync(0xffffffffu, vx, src);
    VY = __shfl_sync(0xffffffffu, vy, src);
    VZ = __shfl_sync(0xffffffffu, vz, src);
    fulldt += __shfl_sync(0xffffffffu, fd, src);
    cur += src + 1;
  }
}

// what the near-membrane kernels read of one simulation
struct NearArgs {
  const int *lstart, *lidx, *acell;
  const int2* arng;
  const TriPre* pre;
  const unsigned char* bands;
  int64_t nt, nv;
  Snap snap;
  HandOff h;
};
inline __host__ __device__ NearArgs near_of(const DevParams& p, const Cells& c, const FastBufs& f, int par) {
  return NearArgs{c.lstart, c.lidx, c.acell, f.arng, f.pre, f.bands, p.nt, p.nv, f.snap, hand_off_of(c, f, par)};
}
__device__ __forceinline__ Snap near_snap(const NearArgs& a, int t) {
  Snap s = a.snap;
  const int64_t o = (int64_t)t * a.nv;
  s.x += o; s.y += o; s.z += o; s.vx += o; s.vy += o; s.vz += o;
  return s;
}

// The particles of one listed cell through the rest of the stretch, by W warps
// (reflectionFed, :400-598, then the walls and wrap).  Each thread holds the
// record of a list entry in registers and runs the crossing test on the cell's
// particles, whose states lie in shared memory.  Nothing is staged, and the particles' states
// stay here between the steps.  Then
//   FULL (long lists; about 0.4 candidates per particle and step, most of them
//   crossing the plane of a triangle elsewhere): every candidate gets the full
//   test by a thread of its own; a particle that hits something walks the list
//   as the reference does (heavy_walk).
//   otherwise (short lists, 0.6% of particles have a candidate): a particle with
//   a candidate goes onto the queue, for the rest of the stretch, so that the
//   full test's registers stay out of this kernel.
// A particle that leaves the cell goes onto the queue too.
constexpr int kCand = 128;
struct NearCell {
  double st[6][kBucket], to[3][kBucket];
  int id[kBucket], k0[kBucket], indio[kBucket], band[kBucket], hit[kBucket];
  unsigned cand[kCand];
  int nc, done;
  unsigned act, leave;
};
template <int W>
__device__ __forceinline__ void near_sync() {
  if (W == 1) __syncwarp();
  else __syncthreads();
}
template <typename R, int W, bool FULL>
__device__ __forceinline__ void near_cell(const DevParams& p, const SolventArrays& s, const NearArgs& A, int a, int n,
                                          int H, NearCell& S) {
  const int tid = W == 1 ? (threadIdx.x & 31) : threadIdx.x, lane = threadIdx.x & 31;
  constexpr int T = 32 * W;
  const int2 rg = __ldg(A.arng + a);
  const int l0 = rg.x, len = rg.y, home = __ldg(A.acell + a);
  // thread j < n looks after particle j
  Flight<R> q{};
  int me = -1, from = 0;
  if (tid < n) {
    const int2 b = A.h.bucket[(int64_t)a * kBucket + tid];
    me = b.x;
    from = b.y;
    S.indio[tid] = flight_load(s, me, q);
    S.id[tid] = me;
  }
  const int jj0 = tid < len ? __ldg(A.lidx + l0 + tid) : 0;
  TriPre next{};
  int nband = 0;
  if (FULL && tid < len) { next = ldg_tri(A.pre + jj0); nband = __ldg(A.bands + jj0); }
  bool here = me >= 0;
  for (int t = 0; t < H; ++t) {
    if (tid < 32) {
      const bool on = here && t >= from;
      if (on) {
        S.st[0][tid] = q.X; S.st[1][tid] = q.Y; S.st[2][tid] = q.Z;
        if (FULL) { S.st[3][tid] = q.VX; S.st[4][tid] = q.VY; S.st[5][tid] = q.VZ; S.hit[tid] = 0x7fffffff; }
        S.to[0][tid] = (double)q.X + (double)q.VX * p.dtmd;
        S.to[1][tid] = (double)q.Y + (double)q.VY * p.dtmd;
        S.to[2][tid] = (double)q.Z + (double)q.VZ * p.dtmd;
        S.band[tid] = band_of(p, q.X, q.Y);
      }
      const unsigned act = __ballot_sync(0xffffffffu, on), any = __ballot_sync(0xffffffffu, here);
      if (lane == 0) { S.act = act; S.leave = 0u; S.nc = 0; S.done = any == 0u; }
    }
    near_sync<W>();
    if (S.done) return;  // every particle has left
    const unsigned act = S.act;
    const TriPre* pre = A.pre + (int64_t)t * A.nt;
    const unsigned char* bands = A.bands + (int64_t)t * A.nt;
    for (int e = tid; e < len; e += T) {
      TriPre r;
      int rb;
      if (FULL && e == tid) {
        r = next;
        rb = nband;
        if (t + 1 < H) { next = ldg_tri(pre + A.nt + jj0); nband = __ldg(bands + A.nt + jj0); }
      } else {
        const int jj = e == tid ? jj0 : __ldg(A.lidx + l0 + e);
        r = ldg_tri(pre + jj);
        rb = __ldg(bands + jj);
      }
      for (unsigned todo = act; todo; todo &= todo - 1) {
        const int j = __ffs(todo) - 1;
        if ((rb & S.band[j]) || tri_crossing(r, S.st[0][j], S.st[1][j], S.st[2][j], S.to[0][j], S.to[1][j], S.to[2][j],
                                             S.indio[j])) {
          if (FULL) {
            const int c = atomicAdd(&S.nc, 1);
            if (c < kCand) S.cand[c] = (unsigned)e | ((unsigned)j << 16);
            else atomicMin(&S.hit[j], e);  // no room: the particle walks the list
          } else {
            atomicOr(&S.leave, 1u << j);
          }
        }
      }
    }
    near_sync<W>();
    if (FULL) {
      const int nc = min(S.nc, kCand);
      if (nc > 0) {
        const Snap sn = near_snap(A, t);
        for (int c = tid; c < nc; c += T) {
          const int e = (int)(S.cand[c] & 0xffffu), j = (int)(S.cand[c] >> 16);
          const int jj = __ldg(A.lidx + l0 + e);
          double x = S.st[0][j], y = S.st[1][j], z = S.st[2][j], vx = S.st[3][j], vy = S.st[4][j], vz = S.st[5][j], fd = 0.0;
          if (tri_visit(p, sn, ldg_tri(pre + jj), jj, x, y, z, vx, vy, vz, S.indio[j], fd,
                        !(__ldg(bands + jj) & S.band[j])))
            atomicMin(&S.hit[j], e);
        }
        near_sync<W>();
        // particles that hit something, a warp each
        for (int j = tid >> 5; j < n; j += W) {
          if (!((act >> j) & 1) || S.hit[j] == 0x7fffffff) continue;
          double x = S.st[0][j], y = S.st[1][j], z = S.st[2][j], vx = S.st[3][j], vy = S.st[4][j], vz = S.st[5][j], fd = 0.0;
          heavy_walk(p, sn, pre, bands, A.lidx + l0, len, lane, S.indio[j], x, y, z, vx, vy, vz, fd);
          if (lane == 0) {
            S.st[0][j] = x; S.st[1][j] = y; S.st[2][j] = z; S.st[3][j] = vx; S.st[4][j] = vy; S.st[5][j] = vz;
            S.to[0][j] = fd;
          }
        }
        near_sync<W>();
      }
    }
    if (here && t >= from) {
      if (!FULL && ((S.leave >> tid) & 1)) {
        flight_store(s, me, q);
        enqueue(A.h, me, t);
        here = false;
      } else {
        if (FULL && S.hit[tid] != 0x7fffffff) {
          double X = S.st[0][tid], Y = S.st[1][tid], Z = S.st[2][tid], VX = S.st[3][tid], VY = S.st[4][tid],
                 VZ = S.st[5][tid];
          finish_stream(p, S.to[0][tid], X, Y, Z, VX, VY, VZ);
          raise_health(p, solvent_bad(p, X, Y, Z, VX, VY, VZ), HEALTH_SOLVENT);
          q = {(R)X, (R)Y, (R)Z, (R)VX, (R)VY, (R)VZ};
        } else {
          end_step(p, 0.0, q);
        }
        if (t + 1 == H) {
          flight_store(s, me, q);
        } else if (cell_at(p, q.X, q.Y, q.Z) != home) {
          flight_store(s, me, q);
          enqueue(A.h, me, t + 1);
          here = false;
        }
      }
    }
    near_sync<W>();  // the shared state is written again
  }
}

// the cells with short lists: a warp each, four to a block.  64 registers:
// eight blocks (32 warps) per SM
template <typename R>
__device__ __forceinline__ void near_short_warp(const DevParams& p, const SolventArrays& s, const NearArgs& A, int a,
                                                int nact, int H, NearCell& S) {
  if (a >= nact) return;
  int n = 0;
  if ((threadIdx.x & 31) == 0) {
    n = A.h.bcnt[a];
    if (n) A.h.bcnt[a] = 0;  // for the next stretch
  }
  n = min(__shfl_sync(0xffffffffu, n, 0), kBucket);
  if (n) near_cell<R, 1, false>(p, s, A, a, n, H, S);
}
template <typename R>
__global__ void __launch_bounds__(32 * kShortWarps, kShortMinBlocks)
    k_near_short(DevParams p, SolventArrays s, NearArgs A, const int* __restrict__ nactp, int H) {
  __shared__ NearCell S[kShortWarps];
  const int w = (int)(threadIdx.x >> 5);
  near_short_warp<R>(p, s, A, (int)blockIdx.x * kShortWarps + w, *nactp, H, S[w]);
}
// the cells with long lists: kLongWarps warps each, longest list first
template <typename R>
__device__ __forceinline__ void near_long_block(const DevParams& p, const SolventArrays& s, const NearArgs& A, int b,
                                                const int* __restrict__ border, int nact, int H, NearCell& S) {
  if (b >= nact) return;
  const int a = border[b], n = min(A.h.bcnt[a], kBucket);
  __syncthreads();
  if (threadIdx.x == 0 && n) A.h.bcnt[a] = 0;
  if (n) near_cell<R, kLongWarps, true>(p, s, A, a, n, H, S);
}
template <typename R>
__global__ void __launch_bounds__(32 * kLongWarps, kLongMinBlocks)
    k_near_long(DevParams p, SolventArrays s, NearArgs A, const int* __restrict__ border, const int* __restrict__ nactp,
                int H) {
  __shared__ NearCell S;
  near_long_block<R>(p, s, A, (int)blockIdx.x, border, *nactp, H, S);
}

// The queue: particles that left their cell or (short lists) have a crossing
// candidate, of full buckets, and in lists longer than the capacity; warp gw
// of tw takes particles gw, gw + tw, ... through the rest of the stretch.
template <typename R>
__device__ __forceinline__ void queue_walk(const DevParams& p, const SolventArrays& s, const NearArgs& A,
                                           const unsigned char* __restrict__ cflag, int H, int64_t gw, int64_t tw) {
  const int lane = threadIdx.x & 31;
  const int nq = *A.h.qn;
  for (int64_t w = gw; w < nq; w += tw) {
    const int64_t i = A.h.queue[w];
    Flight<R> q;
    const int indio = flight_load(s, i, q);
    for (int t = A.h.qk[w]; t < H; ++t) {
      const int pid = cell_at(p, q.X, q.Y, q.Z);
      if (!(__ldg(cflag + pid) & 1)) {
        free_step(p, q);
        raise_health(p, solvent_bad(p, q.X, q.Y, q.Z, q.VX, q.VY, q.VZ), HEALTH_SOLVENT);
        continue;
      }
      const int l0 = __ldg(A.lstart + pid), len = __ldg(A.lstart + pid + 1) - l0;
      double x = q.X, y = q.Y, z = q.Z, vx = q.VX, vy = q.VY, vz = q.VZ, fd = 0.0;
      heavy_walk(p, near_snap(A, t), A.pre + (int64_t)t * A.nt, A.bands + (int64_t)t * A.nt, A.lidx + l0, len, lane,
                 indio, x, y, z, vx, vy, vz, fd);
      finish_stream(p, fd, x, y, z, vx, vy, vz);
      raise_health(p, solvent_bad(p, x, y, z, vx, vy, vz), HEALTH_SOLVENT);
      q = {(R)x, (R)y, (R)z, (R)vx, (R)vy, (R)vz};
    }
    if (lane == 0) flight_store(s, i, q);
  }
}
template <typename R>
__global__ void __launch_bounds__(256, 2) k_near_queue(DevParams p, SolventArrays s, NearArgs A,
                                                      const unsigned char* __restrict__ cflag, int H) {
  const int64_t tw = (int64_t)gridDim.x * (blockDim.x >> 5);
  const int64_t gw = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  queue_walk<R>(p, s, A, cflag, H, gw, tw);
}

}  // namespace irbc

// the membrane of a stretch of steps
#include "segment.cuh"

namespace irbc {

// ================================================================ launch ======
// the side stream's work: a captured graph gives it the side stream's high
// priority
bool is_membrane_kernel(const void* fn) { return fn == (const void*)k_membrane || fn == (const void*)k_tri_records; }

__global__ void k_rank_lengths(Cells c, int nact, int* len, int2* rng) {
  const int a = blockIdx.x * blockDim.x + threadIdx.x;
  if (a >= nact) return;
  const int cell = c.acell[a];
  const int l0 = c.lstart[cell];
  len[a] = c.lstart[cell + 1] - l0;
  rng[a] = make_int2(l0, c.lstart[cell + 1] - l0);
}
void launch_rank_lengths(const Cells& c, int* len, int2* rng, cudaStream_t st) {
  if (c.nact > 0) k_rank_lengths<<<nb(c.nact, 256), 256, 0, st>>>(c, c.nact, len, rng);
}

// snapshot and triangle records of the membrane as it is (irbc_stream), as
// step 0 of a stretch
__global__ void k_snap(DevParams p, Membrane m, FastBufs f) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= p.nv) return;
  const Snap sn = f.snap;
  const int q = f.pidx[i];
  sn.x[q] = m.x[i]; sn.y[q] = m.y[i]; sn.z[q] = m.z[i];
  sn.vx[q] = m.vx[i]; sn.vy[q] = m.vy[i]; sn.vz[q] = m.vz[i];
}
void fast_snap_prep(const DevParams& p, Membrane& m, FastBufs& f, cudaStream_t st) {
  k_snap<<<nb(p.nv, 128), 128, 0, st>>>(p, m, f);
  k_tri_records<<<nb(p.nt, 128), 128, 0, st>>>(p, f, 1);
}

// the near-membrane kernels of a stretch; returns the number launched
template <typename R>
static int launch_near(const DevParams& p, const Solvent& s, const SolventF& sf, const Cells& c, const FastBufs& f,
                       int H, cudaStream_t st) {
  const SolventArrays arr = arrays_of(s, sf);
  const NearArgs A = near_of(p, c, f, 0);
  int n = 1;
  if (f.bcap > 0) {
    if (short_lists(f.hcap))
      k_near_short<R><<<nb(f.bcap, kShortWarps), 32 * kShortWarps, 0, st>>>(p, arr, A, c.totals + 4, H);
    else
      k_near_long<R><<<(unsigned)f.bcap, 32 * kLongWarps, 0, st>>>(p, arr, A, f.border, c.totals + 4, H);
    ++n;
  }
  k_near_queue<R><<<kQueueBlocks, 256, 0, st>>>(p, arr, A, c.flag, H);
  return n;
}

int fast_stream(const DevParams& p, const Solvent& s, const SolventF* sf, const Cells& c, FastBufs& f, int H,
                cudaStream_t st, cudaEvent_t ev0, cudaEvent_t ev1, cudaEvent_t snap) {
  cudaMemsetAsync(f.qn, 0, sizeof(int), st);
  if (!s.n) return 0;
  const HandOff h = hand_off_of(c, f, 0);
  const SolventF none;
  const SolventArrays arr = arrays_of(s, sf ? *sf : none);
  if (ev0) cudaEventRecord(ev0, st);
  if (sf) k_stream_bulk_f<<<nb(s.n, 256), 256, 0, st>>>(p, arr, s.n, c.flag, h, H);
  else k_stream_bulk<<<nb(s.n, 256), 256, 0, st>>>(p, arr, s.n, c.flag, h, H);
  if (ev1) cudaEventRecord(ev1, st);
  if (snap) cudaStreamWaitEvent(st, snap, 0);
  return 1 + (sf ? launch_near<float>(p, s, *sf, c, f, H, st) : launch_near<double>(p, s, none, c, f, H, st));
}

}  // namespace irbc

// FP32-bulk solvent kernels share the device helpers above
#include "fp32.cuh"

// one launch per phase over a cohort of FP32 simulations
#include "multi.cuh"
