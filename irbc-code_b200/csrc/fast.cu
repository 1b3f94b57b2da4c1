// fast.cu -- the production step, a stretch of timesteps at a time: the bulk
// streaming of every particle, the near-membrane streaming of those in cells
// with triangles, and the membrane (segment.cuh) on a side stream beside the
// bulk.
//
// The membrane's and the streaming's single phases that the C ABI also offers are
// in kernels.cu.
#include <algorithm>
#include <cstdio>
#include "fast.h"
#include "fp32.h"

namespace irbc {

static inline unsigned nb(int64_t n, int t) { return (unsigned)((n + t - 1) / t); }

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

__device__ __forceinline__ double longest_side(const DevParams& p) { return fmax(p.Lx, fmax(p.Ly, p.Lz)); }
// A particle's state through a stretch, in the arithmetic of the solvent's
// precision R: double, or float for the FP32-bulk solvent, which is promoted to
// double for reflectionFed and rounded back after every step.
template <typename R>
struct Flight {
  R X, Y, Z, VX, VY, VZ;
};
// its cell; on: whether that is where it lies (positions off the grid count as
// cell 0, and positions beyond a side as their image's cell)
template <typename R>
__device__ __forceinline__ int cell_at(const DevParams& p, R X, R Y, R Z, bool& on) {
  const int fx = (int)floor(bbound(X, (R)p.Lx));
  const int fy = (int)floor(bbound(Y, (R)p.Ly));
  const int fz = (int)floor(Z + R(1));
  on = X >= R(0) && X <= (R)p.Lx && fx < p.nx && Y >= R(0) && Y <= (R)p.Ly && fy < p.ny && fz >= 0 && fz < p.nz;
  return cell_of(p, fx, fy, fz);
}
template <typename R>
__device__ __forceinline__ int cell_at(const DevParams& p, R X, R Y, R Z) {
  bool on;
  return cell_at(p, X, Y, Z, on);
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

// ---- hand-over to the near-membrane kernel -------------------------------------------
// particle i, in a listed cell from step k of the stretch on, onto the queue
struct NearQueue {
  int* i;
  unsigned char* k;
  int* n;  // their number
};
inline __host__ __device__ NearQueue queue_of(const FastBufs& f, int par) { return NearQueue{f.queue, f.qk, f.qn + par}; }
__device__ __forceinline__ void enqueue(const NearQueue& h, int i, int k) {
  const int q = atomicAdd(h.n, 1);
  h.i[q] = i;
  h.k[q] = (unsigned char)k;
}

// ---- the bulk of a stretch --------------------------------------------------------------
// Between two collisions a particle away from the membrane only flies, so one
// pass takes each particle through all H steps of the stretch: its state is
// read and written once instead of H times.  The arithmetic is the steps', one
// after the other.  A particle that a step finds in a listed cell is handed over
// at that step, with its state.  The cell flags (CF_*, launch_llist_flags) tell
// what a particle that flies less than a cell can meet from each cell: most need
// neither a look at the cells on their way nor wraps nor walls, and 36 additions
// are all the 12 steps cost.  Bound by HBM: FP64 80 bytes a particle (the
// 32-byte record carries the index), FP32 48.
template <typename R>
__device__ __forceinline__ bool flies_free(const DevParams& p, const Flight<R>& q, unsigned char cf, int H) {
  // (a moving top wall gives its speed to what it reflects)
  const R reach = fmax(fmax(fabs(q.VX), fabs(q.VY)), fmax(fabs(q.VZ), fabs((R)p.wallspeed))) * (R)(H * p.dtmd);
  // (above 2^16 a float's rounding after each step can carry 0.99 of a cell
  // beyond a whole one: 11 steps of 0.0899 are 11 of 12 / 128)
  const bool fine = sizeof(R) > sizeof(float) || longest_side(p) <= 65536.0;
  return !(cf & CF_MEETS) && reach < R(0.99) && fine;
}
__device__ __forceinline__ void wall_of(const DevParams& p, Flight<double>& q) {
  wall_step(p, p.dtmd, q.X, q.Y, q.Z, q.VX, q.VY, q.VZ);
}
__device__ __forceinline__ void wall_of(const DevParams& p, Flight<float>& q) {
  wall_step_f((float)p.wallspeed, (float)p.Lz, (float)p.dtmd, q.X, q.Y, q.Z, q.VX, q.VY, q.VZ);
}
// H steps away from every listed cell
template <typename R>
__device__ __forceinline__ void fly_free(const DevParams& p, Flight<R>& q, unsigned char cf, int H) {
  const R dt = (R)p.dtmd;
  R dx = q.VX * dt, dy = q.VY * dt, dz = q.VZ * dt;
  if (!(cf & (CF_SIDE | CF_WALL))) {
    for (int k = 0; k < H; ++k) { q.X += dx; q.Y += dy; q.Z += dz; }
    return;
  }
  const R Lx = (R)p.Lx, Ly = (R)p.Ly, Lz = (R)p.Lz;
  for (int k = 0; k < H; ++k) {
    q.X += dx; q.Y += dy; q.Z += dz;
    if (q.Z > Lz || q.Z < R(0)) {
      wall_of(p, q);
      dx = q.VX * dt; dy = q.VY * dt; dz = q.VZ * dt;
    }
    // (bbound: less than a period away)
    if (q.X > Lx) q.X -= Lx;
    if (q.X < R(0)) q.X += Lx;
    if (q.Y > Ly) q.Y -= Ly;
    if (q.Y < R(0)) q.Y += Ly;
  }
}
// through the stretch; returns H, or the step that finds the particle in a
// listed cell.  ONE: H is 1, where looking ahead saves nothing
template <typename R, bool ONE>
__device__ __forceinline__ int fly(const DevParams& p, Flight<R>& q, const unsigned char* __restrict__ cflag, int H) {
  if (ONE) {
    if (__ldg(cflag + cell_at(p, q.X, q.Y, q.Z)) & CF_LISTED) return 0;
    free_step(p, q);
    raise_health(p, solvent_bad(p, q.X, q.Y, q.Z, q.VX, q.VY, q.VZ), HEALTH_SOLVENT);
    return 1;
  }
  bool on;
  unsigned char cf = __ldg(cflag + cell_at(p, q.X, q.Y, q.Z, on));
  if (on && flies_free(p, q, cf, H)) {
    fly_free(p, q, cf, H);
    raise_health(p, solvent_bad(p, q.X, q.Y, q.Z, q.VX, q.VY, q.VZ), HEALTH_SOLVENT);
    return H;
  }
  for (int k = 0;;) {
    if (cf & CF_LISTED) return k;
    free_step(p, q);
    raise_health(p, solvent_bad(p, q.X, q.Y, q.Z, q.VX, q.VY, q.VZ), HEALTH_SOLVENT);
    if (++k == H) return H;
    cf = __ldg(cflag + cell_at(p, q.X, q.Y, q.Z));
  }
}

// The blocks an SM holds bound how many loads are in flight.  One step of 20 M
// particles: FP64 64 registers (4 blocks) 299 us, 40 (6 blocks) 264, with ONE 248;
// FP32 55 registers 246, 32 (8 blocks) 172, with ONE 164.  A stretch's kernel is the
// faster for it too (12 steps 328 and 280, 266 and 196), but so many blocks keep
// the membrane's from starting: 780 steps of 5.2 M particles 62.6 and 62.8 ms.
template <bool ONE>
__global__ void __launch_bounds__(256, ONE ? 6 : 4) k_stream_bulk(DevParams p, SolventArrays s, int64_t n,
                                                        const unsigned char* __restrict__ cflag, NearQueue h, int H) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double X = s.x[i], Y = s.y[i], Z = s.z[i];
  const SolVel r = s.v[i];
  Flight<double> q{X, Y, Z, r.vx, r.vy, r.vz};
  const int k = fly<double, ONE>(p, q, cflag, H);
  if (k > 0) {
    s.x[i] = q.X; s.y[i] = q.Y; s.z[i] = q.Z;
    if (q.VX != r.vx || q.VY != r.vy || q.VZ != r.vz || r.vx != r.vx) {
      s.v[i].vx = q.VX; s.v[i].vy = q.VY; s.v[i].vz = q.VZ;
    }
  }
  if (k < H) enqueue(h, (int)i, k);
}
// one particle of the FP32-bulk solvent, loaded as (a, b)
template <bool ONE>
__device__ __forceinline__ void bulk_f_item(const DevParams& p, const SolventArrays& s,
                                            const unsigned char* __restrict__ cflag, const NearQueue& h, int H, int64_t i,
                                            float4 a, float4 b) {
  Flight<float> q{a.x, a.y, a.z, b.x, b.y, b.z};
  const int k = fly<float, ONE>(p, q, cflag, H);
  if (k > 0) {
    s.pos[i] = make_float4(q.X, q.Y, q.Z, a.w);
    if (q.VX != b.x || q.VY != b.y || q.VZ != b.z || b.x != b.x) s.vel[i] = make_float4(q.VX, q.VY, q.VZ, b.w);
  }
  if (k < H) enqueue(h, (int)i, k);
}
template <bool ONE>
__global__ void __launch_bounds__(256, ONE ? 8 : 4) k_stream_bulk_f(DevParams p, SolventArrays s, int64_t n,
                                                          const unsigned char* __restrict__ cflag, NearQueue h, int H) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) bulk_f_item<ONE>(p, s, cflag, h, H, i, s.pos[i], s.vel[i]);
}

// ---- near the membrane ---------------------------------------------------------------------
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
// bands a particle's corners would be shifted from, as the records' bands
// (records_block) report them.
__device__ __forceinline__ int band_of(const DevParams& p, double x, double y) {
  const double rx = p.Lx - (3.0 * p.a), ry = p.Ly - (3.0 * p.a), l = 3.0 * p.a;
  return (x < l ? BAND_HX : (x > rx ? BAND_LX : 0)) | (y < l ? BAND_HY : (y > ry ? BAND_LY : 0));
}

__device__ __forceinline__ TriCull ldg_cull(const float4* __restrict__ r) {
  const float4 a = __ldg(r), b = __ldg(r + 1), c = __ldg(r + 2);
  return TriCull{{a.x, a.y, a.z}, a.w, {b.x, b.y, b.z}, b.w, c.x, c.y, __float_as_int(c.z)};
}
__device__ __forceinline__ void cull_store(const DevParams& p, float4* to, const TriPre& t0, const CullMove& mv) {
  // (tree_sums: the FP32-bulk solvent)
  const TriCull c = cull_of(t0, mv, longest_side(p), p.tree_sums ? kSegMax : 0);
  to[0] = make_float4(c.X[0], c.X[1], c.X[2], c.nX);
  to[1] = make_float4(c.A[0], c.A[1], c.A[2], c.dX);
  to[2] = make_float4(c.dA, c.m, __int_as_float(c.bands), 0.0f);
}

// what the near-membrane kernel reads of one simulation
struct NearArgs {
  const int *lstart, *lidx;
  const unsigned char *flag, *bands;
  const TriPre* pre;
  const float4* cull;
  int64_t nt, nv;
  Snap snap;
  NearQueue q;
  int first;   // the part's first step
  int* taken;  // particles taken from the queue
};
// part: of a stretch in two parts (k_near runs once for each)
inline __host__ __device__ NearArgs near_of(const DevParams& p, const Cells& c, const FastBufs& f, int par, int first,
                                            int part) {
  return NearArgs{c.lstart, c.lidx, c.flag, f.bands, f.pre, f.cull + (int64_t)part * 3 * p.nt, p.nt, p.nv, f.snap,
                  queue_of(f, par), first, f.qn + 4 - 2 * part + par};
}
__device__ __forceinline__ Snap near_snap(const NearArgs& a, int t) {
  Snap s = a.snap;
  const int64_t o = (int64_t)t * a.nv;
  s.x += o; s.y += o; s.z += o; s.vx += o; s.vy += o; s.vz += o;
  return s;
}

// reflectionFed's test of entry e (triangle jj) at step t for a particle:
// whether it hits; then the state after it and the time fd to it
__device__ __forceinline__ bool near_hit(const DevParams& p, const NearArgs& A, int t, int jj, int band, int indio,
                                         double& x, double& y, double& z, double& vx, double& vy, double& vz,
                                         double& fd) {
  const int64_t at = (int64_t)t * A.nt + jj;
  const TriPre r = ldg_tri(A.pre + at);
  const bool plain = !(__ldg(A.bands + at) & band);
  if (plain && !tri_crossing(r, x, y, z, x + vx * p.dtmd, y + vy * p.dtmd, z + vz * p.dtmd, indio)) return false;
  return tri_visit(p, near_snap(A, t), r, jj, x, y, z, vx, vy, vz, indio, fd, plain);
}

// The triangle walk of reflectionFed for one particle, by G lanes (mask): the
// lanes test G list entries at a time, all from the same particle state.  The
// reference's loop changes the state only at a hit, so up to and including the
// first hit of the G these are exactly its tests: the lowest hit is applied and
// the walk resumes after it with the updated state -- the same sequence of
// states as the sequential loop.  From entry cur on.
template <int G>
__device__ void near_walk(const DevParams& p, const NearArgs& A, int t, int l0, int cur, int len, int g, unsigned mask,
                          int indio, double& X, double& Y, double& Z, double& VX, double& VY, double& VZ,
                          double& fulldt) {
  while (cur < len) {
    double x = X, y = Y, z = Z, vx = VX, vy = VY, vz = VZ, fd = 0.0;
    const bool hit = cur + g < len && near_hit(p, A, t, __ldg(A.lidx + l0 + cur + g), band_of(p, X, Y), indio, x, y, z,
                                               vx, vy, vz, fd);
    const unsigned hb = __ballot_sync(mask, hit) & mask;
    if (hb == 0u) {
      cur += G;
      continue;
    }
    const int src = __ffs(hb) - 1;
    X = __shfl_sync(mask, x, src);
    Y = __shfl_sync(mask, y, src);
    Z = __shfl_sync(mask, z, src);
    VX = __shfl_sync(mask, vx, src);
    VY = __shfl_sync(mask, vy, src);
    VZ = __shfl_sync(mask, vz, src);
    fulldt += __shfl_sync(mask, fd, src);
    cur += (src & (G - 1)) + 1;
  }
}

// One particle near the membrane from step `from` to the end of the stretch
// (reflectionFed, :400-598, then the walls and wrap), by G lanes (g of mask) that
// all keep its state.  On entering a cell the lanes go through its list once and
// keep the entries that the cull leaves (kept: room for KEEP of them); each step
// then tests those, a lane each, all from the same state.  The reference's loop
// changes the state only at a hit, so the lowest entry that hits is its first
// one: it is applied, the list is culled again with the new velocity, and the
// entries after it are tested from there.  ONE: a stretch of one step with short
// lists, where the cull costs what it saves: the list is walked as it is.
template <typename R, int G, int KEEP, bool ONE>
__device__ __forceinline__ void near_particle(const DevParams& p, const SolventArrays& s, const NearArgs& A, int H,
                                              int64_t i, int from, int g, unsigned mask, unsigned short* kept) {
  Flight<R> q;
  const int indio = flight_load(s, i, q);
  int cell = -1, l0 = 0, len = 0, nk = 0, mine = 0;  // mine: this lane's first kept triangle
  for (int t = from; t < H; ++t) {
    // the record of the first kept triangle, wanted if the cell is still the same
    bool early = cell >= 0 && g < nk;
    TriPre first{};
    int fband = 0;
    if (early) {
      const int64_t at = (int64_t)t * A.nt + mine;
      first = ldg_tri(A.pre + at);
      fband = __ldg(A.bands + at);
    }
    bool on;
    const int pid = cell_at(p, q.X, q.Y, q.Z, on);
    if (!(__ldg(A.flag + pid) & CF_LISTED)) {
      free_step(p, q);
      raise_health(p, solvent_bad(p, q.X, q.Y, q.Z, q.VX, q.VY, q.VZ), HEALTH_SOLVENT);
      cell = -1;
      continue;
    }
    double x = q.X, y = q.Y, z = q.Z, vx = q.VX, vy = q.VY, vz = q.VZ, fd = 0.0;
    bool fresh = pid != cell;  // the list is to be culled
    if (fresh) {
      cell = on ? pid : -1;
      l0 = __ldg(A.lstart + pid);
      len = __ldg(A.lstart + pid + 1) - l0;
    }
    if (ONE) near_walk<G>(p, A, t, l0, 0, len, g, mask, indio, x, y, z, vx, vy, vz, fd);
    for (int after = -1; !ONE;) {  // the last entry that hit in this step
      const int band = band_of(p, x, y);
      if (fresh) {
        nk = 0;
        // (a band ends inside a cell only in a box that is no whole number of
        // cells; a wrap ends in another cell, except in a box of one)
        float dP = cull_path(vx, vy, vz, p.wallspeed, p.dtmd, H - t);
        if (p.nx < 2 || p.ny < 2) dP = __int_as_float(0x7f800000);
        const int wide = band | band_of(p, x - dP, y - dP) | band_of(p, x + dP, y + dP);
        constexpr int U = 4;  // entries in flight per lane
        for (int e0 = 0; e0 < len; e0 += U * G) {
          int jj[U];
#pragma unroll
          for (int u = 0; u < U; ++u) jj[u] = e0 + u * G + g < len ? __ldg(A.lidx + l0 + e0 + u * G + g) : -1;
          TriCull c[U];
#pragma unroll
          for (int u = 0; u < U; ++u) c[u] = ldg_cull(A.cull + 3 * (int64_t)max(jj[u], 0));
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const bool keep = jj[u] >= 0 && cull_keeps(c[u], (float)x, (float)y, (float)z, dP, wide);
            const unsigned kb = (__ballot_sync(mask, keep) & mask) >> (threadIdx.x & 31 & ~(G - 1));
            const int at = nk + __popc(kb & ((1u << g) - 1u));
            if (keep && at < KEEP) kept[at] = (unsigned short)(e0 + u * G + g);
            nk += __popc(kb);
          }
        }
        if (len > 65535) nk = KEEP + 1;
        __syncwarp(mask);
        if (g < min(nk, KEEP)) mine = __ldg(A.lidx + l0 + kept[g]);
        early = false;
        fresh = false;
      }
      if (nk > KEEP) {  // more than there is room for: the whole list
        near_walk<G>(p, A, t, l0, after + 1, len, g, mask, indio, x, y, z, vx, vy, vz, fd);
        break;
      }
      const double U = x + vx * p.dtmd, V = y + vy * p.dtmd, W = z + vz * p.dtmd;
      double hx = x, hy = y, hz = z, hvx = vx, hvy = vy, hvz = vz, hfd = 0.0;
      int hit = 0x7fffffff;
      for (int u = g; u < nk && hit == 0x7fffffff; u += G) {
        const int e = kept[u];
        if (e <= after) continue;
        const int jj = u == g ? mine : __ldg(A.lidx + l0 + e);
        TriPre r = first;
        int rb = fband;
        if (u != g || !early) {
          const int64_t at = (int64_t)t * A.nt + jj;
          r = ldg_tri(A.pre + at);
          rb = __ldg(A.bands + at);
        }
        const bool plain = !(rb & band);
        if (plain && !tri_crossing(r, x, y, z, U, V, W, indio)) continue;
        if (tri_visit(p, near_snap(A, t), r, jj, hx, hy, hz, hvx, hvy, hvz, indio, hfd, plain)) hit = e;
      }
      const unsigned hb = __ballot_sync(mask, hit != 0x7fffffff) & mask;
      if (hb == 0u) break;
      const int lowest = (int)__reduce_min_sync(mask, (unsigned)hit);
      const int src = __ffs(__ballot_sync(mask, hit == lowest) & mask) - 1;
      x = __shfl_sync(mask, hx, src);
      y = __shfl_sync(mask, hy, src);
      z = __shfl_sync(mask, hz, src);
      vx = __shfl_sync(mask, hvx, src);
      vy = __shfl_sync(mask, hvy, src);
      vz = __shfl_sync(mask, hvz, src);
      fd += __shfl_sync(mask, hfd, src);
      after = lowest;
      fresh = true;
    }
    finish_stream(p, fd, x, y, z, vx, vy, vz);
    raise_health(p, solvent_bad(p, x, y, z, vx, vy, vz), HEALTH_SOLVENT);
    q = {(R)x, (R)y, (R)z, (R)vx, (R)vy, (R)vz};
  }
  if (g == 0) flight_store(s, i, q);
}
// the queue's particles through the steps before H, each by the next group of G
// lanes that is free; ONE: by block bid of nb in turns, as their work differs
// little and is short against the counter's latency
template <typename R, int G, int KEEP, bool ONE>
__device__ __forceinline__ void near_groups(const DevParams& p, const SolventArrays& s, const NearArgs& A, int H,
                                            unsigned short* kept, int bid, int nb) {
  const int lane = threadIdx.x & 31, g = lane & (G - 1), lead = lane & ~(G - 1);
  const unsigned mask = G == 32 ? 0xffffffffu : ((1u << G) - 1u) << lead;
  const int nq = *A.q.n;
  if (ONE) {
    for (int w = bid * (kNearT / G) + threadIdx.x / G; w < nq; w += nb * (kNearT / G)) {
      near_particle<R, G, KEEP, true>(p, s, A, 1, A.q.i[w], 0, g, mask, kept);
      __syncwarp(mask);
    }
    return;
  }
  while (true) {
    int w = 0;
    if (g == 0) w = atomicAdd(A.taken, 1);
    w = __shfl_sync(mask, w, lead);
    if (w >= nq) break;
    const int from = max((int)A.q.k[w], A.first);
    if (from >= H) continue;
    near_particle<R, G, KEEP, false>(p, s, A, H, A.q.i[w], from, g, mask, kept);
    __syncwarp(mask);
  }
}
template <typename R, int G, int KEEP, bool ONE>
__global__ void __launch_bounds__(kNearT, kNearMinBlocks) k_near(DevParams p, SolventArrays s, NearArgs A, int H) {
  __shared__ unsigned short kept[kNearT / G][KEEP];
  near_groups<R, G, KEEP, ONE>(p, s, A, H, kept[threadIdx.x / G], blockIdx.x, gridDim.x);
}
template <typename R>
static void launch_near(const DevParams& p, const SolventArrays& s, const NearArgs& A, bool few, bool one, int H,
                        cudaStream_t st) {
  const auto k = !few ? k_near<R, kLongG, kLongKeep, false>
                      : (one ? k_near<R, kShortGOne, kShortKeep, true> : k_near<R, kShortG, kShortKeep, false>);
  k<<<kNearBlocks, kNearT, 0, st>>>(p, s, A, H);
}

}  // namespace irbc

// the membrane of a stretch of steps
#include "segment.cuh"

namespace irbc {

// ================================================================ launch ======
// the side stream's work: a captured graph gives it the side stream's high
// priority
bool is_membrane_kernel(const void* fn) {
  for (const void* k : {(const void*)k_membrane, (const void*)k_wide_first, (const void*)k_wide_tri,
                        (const void*)k_wide_terms, (const void*)k_wide_gather})
    if (fn == k) return true;
  return false;
}

// snapshot of the membrane as it is (irbc_stream), as step 0 of a stretch
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
}

void launch_records(const DevParams& p, const FastBufs& f, int s0, int s1, int part, cudaStream_t st) {
  k_tri_records<<<nb(p.nt, kRecordTris), kRecordT, 0, st>>>(p, f, s0, s1, part);
}

int fast_stream(const DevParams& p, const Solvent& s, const SolventF* sf, const Cells& c, FastBufs& f, int H,
                cudaStream_t st, cudaEvent_t ev0, cudaEvent_t ev1, cudaEvent_t snap, int first, cudaEvent_t snap1, bool recorded) {
  cudaMemsetAsync(f.qn, 0, 8 * sizeof(int), st);
  if (!s.n) return 0;
  const NearQueue h = queue_of(f, 0);
  const SolventF none;
  const SolventArrays arr = arrays_of(s, sf ? *sf : none);
  if (ev0) cudaEventRecord(ev0, st);
  const auto bulk = sf ? (H == 1 ? k_stream_bulk_f<true> : k_stream_bulk_f<false>)
                       : (H == 1 ? k_stream_bulk<true> : k_stream_bulk<false>);
  bulk<<<nb(s.n, 256), 256, 0, st>>>(p, arr, s.n, c.flag, h, H);
  if (ev1) cudaEventRecord(ev1, st);
  const bool few = short_lists(f.lmax);
  const int parts = first > 0 ? 2 : 1;
  for (int part = 0; part < parts; ++part) {
    const int s0 = part ? first : 0, s1 = part + 1 < parts ? first : H;
    const cudaEvent_t ready = part + 1 < parts ? snap1 : snap;
    if (ready) cudaStreamWaitEvent(st, ready, 0);
    if (!recorded) launch_records(p, f, s0, s1, part, st);
    const NearArgs A = near_of(p, c, f, 0, s0, part);
    if (sf) launch_near<float>(p, arr, A, few, H == 1, s1, st);
    else launch_near<double>(p, arr, A, few, H == 1, s1, st);
  }
  return 1 + (recorded ? 1 : 2) * parts;
}

}  // namespace irbc

// FP32-bulk solvent kernels share the device helpers above
#include "fp32.cuh"

// one launch per phase over a cohort of FP32 simulations
#include "multi.cuh"
