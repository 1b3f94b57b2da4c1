// cull.h -- which triangles of a list a particle can reach in a stretch of
// timesteps (k_near): plain C++ too, so that the bound is tested on the host.
#pragma once
#include "hd.h"

namespace irbc {

// per-triangle data of reflectionFed at rstep = 0 (Src/solfuncs.cpp:457-517)
struct TriPre {
  double X[3], Xdt[3], A1[3], A2[3];
};

// reflectionFed's crossing test on a record's precomputed normals (the use_pre
// case of tri_visit, Src/solfuncs.cpp:461-517): whether the full test can hit.
// (X, Y, Z): the particle; (U, V, W): where it would fly in this step
IRBC_HD bool tri_crossing(const TriPre& q, double X, double Y, double Z, double U, double V, double W, int indio) {
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

// What no step of a stretch can make a crossing candidate, found once per
// particle and stretch instead of in every step.  A candidate crosses the
// triangle's plane: b_t = X_t . (P_t - A_t) changes sign, X_t the normal and A_t
// the corner at step t, P_t the particle.  With the triangle's largest changes
// over the stretch, dX of the normal and dA of the corner, and the particle's
// path dP (cull_path),
//   |b_t - X_0 . (P - A_0)| <= dX (|P - A_0| + dP + dA) + |X_0| (dP + dA),
// so an entry whose plane is farther away needs no test.  About 5% of the
// 600-vertex mesh's entries and 10% of the discocyte's are left.  TriCull holds
// what that takes in float; m covers the rounding.  In units of 2^-24 of the
// normal's 1-norm, in a box whose longest side is L, it is at most L + 1 of the
// particle's and of the corner's coordinates in float, and with differences up
// to L another L each of the normal in float, the differences and the products
// and 2 L of the sums: 7 L + 2, and m is 8 (L + 16).  The FP32-bulk solvent is
// also rounded to float after every step, by up to 2^-24 of each coordinate and
// at a constant velocity always the same way, which lengthens the path: for the
// steps of a stretch (roundings) m is sqrt(3) (L + 1) larger each.  (Without that a
// stretch of 12 steps lost reflections in boxes longer than 128.  NaN and
// infinities fail the comparison and are kept.)  bands: of the triangle's corners
// in any of the steps.
struct TriCull {
  float X[3], nX, A[3], dX, dA, m;
  int bands;
};
IRBC_HD bool cull_keeps(const TriCull& c, float X, float Y, float Z, float dP, int band) {
  const float x = X - c.A[0], y = Y - c.A[1], z = Z - c.A[2];
  const float b = fabsf(c.X[0] * x + c.X[1] * y + c.X[2] * z);
  const float d = sqrtf(x * x + y * y + z * z), move = dP + c.dA;
  return (c.bands & band) || !(b > 1.0001f * (c.dX * (d + move) + c.nX * move) + c.m);
}
// The longest path of a particle with velocity (vx, vy, vz) in the `left` steps
// that a stretch still has: its speed, or the top wall's, which it gives to what
// it reflects
IRBC_HD float cull_path(double vx, double vy, double vz, double wallspeed, double dtmd, int left) {
  return (float)(fmax(sqrt(vx * vx + vy * vy + vz * vz), fabs(wallspeed)) * dtmd * left) * 1.0001f;
}
// a step's record against that of the first one
struct CullMove {
  double dX, dA;
  int bands;
};
IRBC_HD double norm3(double x, double y, double z) { return sqrt(x * x + y * y + z * z); }
IRBC_HD void cull_fold(CullMove& c, const TriPre& t0, const TriPre& t, int bands) {
  c.dX = fmax(c.dX, fmax(norm3(t.X[0] - t0.X[0], t.X[1] - t0.X[1], t.X[2] - t0.X[2]),
                         norm3(t.Xdt[0] - t0.X[0], t.Xdt[1] - t0.X[1], t.Xdt[2] - t0.X[2])));
  c.dA = fmax(c.dA, fmax(norm3(t.A1[0] - t0.A1[0], t.A1[1] - t0.A1[1], t.A1[2] - t0.A1[2]),
                         norm3(t.A2[0] - t0.A1[0], t.A2[1] - t0.A1[1], t.A2[2] - t0.A1[2])));
  // a record that is not finite stays in every test
  const double s = t.X[0] + t.X[1] + t.X[2] + t.Xdt[0] + t.Xdt[1] + t.Xdt[2] + t.A1[0] + t.A1[1] + t.A1[2] + t.A2[0] +
                   t.A2[1] + t.A2[2];
  if (!(fabs(s) <= 1.7976931348623157e308)) c.dX = c.dA = HUGE_VAL;
  c.bands |= bands;
}
// L: the box's longest side; roundings: see above
IRBC_HD TriCull cull_of(const TriPre& t0, const CullMove& c, double L, int roundings) {
  const double n1 = fabs(t0.X[0]) + fabs(t0.X[1]) + fabs(t0.X[2]) + c.dX;
  return TriCull{{(float)t0.X[0], (float)t0.X[1], (float)t0.X[2]},
                 (float)norm3(t0.X[0], t0.X[1], t0.X[2]) * 1.00001f,
                 {(float)t0.A1[0], (float)t0.A1[1], (float)t0.A1[2]},
                 (float)c.dX * 1.00001f,
                 (float)c.dA * 1.00001f,
                 (float)(n1 * ((L + 16.0) * (1.0 / 2097152.0) + 1.74 * (L + 1.0) * roundings * (1.0 / 16777216.0))),
                 c.bands};
}

}  // namespace irbc
