"""The near-membrane streaming tests only the triangles that the cull
(csrc/cull.h) leaves a particle for the rest of its stretch.  Here the header
itself is compiled for the host and every step of a stretch is tested in the
way k_near does (tri_crossing on the step's record, the state rounded to the
solvent's precision after every step): no triangle that is a crossing candidate
in any step may have been left out."""
import ctypes as C
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

HARNESS = r"""
#include <algorithm>
#include <random>
#include "cull.h"
using namespace irbc;
template <typename R>
static int run(int roundings, double L, int H, int n, unsigned seed, int* candidates) {
  std::mt19937_64 g(seed);
  std::uniform_real_distribution<double> U(0.0, 1.0);
  const double dt = 0.002;
  int missed = 0, cand = 0;
  for (int c = 0; c < n; ++c) {
    // a triangle at the far end of the box, at rest in half of the cases
    const bool axis = U(g) < 0.5, rest = U(g) < 0.5;
    double A[3], N[3], W[3], D[3];
    for (int k = 0; k < 3; ++k) {
      A[k] = k == 0 ? L - 4.0 * U(g) : 2.0 + (L - 4.0) * U(g);
      N[k] = axis ? (k == 0 ? 1.0 : 0.0) : 2.0 * U(g) - 1.0;
      W[k] = rest ? 0.0 : 0.3 * (2.0 * U(g) - 1.0);
      D[k] = rest ? 0.0 : 1e-3 * (2.0 * U(g) - 1.0);
    }
    const double size = std::pow(10.0, -2.0 + 2.0 * U(g));
    std::vector<TriPre> rec(H);
    for (int t = 0; t < H; ++t)
      for (int k = 0; k < 3; ++k) {
        rec[t].X[k] = size * (N[k] + D[k] * t);
        rec[t].Xdt[k] = size * (N[k] + D[k] * (t + 1));
        rec[t].A1[k] = A[k] + W[k] * dt * t;
        rec[t].A2[k] = A[k] + W[k] * dt * (t + 1);
      }
    CullMove mv{0.0, 0.0, 0};
    for (int t = 0; t < H; ++t) cull_fold(mv, rec[0], rec[t], 0);
    const TriCull cl = cull_of(rec[0], mv, L, roundings);
    // a particle flying at the plane, its path a little longer or shorter than
    // the way to it; with v dt just above a half unit in the last place of x
    // each rounding to float lengthens it
    double v[3], x[3], nn = 0.0;
    const double ulp = std::ldexp(1.0, std::ilogb(A[0]) - 23);
    const double sx = N[0] > 0 ? 1.0 : -1.0;
    v[0] = -sx * (double)(float)((std::floor(400.0 * U(g)) + 0.501 + 0.02 * U(g)) * ulp / dt);
    for (int k = 1; k < 3; ++k) v[k] = axis ? 0.0 : (double)(float)(2.0 * (2.0 * U(g) - 1.0));
    for (int k = 0; k < 3; ++k) nn += N[k] * N[k];
    double way = 0.0;  // towards the plane in H steps
    for (int k = 0; k < 3; ++k) way -= N[k] * (v[k] - W[k]) * dt * H;
    way += (U(g) * 2.0 - 0.5) * H * 0.5 * ulp * std::fabs(N[0]);
    for (int k = 0; k < 3; ++k) x[k] = (double)(R)(A[k] + N[k] * way / nn);
    const double x0[3] = {x[0], x[1], x[2]};
    const float dP = cull_path(v[0], v[1], v[2], 0.1, dt, H);
    const bool kept = cull_keeps(cl, (float)x0[0], (float)x0[1], (float)x0[2], dP, 0);
    bool crosses = false;
    for (int t = 0; t < H; ++t) {
      const double u[3] = {x[0] + v[0] * dt, x[1] + v[1] * dt, x[2] + v[2] * dt};
      crosses = crosses || tri_crossing(rec[t], x[0], x[1], x[2], u[0], u[1], u[2], 1);
      for (int k = 0; k < 3; ++k) x[k] = (double)(R)u[k];
    }
    cand += crosses;
    missed += crosses && !kept;
  }
  *candidates = cand;
  return missed;
}
extern "C" int misses(int single, int rounding, double L, int H, int n, unsigned seed, int* candidates) {
  // (sixteen steps, the most a stretch has)
  if (!single) return run<double>(0, L, H, n, seed, candidates);
  return run<float>(rounding ? 16 : 0, L, H, n, seed, candidates);
}
"""


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    d = tmp_path_factory.mktemp("cull")
    src, so = str(d / "h.cpp"), str(d / "h.so")
    with open(src, "w") as f:
        f.write("#include <vector>\n" + HARNESS)
    subprocess.run([os.environ.get("IRBC_CXX", "g++"), "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC",
                    "-I" + os.path.join(ROOT, "irbc-code_b200", "csrc"), src, "-o", so], check=True)
    lib = C.CDLL(so)
    lib.misses.argtypes = [C.c_int, C.c_int, C.c_double, C.c_int, C.c_int, C.c_uint, C.POINTER(C.c_int)]
    return lib


# boxes below, at and just above a power of two; stretches of one step, of a
# part, and the longest
@pytest.mark.parametrize("L", [20.0, 33.0, 64.0, 130.0, 146.0, 260.0, 1030.0])
@pytest.mark.parametrize("steps", [1, 7, 12, 16])
@pytest.mark.parametrize("single", [0, 1])
def test_no_crossing_candidate_is_culled(harness, L, steps, single):
    cand = C.c_int(0)
    assert harness.misses(single, 1, L, steps, 20000, 7, C.byref(cand)) == 0
    assert cand.value > 4000


def test_the_paths_tried_reach_the_rounding(harness):
    """Without its term for the rounding after every step the bound leaves
    candidates out, so the paths above are sharp enough to see it."""
    cand = C.c_int(0)
    assert harness.misses(1, 0, 260.0, 16, 20000, 7, C.byref(cand)) > 0
    assert harness.misses(1, 0, 130.0, 12, 20000, 7, C.byref(cand)) > 0
