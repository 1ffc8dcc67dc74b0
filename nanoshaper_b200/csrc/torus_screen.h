// Single-precision screen of torus candidates: whether a ray can hit the part of an edge patch that
// its clipping sphere and its plane pair leave.  About 11 % of the (ray, patch) candidates do (a ray
// through the clipping sphere mostly passes beside the patch's wedge); the screen keeps 17 %, and
// only those go to the double-precision quartic.
//
// A hit is accepted where three tests hold: inside the clipping sphere, on the allowed side of the
// planes, and at a root of the quartic.  The screen drops a candidate when the first two leave no
// point of the ray, or when the torus surface stays away from what they leave.  Along the ray the
// distance to the torus' circle changes at most as fast as the ray parameter, so a distance beyond
// the half length of a piece at its middle clears the piece.  The first test's slack covers the
// rounding of FP32; the second one's, 0.5 % of the patch's size (about 0.025 A), covers the root
// error of the reference's quartic solver as well, which is up to 3e-4 A on nearly degenerate
// rays.  The solver has thresholds in absolute units, so that holds for patches of molecular size
// only: where depressed coefficients can exceed 3,000 it takes a reciprocal form whose roots are
// off by as much as the tube (1e-4 of the candidates of tori ten times as large as a molecule's),
// and at a tenth of that size a few of its roots in 1e7 are off by more than the slack.  The
// distance test is left out there; the plane test does not depend on the solver.  A NaN anywhere
// keeps the candidate.
//
// Host and device: the same code is tested on the CPU against the double-precision path.
#pragma once
#include <math.h>

#include "ns_types.h"

namespace nsg {

// Record of a torus patch, about the centre of its clipping sphere:
//   [0..3], [4..7]  the two planes of an acute pair (n, d - slack); (0, 0, 0, -1) without one
//   [8..10] torus centre, [11] major radius, [12..14] torus axis, [15] tube radius (the probe)
//   [16] clipping radius, [17] slack of the distance test, [18..19] 0
constexpr int kTorusScreen = 20;

// f: the patch record; w: its first two pool entries (null without them); wedge: the entries are its
// only pair, and acute (feasible where both tests are <= 0).
NS_HD void torus_screen_record(const double* f, const double* w, bool wedge, double probe, float* out) {
  const double r = f[3];
  for (int q = 0; q < 2; q++) {
    out[4 * q] = out[4 * q + 1] = out[4 * q + 2] = 0.f;
    out[4 * q + 3] = -1.f;
    if (!wedge) continue;
    const double* p = w + 4 * q;
    const double d = p[3] + (p[0] * f[0] + p[1] * f[1] + p[2] * f[2]);
    const double size = (fabs(p[0]) + fabs(p[1]) + fabs(p[2])) * r + fabs(d);
    for (int k = 0; k < 3; k++) out[4 * q + k] = (float)p[k];
    out[4 * q + 3] = (float)(d - 1e-5 * size);
  }
  double off = 0.0;
  for (int k = 0; k < 3; k++) {
    out[8 + k] = (float)(f[4 + k] - f[k]);
    out[12 + k] = (float)f[15 + k];
    off += fabs(f[4 + k] - f[k]);
  }
  out[11] = (float)f[7];
  out[15] = (float)probe;
  out[16] = (float)r;
  // sizes where the solver's absolute thresholds stay out of play: the depressed quartic's last
  // coefficient is a product of four roots within `size`, 7^4 < 3,000
  const double size = fabs(f[7]) + r + probe + off;
  out[17] = size >= 2.0 && size <= 7.0 ? (float)(0.005 * size) : 1e30f;
  out[18] = out[19] = 0.f;
}

// Whether the ray along axis VC at offsets (u, v) from the clipping centre along the pixel axes FD
// and LD may hit the patch.
template <int FD, int LD, int VC>
NS_HD bool torus_may_hit(const float* s, float u, float v) {
  const float r2 = s[16] * s[16];
  const float left = r2 - (u * u + v * v);
  const float h = sqrtf((left > 0.f ? left : 0.f) + 1e-5f * r2);
  float lo = -h, hi = h;
  for (int q = 0; q < 2; q++) {
    const float* p = s + 4 * q;
    const float a = p[FD] * u + p[LD] * v + p[3], n = p[VC];
    const float x = -a / n;
    if (n > 0.f) {
      if (x < hi) hi = x;
    } else if (n < 0.f) {
      if (x > lo) lo = x;
    } else if (a > 0.f) {
      return false;
    }
  }
  if (lo > hi) return false;
  // two pieces: a piece is clear when its middle is farther from both sheets of the surface (the
  // second one is the inner sheet of a spindle torus) than the half piece and the slack
  const float quarter = 0.25f * (hi - lo), reach = quarter + s[17];
  const float R = s[11], far2 = (s[15] + reach) * (s[15] + reach);
  const float near = s[15] - reach, near2 = near > 0.f ? near * near : 0.f;
  const float yu = u - s[8 + FD], yv = v - s[8 + LD];
  const float t = s[12 + FD] * yu + s[12 + LD] * yv, yy = yu * yu + yv * yv;
  bool clear = true;
  for (int q = 0; q < 2; q++) {
    const float yw = (lo + (q ? 3.f : 1.f) * quarter) - s[8 + VC];
    const float z = t + s[12 + VC] * yw;
    const float rho2 = (yy + yw * yw) - z * z;
    const float rho = sqrtf(rho2 > 0.f ? rho2 : 0.f);
    const float a = (rho - R) * (rho - R) + z * z, b = (rho + R) * (rho + R) + z * z;
    clear = clear && (a > far2 || a < near2) && (b > far2 || b < near2);
  }
  return !clear;
}

}  // namespace nsg
