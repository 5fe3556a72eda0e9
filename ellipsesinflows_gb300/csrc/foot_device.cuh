// The foot of the normal from a point to an ellipse (ellipse.c:30-65) in single precision:
// the indicator's distance (ibm_device.cuh) and the start of the double-precision feet.
#pragma once
#include "eif_internal.cuh"

namespace {

// The normal-foot iteration of ellipse.c:30-65 in single precision (the mixed form's
// indicator, and the start of the double-precision iteration below). The distance at
// the foot is stationary in t, so an angle error dt changes it by O(a dt^2): stopping
// once the step is below 1e-3 leaves distance errors near 1e-9 cells (checked against
// fully converged iterations over the aspect ratios 1-3).
constexpr float NORMAL_TOL_F = 1.e-3f;
constexpr int NORMAL_MAX_F = 24;

struct EllF {
  float a, b, cz, sz, kex, key;
};

// The reference's iteration (ellipse.c:30-65) in single precision, on the first-quadrant
// offsets (px, py) = (|x_|, |y_|); normal_t_f unfolds the angle. Its fixed point
// is the normal foot whatever the accuracy of the intermediate sin/cos, square
// roots and arcsine, so the loop uses the hardware approximations (__sincosf,
// rsqrtf) and the Taylor polynomial x + x^3/6 + 3x^5/40 of asin (odd, increasing
// and zero only at zero like asin, so the step keeps its sign and vanishes at the
// foot); the distance at the converged angle is evaluated with the accurate
// sincosf, and the distance is stationary in the angle.
__device__ __forceinline__ float normal_t_f_q1(const EllF &e, float px, float py) {
  float t = 0.78539816339744831f;
  for (int n = 0; n < NORMAL_MAX_F; n++) {
    float st, ct;
    __sincosf(t, &st, &ct);
    const float x = e.a * ct, y = e.b * st;
    const float ex = e.kex * (ct * ct * ct), ey = e.key * (st * st * st);
    const float rx = x - ex, ry = y - ey, qx = px - ex, qy = py - ey;
    const float r2 = ry * ry + rx * rx, q2 = qy * qy + qx * qx;
    const float arg = fminf(fmaxf((rx * qy - ry * qx) * rsqrtf(r2 * q2), -1.f), 1.f);
    const float a2 = arg * arg;
    const float dc = r2 * rsqrtf(r2) * (arg * fmaf(a2, fmaf(a2, 0.075f, 0.16666667f), 1.f));
    // a^2 + b^2 - x^2 - y^2 written without cancellation
    const float dt = dc * rsqrtf(e.a * e.a * (st * st) + e.b * e.b * (ct * ct));
    t += dt;
    t = fminf(1.5707963267948966f, t);
    t = fmaxf(0.f, t);
    if (fabsf(dt) < NORMAL_TOL_F) break;
  }
  return t;
}

}  // namespace
