// Device code of the collision forces and the Crank-Nicolson increments, shared by
// the stand-alone kernels (particles.cu) and the persistent stage kernel (subiter.cu).
//
// Reference functions restated here (NaokiHori/EllipsesInFlows):
//   compute_evolute, find_equivalent_circle(s)   src/suspensions/collision.c:75-154
//   compute_collision_force_p_p / _p_w           src/suspensions/collision.c:156-304
//   suspensions_compute_collision_force          src/suspensions/collision.c:306-367
//   compute_curvature                            src/ellipse.c:17-28
//   suspensions_increment_particles              src/suspensions/increment.c:10-72
//
// The particle records are read with ordinary loads: the persistent sub-iteration
// kernel writes them between its phases.
#pragma once
#include "eif_internal.cuh"
#include "foot_device.cuh"
#include <cfloat>

namespace {

using eifd::pmass;

// ellipse.c:30-65, for the few feet that foot_newton leaves
__device__ __noinline__ double normal_t_d(double a, double b, double x_, double y_) {
  const double px = fabs(x_), py = fabs(y_);
  const double kex = a * (1. - (b / a) * (b / a));
  const double key = b * (1. - (a / b) * (a / b));
  const double ab2 = a * a + b * b;
  double t = 0.25 * M_PI;
  for (int n = 0;; n++) {
    double st, ct;
    sincos(t, &st, &ct);
    const double x = a * ct, y = b * st;
    const double ex = kex * (ct * ct * ct), ey = key * (st * st * st);
    const double rx = x - ex, ry = y - ey, qx = px - ex, qy = py - ey;
    const double r = sqrt(ry * ry + rx * rx);
    const double q = sqrt(qy * qy + qx * qx);
    const double dc = r * asin((rx * qy - ry * qx) / (r * q));
    const double dt = dc / sqrt(ab2 - x * x - y * y);
    t += dt;
    t = fmin(0.5 * M_PI, t);
    t = fmax(0., t);
    if (fabs(dt) < 1.e-8) break;
    if (n > EIF_NORMAL_MAX_ITER - 1) break;
  }
  if (x_ < 0.) t = M_PI - t;
  if (y_ < 0.) t = -t;
  return t;
}

// One ellipse of an equivalent-circle fit: what its evolute points need, formed once per fit
struct FitEllipse {
  double a, b, x, y, cp, sp;     // semi-axes, centre, cos and sin of the angle
  double kex, key, rab;          // a(1-(b/a)^2), b(1-(a/b)^2), 1 / (a b)
  EllF f;
};

__device__ __forceinline__ FitEllipse fit_ellipse(double a, double b, double x, double y, double angle) {
  FitEllipse e;
  e.a = a; e.b = b; e.x = x; e.y = y;
  sincos(angle, &e.sp, &e.cp);
  const double ra = 1. / a, rb = 1. / b, d = (a - b) * (a + b);
  e.kex = d * ra;      // a (1 - (b/a)^2)
  e.key = -(d * rb);
  e.rab = ra * rb;
  e.f.a = eifd::d2f(a); e.f.b = eifd::d2f(b);
  e.f.cz = eifd::d2f(d); e.f.sz = 0.f;   // a^2 - b^2 (the angle's words are not used here)
  e.f.kex = eifd::d2f(e.kex); e.f.key = eifd::d2f(e.key);
  return e;
}

// The foot of the normal from (px, py), first quadrant, as (c, s) = (cos t, sin t), from the
// (c, s) given: with v = (px, py) - (a c, b s) and T the derivative of the ellipse in t, the
// angle to the foot solves g - K t + f t^2 / 2 = 0 up to third order, g = v.T, K = T^2 + v.(a c,
// b s), f = -(g + 3 (a^2 - b^2) c s): t = g / K to double precision and the quadratic term, which
// needs no more than single precision. Below FIT_STEP what is left out is below 1e-16. Returns
// false where K is small (next to the evolute) or the start is too far off.
constexpr double FIT_STEP = 4.e-6;
__device__ __forceinline__ bool foot_newton(const FitEllipse &e, double px, double py, double &c, double &s) {
  for (int n = 0; n < 8; n++) {
    const double ac = e.a * c, bs = e.b * s, as = e.a * s, bc = e.b * c;
    const double vx = px - ac, vy = py - bs;
    const double g = fma(vy, bc, -(vx * as));
    const double w2 = fma(as, as, bc * bc);
    const double K = fma(vx, ac, fma(vy, bs, w2));
    const float Kf = eifd::d2f(K);
    if (!(Kf > 0.02f * eifd::d2f(w2))) return false;
    // g / K from a single-precision reciprocal and one Newton step
    const float rf = __fdividef(1.f, Kf);
    const double r = eifd::f2d(rf), gr = g * r;
    const double d = fma(gr, fma(-K, r, 1.), gr);
    if (!(fabs(d) < 0.1)) return false;
    const float df = eifd::d2f(d), f3 = __fmul_rn(3.f * e.f.cz, __fmul_rn(eifd::d2f(c), eifd::d2f(s)));
    const float q = __fmul_rn(__fmul_rn(0.5f * rf, __fadd_rn(eifd::d2f(g), f3)), __fmul_rn(df, df));
    const double t = d - eifd::f2d(q);
    const double h = fma(t, -0.5 * t, 1.);
    const double c1 = fmax(fma(-t, s, c * h), 0.), s1 = fmax(fma(t, c, s * h), 0.);
    // back onto the unit circle: the step leaves t^4 / 4, a start from single precision 1e-7
    const double dn = fma(c1, c1, fma(s1, s1, -1.));
    const double u = fma(dn, fma(dn, 0.375, -0.5), 1.);
    c = c1 * u;
    s = s1 * u;
    if (fabs(d) < FIT_STEP) return true;
  }
  return false;
}

// compute_evolute, collision.c:75-109: the centre (ex, ey) of the circle of curvature at the
// foot of (x, y). (c, s), both signs positive: the foot of the fit's last iteration on entry
// (first: none yet), this one's on return; cs, ss: with its signs. A serial chain of FP64
// operations, of about 25 ns each here: the foot is iterated on (cos t, sin t), from the last
// foot or the one that single precision finds, so that nothing is left of ellipse.c's sincos,
// asin, square roots and divisions, and evaluated to the same accuracy (the foot to 1e-15 and
// better, where ellipse.c stops once the step is below 1e-8). Every product-sum is an explicit
// fma: the same bits in whatever kernel this is compiled.
__device__ __forceinline__ void evolute(const FitEllipse &e, bool first, double x, double y, double &c, double &s,
                                        double &cs, double &ss, double &ex, double &ey) {
  const double X = x - e.x, Y = y - e.y;
  const double x_ = fma(e.cp, X, e.sp * Y), y_ = fma(e.cp, Y, -(e.sp * X));
  const double px = fabs(x_), py = fabs(y_);
  if (first || !foot_newton(e, px, py, c, s)) {
    float sf, cf;
    sincosf(normal_t_f_q1(e.f, eifd::d2f(px), eifd::d2f(py)), &sf, &cf);
    c = eifd::f2d(cf);
    s = eifd::f2d(sf);
    if (!foot_newton(e, px, py, c, s)) sincos(normal_t_d(e.a, e.b, px, py), &s, &c);
  }
  cs = x_ < 0. ? -c : c;
  ss = y_ < 0. ? -s : s;
  const double vx = e.kex * (cs * cs * cs), vy = e.key * (ss * ss * ss);
  ex = fma(e.cp, vx, fma(-e.sp, vy, e.x));
  ey = fma(e.sp, vx, fma(e.cp, vy, e.y));
}
// the rest of compute_evolute, wanted of the last iteration only: the circle's radius r
// (ellipse.c:17-28) and the foot's offset (ix, iy) from the ellipse's centre
__device__ __forceinline__ void evolute_end(const FitEllipse &e, double cs, double ss, double &ix, double &iy, double &r) {
  const double as = e.a * ss, bc = e.b * cs;
  const double w2 = fma(as, as, bc * bc);
  r = fmin(w2 * sqrt(w2) * e.rab, 1. / DBL_EPSILON);
  const double fx = e.a * cs, fy = e.b * ss;
  ix = fma(e.cp, fx, -(e.sp * fy));
  iy = fma(e.sp, fx, e.cp * fy);
}

// Where the centres X^k + dX are taken from: formed from the records, from X^k alone (zero
// increments), or from a list (the persistent sub-iteration kernel, which writes the records'
// increments while other blocks still read the centres)
struct Places {
  const double2 *pos = nullptr;
  const float4 *near = nullptr;   // with pos: pair_prefilter's values
  bool at_x = false;
};
__device__ __forceinline__ double2 place_of(const Places &s, const double *P, int pc, int n) {
  if (s.pos) return s.pos[n];
  const double x = P[EIF_P_X * pc + n], y = P[EIF_P_Y * pc + n];
  return s.at_x ? make_double2(x, y) : make_double2(x + P[EIF_P_DX * pc + n], y + P[EIF_P_DY * pc + n]);
}

struct PV {  // particle view at the positions X^k + dX
  double den, a, b, x, y, az;
};

__device__ __forceinline__ PV load_pv(const Places &s, const double *P, int pc, int n) {
  PV v;
  v.den = P[EIF_P_DEN * pc + n];
  v.a = P[EIF_P_A * pc + n];
  v.b = P[EIF_P_B * pc + n];
  const double2 c = place_of(s, P, pc, n);
  v.x = c.x;
  v.y = c.y;
  v.az = P[EIF_P_AZ * pc + n];
  return v;
}

// y-offset of the nearest periodic image of p1 seen from p0 (collision.c:158-171)
__device__ __forceinline__ double image_offset(double p0y, double p1y, double ly) {
  double yoff = 0., minval = DBL_MAX;
  for (int per = -1; per <= 1; per++) {
    const double v = fabs((p1y + ly * per) - p0y);
    if (v < minval) { minval = v; yoff = ly * per; }
  }
  return yoff;
}

// exact early-out of collision.c:173-189: true when the bounding circles overlap. The distance
// itself (hypot: a chain of about 40 FP64 operations) only where the squares leave it open.
__device__ __forceinline__ bool bounding_overlap(const PV &p0, const PV &p1, double ly) {
  const double yoff = image_offset(p0.y, p1.y, ly);
  const double nx = p1.x - p0.x, ny = (p1.y + yoff) - p0.y;
  const double sum = fmax(p0.a, p0.b) + fmax(p1.a, p1.b);
  const double d2 = fma(nx, nx, ny * ny), s2 = sum * sum;
  if (d2 < s2 * (1. - 1e-12)) return true;
  if (d2 > s2 * (1. + 1e-12)) return false;
  return !(sum - fmax(hypot(nx, ny), DBL_EPSILON) < 0.);
}

// Pairs whose bounding circles overlap (collision.c:173-189) but whose ellipses are
// apart. The reference then iterates the equivalent-circle fit (collision.c:111-135) to
// the circles of curvature at the mutually nearest points, whose overlap is minus the
// gap, and the pair adds no force; for nearly touching ellipses that fixed point
// converges slowly (thousands of iterations in double precision). A line that separates
// the two ellipses with a gap above a hundredth of the smaller minor semi-axis (far above
// the fit's stopping error) proves the same zero contribution without the iteration.
// Candidate normals: the centre line, the four semi-axis directions and 16 fixed
// directions; along a unit normal n the ellipses' extents are their support values
// sqrt(a^2 (n.u)^2 + b^2 (n.v)^2) about the centres. Single precision: whatever it finds apart
// by the margin, which is at least 2e-5 of the radii, forty times its rounding, is apart.
struct PairFrame {
  float dx, dy, s0, c0, s1, c1, a0, b0, a1, b1, margin;
};
__device__ __forceinline__ PairFrame pair_frame(const PV &p0, const PV &p1, double ly) {
  PairFrame f;
  f.dx = eifd::d2f(p1.x - p0.x);
  f.dy = eifd::d2f((p1.y + image_offset(p0.y, p1.y, ly)) - p0.y);
  sincosf(eifd::d2f(p0.az), &f.s0, &f.c0);
  sincosf(eifd::d2f(p1.az), &f.s1, &f.c1);
  f.a0 = eifd::d2f(p0.a); f.b0 = eifd::d2f(p0.b);
  f.a1 = eifd::d2f(p1.a); f.b1 = eifd::d2f(p1.b);
  f.margin = fmaxf(0.01f * fminf(fminf(f.a0, f.b0), fminf(f.a1, f.b1)),
                   2.e-5f * (fmaxf(f.a0, f.b0) + fmaxf(f.a1, f.b1)));
  return f;
}
__device__ __forceinline__ bool separated(const PairFrame &f, float nx, float ny) {
  const float u0 = nx * f.c0 + ny * f.s0, v0 = ny * f.c0 - nx * f.s0;
  const float u1 = nx * f.c1 + ny * f.s1, v1 = ny * f.c1 - nx * f.s1;
  const float h0 = sqrtf(f.a0 * f.a0 * u0 * u0 + f.b0 * f.b0 * v0 * v0);
  const float h1 = sqrtf(f.a1 * f.a1 * u1 * u1 + f.b1 * f.b1 * v1 * v1);
  return fabsf(nx * f.dx + ny * f.dy) - h0 - h1 > f.margin;
}
// the centre line alone, which settles most pairs: one pair per lane
__device__ __forceinline__ bool apart_centres(const PV &p0, const PV &p1, double ly) {
  const PairFrame f = pair_frame(p0, p1, ly);
  const float d = sqrtf(f.dx * f.dx + f.dy * f.dy);
  return d > 0.f && separated(f, f.dx / d, f.dy / d);
}
// the other directions of one pair, one per lane
__device__ __forceinline__ bool apart_warp(const PV &p0, const PV &p1, double ly, int lane) {
  const PairFrame f = pair_frame(p0, p1, ly);
  float ny, nx;
  sincospif((lane - 4) / 16.f, &ny, &nx);
  if (lane == 0) { nx = f.c0; ny = f.s0; }
  if (lane == 1) { nx = -f.s0; ny = f.c0; }
  if (lane == 2) { nx = f.c1; ny = f.s1; }
  if (lane == 3) { nx = -f.s1; ny = f.c1; }
  return __any_sync(0xffffffffu, lane < 20 && separated(f, nx, ny));
}

constexpr int FIT_SLOTS = 16;   // pairs a warp fits at a time, two lanes each
// The contacts of particle k, its pairs with the listed particles (in partner order) and the
// walls at x = 0 and x = lx: equivalent-circle fits (collision.c:111-154), forces and torques
// (collision.c:190-304), summed in partner order and then the walls (lane 0 has the sums).
// The two ellipses of a pair are iterated by two neighbouring lanes, since each iteration
// needs of the other ellipse only its last centre; the walls take one more pair of lanes, with
// the mirrored centre in the place of the other's. A fit is a serial chain of a hundred and more
// evolute points in double precision and sets the time of the launch.
__device__ __forceinline__ void contact_forces(const Places &where, const double *P, int pcap, int k, const PV &pk, const int *list, int ncon,
                                               double ly, double lx, double (*cval)[3], double acc[3], bool &ok_all) {
  const int lane = threadIdx.x & 31, role = lane & 1;
  const double wallx = role ? lx : 0.;
  const bool near_wall = !(fmax(pk.a, pk.b) - fabs(wallx - pk.x) < 0.);
  const bool walls = __any_sync(0xffffffffu, near_wall);
  const int items = ncon + (walls ? 1 : 0);
  acc[0] = acc[1] = acc[2] = 0.;
  ok_all = true;
  for (int base = 0; base < items; base += FIT_SLOTS) {
    const int q = base + (lane >> 1);
    const bool wall = q == ncon;
    bool act = q < ncon || (wall && near_wall);
    PV p0 = pk, p1 = pk;
    bool self0 = true;
    if (q < ncon) {
      const int m = list[q];
      self0 = k < m;
      const PV o = load_pv(where, P, pcap, m);
      p0 = self0 ? pk : o;
      p1 = self0 ? o : pk;
    }
    const double yoff = wall ? 0. : image_offset(p0.y, p1.y, ly);
    const PV pe = role ? p1 : p0;
    const FitEllipse e = fit_ellipse(pe.a, pe.b, pe.x, pe.y + (role ? yoff : 0.), pe.az);
    double cx = e.x, cy = e.y, r = 0., ix = 0., iy = 0., c = 0., s = 0., cs = 0., ss = 0.;
    bool ok = !act;
    for (int n = 0; n < EIF_FIT_MAX_ITER && __any_sync(0xffffffffu, act); n++) {
      double ox = __shfl_xor_sync(0xffffffffu, cx, 1), oy = __shfl_xor_sync(0xffffffffu, cy, 1);
      if (wall) {
        ox = fma(2., wallx, -cx);
        oy = cy;
      }
      double change = 0.;
      if (act) {
        double nx, ny;
        evolute(e, n == 0, ox, oy, c, s, cs, ss, nx, ny);
        const double dx = nx - cx, dy = ny - cy;
        cx += dx;
        cy += dy;
        change = fmax(fabs(dx), fabs(dy));
      }
      const double other = __shfl_xor_sync(0xffffffffu, change, 1);
      if (act && (wall ? change : fmax(change, other)) < 1.e-8) {
        act = false;
        ok = true;
      }
    }
    ok_all &= ok;
    evolute_end(e, cs, ss, ix, iy, r);
    const double ocx = __shfl_xor_sync(0xffffffffu, cx, 1), ocy = __shfl_xor_sync(0xffffffffu, cy, 1),
                 orr = __shfl_xor_sync(0xffffffffu, r, 1);
    // the force over this particle's mass and the torque over its moment of inertia
    // (collision.c:190-304: k = m (pi / h^(3/2))^2 with the harmonic means m of the masses and
    // h of the radii sqrt(a b)), in few and independent divisions
    double out[3] = {0., 0., 0.};
    const bool mine = q < ncon && (role == 0) == self0;
    if (mine || (wall && near_wall)) {
      double nx = wallx - cx, ny = 0., norm = fabs(nx), overlap = r - norm, w = 1., hs = 1., hp = sqrt(pk.a * pk.b);
      if (mine) {
        // from this particle's circle to the other's
        nx = ocx - cx;
        ny = ocy - cy;
        norm = fmax(sqrt(fma(nx, nx, ny * ny)), DBL_EPSILON);
        overlap = r + orr - norm;
        const PV po = role ? p0 : p1;
        const double ms = pmass(pe.den, pe.a, pe.b), mo = pmass(po.den, po.a, po.b), ho = sqrt(po.a * po.b);
        w = 2. * mo / (ms + mo);
        hs = hp + ho;
        hp = 2. * hp * ho;
      }
      if (overlap > 0.) {
        const double rh = hs / hp;
        const double f = -(M_PI * M_PI * w * overlap * (rh * rh * rh)) / norm;
        out[0] = f * nx;
        out[1] = f * ny;
        out[2] = 4. / fma(pe.a, pe.a, pe.b * pe.b) * fma(ix, out[1], -(iy * out[0]));
      }
    }
    if (mine)
      for (int f = 0; f < 3; f++) cval[lane >> 1][f] = out[f];
    if (wall)
      for (int f = 0; f < 3; f++) cval[FIT_SLOTS + role][f] = out[f];
    __syncwarp();
    if (lane == 0) {
      const int pairs = min(FIT_SLOTS, ncon - base);
      for (int t = 0; t < pairs; t++)
        for (int f = 0; f < 3; f++) acc[f] += cval[t][f];
      if (base + FIT_SLOTS >= items && walls)
        for (int t = 0; t < 2; t++)
          for (int f = 0; f < 3; f++) acc[f] += cval[FIT_SLOTS + t][f];
    }
    __syncwarp();
  }
  ok_all = __all_sync(0xffffffffu, ok_all);
}

// Collision forces (collision.c:306-367) in one launch, one warp per particle k:
//  1. candidate partners: the lanes test the partners m = lane, lane + 32, ... in order
//     against single-precision centres (at X^k + dX) and bounding radii, staged in shared
//     memory tile by tile (every block forms them from the records as it loads a tile);
//     the pairs that pass this conservative test are listed in partner order (ballot and
//     prefix count);
//  2. the lanes give the listed pairs the exact double-precision bounding-circle test of
//     collision.c:173-189 (canonical orientation) and compact the hits in order;
//  3. hits whose ellipses a line separates are dropped, the others and the walls are
//     evaluated (contact_forces).
constexpr int CAND_CAP = EIF_CAND_CAP;   // candidates per particle
constexpr int PAIR_WARPS = 8;
constexpr int PAIR_TILE = 1024;
constexpr int PAIR_LOADS = PAIR_TILE / (PAIR_WARPS * 32);

__device__ __forceinline__ float4 pair_prefilter(const Places &where, const double *P, int pcap, int n) {
  if (where.near) return where.near[n];
  const double2 c = place_of(where, P, pcap, n);
  return make_float4(eifd::d2f(c.x), eifd::d2f(c.y), eifd::d2f(fmax(P[EIF_P_A * pcap + n], P[EIF_P_B * pcap + n])), 0.f);
}

// One block of PAIR_WARPS warps: particles block * PAIR_WARPS ...
__device__ __forceinline__ void collision_block(const Places &where, double *P, int pcap, int np, int cn, double ly, double lx,
                                                unsigned *flags, int block) {
  __shared__ float4 tile[PAIR_TILE];
  __shared__ int list[PAIR_WARPS][CAND_CAP];
  __shared__ double cval[PAIR_WARPS][FIT_SLOTS + 2][3];
  const int lane = threadIdx.x & 31, wl = threadIdx.x >> 5;
  const int k = block * PAIR_WARPS + wl;
  const bool on = k < np;   // uniform over the warp
  const float4 fk = on ? pair_prefilter(where, P, pcap, k) : make_float4(0.f, 0.f, 0.f, 0.f);
  const float lyf = eifd::d2f(ly);
  int nmaybe = 0;
  for (int t0 = 0; t0 < np; t0 += PAIR_TILE) {
    const int nt = min(PAIR_TILE, np - t0);
    float4 st[PAIR_LOADS];
#pragma unroll
    for (int r = 0; r < PAIR_LOADS; r++) {
      const int q = threadIdx.x + r * PAIR_WARPS * 32;
      st[r] = q < nt ? pair_prefilter(where, P, pcap, t0 + q) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < PAIR_LOADS; r++) tile[threadIdx.x + r * PAIR_WARPS * 32] = st[r];
    __syncthreads();
    if (!on) continue;
#pragma unroll 2
    for (int base = 0; base < nt; base += 32) {
      const int m = t0 + base + lane;
      bool maybe = false;
      if (base + lane < nt && m != k) {
        const float4 fm = tile[base + lane];
        // conservative single-precision test: skip only pairs clearly apart for every image
        const float rs = fk.z + fm.z;
        const float dxf = fm.x - fk.x;
        const float lim = rs * rs * 1.001f + 1e-6f;
#pragma unroll
        for (int per = -1; per <= 1; per++) {
          const float dyf = fm.y + lyf * per - fk.y;
          maybe |= dxf * dxf + dyf * dyf <= lim;
        }
      }
      const unsigned mask = __ballot_sync(0xffffffffu, maybe);
      if (maybe) {
        const int r = nmaybe + __popc(mask & ((1u << lane) - 1u));
        if (r < CAND_CAP) list[wl][r] = m;
      }
      nmaybe += __popc(mask);
    }
  }
  if (!on) return;
  __syncwarp();
  if (nmaybe > CAND_CAP && lane == 0) atomicOr(flags, EIF_FLAG_NOCONV);
  nmaybe = min(nmaybe, CAND_CAP);
  const PV pk = load_pv(where, P, pcap, k);
  // exact test and the centre line, hits compacted in place (a write never passes the
  // entries still to read)
  int cnt = 0;
  for (int base = 0; base < nmaybe; base += 32) {
    const int q = base + lane;
    bool hit = false;
    int m = 0;
    if (q < nmaybe) {
      m = list[wl][q];
      const PV o = load_pv(where, P, pcap, m);
      const PV p0 = m < k ? o : pk, p1 = m < k ? pk : o;
      hit = bounding_overlap(p0, p1, ly) && !apart_centres(p0, p1, ly);
    }
    const unsigned mask = __ballot_sync(0xffffffffu, hit);
    if (hit) list[wl][cnt + __popc(mask & ((1u << lane) - 1u))] = m;
    cnt += __popc(mask);
    __syncwarp();
  }
  // the other directions, in order again
  int ncon = 0;
  for (int q = 0; q < cnt; q++) {
    const int m = list[wl][q];
    const PV o = load_pv(where, P, pcap, m);
    const PV p0 = m < k ? o : pk, p1 = m < k ? pk : o;
    if (apart_warp(p0, p1, ly, lane)) continue;
    __syncwarp();
    if (lane == 0) list[wl][ncon] = m;
    ncon++;
  }
  __syncwarp();
  double acc[3];
  bool ok;
  contact_forces(where, P, pcap, k, pk, list[wl], ncon, ly, lx, cval[wl], acc, ok);
  if (lane == 0) {
    P[(EIF_P_CFX0 + cn) * pcap + k] = acc[0];
    P[(EIF_P_CFY0 + cn) * pcap + k] = acc[1];
    P[(EIF_P_CTZ0 + cn) * pcap + k] = acc[2];
    if (!ok) atomicOr(flags, EIF_FLAG_NOCONV);
  }
}

// increment.c:10-72, one component (x, y or the rotation) of a particle: the new velocity
// increment from the collision forces c0, c1, the fluid force f, the inertia integrals i0, i1 and
// the constant part g (gravity_increment in x), and the position increment from it. Every
// rounding is explicit: the kernels that form increments give the same bits.
__device__ __forceinline__ double velocity_increment(double hgd, double dt, double c0, double c1, double f, double i0,
                                                     double i1) {
  return __dadd_rn(fma(hgd, __dadd_rn(c0, c1), __dmul_rn(dt, f)), __dadd_rn(i1, -i0));
}
__device__ __forceinline__ double gravity_increment(double gamma, double dt, double den, double Fr2) {
  return __ddiv_rn(__dmul_rn(__dmul_rn(gamma, dt), __dadd_rn(1., -den)), Fr2);
}
__device__ __forceinline__ double position_increment(double hgd, double u, double du) {
  return __dmul_rn(hgd, __dadd_rn(u, __dadd_rn(u, du)));
}

// the three components of particle n (one thread); returns res raised to the largest change of
// the velocity increments
__device__ __forceinline__ double increment_particle(double *p, int pcap, int n, double gamma, double Fr2, double dt,
                                                     double res) {
  const double px = p[EIF_P_DUX * pcap + n], py = p[EIF_P_DUY * pcap + n], pz = p[EIF_P_DVZ * pcap + n];
  const double hgd = __dmul_rn(0.5 * gamma, dt);
  const double dux =
      __dadd_rn(velocity_increment(hgd, dt, p[EIF_P_CFX0 * pcap + n], p[EIF_P_CFX1 * pcap + n], p[EIF_P_FUX * pcap + n],
                                   p[EIF_P_IUX0 * pcap + n], p[EIF_P_IUX1 * pcap + n]),
                gravity_increment(gamma, dt, p[EIF_P_DEN * pcap + n], Fr2));
  const double duy = velocity_increment(hgd, dt, p[EIF_P_CFY0 * pcap + n], p[EIF_P_CFY1 * pcap + n],
                                        p[EIF_P_FUY * pcap + n], p[EIF_P_IUY0 * pcap + n], p[EIF_P_IUY1 * pcap + n]);
  const double dvz = velocity_increment(hgd, dt, p[EIF_P_CTZ0 * pcap + n], p[EIF_P_CTZ1 * pcap + n],
                                        p[EIF_P_TVZ * pcap + n], p[EIF_P_IVZ0 * pcap + n], p[EIF_P_IVZ1 * pcap + n]);
  p[EIF_P_DUX * pcap + n] = dux;
  p[EIF_P_DUY * pcap + n] = duy;
  p[EIF_P_DVZ * pcap + n] = dvz;
  res = fmax(res, fabs(dux - px));
  res = fmax(res, fabs(duy - py));
  res = fmax(res, fabs(dvz - pz));
  p[EIF_P_DX * pcap + n] = position_increment(hgd, p[EIF_P_UX * pcap + n], dux);
  p[EIF_P_DY * pcap + n] = position_increment(hgd, p[EIF_P_UY * pcap + n], duy);
  p[EIF_P_DAZ * pcap + n] = position_increment(hgd, p[EIF_P_VZ * pcap + n], dvz);
  return res;
}

// reset.c:7-18 for particle n: increments of the new stage start at zero
__device__ __forceinline__ void reset_particle(double *P, int pcap, int n) {
  P[EIF_P_DUX * pcap + n] = 0.; P[EIF_P_DUY * pcap + n] = 0.; P[EIF_P_DVZ * pcap + n] = 0.;
  P[EIF_P_DX * pcap + n] = 0.; P[EIF_P_DY * pcap + n] = 0.; P[EIF_P_DAZ * pcap + n] = 0.;
}

// update.c:8-34 for particle n: velocities and positions advanced by the increments,
// the centre wrapped into [0, ly] and the angle into [0, 2 pi]
__device__ __forceinline__ void update_particle(double *P, int pcap, int n, double ly) {
  P[EIF_P_UX * pcap + n] += P[EIF_P_DUX * pcap + n];
  P[EIF_P_UY * pcap + n] += P[EIF_P_DUY * pcap + n];
  P[EIF_P_VZ * pcap + n] += P[EIF_P_DVZ * pcap + n];
  double x = P[EIF_P_X * pcap + n] + P[EIF_P_DX * pcap + n];
  double y = P[EIF_P_Y * pcap + n] + P[EIF_P_DY * pcap + n];
  double az = P[EIF_P_AZ * pcap + n] + P[EIF_P_DAZ * pcap + n];
  if (y < 0.) y += ly;
  if (y > ly) y -= ly;
  if (az < 0.) az += 2. * M_PI;
  if (az > 2. * M_PI) az -= 2. * M_PI;
  P[EIF_P_X * pcap + n] = x;
  P[EIF_P_Y * pcap + n] = y;
  P[EIF_P_AZ * pcap + n] = az;
}

}  // namespace
