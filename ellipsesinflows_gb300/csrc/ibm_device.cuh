// Device code of the immersed-boundary evaluations shared by the stand-alone
// kernels (ibm.cu) and the persistent stage kernel (subiter.cu):
// geometry helpers, the per-particle boxes, the task table and the per-task and
// per-particle bodies of the volume integrals and the momentum exchange.
//
// Reference functions restated here (NaokiHori/EllipsesInFlows):
//   suspensions_decide_loop_size   src/suspensions/auxiliary.c:11-17
//   compute_signed_dist            src/suspensions/auxiliary.c:19-47
//   suspensions_s_weight/v_weight  src/suspensions/auxiliary.c:51-59
//   mass, moment of inertia        src/suspensions/auxiliary.c:63-75
//   find_normal_t, compute_ex/ey   src/ellipse.c:7-65
//   kernel_exchange_momentum       src/suspensions/exchange.c:13-88
//   compute_inertia                src/suspensions/inertia.c:9-70
//
// Loads through the read-only data path (__ldg) are only valid for data that no
// thread writes while the kernel runs. The bodies take a template flag NC: true in
// the stand-alone single-precision kernels, false in the persistent sub-iteration
// kernel, whose phases write the particle records, boxes, task table and parameters
// that later phases read (there those loads are ordinary, coherent after the grid
// barrier), and false in both for the double-precision task body, so that both run
// one instantiation of it.
#pragma once
#include "eif_internal.cuh"
#include "eif_df.cuh"
#include "foot_device.cuh"
#include <cfloat>

namespace {

// a load through the read-only path when NC, an ordinary load otherwise
template <bool NC, typename T>
__device__ __forceinline__ T ldro(const T *p) {
  if constexpr (NC) return __ldg(p);
  else return *p;
}

constexpr int CHUNK = 64;       // cells per warp task (a box row, or a segment of one)
__device__ __host__ __forceinline__ int box_segs(int w) { return (w + CHUNK - 1) / CHUNK; }
constexpr int NEXTRA = 3;       // auxiliary.c:8
constexpr double BETA = 2.;     // auxiliary.c:49
constexpr int GTX = 128, GTY = 8, GTHREADS = 256;  // gather tile and block
constexpr int GCOLS = 64;   // columns covered by the threads of one pass (GTX / GCOLS passes)
constexpr int LMAX = 256;       // gather entries staged in shared memory at a time (GTHREADS)

__device__ __forceinline__ float normal_t_f(const EllF &e, float x_, float y_) {
  float t = normal_t_f_q1(e, fabsf(x_), fabsf(y_));
  if (x_ < 0.f) t = 3.14159265358979323846f - t;
  if (y_ < 0.f) t = -t;
  return t;
}

// Per-particle parameters of the double-precision form, PD_WORDS doubles per particle,
// written with the boxes (box_part): what every row task of a particle needs, formed once
// per particle instead of once per task by all lanes (about 150 FP64 operations a task:
// the stored-weight sums took 0.95 ms at 2048 x 4096 with 2048 ellipses that way, nearly
// all of it this set-up). Lengths with a bar are in units of h / BETA, so that the distance
// the cells compute is the argument of tanh.
constexpr int PD_WORDS = 20;
enum { PD_X, PD_Y,            // centre (with the increments where the boxes have them)
       PD_CZ, PD_SZ,          // cos(-az), sin(-az) times BETA / h
       PD_A, PD_B,            // semi-axes, barred
       PD_RPM, PD_RPIM,       // 1 / mass, 1 / moment of inertia
       PD_QM, PD_QIM,         // dx dy / 4 over them, the factors of the inertia sums
       PD_F };                // single-precision words from here:
enum { PDF_AL, PDF_KA, PDF_DE, PDF_SO2, PDF_SI2, PDF_RO2,   // row_chords
       PDF_A, PDF_B, PDF_KEX, PDF_KEY,                      // the foot iteration, barred
       PDF_PAIRS,                   // PD_A, PD_B, PD_CZ, PD_SZ as float pairs (dist_mid)
       PDF_WORDS = PDF_PAIRS + 8 };
static_assert(2 * (PD_WORDS - PD_F) >= PDF_WORDS && PD_WORDS % 2 == 0, "per-particle parameter block");

// The iteration of ellipse.c:30-65 in double precision with its stopping rule and cap, from
// the foot t that normal_t_f_q1 finds, for offsets (px, py) in the first quadrant: the foot's
// parameter. Only for the few cells next to the evolute, where foot_d does not settle.
__device__ __noinline__ double normal_t_q1(double a, double b, double px, double py, double t) {
  const double kex = a * (1. - (b / a) * (b / a)), key = b * (1. - (a / b) * (a / b)), ab2 = a * a + b * b;
  for (int n = 0;; n++) {
    double st, ct;
    sincos(t, &st, &ct);
    const double x = a * ct, y = b * st;
    const double ex = kex * (ct * ct * ct);
    const double ey = key * (st * st * st);
    const double rx = x - ex, ry = y - ey;
    const double qx = px - ex, qy = py - ey;
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
  return t;
}

// The normal foot of (px, py), first quadrant, in single precision: (c, s) = (cos t, sin t)
// to about 2e-7 (the iteration above, whose hardware sines shift its fixed point a little,
// and one Newton step, d); returns the distance to the foot, positive outside. Out of line:
// inlined into the loops around it, the compiler makes 45 KB of copies of it.
__device__ __noinline__ float foot_f(const EllF &e, float px, float py, float &c, float &s, float &d) {
  const float t = normal_t_f_q1(e, px, py);
  sincospif(t * 0.318309886f, &s, &c);
  float ac = e.a * c, bs = e.b * s, as = e.a * s, bc = e.b * c;
  float vx = px - ac, vy = py - bs;
  const float K = as * as + bc * bc + vx * ac + vy * bs;
  const float g = vy * bc - vx * as;
  d = K > 0.f ? fminf(fmaxf(__fdividef(g, K), -0.01f), 0.01f) : 0.01f;
  const float c1 = c - d * s;
  s = s + d * c;
  c = c1;
  bc = e.b * c; as = e.a * s;
  vx = px - e.a * c; vy = py - e.b * s;
  return (vx * bc + vy * as) * rsqrtf(bc * bc + as * as);
}

// The same foot and distance in double precision, from foot_f's (c0, s0). Bound by the FP64
// pipe (one warp instruction in 16 cycles), so the double-precision work is kept to what
// carries the precision:
//  * (c, s) is put on the unit circle in double precision; what is left of c^2 + s^2 - 1
//    (its rounding, the largest of the distance's errors) is taken off the distance;
//  * with v = (px, py) - (a c, b s), T the derivative of the ellipse in t (w = |T|) and N
//    its outward normal, the remaining angle to the foot is d = v.T / K,
//    K = w^2 + v.(a c, b s) = w^2 (1 + nu / R) with nu = v.N / w the distance to the
//    tangent and R = w^3 / (a b) the radius of curvature; the distance to the foot is
//    nu + (v.T / w)^2 / (2 (R + nu)) up to terms of third order in d. v.T, N and w^2 need
//    double precision, the correction and d only single;
//  * for |d| <= FOOT_TOL the terms left out are below 1e-16 a; a larger d is taken as a
//    Newton step (rare: the start is closer than that nearly everywhere).
// 31 FP64 instructions against about 460 for two passes of ellipse.c's iteration with their
// sincos, asin, square roots and divisions. NORMAL: the outward normal (nx, ny) as well, for
// which the foot itself is iterated to 1e-12 (one more step). Returns false next to the
// evolute (K small, or no convergence): the caller takes the general iteration.
constexpr float FOOT_TOL = 4.e-6f;
constexpr float FOOT_TOL_N = 1.e-12f;  // with the normal, which is not stationary in t
constexpr int FOOT_MAX = 6;
template <bool NORMAL>
__device__ __forceinline__ bool foot_d(double a, double b, float abf, float c0, float s0, double px, double py,
                                       double &dist, double &nx, double &ny) {
  double c = eifd::f2d(c0), s = eifd::f2d(s0);
  // c, s only a few 1e-5 off the unit circle: three terms of (1 + dn)^(-1/2)
  for (int n = 0; n < FOOT_MAX; n++) {
    const double dn = fma(c, c, fma(s, s, -1.));
    const double r = fma(dn, fma(dn, fma(dn, -0.3125, 0.375), -0.5), 1.);
    c *= r;
    s *= r;
    const double vx = fma(-a, c, px), vy = fma(-b, s, py);
    const double as = a * s, bc = b * c;
    const double g = fma(vy, bc, -(vx * as));
    const double w2 = fma(as, as, bc * bc);
    const double nw = fma(vx, bc, vy * as);
    const float w2f = eifd::d2f(w2), gf = eifd::d2f(g), nwf = eifd::d2f(nw);
    const float rw = rsqrtf(w2f);
    const float K = fmaf(nwf * abf, rw * rw, w2f);
    if (!(K > 0.02f * w2f)) return false;
    const float d = __fdividef(gf, K);
    const bool done = fabsf(d) <= (NORMAL ? FOOT_TOL_N : FOOT_TOL);
    if (done) {
      const float corr = 0.5f * gf * d * abf * (rw * rw * rw);
      // 1 / w from its single-precision value by one third-order step
      const double y0 = eifd::f2d(rw);
      const double e = fma(-(w2 * y0), y0, 1.);
      const double p = e * fma(e, 0.375, 0.5);
      const double u = fma(eifd::f2d(0.5f * abf), fma(c, c, fma(s, s, -1.)), nw) * y0;
      dist = fma(u, p, u) + eifd::f2d(corr);
      if (NORMAL) {
        const double y = fma(y0, p, y0);
        nx = bc * y;
        ny = as * y;
      }
      return true;
    }
    if (!(fabsf(d) < 0.1f)) return false;
    const double dd = eifd::f2d(d), h = fma(dd, -0.5 * dd, 1.);
    const double c1 = fma(-dd, s, c * h);
    s = fma(dd, c, s * h);
    c = c1;
  }
  return false;
}

// tanh(z) for z >= 0 from its values near the multiples of 1/16 (tab, up to TANH_TOP) by the
// addition theorem, tanh(z_k + d) = T + S t / (1 + T t), t = tanh(d) from
// its Taylor series (|d| <= 1/32: the first term left out is 3e-19); the quotient from a
// single-precision reciprocal and one third-order step. The table's T is tanh(k/16) rounded to
// double, z_k the place where tanh has that very value (near k/16; beyond z = 16 up to 1 away,
// where S is below 1e-13), so that the rounding of T does not add to the result's own: with
// z_k = k/16 the largest error at z = 4 to 6 was 1.1e-16, now half of that. 15 FP64 instructions.
constexpr int TANH_STEPS = 16, TANH_TOP = 20, TANH_N = TANH_STEPS * TANH_TOP + 1;
__device__ __forceinline__ double tanh_tab(double z, const double2 *__restrict__ tab) {
  const float zf = eifd::d2f(z);
  if (!(zf < (float)TANH_TOP)) return z > 0. ? 1. : z;   // a NaN stays one
  const int k = (int)rintf(zf * (float)TANH_STEPS);
  const double2 ts = __ldg(tab + 2 * k);   // T, S; the next entry's first is z_k
  const double d = z - __ldg(&tab[2 * k + 1].x);
  const double u = d * d;
  const double p = fma(u, fma(u, fma(u, 62. / 2835., -17. / 315.), 2. / 15.), -1. / 3.);
  const double t = fma(d * u, p, d);
  const double den = fma(ts.x, t, 1.);
  const double r = eifd::f2d(__fdividef(1.f, eifd::d2f(den)));
  const double e = fma(-den, r, 1.);
  const double q = ts.y * t * r;
  return ts.x + fma(q, fma(e, e, e), q);
}

// the distance and the normal next to the evolute, by ellipse.c's iteration
__device__ __noinline__ double foot_general(double a, double b, double px, double py, float c0, float s0, double &nx,
                                            double &ny) {
  const double t = normal_t_q1(a, b, px, py, eifd::f2d(fminf(fmaxf(atan2f(s0, c0), 0.f), 1.5707963f)));
  double st, ct;
  sincos(t, &st, &ct);
  const double fx = px - a * ct, fy = py - b * st;
  const bool in = 1. - (px / a) * (px / a) - (py / b) * (py / b) > 0.;
  const double d = sqrt(fx * fx + fy * fy);
  nx = ct / a;
  ny = st / b;
  const double nn = 1. / sqrt(nx * nx + ny * ny);
  nx *= nn;
  ny *= nn;
  return in ? -d : d;
}

// tanh(BETA D) of the signed distance D in units of h (auxiliary.c:19-59), positive
// inside, from the barred body-frame offset (x_, y_) and foot_f's (c0, s0); NORMAL: the
// outward unit normal at the foot in the body frame
template <bool NORMAL>
__device__ __forceinline__ double indicator_d(double a, double b, float abf, float c0, float s0, double x_, double y_,
                                              const double2 *__restrict__ tab, double &nx, double &ny) {
  const double px = fabs(x_), py = fabs(y_);
  double dist;
  if (!foot_d<NORMAL>(a, b, abf, c0, s0, px, py, dist, nx, ny)) dist = foot_general(a, b, px, py, c0, s0, nx, ny);
  if (NORMAL) {
    if (x_ < 0.) nx = -nx;
    if (y_ < 0.) ny = -ny;
  }
  const double th = tanh_tab(fabs(dist), tab);
  return __double2hiint(dist) < 0 ? th : -th;
}

// Cells whose tanh(BETA D) the FP32 pipe gives as well as the FP64 pipe: with z = |BETA D|,
// tanh z = 1 - x, x = 2 / (exp(2 z) + 1), and an error dz of the distance changes it by
// 4 exp(-2 z) dz. foot_f's foot (once its Newton step is below 1e-3) and the distance in
// double-float arithmetic (dist_mid, good to 1e-13 rms and 2e-12 at A = 48, in proportion to the
// major semi-axis A in the same barred units) then leave less than 1e-17, and tanh_mid rounds x
// once. The line at z = 6.5 + A / 100 is where nothing is seen of dz: against extended precision
// the weights 1 - tanh^2 there are off by 6.4e-17 rms (at most 1.13e-16), as with every cell in
// double precision (6.4e-17, 1.11e-16), for ellipses of 3 to 128 cells and ratios to 20; with
// the line at 6 + A / 400 at most 1.26e-16, and 1.5 % faster (2048 x 4096, 2048 ellipses).
// Only the cells within about three and a half of the interface are left to the FP64 pipe, a pass
// of 32 of them being as long as 3000 instructions of the FP32 pipe.
__device__ __forceinline__ float z_mid(float A) { return fmaf(0.01f, A, 6.5f); }
// (1 - m 2^-53) with the sign of -dist; the doubles below 1 are 2^-53 apart
__device__ __forceinline__ double tanh_of(long long m, float dist) {
  const long long b = 0x3ff0000000000000ll - m;
  return __longlong_as_double(dist < 0.f ? b : b | (long long)0x8000000000000000ull);
}

using eifdf::DF;
// product with a single
__device__ __forceinline__ DF df_mulf(DF x, float y) {
  const float p = x.hi * y;
  return eifdf::fast_sum(p, fmaf(x.lo, y, fmaf(x.hi, y, -p)));
}
// The distance of foot_d (positive outside) for offsets (x, y) in the first quadrant, from
// foot_f's (c, s), put back onto the unit circle as far as single precision goes; what is left
// of c^2 + s^2 - 1 is taken off the distance.
__device__ __forceinline__ DF dist_mid(DF a, DF b, float abf, float c, float s, DF x, DF y) {
  const float n = fmaf(-0.5f, fmaf(c, c, fmaf(s, s, -1.f)), 1.f);
  c *= n;
  s *= n;
  const DF vx = eifdf::df_add_nw(x, eifdf::df_neg(df_mulf(a, c))), vy = eifdf::df_add_nw(y, eifdf::df_neg(df_mulf(b, s)));
  const DF as = df_mulf(a, s), bc = df_mulf(b, c);
  const DF nw = eifdf::df_add_nw(eifdf::df_mul(vx, bc), eifdf::df_mul(vy, as));
  const DF w2 = eifdf::df_add_nw(eifdf::df_mul(as, as), eifdf::df_mul(bc, bc));
  const float p = c * c, q = s * s;
  const float rho = ((fmaxf(p, q) - 1.f) + fminf(p, q)) + (fmaf(c, c, -p) + fmaf(s, s, -q));
  // 1 / w = y (1 + e / 2), e = 1 - w^2 y^2
  const float y0 = rsqrtf(w2.hi);
  const DF t = df_mulf(df_mulf(w2, y0), y0);
  const float e = (1.f - t.hi) - t.lo;
  const float g = eifdf::df_add_nw(eifdf::df_mul(vy, bc), eifdf::df_neg(eifdf::df_mul(vx, as))).hi, iw2 = y0 * y0;
  const float K = fmaf(nw.hi * abf, iw2, w2.hi);
  const float corr = 0.5f * g * __fdividef(g, K) * abf * (y0 * iw2) + abf * y0 * (0.5f * rho);
  const DF d = df_mulf(nw, y0);
  return eifdf::fast_sum(d.hi, d.lo + fmaf(d.hi, 0.5f * e, corr));
}
// tanh z of z = |d| from 2 exp(-2 z) at multiples of 1 / MID_STEPS (tab, from MID_Z0 up), within
// 0.52 of the doubles' spacing below 1 at z = 6 and 0.51 from 6.5 on (half of it is the rounding)
constexpr int MID_STEPS = 128, MID_Z0 = 6, MID_Z1 = 20, MID_N = (MID_Z1 - MID_Z0) * MID_STEPS + 1;
__device__ __forceinline__ double tanh_mid(DF d, const float2 *__restrict__ tab) {
  const float zh = fmaxf(fminf(fabsf(d.hi), (float)MID_Z1), (float)MID_Z0), zl = d.hi < 0.f ? -d.lo : d.lo;
  const float kf = rintf((zh - (float)MID_Z0) * (float)MID_STEPS);
  const float2 E = __ldg(tab + (int)kf);
  // e = exp(-2 (z - z_k)) = (1 + y + y^2 / 2 + r)(1 + yl) with y exact. At z = 6 the spacing of
  // the doubles is 2^-37 of x, so that what is above 2^-25 of E is summed as pairs: E, E y,
  // E y^2 / 2 and then the square in x = E e - (E e)^2 / 2 + (E e)^3 / 4
  const float y = -2.f * (zh - fmaf(kf, 1.f / MID_STEPS, (float)MID_Z0)), yl = -2.f * zl;
  const float h = 0.5f * y, q = h * y, s = y + q;
  const float r = q * y * fmaf(y, fmaf(y, 1.f / 60.f, 1.f / 12.f), 1.f / 3.f) + fmaf(h, y, -q);
  const float p1 = E.x * y, p2 = E.x * q;
  const DF e1 = eifdf::fast_sum(E.x, p1), e2 = eifdf::fast_sum(e1.hi, p2);
  const float el = (e1.lo + e2.lo) +
                   ((fmaf(E.x, y, -p1) + fmaf(E.x, q, -p2)) + fmaf(E.x, fmaf(yl, s, yl) + r, fmaf(E.y, s, E.y)));
  const float eh = 0.5f * e2.hi, t = eh * e2.hi;
  const DF m = eifdf::fast_sum(e2.hi, -t);
  const float lo = m.lo + (el - (fmaf(eh, e2.hi, -t) + e2.hi * (el - 0.5f * t)));
  // in units of the doubles' spacing, rounded once
  constexpr float U = 9007199254740992.f;   // 2^53
  const float mu = m.hi * U, mr = rintf(mu);
  return tanh_of(__float2ll_rn(mr) + __float2int_rn(fmaf(lo, U, mu - mr)), d.hi);
}

// Cells far from the interface. With rho = sqrt((x/a)^2 + (y/b)^2) (the gauge of
// the ellipse, Lipschitz with constant 1/min(a,b)) the distance to the boundary is
// at least min(a,b) |rho - 1|, and at least r - max(a,b) outside / min(a,b) - r
// inside (r = |(x, y)|). When that bound times 2/h reaches the value at which
// tanh rounds to +-1 in the working precision, the weights are exactly those of
// the saturated tanh and the normal-foot iteration is not needed. row_chords
// turns these bounds into column ranges of a box row.
//
// double-precision tanh(2d) equals +-1 exactly for |2d| >= 20 (the correction
// 2/(exp(2|x|)+1) is below half an ulp of 1); with a margin for rounding of the bound
constexpr double FAR_CELLS_D = 10.5;
constexpr float FAR_CELLS_F = 5.f;

// auxiliary.c:11-17
__device__ __forceinline__ void loop_size(int lb, int ub, double h, double r, double gc, int &mn, int &mx) {
  mn = (int)(floor((gc - r) / h) - NEXTRA);
  mx = (int)(ceil((gc + r) / h) + NEXTRA);
  mn = mn < lb ? lb : mn;
  mx = mx > ub ? ub : mx;
}

using eifd::pmass;
using eifd::pmoi;

// sizes of the buffers the IBM kernels touch (used by EIF_CHECK builds)
struct Bounds {
  long long P, box, off, partial, wbuf, field, xc, yc;
  unsigned long long *rec;
};

// Per-particle single-precision parameters of the mixed-precision indicator,
// PF_WORDS words per particle (see k_boxes).
constexpr int PF_WORDS = 28;
enum { PF_A, PF_B, PF_CZ, PF_SZ, PF_KEX, PF_KEY, PF_RPM, PF_RPIM, PF_UX, PF_UY, PF_VZ, PF_GX, PF_I0,
       PF_J0, PF_GY = PF_J0 + 3,
       // quadratic form of the ellipse in the lab frame and the far-cell scales (row_chords)
       PF_AL = PF_GY + 3, PF_KA, PF_DE, PF_SO2, PF_SI2, PF_RO2 };
static_assert(PF_RO2 < PF_WORDS && PF_WORDS % 4 == 0, "per-particle parameter block");

struct BoxArgs {
  const double *P;
  int pcap, np, itot, jtot, use_increment;
  double dx, dy, ly, yf1;
  float *pf;                // PF_WORDS per particle, or null (double-precision form)
  double *pd;               // PD_WORDS per particle (double-precision form), or null
  double kb;                // BETA / h: scale of the barred lengths
  int *box, *nchunk;
  const int *bd_off_base;   // start of the buffer nchunk points into
  // inside the sub-iteration loop of a step graph: the loop's counter. In the first
  // sub-iteration the increments are zero, the positions are X and the boxes built at
  // X before the loop are still in place, so the box kernels return at once.
  const unsigned *iter;
  Bounds bd;
};

// Per-particle boxes of the three periodic images and their task counts, and the
// single-precision parameters. The double-precision work of one particle is a long
// chain (divisions, sincos) and the FP64 pipe takes a warp instruction at a time, so
// the work is split into eight parts run by different warps, each over 32
// particles: parts 0-2 the boxes of images -1, 0, +1 (the task count of image q - 1 goes to
// nchunk[q np + n]: a sum formed here would have to be cleared before, and the clearing node
// ahead of this kernel held every stage up for 4 us), parts 3-7 groups of parameters. One
// thread: particle n, part sub.
constexpr int BOX_PARTS = 8;
__device__ __forceinline__ void put_pair(float *p, double v) {
  const eifdf::DF t = eifdf::df_of(v);
  p[0] = t.hi;
  p[1] = t.lo;
}
__device__ __forceinline__ void box_part(const BoxArgs &a, int n, int sub) {
  const double *P = a.P;
  const int pc = a.pcap;
  bool on = n < a.np;
  if (on && !EIF_CHK(a.bd.rec, EIF_P_DY * pc + n, a.bd.P, 1)) on = false;
  int tasks = 0;
  if (on) {
    const double pa = P[EIF_P_A * pc + n], pb = P[EIF_P_B * pc + n];
    double px = P[EIF_P_X * pc + n], py = P[EIF_P_Y * pc + n];
    if (a.use_increment) {
      px = px + P[EIF_P_DX * pc + n];
      py = py + P[EIF_P_DY * pc + n];
    }
    const double r = fmax(pa, pb);
    float *q = a.pf ? a.pf + (size_t)PF_WORDS * n : nullptr;
    double *d = a.pd ? a.pd + (size_t)PD_WORDS * n : nullptr;
    float *df = reinterpret_cast<float *>(d + PD_F);
    if (sub < 3) {
      const int per = sub - 1;
      int imin, imax, jmin, jmax;
      loop_size(1, a.itot, a.dx, r, px, imin, imax);
      loop_size(1, a.jtot, a.dy, r, py + a.ly * per - a.yf1, jmin, jmax);
      if (EIF_CHK(a.bd.rec, 12 * n + 4 * sub + 3, a.bd.box, 2)) {
        int *bx = a.box + 12 * n + 4 * sub;
        bx[0] = imin; bx[1] = imax; bx[2] = jmin; bx[3] = jmax;
        if (imax >= imin && jmax >= jmin) tasks = (jmax - jmin + 1) * box_segs(imax - imin + 1);
      }
    } else if (q && sub == 3) {
      // orientation and the quadratic form rho^2 = al X^2 + 2 ka X Y + de Y^2 of the
      // ellipse for lab-frame offsets (X, Y)
      double az = P[EIF_P_AZ * pc + n];
      if (a.use_increment) az = az + P[EIF_P_DAZ * pc + n];
      double sz, cz;
      sincos(-az, &sz, &cz);
      q[PF_CZ] = (float)cz;
      q[PF_SZ] = (float)sz;
      q[PF_AL] = (float)(cz * cz / (pa * pa) + sz * sz / (pb * pb));
      q[PF_KA] = (float)(cz * sz * (1. / (pb * pb) - 1. / (pa * pa)));
      q[PF_DE] = (float)(sz * sz / (pa * pa) + cz * cz / (pb * pb));
    } else if (q && sub == 4) {
      q[PF_A] = (float)pa;
      q[PF_B] = (float)pb;
      q[PF_KEX] = (float)(pa * (1. - (pb / pa) * (pb / pa)));
      q[PF_KEY] = (float)(pb * (1. - (pa / pb) * (pa / pb)));
    } else if (q && sub == 5) {
      const double den = P[EIF_P_DEN * pc + n];
      q[PF_RPM] = (float)(1. / pmass(den, pa, pb));
      q[PF_RPIM] = (float)(1. / pmoi(den, pa, pb));
      q[PF_UX] = (float)P[EIF_P_UX * pc + n];
      q[PF_UY] = (float)P[EIF_P_UY * pc + n];
      q[PF_VZ] = (float)P[EIF_P_VZ * pc + n];
    } else if (q && sub == 6) {
      // cell centres XC(i) = (i - 1/2) dx, YC(j) = (j - 1/2) dy: offsets in grid units are
      // (i - i0) - gx and (j - j0[m]) - gy[m] for the periodic images m = -1, 0, +1
      const double sx = px / a.dx;
      const int i0 = (int)floor(sx);
      q[PF_GX] = (float)(sx - i0 + 0.5);
      q[PF_I0] = __int_as_float(i0);
      for (int m = 0; m < 3; m++) {
        const double sy = (py + a.ly * (m - 1)) / a.dy;
        const int j0 = (int)floor(sy);
        q[PF_J0 + m] = __int_as_float(j0);
        q[PF_GY + m] = (float)(sy - j0 + 0.5);
      }
    } else if (q && sub == 7) {
      // far-cell scales (row_chords)
      const double mn = fmin(pa, pb), mx = fmax(pa, pb);
      const double md = FAR_CELLS_F * fmin(a.dx, a.dy);
      const double so = 1. + md / mn, si = 1. - md / mn;
      q[PF_SO2] = (float)(so * so);
      q[PF_SI2] = si > 0. ? (float)(si * si) : -1.f;
      q[PF_RO2] = (float)((mx + md) * (mx + md));
    } else if (d && sub == 3) {
      double az = P[EIF_P_AZ * pc + n];
      if (a.use_increment) az = az + P[EIF_P_DAZ * pc + n];
      double sz, cz;
      sincos(-az, &sz, &cz);
      d[PD_CZ] = cz * a.kb;
      d[PD_SZ] = sz * a.kb;
      put_pair(df + PDF_PAIRS + 4, d[PD_CZ]);
      put_pair(df + PDF_PAIRS + 6, d[PD_SZ]);
      // the far cells' row bounds in single precision: the far distance (10.5 cells) exceeds
      // the saturation distance of tanh (9.53 cells) by far more than their rounding
      const float fa = eifd::d2f(pa), fb = eifd::d2f(pb), cf = eifd::d2f(cz), sf = eifd::d2f(sz);
      df[PDF_AL] = cf * cf / (fa * fa) + sf * sf / (fb * fb);
      df[PDF_KA] = cf * sf * (1.f / (fb * fb) - 1.f / (fa * fa));
      df[PDF_DE] = sf * sf / (fa * fa) + cf * cf / (fb * fb);
    } else if (d && sub == 4) {
      const double ba = pa * a.kb, bb = pb * a.kb;
      d[PD_A] = ba;
      d[PD_B] = bb;
      put_pair(df + PDF_PAIRS, ba);
      put_pair(df + PDF_PAIRS + 2, bb);
      const float fa = eifd::d2f(ba), fb = eifd::d2f(bb);
      df[PDF_A] = fa;
      df[PDF_B] = fb;
      df[PDF_KEX] = (fa - fb) * (fa + fb) / fa;
      df[PDF_KEY] = (fb - fa) * (fb + fa) / fb;
    } else if (d && sub == 5) {
      const double m = pmass(P[EIF_P_DEN * pc + n], pa, pb);
      d[PD_RPM] = 1. / m;
      d[PD_QM] = 0.25 * a.dx * a.dy / m;
    } else if (d && sub == 6) {
      const double m = pmoi(P[EIF_P_DEN * pc + n], pa, pb);
      d[PD_RPIM] = 1. / m;
      d[PD_QIM] = 0.25 * a.dx * a.dy / m;
    } else if (d && sub == 7) {
      d[PD_X] = px;
      d[PD_Y] = py;
      const float fa = eifd::d2f(pa), fb = eifd::d2f(pb), md = eifd::d2f(FAR_CELLS_D * fmin(a.dx, a.dy));
      const float mn = fminf(fa, fb), mx = fmaxf(fa, fb);
      const float so = 1.f + md / mn, si = 1.f - md / mn;
      df[PDF_SO2] = so * so;
      df[PDF_SI2] = si > 0.f ? si * si : -1.f;
      df[PDF_RO2] = (mx + md) * (mx + md);
    }
  }
  if (on && sub < 3 && EIF_CHK(a.bd.rec, (a.nchunk - a.bd_off_base) + sub * a.np + n, a.bd.off, 3))
    a.nchunk[sub * a.np + n] = tasks;
}

__device__ __forceinline__ eifdf::DF get_pair(const float *p) { return eifdf::DF{p[0], p[1]}; }

// The same for one particle by the first four warps of a CTA, into shared memory (bx: 12 ints,
// pf or pd: its parameter block), at X + dX in a sub-iteration: the values of box_part bit for
// bit. An FP64 instruction holds its scheduler 64 cycles whether one lane or all take part and
// whatever else the warp has ready, so the work is one instruction stream per scheduler: the
// angle and the quadratic form (six divisions in six lanes), the boxes' bounds (twelve lanes),
// the grid offsets (four); the words that do not change within a stage are copied from the
// blocks at X. About 45 FP64 instructions in the longest; all in one warp took 7400 cycles, and
// with a part of box_part per warp, one lane each, 30 000.
__device__ __forceinline__ void box_warps(const BoxArgs &a, int n, int part, int *bx, float *pf, double *pd) {
  const double *P = a.P;
  const int pc = a.pcap, lane = threadIdx.x & 31;
  if (part == 0) {
    const double pa = P[EIF_P_A * pc + n], pb = P[EIF_P_B * pc + n];
    double sz, cz;
    sincos(-(P[EIF_P_AZ * pc + n] + P[EIF_P_DAZ * pc + n]), &sz, &cz);
    if (pf) {
      // cz^2/pa^2, sz^2/pb^2, sz^2/pa^2, cz^2/pb^2, 1/pb^2, 1/pa^2
      const double x = lane == 0 || lane == 3 ? cz : (lane < 3 ? sz : 1.);
      const double y = lane == 0 || lane == 2 || lane == 5 ? pa : pb;
      const double v = x * x / (y * y), v1 = __shfl_down_sync(0xffffffffu, v, 1);
      // AL, -, DE, -, KA; CZ and SZ in the lanes between
      const double w = lane == 4 ? cz * sz * (v - v1) : (lane == 1 ? cz : (lane == 3 ? sz : v + v1));
      if (lane < 5) pf[lane == 0 ? PF_AL : (lane == 1 ? PF_CZ : (lane == 2 ? PF_DE : (lane == 3 ? PF_SZ : PF_KA)))] = (float)w;
    } else if (lane == 0) {
      const double bc = cz * a.kb, bs = sz * a.kb;
      pd[PD_CZ] = bc;
      pd[PD_SZ] = bs;
      float *df = reinterpret_cast<float *>(pd + PD_F);
      put_pair(df + PDF_PAIRS + 4, bc);
      put_pair(df + PDF_PAIRS + 6, bs);
      const float fa = eifd::d2f(pa), fb = eifd::d2f(pb), cf = eifd::d2f(cz), sf = eifd::d2f(sz);
      df[PDF_AL] = cf * cf / (fa * fa) + sf * sf / (fb * fb);
      df[PDF_KA] = cf * sf * (1.f / (fb * fb) - 1.f / (fa * fa));
      df[PDF_DE] = sf * sf / (fa * fa) + cf * cf / (fb * fb);
    }
  } else if (part == 1) {
    // lane: image lane / 4 - 1; imin, imax, jmin, jmax (loop_size)
    const double px = P[EIF_P_X * pc + n] + P[EIF_P_DX * pc + n], py = P[EIF_P_Y * pc + n] + P[EIF_P_DY * pc + n];
    const double r = fmax(P[EIF_P_A * pc + n], P[EIF_P_B * pc + n]);
    const bool row = lane & 2;
    const double gc = row ? py + a.ly * (double)(lane / 4 - 1) - a.yf1 : px;
    const double v = (gc + (lane & 1 ? r : -r)) / (row ? a.dy : a.dx);
    if (lane < 12) {
      const int lb = 1, ub = row ? a.jtot : a.itot;
      // floor, or ceil as -floor(-v)
      const double e = floor(lane & 1 ? -v : v);
      int w;
      if (lane & 1) {
        w = (int)(-e + NEXTRA);
        w = w > ub ? ub : w;
      } else {
        w = (int)(e - NEXTRA);
        w = w < lb ? lb : w;
      }
      bx[lane] = w;
    }
  } else if (part == 2) {
    const double px = P[EIF_P_X * pc + n] + P[EIF_P_DX * pc + n], py = P[EIF_P_Y * pc + n] + P[EIF_P_DY * pc + n];
    if (pf) {
      const double v = (lane == 0 ? px : py + a.ly * (double)(lane - 2)) / (lane == 0 ? a.dx : a.dy);
      const int i0 = (int)floor(v);
      const float g = (float)(v - i0 + 0.5);
      if (lane < 4) {
        pf[lane == 0 ? PF_I0 : PF_J0 + (lane - 1)] = __int_as_float(i0);
        pf[lane == 0 ? PF_GX : PF_GY + (lane - 1)] = g;
      }
    } else if (lane == 0) {
      pd[PD_X] = px;
      pd[PD_Y] = py;
    }
  } else if (pf) {
    const float *c = a.pf + (size_t)PF_WORDS * n;
    constexpr unsigned keep = 1u << PF_A | 1u << PF_B | 1u << PF_KEX | 1u << PF_KEY | 1u << PF_RPM | 1u << PF_RPIM |
                              1u << PF_UX | 1u << PF_UY | 1u << PF_VZ | 1u << PF_SO2 | 1u << PF_SI2 | 1u << PF_RO2;
    if ((keep >> lane) & 1u) pf[lane] = c[lane];
  } else {
    // everything but the first words and those of the quadratic form
    const double *c = a.pd + (size_t)PD_WORDS * n;
    if (lane >= PD_A && lane < PD_F) pd[lane] = c[lane];
    float *df = reinterpret_cast<float *>(pd + PD_F);
    if (lane >= PDF_SO2 && lane < PDF_PAIRS + 4) df[lane] = reinterpret_cast<const float *>(c + PD_F)[lane];
  }
}
__device__ __forceinline__ int box_tasks(const int *bx) {
  int t = 0;
#pragma unroll
  for (int q = 0; q < 3; q++) {
    const int w = bx[4 * q + 1] - bx[4 * q] + 1, h = bx[4 * q + 3] - bx[4 * q + 2] + 1;
    if (w > 0 && h > 0) t += h * box_segs(w);
  }
  return t;
}

// A particle's tasks: image by image, row by row, segment by segment.
struct RowTask {
  int img, j, ib, ie;   // image -1..1, row, first and last column of the segment
};
// one image's box (columns bi0..bi1, rows bj0..bj1): true when task r lies in it,
// otherwise r is reduced by the image's task count
__device__ __forceinline__ bool row_task_in(int4 b, int img, int &r, RowTask &t) {
  const int w = b.y - b.x + 1, h = b.w - b.z + 1;
  if (w <= 0 || h <= 0) return false;
  const int segs = box_segs(w);
  const int cnt = h * segs;
  if (r >= cnt) {
    r -= cnt;
    return false;
  }
  const int row = segs == 1 ? r : r / segs;
  const int seg = r - row * segs;
  t.img = img;
  t.j = b.z + row;
  t.ib = b.x + seg * CHUNK;
  t.ie = min(t.ib + CHUNK - 1, b.y);
  return true;
}
// task r of a particle whose image boxes are bm, b0, bp (images -1, 0, +1)
__device__ __forceinline__ bool row_task(int4 bm, int4 b0, int4 bp, int r, RowTask &t) {
  return row_task_in(bm, -1, r, t) || row_task_in(b0, 0, r, t) || row_task_in(bp, 1, r, t);
}

// The same table with the task offsets formed in the same kernel, for particle
// counts up to TT_MAX_NP: every block sums the task counts of the particles before
// its own (a few thousand integers from L2), then each warp writes its particle's
// offset and table entries. Replaces k_scan + k_task_table (one launch and one
// single-block pass fewer on the path of every box build). One block of TT_WARPS
// warps: particles block * TT_WARPS ... cnt: the counts of the three images, np each.
constexpr int TT_WARPS = 8;
constexpr int TT_MAX_NP = 8192;
__device__ __forceinline__ void task_table_block(const int *box, const int *cnt, int *off, int4 *tdesc, int np,
                                                 const Bounds &bd, int cap, int block) {
  __shared__ int red[TT_WARPS], wcnt[TT_WARPS];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int n0 = block * TT_WARPS;
  int s = 0;
  for (int q = threadIdx.x; q < n0; q += blockDim.x) s += cnt[q] + cnt[np + q] + cnt[2 * np + q];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  const int n = n0 + w;
  const int my = n < np ? cnt[n] + cnt[np + n] + cnt[2 * np + n] : 0;
  if (lane == 0) {
    red[w] = s;
    wcnt[w] = my;
  }
  __syncthreads();
  int c0 = 0;
#pragma unroll
  for (int q = 0; q < TT_WARPS; q++) c0 += red[q] + (q < w ? wcnt[q] : 0);
  if (n >= np) return;
  if (lane == 0) {
    if (EIF_CHK(bd.rec, n, bd.off, 5)) off[n] = c0;
    if (n == np - 1 && EIF_CHK(bd.rec, np, bd.off, 6)) off[np] = c0 + my;
  }
  const int4 *b4 = reinterpret_cast<const int4 *>(box + 12 * n);
  const int4 bA = b4[0], bB = b4[1], bC = b4[2];
  for (int c = c0 + lane; c < c0 + my; c += 32) {
    RowTask t;
    int4 d = make_int4(-1, 0, 0, 0);
    if (row_task(bA, bB, bC, c - c0, t)) d = make_int4(n, t.j, t.ib, t.ie * 4 + t.img + 1);
    if (EIF_CHK(bd.rec, c, cap, 59)) tdesc[c] = d;
  }
}
__device__ __forceinline__ bool task_of(int4 d, int np, RowTask &t) {
  t.j = d.y;
  t.ib = d.z;
  t.ie = d.w >> 2;
  t.img = (d.w & 3) - 1;
  return d.x >= 0 && d.x < np;
}

// The far-cell bounds above along one row, as ranges of the lab-frame offset
// X from the centre at the row's offset Y: cells outside (olo, ohi) are far
// outside (rho >= so or r >= ro), cells in [ilo, ihi] are far inside (rho <= si;
// the disc r <= mn - md lies inside that ellipse). rho^2 = al X^2 + 2 ka X Y + de Y^2.
template <typename T>
__device__ __forceinline__ void row_chords(T al, T ka, T de, T so2, T si2, T ro2, T Y, T &olo, T &ohi, T &ilo,
                                           T &ihi) {
  const T big = T(1e30);
  olo = big; ohi = -big; ilo = big; ihi = -big;
  const T bY = ka * Y;
  const T Do = bY * bY - al * (de * Y * Y - so2);
  const T c2 = ro2 - Y * Y;
  if (Do > T(0) && c2 > T(0)) {
    const T sq = sqrt(Do), xc = sqrt(c2);
    olo = fmax((-bY - sq) / al, -xc);
    ohi = fmin((-bY + sq) / al, xc);
  }
  if (si2 > T(0)) {
    const T Di = bY * bY - al * (de * Y * Y - si2);
    if (Di >= T(0)) {
      const T sq = sqrt(Di);
      ilo = (-bY - sq) / al;
      ihi = (-bY + sq) / al;
    }
  }
}

// The last indicator evaluation of the mixed form inside a sub-iteration loop (at the
// positions X + dX of a sub-iteration after the first): its weights, one per task slot,
// and the particles' geometry parameters (the PF_WORDS block), boxes and first task,
// with a flag set once a complete evaluation is stored. The loop stops when the
// increments have settled, so the positions X of the next stage differ from those by
// the last change of the increments (below 1e-8 dt in velocity); the single-precision
// geometry of nearly every particle is then bitwise the stored one, and so are its
// weights, which the next stage's first evaluation copies instead of recomputing.
struct WeightMemo {
  float *w;
  float *pf;
  int *box, *off;
  int *valid;
};
// geometry words of the per-particle parameter block (everything but the mass, inertia
// and velocity words PF_RPM .. PF_VZ); with the 12 box bounds, 32 words: one per lane
__device__ __forceinline__ int memo_word(int lane) { return lane < 6 ? lane : lane + 5; }

struct WorkArgs {
  const double *P;
  const double *ux, *uy, *xc, *yc, *dt;
  // mixed form: ux, uy rounded to float (eifd::d2f), kept with them by the kernels that
  // write the velocities; the single-precision bodies read these
  const float *uxf, *uyf;
  const int *box, *off;
  double *partial;   // 3 per chunk
  double2 *wbuf;     // CHUNK per chunk (exchange only)
  int pcap, np, ld, mode, cn;   // mode 0: inertia (cn), 1: exchange
  double dx, dy, ly, h;
  const float *pf;       // per-particle single-precision parameters (mixed form)
  const double *pd;      // per-particle parameters (double-precision form)
  const double2 *tanh_tab;   // tanh_tab's values (double-precision form)
  const float2 *mid_tab;     // tanh_mid's
  const int4 *tdesc;     // task table (k_task_table)
  const float *coef;     // single-precision dt products; [9] = 1/dt
  float rh_f, dx_f, dy_f, dxdy_f;
  // Indicator weights of the cells at the positions X are kept in wcache (one per
  // task slot, like wbuf) and reused by the evaluations that see the same
  // geometry: wmode 0 computes, 1 computes and stores, 2 loads; when iter is set
  // (the sub-iteration loop of a step graph) the kernel loads in the first
  // sub-iteration (*iter == 0, increments still zero) and computes afterwards.
  void *wcache;
  int wmode;
  const unsigned *iter;
  int weights_only;   // exchange (double precision): the cell contributions are the weights (w, w)
  // box cells whose geometry is evaluated and, of those, the near cells that run the
  // normal-foot iteration, added to count[0] and count[1], and the tasks whose weights
  // come from the memo, added to count[2] (null: not counted)
  unsigned long long *count;
  // mixed form: memo_mode 1 (the stage start, ibm_memo_f_tasks) takes the weights of a
  // task from the memo when its particle's geometry and boxes are the memo's; 2
  // (ibm_work_f_tasks in the loops) stores computed weights in it
  WeightMemo memo;
  int memo_mode;
  // the stage start of the mixed form (ibm_memo_f_tasks): miss[0] counts the tasks the
  // memo did not serve, miss[1 ..] lists them; with `only` set, ibm_work_f_tasks
  // evaluates just the tasks listed there (same layout)
  int *miss;
  const int *only;
  Bounds bd;
};

// The tasks of one particle for the persistent sub-iteration kernel, which forms the boxes and
// parameters of the particle at hand in shared memory instead of tables over all particles:
// tasks r = 0 .. of the boxes, numbered base + r in the scratch buffers. box null: the tasks of
// the table up to number `total`.
struct OneParticle {
  const int4 *box;      // the three images' boxes, or null
  const float *pf;
  const double *pd;
  int n, base, total;
};
__device__ __forceinline__ int4 task_desc(const OneParticle &o, int r) {
  RowTask t;
  return row_task(o.box[0], o.box[1], o.box[2], r, t) ? make_int4(o.n, t.j, t.ib, t.ie * 4 + t.img + 1)
                                                      : make_int4(-1, 0, 0, 0);
}

// Sums of three values over the warp, in 6 additions instead of 15: in each of the first
// two steps the two halves of a group of lanes keep different values. The additions pair the
// same lanes as warp_sum's. The sums are in lane 0 (v0), 16 (v1) and 8 (v2).
template <typename T>
__device__ __forceinline__ T warp_sum3(T v0, T v1, T v2, int lane) {
  const bool h16 = lane & 16, h8 = lane & 8;
  const T o = __shfl_xor_sync(0xffffffffu, h16 ? v0 : v1, 16);
  T v = (h16 ? v1 : v0) + o;
  v2 += __shfl_xor_sync(0xffffffffu, v2, 16);
  // lanes 0-7, 16-23 go on with v, lanes 8-15, 24-31 with v2
  const T q = __shfl_xor_sync(0xffffffffu, h8 ? v : v2, 8);
  v = (h8 ? v2 : v) + q;
#pragma unroll
  for (int d = 4; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
  return v;
}

// One warp per row task: indicator weights, partial sums, and (for the exchange)
// per-cell field contributions. The warp runs the tasks first, first + stride, ...
// with the weight mode wmode, WORK_ROWS at a time: the cells of theirs that need double
// precision are evaluated together, packed onto the lanes.
// Bound by the FP64 pipe: an instruction of a warp holds its scheduler 64 cycles. About 27 FP64
// instructions per task for the sums and 48 for each pass of 32 cells next to the interface,
// of which a task has 15 or so. Not inlined, and every product that could be fused is written
// as fma: the stage kernel gives the bits of the stand-alone kernel. Kept short (loops not
// unrolled, the guards' records out of line): with 30 KB of straight code the warps waited for
// instructions more than half of the time.
__device__ __noinline__ bool work_chk_fail(unsigned long long *rec, long long idx, long long bound, int tag) {
  return EIF_CHK(rec, idx, bound, tag);
}
__device__ __forceinline__ void prefetch_l1(const double *p) {
  asm volatile("prefetch.global.L1 [%0];" : : "l"(p));
}
#define WORK_CHK(rec, idx, bound, tag) \
  ((unsigned long long)(idx) < (unsigned long long)(bound) || work_chk_fail((rec), (long long)(idx), (long long)(bound), (tag)))
constexpr int WORK_ROWS = 4;
struct alignas(16) WorkSlots {     // shared memory of a warp (or a WorkSlotsF)
  double th[WORK_ROWS][CHUNK];        // weights; before pass 3 the feet (c, s) of its cells
  double px[WORK_ROWS], Y[WORK_ROWS];
  const double *pd[WORK_ROWS];
  int ib[WORK_ROWS];
  unsigned char near[CHUNK];          // cells of a row for pass 2
  unsigned char list[WORK_ROWS * CHUNK];   // row * CHUNK + cell for pass 3
};
template <bool NC>
__device__ __noinline__ void ibm_work_tasks(const WorkArgs &a, int wmode, int first, int stride, WorkSlots &ws,
                                            const OneParticle *one) {
  const int lane = threadIdx.x & 31;
  const int total = one ? one->total : (WORK_CHK(a.bd.rec, a.np, a.bd.off, 10) ? ldro<NC>(a.off + a.np) : 0);
  const bool own = one && one->box;
  // factor of the exchange's sums (exchange.c:61-76) over the particle's PD_QM, PD_QIM
  const double xscale = a.mode == 0 ? 1. : -4. / __ldg(a.dt);
  const int pc = a.pcap, ld = a.ld;
  double *wcache = static_cast<double *>(a.wcache);
  // task k: its number c, descriptor and row; false when it is to be skipped
  auto task_at = [&](int k, int &c, int &n, RowTask &t, bool &task) {
    c = own ? one->base + k : k;
    if (!WORK_CHK(a.bd.rec, c, a.bd.partial / 3, 21)) return false;
    const int4 dsc = own ? task_desc(*one, k) : ldro<NC>(a.tdesc + c);
    n = dsc.x;
    if (!WORK_CHK(a.bd.rec, n, a.np, 11)) return false;
    if (!WORK_CHK(a.bd.rec, EIF_P_VZ * pc + n, a.bd.P, 13)) return false;
    task = task_of(dsc, a.np, t) && WORK_CHK(a.bd.rec, t.j, a.bd.yc - 1, 15);
    if (!task) {
      t.img = 0;
      t.j = t.ib = 1;
      t.ie = 0;
    }
    return true;
  };
  auto centre_y = [&](const double *pd, int img) {
    return ldro<NC>(pd + PD_Y) + (img == 0 ? 0. : (img > 0 ? a.ly : -a.ly));
  };
  for (int k0 = first; k0 < total; k0 += WORK_ROWS * stride) {
    const int nq = min(WORK_ROWS, (total - k0 + stride - 1) / stride);
    if (wmode != 2) {
      int ndbl = 0;
      for (int q = 0; q < nq; q++) {
        int c, n;
        RowTask t;
        bool task;
        if (!task_at(k0 + q * stride, c, n, t, task)) continue;
        const double *pd = own ? one->pd : a.pd + (size_t)PD_WORDS * n;
        const float *pdf = reinterpret_cast<const float *>(pd + PD_F);
        const double px = ldro<NC>(pd + PD_X);
        const double Y = __ldg(a.yc + t.j) - centre_y(pd, t.img);
        // the columns are dx apart
        const DF X0 = eifdf::df_of(__ldg(a.xc + t.ib) - px), dxp = eifdf::df_of(a.dx), Yp = eifdf::df_of(Y);
        if (lane == 0) {
          ws.px[q] = px;
          ws.Y[q] = Y;
          ws.pd[q] = pd;
          ws.ib[q] = t.ib;
        }
        // pass 1: cells of the row, far cells settled (tanh +-1), the near ones listed
        int nnear = 0;
        float olo, ohi, ilo, ihi;
        row_chords(ldro<NC>(pdf + PDF_AL), ldro<NC>(pdf + PDF_KA), ldro<NC>(pdf + PDF_DE), ldro<NC>(pdf + PDF_SO2),
                   ldro<NC>(pdf + PDF_SI2), ldro<NC>(pdf + PDF_RO2), Yp.hi, olo, ohi, ilo, ihi);
#pragma unroll 1
        for (int half = 0; half < CHUNK / 32; half++) {
          const int at = half * 32 + lane;
          const bool in = t.ib + at <= t.ie;
          const float Xf = fmaf((float)at, dxp.hi, X0.hi);
          // reference sign convention: +1 inside (auxiliary.c:36-38)
          const int side = !(Xf > olo && Xf < ohi) ? -1 : ((Xf >= ilo && Xf <= ihi) ? 1 : 0);
          const bool near = in && side == 0;
          if (in) {
            // the sums' velocities, needed some thousand cycles later
            prefetch_l1(a.ux + t.j * ld + t.ib + at);
            prefetch_l1(a.uy + t.j * ld + t.ib + at);
            prefetch_l1(a.uy + (t.j + 1) * ld + t.ib + at);
          }
          ws.th[q][at] = in ? (side > 0 ? 1. : (side < 0 ? -1. : 0.)) : 0.;
          const unsigned mask = __ballot_sync(0xffffffffu, near);
          if (near) ws.near[nnear + __popc(mask & ((1u << lane) - 1u))] = (unsigned char)at;
          nnear += __popc(mask);
        }
        if (a.count && lane == 0) {
          atomicAdd(a.count, (unsigned long long)max(0, min(CHUNK, t.ie - t.ib + 1)));
          atomicAdd(a.count + 1, (unsigned long long)nnear);
        }
        __syncwarp();
        if (nnear == 0) continue;
        // pass 2: the near cells packed onto consecutive lanes, on the FP32 pipe; the cells it
        // settles get their weights, the others are listed for pass 3 with their feet
        EllF ef;
        ef.a = ldro<NC>(pdf + PDF_A); ef.b = ldro<NC>(pdf + PDF_B);
        ef.kex = ldro<NC>(pdf + PDF_KEX); ef.key = ldro<NC>(pdf + PDF_KEY);
        ef.cz = ef.sz = 0.f;
        const DF ap = get_pair(pdf + PDF_PAIRS), bp = get_pair(pdf + PDF_PAIRS + 2), czp = get_pair(pdf + PDF_PAIRS + 4),
                 szp = get_pair(pdf + PDF_PAIRS + 6);
        const DF szY = eifdf::df_mul(szp, Yp), czY = eifdf::df_mul(czp, Yp);
        const float zm = z_mid(fmaxf(ef.a, ef.b));
        for (int base = 0; base < nnear; base += 32) {
          const int k = base + lane;
          bool dbl = false;
          int at = 0;
          float c0 = 0.f, s0 = 0.f;
          if (k < nnear) {
            at = ws.near[k];
            // offset X0 + at dx, then the body frame
            const float f = (float)at, p = f * dxp.hi;
            const DF sm = eifdf::two_sum(X0.hi, p);
            const DF X = eifdf::fast_sum(sm.hi, sm.lo + (fmaf(f, dxp.hi, -p) + fmaf(f, dxp.lo, X0.lo)));
            DF x = eifdf::df_add_nw(eifdf::df_mul(czp, X), eifdf::df_neg(szY));
            DF y = eifdf::df_add_nw(eifdf::df_mul(szp, X), czY);
            if (x.hi < 0.f) x = eifdf::df_neg(x);
            if (y.hi < 0.f) y = eifdf::df_neg(y);
            float d;
            const float dist = foot_f(ef, x.hi, y.hi, c0, s0, d);
            dbl = !(fabsf(dist) >= zm && fabsf(d) < 1.e-3f);
            if (!dbl) ws.th[q][at] = tanh_mid(dist_mid(ap, bp, ef.a * ef.b, c0, s0, x, y), a.mid_tab);
          }
          const unsigned mask = __ballot_sync(0xffffffffu, dbl);
          if (dbl) {
            ws.th[q][at] = __hiloint2double(__float_as_int(c0), __float_as_int(s0));
            ws.list[ndbl + __popc(mask & ((1u << lane) - 1u))] = (unsigned char)(q * CHUNK + at);
          }
          ndbl += __popc(mask);
        }
        __syncwarp();
      }
      __syncwarp();
      // pass 3: double precision
      for (int k = lane; k < ndbl; k += 32) {
        const int e = ws.list[k], q = e / CHUNK, at = e % CHUNK;
        const double *pd = ws.pd[q];
        const double cs = ws.th[q][at];
        const double cz = ldro<NC>(pd + PD_CZ), sz = ldro<NC>(pd + PD_SZ);
        const double X = __ldg(a.xc + ws.ib[q] + at) - ws.px[q], Y = ws.Y[q];
        const float *pdf = reinterpret_cast<const float *>(pd + PD_F);
        double nx, ny;
        ws.th[q][at] = indicator_d<false>(ldro<NC>(pd + PD_A), ldro<NC>(pd + PD_B), ldro<NC>(pdf + PDF_A) * ldro<NC>(pdf + PDF_B),
                                          __int_as_float(__double2hiint(cs)), __int_as_float(__double2loint(cs)),
                                          fma(cz, X, -(sz * Y)), fma(sz, X, cz * Y), a.tanh_tab, nx, ny);
      }
      __syncwarp();
    }
    // the sums
    for (int q = 0; q < nq; q++) {
      int c, n;
      RowTask t;
      bool task;
      if (!task_at(k0 + q * stride, c, n, t, task)) continue;
      const double *pd = own ? one->pd : a.pd + (size_t)PD_WORDS * n;
      const double px = ldro<NC>(pd + PD_X);
      const int j = t.j;
      const double Y = __ldg(a.yc + j) - centre_y(pd, t.img);
      const double pux = ldro<NC>(a.P + EIF_P_UX * pc + n), puy = ldro<NC>(a.P + EIF_P_UY * pc + n),
                   pvz = ldro<NC>(a.P + EIF_P_VZ * pc + n);
      double s0 = 0., s1 = 0., s2 = 0.;
#pragma unroll 1
      for (int half = 0; half < CHUNK / 32; half++) {
        const int at = half * 32 + lane, i = t.ib + at;
        // nothing but the stored weights and contributions of a short row's second half
        if (half > 0 && t.ib + 32 > t.ie && a.mode == 0 && wmode != 1) break;
        const long long slot = (long long)c * CHUNK + at;
        bool in = i <= t.ie;
        if (in) {
          in = WORK_CHK(a.bd.rec, i, a.bd.xc - 1, 14) && WORK_CHK(a.bd.rec, j * ld + i, a.bd.field, 16) &&
               WORK_CHK(a.bd.rec, (j + 1) * ld + i, a.bd.field, 17) && WORK_CHK(a.bd.rec, j * ld + (i - 1), a.bd.field, 18);
        }
        double th = 0.;
        if (wmode == 2) {
          // weights of the same geometry from an earlier evaluation
          if (in) in = WORK_CHK(a.bd.rec, slot, a.bd.wbuf, 22);
          if (in) th = wcache[slot];
        } else {
          if (in) th = ws.th[q][at];
          if (wmode == 1 && WORK_CHK(a.bd.rec, slot, a.bd.wbuf, 23)) wcache[slot] = th;
        }
        double2 contrib = make_double2(0., 0.);
        // cells of weight exactly zero (inertia: far outside; exchange: any far cell) are
        // skipped; compared as integers, the FP64 pipe does comparisons too
        const int hi = __double2hiint(th), lo = __double2loint(th);
        const bool zero = (a.mode == 0 ? hi : hi | (int)0x80000000) == (int)0xbff00000 && lo == 0;
        if (in && !zero) {
          const double X = __ldg(a.xc + i) - px;
          const double us = __ldg(a.ux + j * ld + (i - 1)) + __ldg(a.ux + j * ld + i);
          const double vs = __ldg(a.uy + j * ld + i) + __ldg(a.uy + (j + 1) * ld + i);
          if (a.mode == 0) {
            // inertia.c:51-59: the constant factors, and the row's Y in the moment, after the sum
            const double w = 1. + th, wv = w * vs;
            s0 = fma(w, us, s0);
            s1 += wv;
            s2 = fma(X, wv, s2);
          } else {
            // exchange.c:61-76 (BETA / 2 = 1)
            const double w = fma(-th, th, 1.);
            const double gx = w * fma(-0.5, us, fma(-pvz, Y, pux));
            const double gy = w * fma(-0.5, vs, fma(pvz, X, puy));
            contrib = a.weights_only ? make_double2(w, w) : make_double2(gx, gy);
            s0 += gx;
            s1 += gy;
            s2 = fma(X, gy, s2);
          }
        }
        if (a.mode == 1 && WORK_CHK(a.bd.rec, slot, a.bd.wbuf, 19)) a.wbuf[slot] = contrib;
      }
      // sum_x, sum_y in lanes 0 and 16, the moment sum X f_y in lane 8, which takes Y sum_x off it
      double v = warp_sum3(s0, s1, s2, lane);
      const double sx = __shfl_sync(0xffffffffu, v, 0);
      const int slot = lane == 0 ? 0 : (lane == 16 ? 1 : (lane == 8 ? 2 : -1));
      if (slot >= 0 && WORK_CHK(a.bd.rec, 3LL * c + 2, a.bd.partial, 20)) {
        if (slot == 2) v = fma(-Y, sx, v);
        const double f = ldro<NC>(pd + (slot == 2 ? PD_QIM : PD_QM));
        a.partial[3 * (size_t)c + slot] = a.mode == 0 ? v * f : v * (f * xscale);
      }
    }
    __syncwarp();
  }
}

// ---------------------------------------------------------------------------
// Single-precision indicator (EIF_PREC_MIXED). Cell offsets from the particle
// centre are formed in grid units, (x - px)/dx = (i - i0) - g with the integer
// i0 and the fraction g computed once per chunk in double precision, so the
// per-cell arithmetic is single precision without cancellation. The normal
// foot iteration is normal_t_f (above).

// tanh(2 d / h) of the signed distance (positive inside), d from the body-frame
// offset; tanh through one exponential, accurate to a few units of 1e-7 absolute
__device__ __forceinline__ float indicator_f(const EllF &e, float x_, float y_, float rh) {
  const float f0 = 1.f - (x_ / e.a) * (x_ / e.a) - (y_ / e.b) * (y_ / e.b);
  const float t = normal_t_f(e, x_, y_);
  float st, ct;
  sincosf(t, &st, &ct);
  const float dxx = e.a * ct - x_, dyy = e.b * st - y_;
  // |2d/h|; tanh is 1 in single precision beyond 10, the clamp keeps exp finite
  const float z = fminf(2.f * sqrtf(dxx * dxx + dyy * dyy) * rh, 20.f);
  const float ez = __expf(2.f * z);
  const float th = __fdividef(ez - 1.f, ez + 1.f);
  return f0 > 0.f ? th : -th;
}

// One cell's contributions to the inertia integrals (inertia.c:9-70) in single precision,
// with every rounding explicit: the bodies that form these sums (the full evaluation, the
// memo-served stage start, the cached-weight sums) then give the same bits in whatever
// kernel they are compiled, whichever products the compiler would fuse there.
__device__ __forceinline__ void inertia_cell_f(float th, float X, float Y, float uxs, float uys, float dxdy,
                                               float rpm, float rpim, float &s0, float &s1, float &s2) {
  const float w = __fmul_rn(0.5f, __fadd_rn(1.f, th));
  const float valx = __fmul_rn(__fmul_rn(__fmul_rn(w, 0.5f), uxs), dxdy);
  const float valy = __fmul_rn(__fmul_rn(__fmul_rn(w, 0.5f), uys), dxdy);
  s0 = __fmaf_rn(valx, rpm, s0);
  s1 = __fmaf_rn(valy, rpm, s1);
  s2 = __fmaf_rn(__fmaf_rn(X, valy, __fmul_rn(-Y, valx)), rpim, s2);
}

// The bounds of a row's accesses, checked once for the row: cells ib - 1 .. ie of rows j and
// j + 1, and the CHUNK slots of task c in a buffer of n. (A check of every cell's was two
// compares and a divergence point each: 95 us of a full evaluation with 2048 ellipses, by the
// row 88.)
__device__ __forceinline__ bool row_cells_in(const Bounds &bd, const RowTask &t, int ld, int tag) {
  return EIF_CHK(bd.rec, (long long)t.j * ld + t.ib - 1, bd.field, tag) &&
         EIF_CHK(bd.rec, (long long)(t.j + 1) * ld + t.ie, bd.field, tag + 1);
}
__device__ __forceinline__ bool row_slots_in(const Bounds &bd, long long c, long long n, int tag) {
  return EIF_CHK(bd.rec, c * CHUNK, n, tag) && EIF_CHK(bd.rec, c * CHUNK + CHUNK - 1, n, tag);
}

// single-precision partial sums of task c, reduced per particle by k_chunk_reduce_f
__device__ __forceinline__ void store_sums_f(const WorkArgs &a, int c, float s0, float s1, float s2, int lane, int tag) {
  const float sum = warp_sum3(s0, s1, s2, lane);
  const int slot = lane == 0 ? 0 : (lane == 16 ? 1 : (lane == 8 ? 2 : -1));
  if (slot >= 0 && EIF_CHK(a.bd.rec, 3LL * c + 2, a.bd.partial, tag))
    reinterpret_cast<float *>(a.partial)[3 * (size_t)c + slot] = sum;
}
struct RowF {
  float4 ell;      // a, b, kex, key
  float4 geo;      // cz, sz, Y, gx
  float4 chords;   // row_chords' olo, ohi, ilo, ihi
  float4 par;      // rpm, rpim, ux, uy
  int4 cells;      // i0, first and last column, row
  float vz;
  int c;           // task number, or -1: skipped
};
struct WorkSlotsF {   // shared memory of a warp
  float th[WORK_ROWS][CHUNK];              // weights
  RowF row[WORK_ROWS];
  unsigned char list[WORK_ROWS * CHUNK];   // row * CHUNK + cell of the near cells
};
static_assert(sizeof(WorkSlotsF) <= sizeof(WorkSlots) && alignof(WorkSlotsF) <= alignof(WorkSlots),
              "the persistent kernel has one array for both");
// One warp per row task, single precision, WORK_ROWS rows at a time as in ibm_work_tasks (ONE:
// the tasks of one particle). Bound by instruction issue: the foot iteration of the near cells,
// and what a row needs before it (descriptor, parameters, the chords' roots and divisions). One
// lane prepares a row, four rows at once, instead of every lane the same row; the near cells of
// the four rows, about 25 a row, are packed onto the lanes together. 2048 ellipses of 12 to 25
// cells: 108 -> 95 us (88 with the bounds checked by the row), 63-70 % of the issue slots; the
// persistent kernel of 12 suspensions 611 -> 575 us a stage (24 ellipses alone, a row to a warp:
// 1 % slower). The products of x_, y_ are written out with the roundings that every form of this
// body has had.
template <bool NC, bool ONE = false>
__device__ __forceinline__ void ibm_work_f_tasks(const WorkArgs &a, int wmode, int first, int stride, WorkSlotsF &ws,
                                                 const OneParticle *one = nullptr) {
  const int lane = threadIdx.x & 31;
  // all tasks, or (with a.only) the listed ones: task number c of list entry k
  const int total = ONE ? one->total
                        : (a.only ? (int)min((long long)ldro<NC>(a.only), (long long)(a.bd.partial / 3))
                                  : (EIF_CHK(a.bd.rec, a.np, a.bd.off, 50) ? ldro<NC>(a.off + a.np) : 0));
  const float rh = a.rh_f, dxf = a.dx_f, dyf = a.dy_f, dxdy = a.dxdy_f;
  const float rdtv = a.mode == 1 ? __ldg(a.coef + 9) : 0.f;
  const int ld = a.ld;
  float2 *wb = reinterpret_cast<float2 *>(a.wbuf);
  float *wcache = static_cast<float *>(a.wcache);
  if (first >= total) return;
  // the warp's tasks in groups of nearly the same size
  int left = (total - first + stride - 1) / stride, rows = left;
  if (left > WORK_ROWS) {
    const int groups = (left + WORK_ROWS - 1) / WORK_ROWS;
    rows = (left + groups - 1) / groups;
  }
  // lane q: task number and descriptor of row q of the group from k0 on
  auto fetch = [&](int k0, int &c, int4 &dsc) {
    const int k = k0 + lane * stride;
    c = -1;
    dsc = make_int4(-1, 0, 0, 0);
    if (lane < rows && k < total) {
      c = ONE ? one->base + k : (a.only ? ldro<NC>(a.only + 1 + k) : k);
      if (!EIF_CHK(a.bd.rec, c, a.bd.partial / 3, 51)) c = -1;
      else if constexpr (ONE) dsc = task_desc(*one, k);
      else dsc = ldro<NC>(a.tdesc + c);
    }
  };
  int nxt_c;
  int4 nxt;
  fetch(first, nxt_c, nxt);
  // a row's field values
  struct Vel {
    float uw[CHUNK / 32], ue[CHUNK / 32], vs[CHUNK / 32], vn[CHUNK / 32];
    bool in[CHUNK / 32];
  };
  auto load = [&](int q, Vel &v) {
    const RowF &r = ws.row[q];
    const int4 ce = r.cells;
    const int j = ce.w;
#pragma unroll
    for (int half = 0; half < CHUNK / 32; half++) {
      const int i = ce.y + half * 32 + lane;
      const bool in = r.c >= 0 && i <= ce.z;
      v.in[half] = in;
      v.uw[half] = v.ue[half] = v.vs[half] = v.vn[half] = 0.f;
      if (in) {
        v.uw[half] = __ldg(a.uxf + j * ld + (i - 1));
        v.ue[half] = __ldg(a.uxf + j * ld + i);
        v.vs[half] = __ldg(a.uyf + j * ld + i);
        v.vn[half] = __ldg(a.uyf + (j + 1) * ld + i);
      }
    }
  };
  for (int k0 = first; left > 0; k0 += rows * stride, left -= rows) {
    const int nq = min(rows, left);
    // the next rows' table entries are loaded while these are processed
    int c = nxt_c;
    const int4 dsc = nxt;
    fetch(k0 + rows * stride, nxt_c, nxt);
    if (lane < nq) {
      const int n = dsc.x;
      if (c >= 0 && !(EIF_CHK(a.bd.rec, n, a.np, 52) && row_slots_in(a.bd, c, a.bd.wbuf, 60))) c = -1;
      RowF &r = ws.row[lane];
      r.c = c;
      r.cells = make_int4(1, 1, 0, 1);
      if (c >= 0) {
        RowTask t;
        const bool task = task_of(dsc, a.np, t) && (t.ib > t.ie || row_cells_in(a.bd, t, ld, 54));
        const float4 *q4 = reinterpret_cast<const float4 *>(ONE ? one->pf : a.pf + (size_t)PF_WORDS * n);
        const float4 qA = ldro<NC>(q4), qB = ldro<NC>(q4 + 1), qC = ldro<NC>(q4 + 2), qD = ldro<NC>(q4 + 3),
                     qE = ldro<NC>(q4 + 4), qF = ldro<NC>(q4 + 5), qG = ldro<NC>(q4 + 6);
        const int m = task ? t.img + 1 : 1;
        // image row origin and fraction selected without a local array
        const int j0i = __float_as_int(m == 0 ? qD.y : (m == 1 ? qD.z : qD.w));
        const float gyi = m == 0 ? qE.x : (m == 1 ? qE.y : qE.z);
        const int j = task ? t.j : 1;
        const float Y = ((float)(j - j0i) - gyi) * dyf;
        r.ell = make_float4(qA.x, qA.y, qB.x, qB.y);
        r.geo = make_float4(qA.z, qA.w, Y, qC.w);
        r.par = make_float4(qB.z, qB.w, qC.x, qC.y);
        r.vz = qC.z;
        r.cells = make_int4(__float_as_int(qD.x), task ? t.ib : 1, task ? t.ie : 0, j);
        // far cells of the row (PF_AL .. PF_RO2: al, ka, de, so^2, si^2, ro^2)
        float olo, ohi, ilo, ihi;
        row_chords(qE.w, qF.x, qF.y, qF.z, qF.w, qG.x, Y, olo, ohi, ilo, ihi);
        r.chords = make_float4(olo, ohi, ilo, ihi);
      }
    }
    __syncwarp();
    // the rows' field values are loaded a row ahead
    Vel vel;
    load(0, vel);
    // pass 1: far cells settled, the near ones listed
    int nnear = 0;
#pragma unroll 1
    for (int q = 0; q < nq; q++) {
      const RowF &r = ws.row[q];
      if (r.c < 0) continue;
      const int4 ce = r.cells;
      const float4 ch = r.chords;
      const float gx = r.geo.w;
      const int near0 = nnear;
#pragma unroll
      for (int half = 0; half < CHUNK / 32; half++) {
        const int at = half * 32 + lane, i = ce.y + at;
        const bool in = i <= ce.z;
        const float X = ((float)(i - ce.x) - gx) * dxf;
        const int side = !(X > ch.x && X < ch.y) ? -1 : ((X >= ch.z && X <= ch.w) ? 1 : 0);
        const bool near = in && side == 0;
        ws.th[q][at] = in ? (float)side : 0.f;
        const unsigned mask = __ballot_sync(0xffffffffu, near);
        if (near) ws.list[nnear + __popc(mask & ((1u << lane) - 1u))] = (unsigned char)(q * CHUNK + at);
        nnear += __popc(mask);
      }
      if (a.count && lane == 0) {
        atomicAdd(a.count, (unsigned long long)max(0, min(CHUNK, ce.z - ce.y + 1)));
        atomicAdd(a.count + 1, (unsigned long long)(nnear - near0));
      }
    }
    __syncwarp();
    // pass 2: the near cells, packed onto the lanes
    for (int k = lane; k < nnear; k += 32) {
      const int id = ws.list[k], q = id / CHUNK, at = id % CHUNK;
      const RowF &r = ws.row[q];
      const float4 el = r.ell, ge = r.geo;
      EllF e;
      e.a = el.x; e.b = el.y; e.kex = el.z; e.key = el.w; e.cz = ge.x; e.sz = ge.y;
      const float X = ((float)(r.cells.y + at - r.cells.x) - ge.w) * dxf, Y = ge.z;
      const float x_ = __fmaf_rn(e.cz, X, -__fmul_rn(e.sz, Y));
      const float y_ = __fmaf_rn(e.sz, X, __fmul_rn(e.cz, Y));
      ws.th[q][at] = indicator_f(e, x_, y_, rh);
    }
    __syncwarp();
    // the sums
#pragma unroll 1
    for (int q = 0; q < nq; q++) {
      const Vel v = vel;
      if (q + 1 < nq) load(q + 1, vel);
      const RowF &r = ws.row[q];
      const int c = r.c;
      if (c < 0) continue;
      const float4 par = r.par;
      const float Y = r.geo.z, gx = r.geo.w, pvz = r.vz;
      const int at0 = r.cells.y - r.cells.x;
      float sacc0 = 0.f, sacc1 = 0.f, sacc2 = 0.f;
#pragma unroll
      for (int half = 0; half < CHUNK / 32; half++) {
        const int at = half * 32 + lane;
        float2 contrib = make_float2(0.f, 0.f);
        const float th = ws.th[q][at];
        // (the stage start's weights from the memo are taken by ibm_memo_f_tasks, which
        // leaves this body only the tasks the memo did not serve)
        if (a.memo_mode == 2) a.memo.w[(size_t)c * CHUNK + at] = th;
        if (wmode == 1) wcache[(size_t)c * CHUNK + at] = th;
        // cells of weight exactly zero (inertia: far outside; exchange: any far cell) are skipped
        const bool live = a.mode == 0 ? th != -1.f : fabsf(th) != 1.f;
        if (v.in[half] && live) {
          const float X = ((float)(at0 + at) - gx) * dxf;
          const float uxs = v.uw[half] + v.ue[half];
          const float uys = v.vs[half] + v.vn[half];
          if (a.mode == 0) {
            inertia_cell_f(th, X, Y, uxs, uys, dxdy, par.x, par.y, sacc0, sacc1, sacc2);
          } else {
            const float w = 1.f - th * th;
            const float uxp = par.z - pvz * Y;
            const float uyp = par.w + pvz * X;
            const float gxv = w * (uxp - 0.5f * uxs);   // fx * dt
            const float gyv = w * (uyp - 0.5f * uys);   // fy * dt
            contrib = make_float2(gxv, gyv);
            const float Fx = gxv * rdtv * dxdy, Fy = gyv * rdtv * dxdy;
            sacc0 -= Fx * par.x;
            sacc1 -= Fy * par.x;
            sacc2 += (Y * Fx - X * Fy) * par.y;
          }
        }
        if (a.mode == 1) wb[(size_t)c * CHUNK + at] = contrib;
      }
      store_sums_f(a, c, sacc0, sacc1, sacc2, lane, 58);
    }
    __syncwarp();
  }
}

// The stage start of the mixed form (inertia at X with zero increments, weights stored for
// the stage: wmode 1, memo_mode 1 of ibm_work_f_tasks) without the geometry code: a task
// whose particle geometry words and boxes are bitwise those of the memo takes the memo's
// weights, stores them in wcache and forms its sums exactly as ibm_work_f_tasks does;
// any other task is appended to a.miss for k_ibm_work_f, which evaluates those in full.
// It runs with the registers of the sums kernel, so more warps hide its loads.
template <bool NC>
__device__ __forceinline__ void ibm_memo_f_tasks(const WorkArgs &a, int first, int stride) {
  const int lane = threadIdx.x & 31;
  const int total = EIF_CHK(a.bd.rec, a.np, a.bd.off, 90) ? ldro<NC>(a.off + a.np) : 0;
  const float dxf = a.dx_f, dyf = a.dy_f, dxdy = a.dxdy_f;
  const int ld = a.ld;
  float *wcache = static_cast<float *>(a.wcache);
  const bool valid = ldro<NC>(a.memo.valid) != 0;
  for (int c = first; c < total; c += stride) {
    if (!EIF_CHK(a.bd.rec, c, a.bd.partial / 3, 91)) continue;
    const int4 dsc = ldro<NC>(a.tdesc + c);
    const int n = dsc.x;
    if (!EIF_CHK(a.bd.rec, n, a.np, 92)) continue;
    bool eq = false;
    if (valid) {
      if (lane < 20) {
        const size_t q = (size_t)PF_WORDS * n + memo_word(lane);
        eq = __float_as_uint(ldro<NC>(a.pf + q)) == __float_as_uint(ldro<NC>(a.memo.pf + q));
      } else {
        const size_t q = 12 * (size_t)n + (lane - 20);
        eq = ldro<NC>(a.box + q) == ldro<NC>(a.memo.box + q);
      }
    }
    if (!__all_sync(0xffffffffu, eq)) {
      if (lane == 0) {
        const int k = atomicAdd(a.miss, 1);
        if (EIF_CHK(a.bd.rec, k, a.bd.partial / 3, 93)) a.miss[1 + k] = c;
      }
      continue;
    }
    if (a.count && lane == 0) atomicAdd(a.count + 2, 1ull);
    const long long src = (long long)c + (ldro<NC>(a.memo.off + n) - ldro<NC>(a.off + n));
    RowTask t;
    const bool task = task_of(dsc, a.np, t) && (t.ib > t.ie || row_cells_in(a.bd, t, ld, 94));
    const float4 *q4 = reinterpret_cast<const float4 *>(a.pf + (size_t)PF_WORDS * n);
    const float4 qB = ldro<NC>(q4 + 1), qC = ldro<NC>(q4 + 2), qD = ldro<NC>(q4 + 3), qE = ldro<NC>(q4 + 4);
    const float rpm = qB.z, rpim = qB.w, gx = qC.w;
    const int i0 = __float_as_int(qD.x);
    const int m = task ? t.img + 1 : 1;
    const int j0i = __float_as_int(m == 0 ? qD.y : (m == 1 ? qD.z : qD.w));
    const float gyi = m == 0 ? qE.x : (m == 1 ? qE.y : qE.z);
    const int j = task ? t.j : 1;
    const float Y = ((float)(j - j0i) - gyi) * dyf;
    bool cin[2];
    float cX[2], th2[2], fuw[2], fue[2], fvs[2], fvn[2];
#pragma unroll
    for (int half = 0; half < CHUNK / 32; half++) {
      const int i = (task ? t.ib : 1) + half * 32 + lane;
      const bool in = task && i <= t.ie;
      fuw[half] = fue[half] = fvs[half] = fvn[half] = 0.f;
      if (in) {
        fuw[half] = __ldg(a.uxf + j * ld + (i - 1));
        fue[half] = __ldg(a.uxf + j * ld + i);
        fvs[half] = __ldg(a.uyf + j * ld + i);
        fvn[half] = __ldg(a.uyf + (j + 1) * ld + i);
      }
      cin[half] = in;
      cX[half] = ((float)(i - i0) - gx) * dxf;
    }
    // (after the field loads, which do not wait for the offsets)
    if (!row_slots_in(a.bd, c, a.bd.wbuf, 98) || !row_slots_in(a.bd, src, a.bd.wbuf, 97)) continue;
#pragma unroll
    for (int half = 0; half < CHUNK / 32; half++)
      th2[half] = cin[half] ? a.memo.w[(size_t)src * CHUNK + half * 32 + lane] : 0.f;
#pragma unroll
    for (int half = 0; half < CHUNK / 32; half++) wcache[(size_t)c * CHUNK + half * 32 + lane] = th2[half];
    float sacc0 = 0.f, sacc1 = 0.f, sacc2 = 0.f;
#pragma unroll
    for (int half = 0; half < CHUNK / 32; half++) {
      const float th_ = th2[half];
      if (cin[half] && th_ != -1.f) {
        const float uxs = fuw[half] + fue[half];
        const float uys = fvs[half] + fvn[half];
        inertia_cell_f(th_, cX[half], Y, uxs, uys, dxdy, rpm, rpim, sacc0, sacc1, sacc2);
      }
    }
    store_sums_f(a, c, sacc0, sacc1, sacc2, lane, 99);
  }
}

// The mixed form's evaluation with cached weights (wmode 2 of k_ibm_work_f): the
// same sums and field contributions, without the geometry work, so it runs with
// few registers and many resident warps, which hide the latency of its loads.
// The warp runs the tasks first, first + stride, ...
template <bool NC>
__device__ __forceinline__ void ibm_sum_f_tasks(const WorkArgs &a, int first, int stride, int total) {
  const int lane = threadIdx.x & 31;
  const int warp = first, nwarps = stride;
  const float dxf = a.dx_f, dyf = a.dy_f, dxdy = a.dxdy_f;
  const float rdtv = a.mode == 1 ? __ldg(a.coef + 9) : 0.f;
  const int ld = a.ld;
  float2 *wb = reinterpret_cast<float2 *>(a.wbuf);
  const float *wcache = static_cast<const float *>(a.wcache);
  // the next task's table entry and cached weights are loaded while the current task
  // is processed, so that its field loads need not wait for them
  int4 nxt = make_int4(-1, 0, 0, 0);
  float nth0 = 0.f, nth1 = 0.f;
  if (warp < total && EIF_CHK(a.bd.rec, warp, a.bd.partial / 3, 71) &&
      EIF_CHK(a.bd.rec, (long long)warp * CHUNK + CHUNK - 1, 2 * a.bd.wbuf, 77)) {
    nxt = ldro<NC>(a.tdesc + warp);
    nth0 = wcache[(size_t)warp * CHUNK + lane];
    nth1 = wcache[(size_t)warp * CHUNK + 32 + lane];
  }
  for (int c = warp; c < total; c += nwarps) {
    const int4 dsc = nxt;
    const float th_pre[2] = {nth0, nth1};
    const int cn = c + nwarps;
    if (cn < total && EIF_CHK(a.bd.rec, cn, a.bd.partial / 3, 71) &&
        EIF_CHK(a.bd.rec, (long long)cn * CHUNK + CHUNK - 1, 2 * a.bd.wbuf, 77)) {
      nxt = ldro<NC>(a.tdesc + cn);
      nth0 = wcache[(size_t)cn * CHUNK + lane];
      nth1 = wcache[(size_t)cn * CHUNK + 32 + lane];
    }
    const int n = dsc.x;
    if (!EIF_CHK(a.bd.rec, n, a.np, 72) || !row_slots_in(a.bd, c, 2 * a.bd.wbuf, 78)) continue;
    RowTask t;
    const bool task = task_of(dsc, a.np, t) && (t.ib > t.ie || row_cells_in(a.bd, t, ld, 74));
    const float4 *q4 = reinterpret_cast<const float4 *>(a.pf + (size_t)PF_WORDS * n);
    const float4 qB = ldro<NC>(q4 + 1), qC = ldro<NC>(q4 + 2), qD = ldro<NC>(q4 + 3), qE = ldro<NC>(q4 + 4);
    const float rpm = qB.z, rpim = qB.w, pux = qC.x, puy = qC.y, pvz = qC.z, gx = qC.w;
    const int i0 = __float_as_int(qD.x);
    const int m = task ? t.img + 1 : 1;
    const int j0i = __float_as_int(m == 0 ? qD.y : (m == 1 ? qD.z : qD.w));
    const float gyi = m == 0 ? qE.x : (m == 1 ? qE.y : qE.z);
    const int j = task ? t.j : 1;
    const float Y = ((float)(j - j0i) - gyi) * dyf;
    // the field values of both halves are loaded before either is used, so that the
    // warp has all eight loads of the task in flight at once
    bool live[2];
    float thv[2];
    float uw[2], ue[2], vs[2], vn[2];
#pragma unroll
    for (int half = 0; half < CHUNK / 32; half++) {
      const int i = (task ? t.ib : 1) + half * 32 + lane;
      const bool in = task && i <= t.ie;
      const float th = in ? th_pre[half] : 0.f;
      thv[half] = th;
      // cells of weight exactly zero (inertia: far outside; exchange: any far cell) are skipped
      live[half] = in && (a.mode == 0 ? th != -1.f : fabsf(th) != 1.f);
      uw[half] = ue[half] = vs[half] = vn[half] = 0.f;
      if (live[half]) {
        uw[half] = __ldg(a.uxf + j * ld + (i - 1));
        ue[half] = __ldg(a.uxf + j * ld + i);
        vs[half] = __ldg(a.uyf + j * ld + i);
        vn[half] = __ldg(a.uyf + (j + 1) * ld + i);
      }
    }
    float sacc0 = 0.f, sacc1 = 0.f, sacc2 = 0.f;
#pragma unroll
    for (int half = 0; half < CHUNK / 32; half++) {
      const int i = (task ? t.ib : 1) + half * 32 + lane;
      const long long slot = (long long)c * CHUNK + half * 32 + lane;
      float2 contrib = make_float2(0.f, 0.f);
      const float th = thv[half];
      if (live[half]) {
        const float X = ((float)(i - i0) - gx) * dxf;
        const float uxs = uw[half] + ue[half];
        const float uys = vs[half] + vn[half];
        if (a.mode == 0) {
          inertia_cell_f(th, X, Y, uxs, uys, dxdy, rpm, rpim, sacc0, sacc1, sacc2);
        } else {
          const float w = 1.f - th * th;
          const float uxp = pux - pvz * Y;
          const float uyp = puy + pvz * X;
          const float gxv = w * (uxp - 0.5f * uxs);   // fx * dt
          const float gyv = w * (uyp - 0.5f * uys);   // fy * dt
          contrib = make_float2(gxv, gyv);
          const float Fx = gxv * rdtv * dxdy, Fy = gyv * rdtv * dxdy;
          sacc0 -= Fx * rpm;
          sacc1 -= Fy * rpm;
          sacc2 += (Y * Fx - X * Fy) * rpim;
        }
      }
      if (a.mode == 1) wb[slot] = contrib;
    }
    store_sums_f(a, c, sacc0, sacc1, sacc2, lane, 79);
  }
}

// sums over the chunks c0 .. c1 - 1 in a fixed order (one warp): lane k < 3 has sum k
__device__ __forceinline__ double chunk_sum_warp(const double *partial, int c0, int c1, const Bounds &bd) {
  const int lane = threadIdx.x & 31;
  double s0 = 0., s1 = 0., s2 = 0.;
  for (int c = c0 + lane; c < c1; c += 32) {
    if (!EIF_CHK(bd.rec, 3LL * c + 2, bd.partial, 31)) break;
    s0 += partial[3 * (size_t)c + 0];
    s1 += partial[3 * (size_t)c + 1];
    s2 += partial[3 * (size_t)c + 2];
  }
  // the sums are in lanes 0, 16 and 8
  return __shfl_sync(0xffffffffu, warp_sum3(s0, s1, s2, lane), lane == 0 ? 0 : (lane == 1 ? 16 : 8));
}

// The same per-particle sums from the single-precision partials of the mixed form,
// accumulated in double-float arithmetic (TwoSum) on the FP32 pipe: the sum of at most
// a few hundred floats is kept to about 48 bits, and the result is rounded once to
// double.
__device__ __forceinline__ double chunk_sum_f_warp(const float *partial, int c0, int c1, const Bounds &bd) {
  const int lane = threadIdx.x & 31;
  float h[3] = {0.f, 0.f, 0.f}, l[3] = {0.f, 0.f, 0.f};
  for (int c = c0 + lane; c < c1; c += 32) {
    if (!EIF_CHK(bd.rec, 3LL * c + 2, 2 * bd.partial, 34)) break;
#pragma unroll
    for (int k = 0; k < 3; k++) {
      const float v = partial[3 * (size_t)c + k];
      const float s = h[k] + v, bb = s - h[k];
      l[k] += (h[k] - (s - bb)) + (v - bb);
      h[k] = s;
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
    for (int k = 0; k < 3; k++) {
      const float vh = __shfl_xor_sync(0xffffffffu, h[k], o), vl = __shfl_xor_sync(0xffffffffu, l[k], o);
      const float s = h[k] + vh, bb = s - h[k];
      l[k] += ((h[k] - (s - bb)) + (vh - bb)) + vl;
      h[k] = s;
    }
  }
  // lane 0's (the lanes' trailing parts differ in their last bits)
#pragma unroll
  for (int k = 0; k < 3; k++) {
    h[k] = __shfl_sync(0xffffffffu, h[k], 0);
    l[k] = __shfl_sync(0xffffffffu, l[k], 0);
  }
  const float hk = lane == 0 ? h[0] : (lane == 1 ? h[1] : h[2]), lk = lane == 0 ? l[0] : (lane == 1 ? l[1] : l[2]);
  return eifd::f2d(hk) + eifd::f2d(lk);
}

// The geometry words (pf: PF_WORDS words), boxes (12 ints) and first task c0 of particle n to
// the memo, after a sub-iteration's indicator evaluation that stored its weights there (one warp).
__device__ __forceinline__ void memo_particle(const WeightMemo &memo, const float *pf, const int *box, int c0, int n) {
  const int lane = threadIdx.x & 31;
  if (lane < 20) memo.pf[(size_t)PF_WORDS * n + memo_word(lane)] = pf[memo_word(lane)];
  else memo.box[12 * (size_t)n + (lane - 20)] = box[lane - 20];
  if (lane == 0) memo.off[n] = c0;
  if (lane == 0 && n == 0) *memo.valid = 1;
}

// ---- arguments of the box, table and task bodies from a context (host) ----

inline Bounds bounds_of(const eif_ctx *c) {
  Bounds b;
  b.P = (long long)EIF_NFIELDS * c->pcap;
  b.box = 12LL * c->np;
  b.off = (c->np + 1) + 3LL * c->np;
  b.partial = 3LL * c->chunk_cap;
  b.wbuf = (long long)c->wcap;
  b.field = (long long)c->nfield;
  b.xc = c->itot + 3;   // entries 0..itot+1 (EIF_CHK is given xc-1 as the bound of valid i)
  b.yc = c->jtot + 3;
  b.rec = c->d_check;
  return b;
}

inline WeightMemo memo_of(const eif_ctx *c) {
  WeightMemo m;
  m.w = c->memo_w;
  m.pf = c->memo_pf;
  m.box = c->memo_box;
  m.off = c->memo_off;
  m.valid = c->memo_valid;
  return m;
}

// boxes of the particles at X (+ dX with use_increment); the task counts of their images go
// to nchunk = chunk_off + np + 1
inline BoxArgs box_args(const eif_ctx *c, bool use_increment) {
  BoxArgs b;
  b.bd = bounds_of(c);
  b.bd_off_base = c->chunk_off;
  b.P = c->P; b.pcap = c->pcap; b.np = c->np; b.itot = c->itot; b.jtot = c->jtot;
  b.use_increment = use_increment ? 1 : 0;
  b.dx = c->dx; b.dy = c->dy; b.ly = c->ly; b.yf1 = c->h_yf[0];
  b.box = c->box;
  b.pf = c->cfg.precision == EIF_PREC_MIXED ? c->pf : nullptr;
  b.pd = c->cfg.precision == EIF_PREC_MIXED ? nullptr : c->pd;
  b.kb = BETA / (c->dx < c->dy ? c->dx : c->dy);
  b.iter = nullptr;
  b.nchunk = c->chunk_off + (c->np + 1);
  return b;
}

// the task sums of mode 0 or 1: arrays of their own, so that the inertia's are reduced beside
// the exchange's evaluation (rk_stage_front)
inline double *partial_of(const eif_ctx *c, int mode) { return c->partial + (mode == 0 ? 0 : 3 * (size_t)c->chunk_cap); }

// task evaluations of mode 0 (inertia into the integrals cn) or 1 (exchange) over the
// current velocity buffers; wmode 0, no loop counter, no counts
inline WorkArgs work_args(const eif_ctx *c, int mode, int cn) {
  WorkArgs w;
  w.P = c->P; w.ux = c->ux[c->cur]; w.uy = c->uy[c->cur]; w.xc = c->xc; w.yc = c->yc; w.dt = c->d_scal;
  w.uxf = c->uxf[c->cur]; w.uyf = c->uyf[c->cur];
  w.box = c->box; w.off = c->chunk_off; w.partial = partial_of(c, mode); w.wbuf = reinterpret_cast<double2 *>(c->wbuf);
  w.pcap = c->pcap; w.np = c->np; w.ld = c->ld; w.mode = mode; w.cn = cn;
  w.dx = c->dx; w.dy = c->dy; w.ly = c->ly; w.h = c->dx < c->dy ? c->dx : c->dy;
  w.bd = bounds_of(c);
  w.pf = c->pf;
  w.pd = c->pd;
  w.tanh_tab = c->tanh_tab;
  w.mid_tab = reinterpret_cast<const float2 *>(c->tanh_tab + 2 * TANH_N);
  w.tdesc = c->tdesc;
  w.coef = c->d_coef;
  w.rh_f = (float)(1. / w.h);
  w.dx_f = (float)c->dx;
  w.dy_f = (float)c->dy;
  w.dxdy_f = (float)(c->dx * c->dy);
  w.wcache = c->wcache;
  w.wmode = 0;
  w.iter = nullptr;
  w.weights_only = c->ibm_weights_only ? 1 : 0;
  w.count = nullptr;
  w.memo = memo_of(c);
  w.memo_mode = 0;
  w.miss = nullptr;
  w.only = nullptr;
  return w;
}

}  // namespace
