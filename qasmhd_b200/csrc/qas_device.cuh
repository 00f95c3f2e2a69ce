// qas_device.cuh -- FP64 point functions of the qasMHD step for sm_100a.
//
// Every expression keeps the reference's IEEE operation sequence (same
// constants, same association, no contraction: the library is compiled with
// --fmad=false and IEEE division/sqrt), so results are bit-identical to the
// reference CPU build.  What differs is structure: the 7x7 eigen-projections
// of the characteristic reconstruction are written out sparsely (only the
// non-zero terms, summed in the reference's left-to-right order; an omitted
// 0*x term can only change the sign of an exact zero), the spatial order is a
// template parameter and the stencils live in registers.
#pragma once

#include <math.h>
#include <string.h>

#if defined(__CUDACC__)
#include <cuda_runtime.h>
#define QAS_HD __host__ __device__ __forceinline__
#else
#define QAS_HD inline
#endif

namespace qas {


// ---------------------------------------------------------------------------
// common/common_func.h:4-31
// ---------------------------------------------------------------------------
QAS_HD bool is_zero(double x) { return x == 0.0; }

// c*a + b for c a power of two: the product is exact, so the one rounding of the FMA is the
// reference's (c*a overflowing or falling below the normal range aside, see wcns4_lr_fast)
QAS_HD double p2fma(double c, double a, double b)
{
#if defined(__CUDA_ARCH__)
  return fma(c, a, b);
#else
  return c * a + b;
#endif
}

// high word of x, for range tests on the integer pipe
QAS_HD unsigned hiword(double x)
{
#if defined(__CUDA_ARCH__)
  return (unsigned)__double2hiint(x);
#else
  unsigned long long b;
  memcpy(&b, &x, 8);
  return (unsigned)(b >> 32);
#endif
}
QAS_HD unsigned umax3(unsigned a, unsigned b, unsigned c)
{
  const unsigned t = a > b ? a : b;
  return t > c ? t : c;
}

// 1/x rounded to nearest for 2^-1000 < x < 2^1000: Newton's iteration for a reciprocal with a last step that
// rounds correctly (P. Markstein, IBM J. Res. Dev. 34, 1990; Muller et al., Handbook of Floating-Point
// Arithmetic, division by Newton-Raphson with an FMA).  Step by step, d the relative error of the seed:
//  * the seed, PTX's approximation of the reciprocal: all that is used of it is |d| < 2^-14;
//  * one step, y + y*(1 - x*y), squares the error: y = (1 - d^2)/x, to within 2^-28;
//  * a second gives (1 - d^4)/x, at most 2^-56 below 1/x, and is rounded UP: less than one ulp from 1/x.  (1 - x*y
//    is itself rounded in it, which moves the result by less than 2^-80; where that makes it more than one ulp,
//    1/x lies next to a double, nowhere near a midpoint.)
//  * Markstein: from there 1 - x*y is exact and y + y*(1 - x*y) rounds to the double nearest 1/x, unless x has
//    the largest significand of all.  For that one, x = 2 - 2^-52 (times a power of two), 1/x = (1 + 2^-53 +
//    ...)/2 lies just above the midpoint of 1/2 and its successor 1/2 + 2^-53.  The second step's value before
//    rounding is above 1/2, so that rounding up gives the successor, which is the right result, and the last step
//    keeps it: 1 - x*y = -2^-53 + 2^-105 leads to 1/2 + 2^-54 + 2^-158, still above the midpoint.
// Compared with 1.0/x bit for bit in the GPU tests, the seed's error (2^-19.9) too.  The reconstruction forms 35 of
// these per cell and axis; a step with them / with 1.0/x, whose range test the compiler writes at every use: KH
// 160^3 8.01 / 8.36 ms, OT 1024^2 1174 / 1221 us, KH 117x75x93 1907 / 1983 us.
#if defined(__CUDACC__)
__device__ __forceinline__ double rcp_seed(double x)
{
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  return y;
}
#endif
QAS_HD double rcp_positive(double x)
{
#if defined(__CUDA_ARCH__)
  double y = rcp_seed(x);
  y = fma(y, fma(-x, y, 1.0), y);
  y = __fma_ru(y, fma(-x, y, 1.0), y);
  return fma(y, fma(-x, y, 1.0), y);
#else
  return 1.0 / x;
#endif
}
// the same for either sign
QAS_HD double rcp_normal(double x) { return copysign(rcp_positive(fabs(x)), x); }

// x with its sign flipped where neg (the reference's multiplication by +-1.0), on the integer pipe
QAS_HD double flip(double x, bool neg)
{
#if defined(__CUDA_ARCH__)
  return __hiloint2double(__double2hiint(x) ^ (neg ? (int)0x80000000 : 0), __double2loint(x));
#else
  return neg ? -x : x;
#endif
}

// x/24 rounded to nearest by two operations instead of a division: with h + l = 1/24 to 106
// bits, x*h + RN(x*l) is within 2^-50 ulp of x/24, and no x/24 lies nearer than 1/6 ulp to a
// rounding boundary (24 = 3*8; Brisebarre, Muller, Raina, IEEE Trans. Comput. 53, 2004, division
// by a constant).  Below 2^-900, where x*l would lose bits, the division itself.
QAS_HD double div24(double x)
{
#if defined(__CUDA_ARCH__)
  const double h = 1.0 / 24.0;                  // RN(1/24) = (1 - 2^-54)/24: 24 h = 1 - 2^-54
  const double l = 5.5511151231257827e-17 / 24.0;  // (1 - 24 h)/24, 2^-54/24
  const unsigned hi = (unsigned)__double2hiint(x) & 0x7fffffffu;
  if (hi < 0x07b00000u && (hi | (unsigned)__double2loint(x)) != 0u) return x / 24.0;  // tiny, not zero
  return fma(x, h, x * l);
#else
  return x / 24.0;
#endif
}

QAS_HD double qmax(double a, double b) { return (a >= b) ? a : b; }
QAS_HD double qmin(double a, double b) { return (a >= b) ? b : a; }
QAS_HD double minmod(double a, double b)
{
  return +qmin(qmax(a, b), 0.0) + qmax(qmin(a, b), 0.0);
}

// ---------------------------------------------------------------------------
// face <-> centre stencils, common/common_interp.h:6-24.
// f0 is the value at face i-1/2, f1 at i+1/2, fm at i-3/2, f2 at i+3/2.
// ---------------------------------------------------------------------------
template <int ODR>
QAS_HD double fcen(double fm, double f0, double f1, double f2)
{
  if (ODR >= 3) return (0.0625 * (9.0 * (f0 + f1) - (fm + f2)));
  return (0.5 * (f0 + f1));
}
template <int ODR>
QAS_HD double dfc(double fm, double f0, double f1, double f2)
{
  if (ODR >= 3) return div24(27.0 * (f1 - f0) - (f2 - fm));
  return (f1 - f0);
}

// ---------------------------------------------------------------------------
// linear interpolation to the faces, common/common_interp.c:7-28
// f[0..4] = values at i-2..i+2; fl at i+1/2, fr at i-1/2
// ---------------------------------------------------------------------------
template <int ODR>
QAS_HD void lin_lr(const double f[5], double &fl, double &fr)
{
  if (ODR == 1) {
    fl = f[2];
    fr = f[2];
  } else if (ODR == 2) {
    fl = (-f[1] + 5.0 * f[2] + 2.0 * f[3]) / 6.0;
    fr = (-f[3] + 5.0 * f[2] + 2.0 * f[1]) / 6.0;
  } else if (ODR == 3) {
    fl = 0.125 * (-f[1] + 6.0 * f[2] + 3.0 * f[3]);
    fr = 0.125 * (-f[3] + 6.0 * f[2] + 3.0 * f[1]);
  } else {
    fl = 0.003125 * (9.0 * f[0] - 56.0 * f[1] + 234.0 * f[2] + 144.0 * f[3] - 11.0 * f[4]);
    fr = 0.003125 * (9.0 * f[4] - 56.0 * f[3] + 234.0 * f[2] + 144.0 * f[1] - 11.0 * f[0]);
  }
}
template <int ODR>
QAS_HD double lin_left(const double f[5])
{
  double l, r;
  lin_lr<ODR>(f, l, r);
  return l;
}
template <int ODR>
QAS_HD double lin_right(const double f[5])
{
  double l, r;
  lin_lr<ODR>(f, l, r);
  return r;
}

// ---------------------------------------------------------------------------
// nonlinear interpolation interpol[ODR-1] (common/mhd_class.hpp:109):
// 1st order, MUSCL minmod (common_interp.c:32-37), WCNS3 (:65-101),
// WCNS4 (:102-150)
// ---------------------------------------------------------------------------
QAS_HD void wcns4_lr(const double f[5], double &fl, double &fr)
{
  const double eps = 1e-40;
  double c1, c2;
  c1 = f[0] - 4.0 * f[1] + 3.0 * f[2];
  c2 = f[0] - 2.0 * f[1] + f[2];
  double s0 = (13. / 12.) * c2 * c2 + 0.25 * c1 * c1;
  c1 = f[1] - f[3];
  c2 = f[1] - 2.0 * f[2] + f[3];
  double s1 = (13. / 12.) * c2 * c2 + 0.25 * c1 * c1;
  c1 = f[4] - 4.0 * f[3] + 3.0 * f[2];
  c2 = f[4] - 2.0 * f[3] + f[2];
  double s2 = (13. / 12.) * c2 * c2 + 0.25 * c1 * c1;
  s0 = 1.0 / (s0 * s0 + eps);
  s1 = 1.0 / (s1 * s1 + eps);
  s2 = 1.0 / (s2 * s2 + eps);
  // candidate polynomials (shared by both sides in the reference's order)
  double pl0 = (3.0 * f[0] - 10.0 * f[1] + 15.0 * f[2]);
  double pl1 = (-f[1] + 6.0 * f[2] + 3.0 * f[3]);
  double pl2 = (+3.0 * f[2] + 6.0 * f[3] - f[4]);
  double w0 = 0.075 * s0, w1 = 0.650 * s1, w2 = 0.275 * s2;
  double dn = 1.0 / (w0 + w1 + w2);
  w0 *= dn;
  w1 *= dn;
  w2 = 1.0 - w0 - w1;
  fl = 0.125 * (+w0 * pl0 + w1 * pl1 + w2 * pl2);
  double pr2 = (3.0 * f[4] - 10.0 * f[3] + 15.0 * f[2]);
  double pr1 = (-f[3] + 6.0 * f[2] + 3.0 * f[1]);
  double pr0 = (+3.0 * f[2] + 6.0 * f[1] - f[0]);
  w0 = 0.275 * s0;
  w1 = 0.650 * s1;
  w2 = 0.075 * s2;
  dn = 1.0 / (w0 + w1 + w2);
  w0 *= dn;
  w1 *= dn;
  w2 = 1.0 - w0 - w1;
  fr = 0.125 * (+w2 * pr2 + w1 * pr1 + w0 * pr0);
}

// wcns4_lr with the same rounded results in fewer FP64 operations (115 -> 106 a field), the form the
// kernels run:
//  * a product by a power of two feeding a sum is one FMA (p2fma);
//  * the candidates carry the final factor 1/8 in their coefficients (3/8 f instead of 3 f, ...;
//    every intermediate is the reference's times an exact power of two), and 6 f, 3 f share
//    one product;
//  * the five reciprocals are rcp_positive: s^2 + 1e-40 is at least 1e-40, so only the upper
//    end needs a test, left to the caller: hx receives the largest high word of the three
//    denominators (of any NaN too, whose sign bit or exponent exceeds every finite value's), and
//    the results hold for hx < WCNS_HX, 2^900.
// Magnitudes below about 2^-1015, where a scaled intermediate leaves the normal range, are the
// one place where the last bit may differ.
constexpr unsigned WCNS_HX = 0x78300000u;
QAS_HD void wcns4_lr_fast(const double f[5], double &fl, double &fr, unsigned &hx)
{
  const double eps = 1e-40;
  const double g1 = 0.375 * f[1], g2 = 0.375 * f[2], g3 = 0.375 * f[3];
  double c1, c2;
  c1 = p2fma(8.0, g2, p2fma(-4.0, f[1], f[0]));
  c2 = p2fma(-2.0, f[1], f[0]) + f[2];
  double s0 = p2fma(0.25, c1 * c1, (13. / 12.) * c2 * c2);
  c1 = f[1] - f[3];
  c2 = p2fma(-2.0, f[2], f[1]) + f[3];
  double s1 = p2fma(0.25, c1 * c1, (13. / 12.) * c2 * c2);
  c1 = p2fma(8.0, g2, p2fma(-4.0, f[3], f[4]));
  c2 = p2fma(-2.0, f[3], f[4]) + f[2];
  double s2 = p2fma(0.25, c1 * c1, (13. / 12.) * c2 * c2);
  s0 = s0 * s0 + eps;
  s1 = s1 * s1 + eps;
  s2 = s2 * s2 + eps;
  hx = umax3(hiword(s0), hiword(s1), umax3(hx, hiword(s2), 0u));
  s0 = rcp_positive(s0);
  s1 = rcp_positive(s1);
  s2 = rcp_positive(s2);
  const double h2 = 1.875 * f[2];
  const double pl0 = 0.375 * f[0] - 1.25 * f[1] + h2;
  const double pl1 = p2fma(2.0, p2fma(-0.0625, f[1], g2), g3);
  const double pl2 = p2fma(-0.125, f[4], p2fma(2.0, g3, g2));
  const double u1 = 0.650 * s1;
  double w0 = 0.075 * s0, w1, w2 = 0.275 * s2;
  double dn = rcp_positive(w0 + u1 + w2);
  w0 *= dn;
  w1 = u1 * dn;
  w2 = 1.0 - w0 - w1;
  fl = (+w0 * pl0 + w1 * pl1 + w2 * pl2);
  const double pr2 = 0.375 * f[4] - 1.25 * f[3] + h2;
  const double pr1 = p2fma(2.0, p2fma(-0.0625, f[3], g2), g1);
  const double pr0 = p2fma(-0.125, f[0], p2fma(2.0, g1, g2));
  w0 = 0.275 * s0;
  w2 = 0.075 * s2;
  dn = rcp_positive(w0 + u1 + w2);
  w0 *= dn;
  w1 = u1 * dn;
  w2 = 1.0 - w0 - w1;
  fr = (+w2 * pr2 + w1 * pr1 + w0 * pr0);
}

QAS_HD void wcns3_lr(const double f[5], double &fl, double &fr)
{
  const double eps = 1e-40;
  double c1 = f[1] - f[2];
  double is0 = c1 * c1;
  c1 = f[3] - f[2];
  double is1 = c1 * c1;
  double tau = f[3] - 2.0 * f[2] + f[1];
  tau = tau * tau;
  is0 = (1.0 + tau / (is0 + eps));
  is1 = (1.0 + tau / (is1 + eps));
  double w0 = 0.25 * is0, w1 = 0.75 * is1;
  w0 /= (w0 + w1);
  w1 = 1.0 - w0;
  fl = 0.5 * (w0 * (-f[1] + 3.0 * f[2]) + w1 * (f[2] + f[3]));
  w0 = 0.75 * is0;
  w1 = 0.25 * is1;
  w0 /= (w0 + w1);
  w1 = 1.0 - w0;
  fr = 0.5 * (w1 * (-f[3] + 3.0 * f[2]) + w0 * (f[2] + f[1]));
}

template <int ODR>
QAS_HD void nl_lr(const double f[5], double &fl, double &fr)
{
  if (ODR == 1) {
    fl = f[2];
    fr = f[2];
  } else if (ODR == 2) {
    double d = 0.5 * minmod(f[2] - f[1], f[3] - f[2]);
    fl = f[2] + d;
    fr = f[2] - d;
  } else if (ODR == 3) {
    wcns3_lr(f, fl, fr);
  } else {
    wcns4_lr(f, fl, fr);
  }
}

// nl_lr in the kernels' form: the 4th order by wcns4_lr_fast (hx: see there)
template <int ODR>
QAS_HD void nl_lr_fast(const double f[5], double &fl, double &fr, unsigned &hx)
{
  if (ODR == 4)
    wcns4_lr_fast(f, fl, fr, hx);
  else
    nl_lr<ODR>(f, fl, fr);
}

// ---------------------------------------------------------------------------
// Characteristic reconstruction of one cell's 5-point stencil.
// q[v][m]: v = ro, vn, vt, vu, bt, bu, pr; m = i-2..i+2.  bn: normal field at
// the centre.  vl: state at the right face (i+1/2), vr: at the left face.
// mhd_lrstate (common/mhd_func.c:108-161) with mhd_m_reconst / mhd_a_reconst
// (common/mhd_eigen.c:513-665) and the eigenvectors of mhd_eigen_mi/ae
// (:175-434), projections written sparsely.
// ---------------------------------------------------------------------------
template <int ODR>
QAS_HD void face_states(const double q[7][5], double bn, double gam, double vl[7],
                                            double vr[7])
{
  const double ro = q[0][2], vn = q[1][2], vt = q[2][2], vu = q[3][2];
  const double by = q[4][2], bz = q[5][2], pr = q[6][2];
  const bool fast = (ro * (vn * vn + vt * vt + vu * vu) > gam * pr);
  // wave speeds (identical prefix of mhd_eigen_mi and mhd_eigen_ae)
  double iro = 1.0 / ro;
  double cs2 = gam * pr * iro;
  double ca2 = bn * bn * iro;
  double ct2 = (by * by + bz * bz) * iro;
  double cb2 = cs2 + ca2 + ct2;
  double cf2 = 0.5 * (cb2 + sqrt(fabs(cb2 * cb2 - 4.0 * cs2 * ca2)));
  double sro = sqrt(ro);
  double isroh = 0.5 / sro;
  double icf2 = 1.0 / cf2;
  double byh = 0.5 * by, bzh = 0.5 * bz;
  double rcf = 0.0, icf2h = 0.0, ircfh = 0.0;
  if (fast) {
    double cf = sqrt(cf2);
    rcf = ro * cf;
    icf2h = 0.5 * icf2;
    ircfh = 0.5 / rcf;
  }
  const double nrcf = -rcf;

  double wl[7], wr[7];
  // characteristic field k over the stencil, then interpolate
#pragma unroll
  for (int k = 0; k < 7; k++) {
    double w[5];
#pragma unroll
    for (int m = 0; m < 5; m++) {
      const double r_ = q[0][m], n_ = q[1][m], t_ = q[2][m], u_ = q[3][m];
      const double b_ = q[4][m], c_ = q[5][m], p_ = q[6][m];
      double s;
      switch (k) {
        case 0: s = fast ? (((nrcf * n_ + by * b_) + bz * c_) + p_) : n_; break;
        case 1: s = ((cf2 * r_ - by * b_) - bz * c_) - p_; break;
        case 2: s = fast ? (((rcf * n_ + by * b_) + bz * c_) + p_) : ((by * b_ + bz * c_) + p_); break;
        case 3: s = sro * t_ + b_; break;
        case 4: s = sro * t_ - b_; break;
        case 5: s = sro * u_ + c_; break;
        default: s = sro * u_ - c_; break;
      }
      w[m] = s;
    }
    nl_lr<ODR>(w, wl[k], wr[k]);
  }
  // back to primitives (right eigenvectors)
  if (fast) {
    vl[0] = icf2h * wl[0] + icf2 * wl[1] + icf2h * wl[2];
    vr[0] = icf2h * wr[0] + icf2 * wr[1] + icf2h * wr[2];
    vl[1] = (-ircfh) * wl[0] + ircfh * wl[2];
    vr[1] = (-ircfh) * wr[0] + ircfh * wr[2];
    vl[6] = ((((0.5 * wl[0] + 0.5 * wl[2]) - byh * wl[3]) + byh * wl[4]) - bzh * wl[5]) + bzh * wl[6];
    vr[6] = ((((0.5 * wr[0] + 0.5 * wr[2]) - byh * wr[3]) + byh * wr[4]) - bzh * wr[5]) + bzh * wr[6];
  } else {
    vl[0] = icf2 * wl[1] + icf2 * wl[2];
    vr[0] = icf2 * wr[1] + icf2 * wr[2];
    vl[1] = wl[0];
    vr[1] = wr[0];
    vl[6] = (((wl[2] - byh * wl[3]) + byh * wl[4]) - bzh * wl[5]) + bzh * wl[6];
    vr[6] = (((wr[2] - byh * wr[3]) + byh * wr[4]) - bzh * wr[5]) + bzh * wr[6];
  }
  vl[2] = isroh * wl[3] + isroh * wl[4];
  vr[2] = isroh * wr[3] + isroh * wr[4];
  vl[3] = isroh * wl[5] + isroh * wl[6];
  vr[3] = isroh * wr[5] + isroh * wr[6];
  vl[4] = 0.5 * wl[3] - 0.5 * wl[4];
  vr[4] = 0.5 * wr[3] - 0.5 * wr[4];
  vl[5] = 0.5 * wl[5] - 0.5 * wl[6];
  vr[5] = 0.5 * wr[5] - 0.5 * wr[6];
  // exactly-zero velocity / transverse field stays exactly zero (mhd_eigen.c:574-587)
#pragma unroll
  for (int v = 1; v <= 5; v++) {
    bool z = (q[v][0] == 0.0) && (q[v][1] == 0.0) && (q[v][2] == 0.0) && (q[v][3] == 0.0) && (q[v][4] == 0.0);
    if (z) {
      vl[v] = 0.0;
      vr[v] = 0.0;
    }
  }
  // positivity fallback to first order (mhd_func.c:150-160)
  const double eps = 1e-12;
  if (vl[0] <= eps || vl[6] <= eps) {
    vl[0] = ro;
    vl[1] = vn;
    vl[6] = pr;
  }
  if (vr[0] <= eps || vr[6] <= eps) {
    vr[0] = ro;
    vr[1] = vn;
    vr[6] = pr;
  }
}

// mhd_lrstate with the primitive reconstruction mhd_reconst (common/mhd_eigen.c:667-706): each
// of (ro, vn, vb, vc, cb, cc, pr) interpolated on its own, then the positivity fallback
// (common/mhd_func.c:150-160)
template <int ODR, class ST>
QAS_HD void face_states_prim(const ST &st, double vl[7], double vr[7])
{
#pragma unroll
  for (int f = 0; f < 7; f++) {
    const double w[5] = {st(f, 0), st(f, 1), st(f, 2), st(f, 3), st(f, 4)};
    nl_lr<ODR>(w, vl[f], vr[f]);
  }
  const double eps = 1e-12;
  if (vl[0] <= eps || vl[6] <= eps) {
    vl[0] = st(0, 2);
    vl[1] = st(1, 2);
    vl[6] = st(6, 2);
  }
  if (vr[0] <= eps || vr[6] <= eps) {
    vr[0] = st(0, 2);
    vr[1] = st(1, 2);
    vr[6] = st(6, 2);
  }
}

// every value added is zero (either sign), tested by one OR of the bits on the integer pipe
struct ZeroTest {
  unsigned long long b = 0;
  QAS_HD void add(double x)
  {
#if defined(__CUDA_ARCH__)
    b |= (unsigned long long)__double_as_longlong(x);
#else
    unsigned long long t;
    memcpy(&t, &x, 8);
    b |= t;
#endif
  }
  QAS_HD bool zero() const { return (b << 1) == 0; }
};

// ---------------------------------------------------------------------------
// Same reconstruction in the kernels' form: the stencil is read per characteristic field
// (`P` is a functor P(v, m) returning primitive v at stencil point m), each component's two
// states are handed to out(v, left-face-of-the-right-neighbour state, own left-face state)
// as soon as they are final, and the fields go through one loop body in pairs: {1, 2} (the
// entropy and the pressure-like row), {3, 4} and {5, 6} (the Alfven rows of either transverse
// axis); field 0 stands alone.  out.again(P, bn, gam) is called, rarely, where the fast
// interpolation does not hold, and stores all the states anew by face_states.  Three copies of the interpolation instead of seven keep the
// code small (the sweeps are held up by instruction fetch) and few values live.
// ---------------------------------------------------------------------------
template <int ODR, class Stencil, class Out>
QAS_HD void face_states_emit(const Stencil &P, double bn, double gam, const Out &out)
{
  unsigned hx = 0;
  double cf2, icf2, sro, isroh, by, bz;
  bool fast;
  double l0, r0, l1, r1, l6, r6;  // components 0 (ro), 1 (vn), 6 (pr)
  {
    const double ro = P(0, 2), vn = P(1, 2), vt = P(2, 2), vu = P(3, 2), pr = P(6, 2);
    by = P(4, 2);
    bz = P(5, 2);
    fast = (ro * (vn * vn + vt * vt + vu * vu) > gam * pr);
    const double iro = 1.0 / ro;
    const double cs2 = gam * pr * iro;
    const double ca2 = bn * bn * iro;
    const double ct2 = (by * by + bz * bz) * iro;
    const double cb2 = cs2 + ca2 + ct2;
    cf2 = 0.5 * (cb2 + sqrt(fabs(p2fma(-4.0, cs2 * ca2, cb2 * cb2))));
    sro = sqrt(ro);
    isroh = 0.5 * (1.0 / sro);
    icf2 = 1.0 / cf2;
  }
  {  // field 0: vn of the slow eigen-system (mhd_eigen_mi), the backward fast wave of mhd_eigen_ae
    double w[5];
    ZeroTest tn;
#pragma unroll
    for (int m = 0; m < 5; m++) {
      w[m] = P(1, m);
      tn.add(w[m]);
    }
    if (fast) {
      const double rcf = P(0, 2) * sqrt(cf2);
#pragma unroll
      for (int m = 0; m < 5; m++) w[m] = (((-rcf) * w[m] + by * P(4, m)) + bz * P(5, m)) + P(6, m);
    }
    nl_lr_fast<ODR>(w, l1, r1, hx);
    if (!fast && tn.zero()) {
      l1 = 0.0;
      r1 = 0.0;
    }
  }
#pragma unroll 1
  for (int g = 0; g < 3; g++) {
    double wa[5], wb[5], la, ra, lb, rb;
    ZeroTest tv, tb;
    if (g == 0) {
#pragma unroll
      for (int m = 0; m < 5; m++) {
        const double p_ = P(6, m), yb = by * P(4, m), zc = bz * P(5, m);
        wa[m] = ((cf2 * P(0, m) - yb) - zc) - p_;
        wb[m] = (yb + zc) + p_;
      }
      if (fast) {
        const double rcf = P(0, 2) * sqrt(cf2);
#pragma unroll
        for (int m = 0; m < 5; m++) wb[m] = ((rcf * P(1, m) + by * P(4, m)) + bz * P(5, m)) + P(6, m);
      }
    } else {
#pragma unroll
      for (int m = 0; m < 5; m++) {
        const double t_ = P(1 + g, m), b_ = P(3 + g, m);
        tv.add(t_);
        tb.add(b_);
        const double st = sro * t_;
        wa[m] = st + b_;
        wb[m] = st - b_;
      }
    }
    nl_lr_fast<ODR>(wa, la, ra, hx);
    nl_lr_fast<ODR>(wb, lb, rb, hx);
    if (g == 0) {
      if (fast) {
        const double icf2h = 0.5 * icf2, ircfh = 0.5 / (P(0, 2) * sqrt(cf2));
        l0 = icf2h * l1 + icf2 * la + icf2h * lb;
        r0 = icf2h * r1 + icf2 * ra + icf2h * rb;
        l6 = 0.5 * (l1 + lb);
        r6 = 0.5 * (r1 + rb);
        l1 = (-ircfh) * l1 + ircfh * lb;
        r1 = (-ircfh) * r1 + ircfh * rb;
        ZeroTest tn;
#pragma unroll
        for (int m = 0; m < 5; m++) tn.add(P(1, m));
        if (tn.zero()) {
          l1 = 0.0;
          r1 = 0.0;
        }
      } else {
        l0 = icf2 * la + icf2 * lb;
        r0 = icf2 * ra + icf2 * rb;
        l6 = lb;
        r6 = rb;
      }
    } else {
      const double bh = 0.5 * (g == 1 ? by : bz);
      l6 = (l6 - bh * la) + bh * lb;
      r6 = (r6 - bh * ra) + bh * rb;
      const bool zv = tv.zero(), zb = tb.zero();  // exactly-zero fields stay exactly zero
      out(1 + g, zv ? 0.0 : isroh * la + isroh * lb, zv ? 0.0 : isroh * ra + isroh * rb);
      out(3 + g, zb ? 0.0 : 0.5 * (la - lb), zb ? 0.0 : 0.5 * (ra - rb));
    }
  }
  const double eps = 1e-12;  // positivity fallback to first order (mhd_func.c:150-160)
  if (l0 <= eps || l6 <= eps) {
    l0 = P(0, 2);
    l1 = P(1, 2);
    l6 = P(6, 2);
  }
  if (r0 <= eps || r6 <= eps) {
    r0 = P(0, 2);
    r1 = P(1, 2);
    r6 = P(6, 2);
  }
  out(0, l0, r0);
  out(1, l1, r1);
  out(6, l6, r6);
  // a smoothness denominator beyond 2^900 or a NaN: all over again with the reference's divisions
  if (ODR == 4 && hx >= WCNS_HX) out.again(P, bn, gam);
}

// face_states from a stencil functor
template <int ODR, class Stencil>
QAS_HD void face_states_of(const Stencil &P, double bn, double gam, double vl[7], double vr[7])
{
  double q[7][5];
#pragma unroll
  for (int f = 0; f < 7; f++)
#pragma unroll
    for (int m = 0; m < 5; m++) q[f][m] = P(f, m);
  face_states<ODR>(q, bn, gam, vl, vr);
}

// the same into arrays
template <int ODR>
struct StatesInto {
  double *vl, *vr;
  QAS_HD void operator()(int m, double l, double r) const
  {
    vl[m] = l;
    vr[m] = r;
  }
  template <class Stencil>
  QAS_HD void again(const Stencil &P, double bn, double gam) const
  {
    face_states_of<ODR>(P, bn, gam, vl, vr);
  }
};
template <int ODR, class Stencil>
QAS_HD void face_states_grouped(const Stencil &P, double bn, double gam, double vl[7], double vr[7])
{
  face_states_emit<ODR>(P, bn, gam, StatesInto<ODR>{vl, vr});
}

// ---------------------------------------------------------------------------
// mhd_lrstate with the Athena-type characteristic reconstruction mhd_c_reconst
// (common/mhd_eigen.c:436-511) and the eigenvectors of mhd_eigen_st (:5-173, Stone et al.
// 2008, ApJS 178, 137), which the reference offers beside mhd_m/a_reconst (the call in
// mhd_lrstate switched): one eigen-system for every state, no fast/slow choice.  L and R are
// 7x7 with literal zeros; each projection keeps the reference's left-to-right sum over the
// non-zero entries (an omitted 0*x term can only change the sign of an exact zero), every
// entry formed by the reference's expression.  Then the exact-zero flags of mhd_c_reconst and
// the positivity fallback of mhd_lrstate.
// ---------------------------------------------------------------------------
template <int ODR, class Stencil>
QAS_HD void face_states_athena(const Stencil &P, double bx, double gamma, double vl[7], double vr[7])
{
  const double ro = P(0, 2), vn = P(1, 2), by = P(4, 2), bz = P(5, 2), pr = P(6, 2);
  // mhd_eigen_st at the centre point
  const double eps = 1e-12;
  const double sqrt2 = sqrt(2.0);
  double iro = 1.0 / ro;
  double sro = sqrt(ro);
  double isro = 1.0 / sro;
  double bxsr = bx * isro;
  double bysr = by * isro;
  double bzsr = bz * isro;
  double bx2 = bxsr * bxsr;
  double bt2 = bysr * bysr + bzsr * bzsr;
  double b2 = bx2 + bt2;
  double a2 = fabs(gamma * pr / ro);
  double aa = sqrt(a2);
  double ca2 = bx2;
  double junk = sqrt(fabs((a2 + b2) * (a2 + b2) - 4.0 * a2 * ca2));
  double cf2 = fabs(0.5 * (a2 + b2 + junk));
  double cf = sqrt(cf2);
  double cs2 = fabs(0.5 * (a2 + b2 - junk));
  double cs = sqrt(cs2);
  bx2 = bx * bx;
  bt2 = by * by + bz * bz;
  b2 = bx2 + bt2;
  double denom = 1.0 / sqrt(bt2);
  bool flag = (bt2 > eps * b2);
  const double betay = flag ? (by * denom) : (0.5 * sqrt2);
  const double betaz = flag ? (bz * denom) : (0.5 * sqrt2);
  denom = 1.0 / sqrt(fabs(cf2 - cs2));
  flag = ((bt2 > eps * b2) || (fabs(gamma * pr - bx2) > eps * gamma * pr));
  const double alphaf = flag ? (sqrt(fabs(a2 - cs2)) * denom) : 1.0;
  const double alphas = flag ? (sqrt(fabs(cf2 - a2)) * denom) : 0.0;
  const double sgnbx = (bx > 0) ? (1.0) : (-1.0);
  const double cfalf = cf * alphaf;
  const double csals = cs * alphas;
  const double aaalf = aa * alphaf;
  const double aaals = aa * alphas;
  denom = 0.5 / a2;
  // left eigenvectors (rows; k = 0..6 are mhd_eigen_st's l1..l7), non-zero entries
  const double l0v = -cfalf * denom, l0t = +csals * denom * sgnbx * betay, l0u = +csals * denom * sgnbx * betaz;
  const double l0b = +aaals * denom * isro * betay, l0c = +aaals * denom * isro * betaz, l0p = alphaf * denom * iro;
  const double l1t = -0.5 * betaz, l1u = +0.5 * betay;
  const double l1b = -0.5 * isro * betaz * sgnbx, l1c = +0.5 * isro * betay * sgnbx;
  const double l2v = -csals * denom, l2t = -cfalf * denom * sgnbx * betay, l2u = -cfalf * denom * sgnbx * betaz;
  const double l2b = -aaalf * denom * isro * betay, l2c = -aaalf * denom * isro * betaz, l2p = alphas * denom * iro;
  const double l3p = -1.0 / a2;
  double wl[7], wr[7];
  bool zvn = true, zvt = true, zvu = true, zbt = true, zbu = true;
  {  // the six waves that see (vn, vt, vu, bt, bu, pr): l1..l3, l5..l7 (mirror signs)
    double w0[5], w6[5], w2[5], w4[5];
#pragma unroll
    for (int m = 0; m < 5; m++) {
      const double n_ = P(1, m), t_ = P(2, m), u_ = P(3, m), b_ = P(4, m), c_ = P(5, m), p_ = P(6, m);
      zvn = zvn && (n_ == 0.0);
      zvt = zvt && is_zero(t_);
      zvu = zvu && is_zero(u_);
      zbt = zbt && (b_ == 0.0);
      zbu = zbu && (c_ == 0.0);
      w0[m] = ((((l0v * n_ + l0t * t_) + l0u * u_) + l0b * b_) + l0c * c_) + l0p * p_;
      w6[m] = (((((-l0v) * n_ + (-l0t) * t_) + (-l0u) * u_) + l0b * b_) + l0c * c_) + l0p * p_;
      w2[m] = ((((l2v * n_ + l2t * t_) + l2u * u_) + l2b * b_) + l2c * c_) + l2p * p_;
      w4[m] = (((((-l2v) * n_ + (-l2t) * t_) + (-l2u) * u_) + l2b * b_) + l2c * c_) + l2p * p_;
    }
    nl_lr<ODR>(w0, wl[0], wr[0]);
    nl_lr<ODR>(w6, wl[6], wr[6]);
    nl_lr<ODR>(w2, wl[2], wr[2]);
    nl_lr<ODR>(w4, wl[4], wr[4]);
  }
  {  // the Alfven waves l2, l6 (vt, vu, bt, bu) and the entropy wave l4 (ro, pr)
    double w1[5], w5[5], w3[5];
#pragma unroll
    for (int m = 0; m < 5; m++) {
      const double t_ = P(2, m), u_ = P(3, m), b_ = P(4, m), c_ = P(5, m);
      w1[m] = ((l1t * t_ + l1u * u_) + l1b * b_) + l1c * c_;
      w5[m] = (((-l1t) * t_ + (-l1u) * u_) + l1b * b_) + l1c * c_;
      w3[m] = P(0, m) + l3p * P(6, m);
    }
    nl_lr<ODR>(w1, wl[1], wr[1]);
    nl_lr<ODR>(w5, wl[5], wr[5]);
    nl_lr<ODR>(w3, wl[3], wr[3]);
  }
  // right eigenvectors (columns; r1..r7 of mhd_eigen_st), non-zero entries
  const double r0r = ro * alphaf, r0v = -cfalf, r0t = +csals * sgnbx * betay, r0u = +csals * sgnbx * betaz;
  const double r0b = +aaals * sro * betay, r0c = +aaals * sro * betaz, r0p = alphaf * gamma * pr;
  const double r1t = -betaz, r1u = +betay, r1b = -sro * betaz * sgnbx, r1c = +sro * betay * sgnbx;
  const double r2r = ro * alphas, r2v = -csals, r2t = -cfalf * sgnbx * betay, r2u = -cfalf * sgnbx * betaz;
  const double r2b = -aaalf * sro * betay, r2c = -aaalf * sro * betaz, r2p = alphas * gamma * pr;
  auto back = [&](const double w[7], double u[7]) {
    u[0] = (((r0r * w[0] + r2r * w[2]) + w[3]) + r2r * w[4]) + r0r * w[6];
    u[1] = ((r0v * w[0] + r2v * w[2]) + (-r2v) * w[4]) + (-r0v) * w[6];
    u[2] = (((((r0t * w[0] + r1t * w[1]) + r2t * w[2]) + (-r2t) * w[4]) + (-r1t) * w[5]) + (-r0t) * w[6]);
    u[3] = (((((r0u * w[0] + r1u * w[1]) + r2u * w[2]) + (-r2u) * w[4]) + (-r1u) * w[5]) + (-r0u) * w[6]);
    u[4] = (((((r0b * w[0] + r1b * w[1]) + r2b * w[2]) + r2b * w[4]) + r1b * w[5]) + r0b * w[6]);
    u[5] = (((((r0c * w[0] + r1c * w[1]) + r2c * w[2]) + r2c * w[4]) + r1c * w[5]) + r0c * w[6]);
    u[6] = ((r0p * w[0] + r2p * w[2]) + r2p * w[4]) + r0p * w[6];
  };
  back(wl, vl);
  back(wr, vr);
  if (zvn) { vl[1] = 0.0; vr[1] = 0.0; }
  if (zvt) { vl[2] = 0.0; vr[2] = 0.0; }
  if (zvu) { vl[3] = 0.0; vr[3] = 0.0; }
  if (zbt) { vl[4] = 0.0; vr[4] = 0.0; }
  if (zbu) { vl[5] = 0.0; vr[5] = 0.0; }
  const double peps = 1e-12;
  if (vl[0] <= peps || vl[6] <= peps) {
    vl[0] = ro;
    vl[1] = vn;
    vl[6] = pr;
  }
  if (vr[0] <= peps || vr[6] <= peps) {
    vr[0] = ro;
    vr[1] = vn;
    vr[6] = pr;
  }
}

// ---------------------------------------------------------------------------
// Riemann solvers, common/mhd_flux.c.  L/R = (ro,vn,vt,vu,bt,bu,pr),
// F = (fro,fmn,fmt,fmu,fbt,fbu,fen).
// ---------------------------------------------------------------------------
#define QAS_FL_EPS (1e-8)

// cb + sqrt(|cb^2 - 4 x ca|), the larger of the two sides (twice the squared speed of the faster
// side): the sum and the root are monotonic also after rounding, so where one side has both the
// larger cb and the larger discriminant its root alone is taken; the second root only where the
// two disagree
QAS_HD double larger_speed2(double cbl, double xl, double cal, double cbr, double xr, double car)
{
  const double dl = fabs(p2fma(-4.0, xl * cal, cbl * cbl)), dr = fabs(p2fma(-4.0, xr * car, cbr * cbr));
  const bool left = cbl >= cbr;
  const double cb = left ? cbl : cbr, d = left ? dl : dr, co = left ? cbr : cbl, o = left ? dr : dl;
  const double f = cb + sqrt(d);
  if (d >= o) return f;
  return qmax(f, co + sqrt(o));  // a NaN on either side comes here too
}

// HLLD (LOW=false, mhd_flux.c:435-561) and low-dissipation LHLLD (LOW=true, :563-698).
// The reference forms all four star states of both sides and adds them with weights of exactly 0
// or 1; here the side of the contact (vnc > 0) and the outer / inner state are chosen first and
// only that side's energy, Alfven-wave speed and products are formed (each by the reference's
// expression): two IEEE divisions and about a third of the FP64 work less.  A weighted sum and
// the choice differ only where an unused state is not finite, which needs a face state with
// ro <= 0 or pr <= 0 (sl < vnc < sr otherwise).
template <bool LOW>
QAS_HD void flux_hlld(const double L[7], const double R[7], double bnc, double gamma, double gammam1i,
                                          double dv0, double dv1, double F[7])
{
  const double rol = L[0], vnl = L[1], vtl = L[2], vul = L[3], btl = L[4], bul = L[5], prl = L[6];
  const double ror = R[0], vnr = R[1], vtr = R[2], vur = R[3], btr = R[4], bur = R[5], prr = R[6];
  const double bnc2 = bnc * bnc;
  const bool neg = !(bnc > 0);  // sgn = -1
  const double roli = 1.0 / rol;
  const double bl2 = btl * btl + bul * bul;  // 2 pml
  const double ptl = p2fma(0.5, bl2, prl);
  const double rori = 1.0 / ror;
  const double br2 = btr * btr + bur * bur;
  const double ptr = p2fma(0.5, br2, prr);
  const double vl2 = vnl * vnl + vtl * vtl + vul * vul;
  const double vr2 = vnr * vnr + vtr * vtr + vur * vur;
  const double cl2 = gamma * prl * roli;
  const double cr2 = gamma * prr * rori;
  const double cal2 = bnc2 * roli;
  const double car2 = bnc2 * rori;
  const double tl = bl2 * roli, tr = br2 * rori;
  const double cmax = sqrt(0.5 * larger_speed2(cl2 + cal2 + tl, cl2, cal2, cr2 + car2 + tr, cr2, car2));
  double sl = qmin(0.0, qmin(vnl, vnr) - cmax);
  double sr = qmax(0.0, qmax(vnl, vnr) + cmax);
  double slvl = sl - vnl;
  double srvr = sr - vnr;
  double rslvl = rol * slvl;
  double rsrvr = ror * srvr;
  double drsvi = 1.0 / (rsrvr - rslvl);
  double vnc, ptc;
  if (LOW) {
    double theta = qmin(1.0, (cmax - qmin(dv0, 0.0)) / (cmax - qmin(dv1, 0.0)));
    theta *= theta;
    theta *= theta;
    vnc = (rsrvr * vnr - rslvl * vnl - theta * (ptr - ptl)) * drsvi;
    const double cc = larger_speed2(vl2 + cal2 + tl, vl2, cal2, vr2 + car2 + tr, vr2, car2);
    double mcc = qmin(1.0, sqrt(0.5 * cc) / cmax);
    ptc = (rsrvr * ptl - rslvl * ptr + (mcc * (2.0 - mcc)) * rsrvr * rslvl * (vnr - vnl)) * drsvi;
  } else {
    vnc = (rsrvr * vnr - rslvl * vnl - ptr + ptl) * drsvi;
    ptc = (rsrvr * ptl - rslvl * ptr + rsrvr * rslvl * (vnr - vnl)) * drsvi;
  }
  double slvc = sl - vnc;
  double srvc = sr - vnc;
  double ro2l = rslvl / slvc;
  double ro2r = rsrvr / srvc;
  double rhdl = rslvl * slvc - bnc2;
  double rhdr = rsrvr * srvc - bnc2;
  double vt2l, vu2l, bt2l, bu2l, vt2r, vu2r, bt2r, bu2r;
  if (fabs(rhdl) > QAS_FL_EPS) {
    double rhdli = 1.0 / rhdl;
    double rhnvl = (vnl - vnc) * bnc;
    double rhnbl = rslvl * slvl - bnc2;
    const double av = rhnvl * rhdli, ab = rhnbl * rhdli;
    vt2l = vtl + av * btl;
    vu2l = vul + av * bul;
    bt2l = ab * btl;
    bu2l = ab * bul;
  } else {
    vt2l = vtl; vu2l = vul; bt2l = btl; bu2l = bul;
  }
  if (fabs(rhdr) > QAS_FL_EPS) {
    double rhdri = 1.0 / rhdr;
    double rhnvr = (vnr - vnc) * bnc;
    double rhnbr = rsrvr * srvr - bnc2;
    const double av = rhnvr * rhdri, ab = rhnbr * rhdri;
    vt2r = vtr + av * btr;
    vu2r = vur + av * bur;
    bt2r = ab * btr;
    bu2r = ab * bur;
  } else {
    vt2r = vtr; vu2r = vur; bt2r = btr; bu2r = bur;
  }
  const double rro2l = sqrt(ro2l);
  const double rro2r = sqrt(ro2r);
  const double rro2i = 1.0 / (rro2r + rro2l);
  const bool left = vnc > 0;
  // the upwind side
  const double ro_ = left ? rol : ror, vn_ = left ? vnl : vnr, vt_ = left ? vtl : vtr, vu_ = left ? vul : vur;
  const double bt_ = left ? btl : btr, bu_ = left ? bul : bur, pr_ = left ? prl : prr, pt_ = left ? ptl : ptr;
  const double b2_ = left ? bl2 : br2, v2_ = left ? vl2 : vr2, sv_ = left ? slvl : srvr, sc_ = left ? slvc : srvc;
  const double vt2 = left ? vt2l : vt2r, vu2 = left ? vu2l : vu2r;
  const double bt2 = left ? bt2l : bt2r, bu2 = left ? bu2l : bu2r;
  const double rro2 = left ? rro2l : rro2r;
  const double en = p2fma(0.5, ro_ * v2_, p2fma(0.5, b2_, gammam1i * pr_));
  const double vb = vt_ * bt_ + vu_ * bu_;
  const double vb2 = vt2 * bt2 + vu2 * bu2;
  const double en2 = (sv_ * en - pt_ * vn_ + ptc * vnc + bnc * (vb - vb2)) / sc_;
  const double ca = fabs(bnc) / rro2;
  const bool outer = left ? (vnc - ca > 0) : !(vnc + ca > 0);
  const double vt3m = (rro2r * vt2r + rro2l * vt2l + flip(bt2r - bt2l, neg)) * rro2i;
  const double vu3m = (rro2r * vu2r + rro2l * vu2l + flip(bu2r - bu2l, neg)) * rro2i;
  const double rr = rro2r * rro2l;
  const double bt3m = (rro2l * bt2r + rro2r * bt2l + flip(rr * (vt2r - vt2l), neg)) * rro2i;
  const double bu3m = (rro2l * bu2r + rro2r * bu2l + flip(rr * (vu2r - vu2l), neg)) * rro2i;
  const double vb3m = vt3m * bt3m + vu3m * bu3m;
  // en2 - rro2*(vb2 - vb3)*sgn on the left, + on the right
  const double en3 = en2 + flip(rro2 * (vb2 - vb3m), neg != left);
  const double rou = left ? ro2l : ro2r;
  const double vtu = outer ? vt2 : vt3m;
  const double vuu = outer ? vu2 : vu3m;
  const double btu = outer ? bt2 : bt3m;
  const double buu = outer ? bu2 : bu3m;
  const double enu = outer ? en2 : en3;
  const double mf = rou * vnc;
  F[0] = mf;
  F[1] = p2fma(-0.5, bnc2, mf * vnc + ptc);
  F[2] = rou * vtu * vnc - bnc * btu;
  F[3] = rou * vuu * vnc - bnc * buu;
  F[4] = btu * vnc - bnc * vtu;
  F[5] = buu * vnc - bnc * vuu;
  F[6] = (enu + ptc) * vnc - bnc * (vtu * btu + vuu * buu);
}

// MLAU all-speed flux, common/mhd_flux.c:7-192.  Every value keeps the reference's expression
// and rounding; what differs is which values are formed.  The reference weighs the two sides with
// dirl, dirr = (1, 0) or (0, 1); here the upwind side's operands are chosen and only its energy,
// products and sums are formed, products by +-1 are sign flips, and the larger of two speeds takes
// one square root where it can (larger_speed2).  Few values are live at once (the kernels run this
// solver at 80 registers): the two transverse components are finished one after the other, and
// each flux goes to out(m, value) as soon as it is final (the kernels store it at once).  out
// receives F = (fro, fmn, fmt, fmu, fbt, fbu, fen) in the order 0, 1, 2, 4, 3, 5, 6.
template <class Out>
QAS_HD void flux_mlau_out(const double L[7], const double R[7], double bnc, double gamma, double gammam1i, double dv0,
                          double dv1, Out &&out)
{
  const double rol = L[0], vnl = L[1], vtl = L[2], vul = L[3], btl = L[4], bul = L[5], prl = L[6];
  const double ror = R[0], vnr = R[1], vtr = R[2], vur = R[3], btr = R[4], bur = R[5], prr = R[6];
  const double bnc2 = bnc * bnc;
  const bool neg = !(bnc > 0);  // sgn = -1
  const double bnca = flip(bnc, neg);
  const double roli = 1.0 / rol;
  const double vl2 = vnl * vnl + vtl * vtl + vul * vul;
  const double bl2 = btl * btl + bul * bul;  // 2 pml
  const double ptl = p2fma(0.5, bl2, prl);
  const double rori = 1.0 / ror;
  const double vr2 = vnr * vnr + vtr * vtr + vur * vur;
  const double br2 = btr * btr + bur * bur;
  const double ptr = p2fma(0.5, br2, prr);
  double cfn, cfmod;
  {
    const double cl2 = gamma * prl * roli, cr2 = gamma * prr * rori;
    const double cal2 = bnc2 * roli, car2 = bnc2 * rori;
    const double tl = bl2 * roli, tr = br2 * rori;
    cfn = sqrt(0.5 * larger_speed2(cl2 + cal2 + tl, cl2, cal2, cr2 + car2 + tr, cr2, car2));
    cfmod = sqrt(0.5 * larger_speed2(vl2 + cal2 + tl, vl2, cal2, vr2 + car2 + tr, vr2, car2));
  }
  const double cfni = 1.0 / cfn;
  const double sl = qmin(0.0, qmin(vnl, vnr) - cfn);
  const double sr = qmax(0.0, qmax(vnl, vnr) + cfn);
  const double mal = vnl * cfni;
  const double mar = vnr * cfni;
  double theta = qmin(1.0, (cfn - qmin(dv0, 0.0)) / (cfn - qmin(dv1, 0.0)));
  theta *= theta;
  theta *= theta;
  const double alpha = 0.1875;
  double bfl, ffl, bfr, ffr;
  if (fabs(mal) > 1.0) {
    bfl = mal > 0 ? 1.0 : 0.0;
    ffl = bfl * mal;
  } else {
    const double p1 = mal + 1.0, m1 = mal * mal - 1.0, pp = p1 * p1, mm = m1 * m1;
    bfl = p2fma(0.25, pp * (2.0 - mal), alpha * mal * m1 * m1);
    ffl = p2fma(0.25, pp, 0.125 * mm);
  }
  if (fabs(mar) > 1.0) {
    bfr = mar > 0 ? 0.0 : 1.0;
    ffr = bfr * mar;
  } else {
    const double p1 = mar - 1.0, m1 = mar * mar - 1.0, pp = p1 * p1, mm = m1 * m1;
    bfr = p2fma(0.25, pp * (2.0 + mar), -(alpha * mar * m1 * m1));
    ffr = p2fma(-0.25, pp, -(0.125 * mm));
  }
  const double mnc = ffl + ffr;
  double mflux = mnc * cfn;
  mflux -= qmax(1.0 - fabs(mnc), 0.0) * theta * cfni * (ptr - ptl) / (rol + ror);
  const bool up = mflux > 0;  // the left side is upwind: dirl = 1, dirr = 0
  mflux *= up ? rol : ror;
  out(0, mflux);
  {
    double ptot = bfl * ptl + bfr * ptr;
    ptot = p2fma(-0.25, bfl * bfr * (rol + ror) * cfmod * (vnr - vnl), ptot);
    ptot = p2fma(-0.5, (1.0 - cfmod * cfni) * (bfl + bfr - 1.0) * (ptl + ptr), ptot);
    out(1, p2fma(-0.5, bnc2, mflux * (up ? vnl : vnr) + ptot));
  }
  const double roui = up ? roli : rori;
  double e6;  // fen = e6 - bnvb
  {
    const double en = p2fma(0.5, (up ? rol : ror) * (up ? vl2 : vr2),
                            p2fma(0.5, up ? bl2 : br2, gammam1i * (up ? prl : prr)));
    e6 = mflux * ((en + (up ? ptl : ptr)) * roui);
  }
  const double slvl = sl - vnl;
  const double srvr = sr - vnr;
  const double snc = up ? sl : sr;
  const double rsl = rol * slvl, rsr = ror * srvr;
  const double vndnm = mflux + (up ? rsl : rsr);
  const double vnc = ((fabs(vndnm) > QAS_FL_EPS) && (snc != 0)) ? (mflux * snc / vndnm) : (up ? vnl : vnr);
  const double slvc = sl - vnc;
  const double srvc = sr - vnc;
  const double slvci = 1.0 / slvc;
  const double srvci = 1.0 / srvc;
  const double rhdl = rsl * slvc - bnc2;
  const double rhdr = rsr * srvc - bnc2;
  // the reference's q of each side, used only where |rhd| > FL_EPS (else the corrections are 0.0)
  const bool hl = fabs(rhdl) > QAS_FL_EPS, hr = fabs(rhdr) > QAS_FL_EPS;
  const double ql = hl ? (vnc - vnl) / rhdl : 0.0;
  const double qr = hr ? (vnc - vnr) / rhdr : 0.0;
  const double cmpl = slvl * slvci;
  const double cmpr = srvr * srvci;
  const double srol = sqrt(rol * cmpl);
  const double sror = sqrt(ror * cmpr);
  const double sroi = 1.0 / (srol + sror);
  const double srollri = srol * sroi;
  const double srorlri = sror * sroi;
  const double bnflb = flip(qmin(qmax(0.0, srollri * (bnca + sror * vnc)), bnca), neg);
  const double bnfrb = flip(qmin(qmax(0.0, srorlri * (bnca - srol * vnc)), bnca), neg);
  const double bnflv = flip(qmin(qmax(0.0, srorlri * (bnca + mflux / sror)), bnca), neg);
  const double bnfrv = flip(qmin(qmax(0.0, srollri * (bnca - mflux / srol)), bnca), neg);
  const double bnsrv = qmax(bnca - flip(vnc * (up ? srol : sror), !up), 0.0);
  const double ccb = sroi * bnsrv;
  const double ccv = srol * sror * ccb;
  // one transverse component (t: vt, bt; u: vu, bu): its momentum and induction fluxes, its
  // terms of vb1 and vb2 (v*b of the upwind side) and of vb3's numerator
  auto comp = [&](double vl_, double bl_, double vr_, double br_, int mf, int mb, double &p1, double &p2,
                  double &q3) {
    const double dvl = hl ? -bnc * bl_ * ql : 0.0;
    const double dbl = hl ? bnc2 * bl_ * ql * slvci : 0.0;
    const double dvr = hr ? -bnc * br_ * qr : 0.0;
    const double dbr = hr ? bnc2 * br_ * qr * srvci : 0.0;
    const double v2l = dvl + vl_;
    const double b2l = dbl + bl_ * cmpl;
    const double v2r = dvr + vr_;
    const double b2r = dbr + br_ * cmpr;
    const double vu_ = up ? vl_ : vr_, bu_ = up ? bl_ : br_;
    double bnv = bnflb * v2l + bnfrb * v2r + ccb * (b2r - b2l);
    double bnb = bnflv * b2l + bnfrv * b2r + ccv * (v2r - v2l);
    bnv -= vnc * (up ? dbl : dbr);
    bnb -= mflux * (up ? dvl : dvr);
    const double fm = mflux * vu_ - bnb;
    const double fb = mflux * bu_ * roui - bnv;
    out(mf, fm);
    out(mb, fb);
    p1 = vu_ * bu_;
    p2 = (up ? v2l : v2r) * (up ? b2l : b2r);
    q3 = (fm * vnc + fb * bnc) * (fm * bnc + fb * mflux);
  };
  double vb1 = 0.0, vb2 = 0.0, q3 = 0.0;
#pragma unroll
  for (int t = 0; t < 2; t++) {
    double p1, p2, q;
    comp(t == 0 ? vtl : vul, t == 0 ? btl : bul, t == 0 ? vtr : vur, t == 0 ? btr : bur, 2 + t, 4 + t, p1, p2, q);
    vb1 = t == 0 ? p1 : vb1 + p1;
    vb2 = t == 0 ? p2 : vb2 + p2;
    q3 = t == 0 ? q : q3 + q;
  }
  double rv2b2 = (mflux * vnc - bnc2);
  rv2b2 *= rv2b2;
  double vb3 = 0.0;
  if (rv2b2 > QAS_FL_EPS * QAS_FL_EPS) vb3 = q3 / rv2b2;
  const double bnvb = flip(bnca * (snc * vb2 - vnc * vb1) * (up ? slvci : srvci) + bnsrv * (vb3 - vb2), neg);
  out(6, e6 - bnvb);
}

QAS_HD void flux_mlau(const double L[7], const double R[7], double bnc, double gamma, double gammam1i, double dv0,
                      double dv1, double F[7])
{
  flux_mlau_out(L, R, bnc, gamma, gammam1i, dv0, dv1, [&](int m, double x) { F[m] = x; });
}

// Roe flux, common/mhd_flux.c:194-433
QAS_HD void flux_roe(const double L[7], const double R[7], double bnc, double gamma, double gammam1i, double F[7])
{
  const double rol = L[0], vnl = L[1], vtl = L[2], vul = L[3], btl = L[4], bul = L[5], prl = L[6];
  const double ror = R[0], vnr = R[1], vtr = R[2], vur = R[3], btr = R[4], bur = R[5], prr = R[6];
  double gammam1 = gamma - 1.0;
  double gammam2 = gamma - 2.0;
  double roli = 1.0 / rol;
  double rori = 1.0 / ror;
  double rrol = sqrt(rol);
  double rror = sqrt(ror);
  double rroi = 1.0 / (rrol + rror);
  double robar = rrol * rror;
  double robari = 1.0 / robar;
  double rrobar = sqrt(robar);
  double rrobai = sqrt(robari);
  double vnbar = (rrol * vnl + rror * vnr) * rroi;
  double vtbar = (rrol * vtl + rror * vtr) * rroi;
  double vubar = (rrol * vul + rror * vur) * rroi;
  double bnbar = bnc;
  double btbar = (rrol * btr + rror * btl) * rroi;
  double bubar = (rrol * bur + rror * bul) * rroi;
  double hl = (+gamma * gammam1i * prl * roli + 0.5 * (vnl * vnl + vtl * vtl + vul * vul) +
               (bnbar * bnbar + btl * btl + bul * bul) * roli);
  double hr = (+gamma * gammam1i * prr * rori + 0.5 * (vnr * vnr + vtr * vtr + vur * vur) +
               (bnbar * bnbar + btr * btr + bur * bur) * rori);
  double hbar = (rrol * hl + rror * hr) * rroi;
  double btave = 0.5 * (btl + btr);
  double buave = 0.5 * (bul + bur);
  double sgn = (bnbar > 0) ? (1.0) : (-1.0);
  double db2 = 0.5 * gammam2 * gammam1i * ((btr - btl) * (btr - btl) + (bur - bul) * (bur - bul)) * rroi * rroi;
  double v2h = 0.5 * (vnbar * vnbar + vtbar * vtbar + vubar * vubar);
  double b2r = (bnbar * bnbar + btbar * btbar + bubar * bubar) * robari;
  double c2 = gammam1 * (+hbar - v2h - db2 - b2r);
  double a2 = (gammam1 * (+hbar - v2h - db2) - gammam2 * (bnbar * bnbar + btbar * btbar + bubar * bubar) * robari);
  double ca2 = bnbar * bnbar * robari;
  double cb2 = (btbar * btbar + bubar * bubar) * robari;
  double cf2 = 0.5 * (a2 + sqrt(cb2 * (a2 + c2 + ca2) + (c2 - ca2) * (c2 - ca2)));
  double cs2 = c2 * ca2 / cf2;
  double cf = sqrt(cf2);
  double cs = sqrt(cs2);
  double ca = sqrt(ca2);
  double c = sqrt(c2);
  double cfi = 1.0 / cf;
  double sgr1 = btbar * btbar + bubar * bubar - QAS_FL_EPS;
  double sf11 = (sgr1 > 0) ? 1.0 : 0.0;
  double sf21 = 1.0 - sf11;
  double beti = 1.0 / sqrt(btbar * btbar + bubar * bubar + sf21);
  const double sqh = sqrt(0.5);
  double bett = sf11 * btbar * beti + sf21 * sqh;
  double betu = sf11 * bubar * beti + sf21 * sqh;
  double sgr2 = (btbar * btbar + bubar * bubar) * robari + fabs(ca2 - c2) - QAS_FL_EPS;
  double sf12 = (sgr2 > 0) ? 1.0 : 0.0;
  double sf22 = 1.0 - sf12;
  double cfca = qmax(0.0, cf2 - ca2);
  double cfcs = qmax(0.0, cf2 - cs2);
  double cfa = qmax(0.0, cf2 - c2);
  double alpi = 1.0 / sqrt(cfcs + sf22);
  double alpf = sf12 * sqrt(cfca) * alpi + sf22;
  double alps = sf12 * sqrt(cfa) * alpi;
  const double eeps = 0.0;
  double evpf = qmax(fabs(vnbar + cf), eeps);
  double evmf = qmax(fabs(vnbar - cf), eeps);
  double evps = qmax(fabs(vnbar + cs), eeps);
  double evms = qmax(fabs(vnbar - cs), eeps);
  double evpa = qmax(fabs(vnbar + ca), eeps);
  double evma = qmax(fabs(vnbar - ca), eeps);
  double ev00 = qmax(fabs(vnbar), eeps);
  double dltro = ror - rol;
  double dltmn = robar * (vnr - vnl);
  double dltmt = robar * (vtr - vtl);
  double dltmu = robar * (vur - vul);
  double dltbt = btr - btl;
  double dltbu = bur - bul;
  double t1 = bett * dltbt + betu * dltbu;
  double t2 = (prr - prl + (btave * dltbt + buave * dltbu) + gammam2 * (btbar * dltbt + bubar * dltbu)) * gammam1i;
  double t3 = betu * dltbt - bett * dltbu;
  double s1 = dltmn;
  double s2 = bett * dltmt + betu * dltmu;
  double s3 = betu * dltmt - bett * dltmu;
  double p11 = alps * cf * rrobai;
  double p12 = -alpf * c2 * cfi * rrobai;
  double p21 = alpf * (cf2 - c2 * gammam2 * gammam1i);
  double p22 = alps * (cs2 - c2 * gammam2 * gammam1i);
  double q11 = alpf * cf;
  double q12 = alps * cs;
  double q21 = -alps * ca * sgn;
  double q22 = alpf * c * sgn;
  double detpi = 1.0 / (p11 * p22 - p12 * p21);
  double detqi = 1.0 / (q11 * q22 - q12 * q21);
  double wvpf = 0.5 * ((p22 * t1 - p12 * t2) * detpi + (q22 * s1 - q12 * s2) * detqi);
  double wvmf = 0.5 * ((p22 * t1 - p12 * t2) * detpi - (q22 * s1 - q12 * s2) * detqi);
  double wvps = 0.5 * ((-p21 * t1 + p11 * t2) * detpi + (-q21 * s1 + q11 * s2) * detqi);
  double wvms = 0.5 * ((-p21 * t1 + p11 * t2) * detpi - (-q21 * s1 + q11 * s2) * detqi);
  double wvpa = 0.5 * (rrobar * t3 - sgn * s3);
  double wvma = 0.5 * (rrobar * t3 + sgn * s3);
  double wv00 = dltro - alpf * (wvpf + wvmf) - alps * (wvps + wvms);
  // eigen-weighted jumps: ev*wv of each family
  double apf = evpf * wvpf, amf = evmf * wvmf, aps = evps * wvps, ams = evms * wvms;
  double apa = evpa * wvpa, ama = evma * wvma, a00 = ev00 * wv00;
  // right eigenvectors of the Roe matrix
  double rvpfmn = alpf * (vnbar + cf);
  double rvpfmt = alpf * vtbar - alps * bett * ca * sgn;
  double rvpfmu = alpf * vubar - alps * betu * ca * sgn;
  double rvpfbt = alps * bett * cf * rrobai;
  double rvpfbu = alps * betu * cf * rrobai;
  double cab = alps * ca * (bett * vtbar + betu * vubar) * sgn;
  double rvpfen = alpf * (v2h + db2 + cf * vnbar + cf2 * gammam1i + (cf2 - c2) * gammam2 * gammam1i) - cab;
  double rvmfmn = alpf * (vnbar - cf);
  double rvmfmt = alpf * vtbar + alps * bett * ca * sgn;
  double rvmfmu = alpf * vubar + alps * betu * ca * sgn;
  double rvmfen = alpf * (v2h + db2 - cf * vnbar + cf2 * gammam1i + (cf2 - c2) * gammam2 * gammam1i) + cab;
  double rvpsmn = alps * (vnbar + cs);
  double rvpsmt = alps * vtbar + c * sgn * alpf * bett;
  double rvpsmu = alps * vubar + c * sgn * alpf * betu;
  double rvpsbt = -rrobai * c2 * alpf * bett * cfi;
  double rvpsbu = -rrobai * c2 * alpf * betu * cfi;
  double cfb = alpf * c * (bett * vtbar + betu * vubar) * sgn;
  double rvpsen = alps * (v2h + db2 + cs * vnbar + cs2 * gammam1i + (cs2 - c2) * gammam2 * gammam1i) + cfb;
  double rvmsmn = alps * (vnbar - cs);
  double rvmsmt = alps * vtbar - c * sgn * alpf * bett;
  double rvmsmu = alps * vubar - c * sgn * alpf * betu;
  double rvmsen = alps * (v2h + db2 - cs * vnbar + cs2 * gammam1i + (cs2 - c2) * gammam2 * gammam1i) - cfb;
  double rvpamt = -sgn * betu;
  double rvpamu = sgn * bett;
  double rvpabt = rrobai * betu;
  double rvpabu = -rrobai * bett;
  double rvpaen = -(betu * vtbar - bett * vubar) * sgn;
  double rv00en = v2h + db2;
  // left/right fluxes
  double frol = rol * vnl;
  double fmnl = rol * vnl * vnl + prl + 0.5 * (-bnbar * bnbar + btl * btl + bul * bul);
  double fmtl = rol * vnl * vtl - bnbar * btl;
  double fmul = rol * vnl * vul - bnbar * bul;
  double fbtl = vnl * btl - vtl * bnbar;
  double fbul = vnl * bul - vul * bnbar;
  double fenl = rol * vnl * hl - bnbar * (bnbar * vnl + btl * vtl + bul * vul);
  double fror = ror * vnr;
  double fmnr = ror * vnr * vnr + prr + 0.5 * (-bnbar * bnbar + btr * btr + bur * bur);
  double fmtr = ror * vnr * vtr - bnbar * btr;
  double fmur = ror * vnr * vur - bnbar * bur;
  double fbtr = vnr * btr - vtr * bnbar;
  double fbur = vnr * bur - vur * bnbar;
  double fenr = ror * vnr * hr - bnbar * (bnbar * vnr + btr * vtr + bur * vur);
  // 0.5*(fl + fr - sum_k ev_k wv_k r_k), terms in the reference's order; the
  // entropy-wave and Alfven-wave entries that are literal zeros keep their
  // 0.0 products so signed zeros match.
  F[0] = 0.5 * (+frol + fror - apf * alpf - amf * alpf - aps * alps - ams * alps - apa * 0.0 - ama * 0.0 - a00 * 1.0);
  F[1] = 0.5 * (+fmnl + fmnr - apf * rvpfmn - amf * rvmfmn - aps * rvpsmn - ams * rvmsmn - apa * 0.0 - ama * 0.0 -
                a00 * vnbar);
  F[2] = 0.5 * (fmtl + fmtr - apf * rvpfmt - amf * rvmfmt - aps * rvpsmt - ams * rvmsmt - apa * rvpamt -
                ama * (-rvpamt) - a00 * vtbar);
  F[3] = 0.5 * (fmul + fmur - apf * rvpfmu - amf * rvmfmu - aps * rvpsmu - ams * rvmsmu - apa * rvpamu -
                ama * (-rvpamu) - a00 * vubar);
  F[4] = 0.5 * (fbtl + fbtr - apf * rvpfbt - amf * rvpfbt - aps * rvpsbt - ams * rvpsbt - apa * rvpabt -
                ama * rvpabt - a00 * 0.0);
  F[5] = 0.5 * (fbul + fbur - apf * rvpfbu - amf * rvpfbu - aps * rvpsbu - ams * rvpsbu - apa * rvpabu -
                ama * rvpabu - a00 * 0.0);
  F[6] = 0.5 * (fenl + fenr - apf * rvpfen - amf * rvmfen - aps * rvpsen - ams * rvmsen - apa * rvpaen -
                ama * (-rvpaen) - a00 * rv00en);
}

QAS_HD void flux_roe(const double L[7], const double R[7], double bnc, double gamma, double F[7])
{
  flux_roe(L, R, bnc, gamma, 1.0 / (gamma - 1.0), F);
}

// gammam1i = 1/(gamma - 1), the same IEEE quotient wherever it is formed: the kernels take it from the host
template <int RMN>
QAS_HD void riemann(const double L[7], const double R[7], double bnc, double gamma, double gammam1i, double dv0,
                                        double dv1, double F[7])
{
  if (RMN == 0)
    flux_roe(L, R, bnc, gamma, gammam1i, F);
  else if (RMN == 1)
    flux_hlld<false>(L, R, bnc, gamma, gammam1i, dv0, dv1, F);
  else if (RMN == 2)
    flux_hlld<true>(L, R, bnc, gamma, gammam1i, dv0, dv1, F);
  else
    flux_mlau(L, R, bnc, gamma, gammam1i, dv0, dv1, F);
}
template <int RMN>
QAS_HD void riemann(const double L[7], const double R[7], double bnc, double gamma, double dv0,
                                        double dv1, double F[7])
{
  riemann<RMN>(L, R, bnc, gamma, 1.0 / (gamma - 1.0), dv0, dv1, F);
}

// the same flux handed to out(m, F[m]) as each component is final (MLAU emits while it runs;
// the other solvers after their last component)
template <int RMN, class Out>
QAS_HD void riemann_out(const double L[7], const double R[7], double bnc, double gamma, double gammam1i, double dv0,
                        double dv1, Out &&out)
{
  if constexpr (RMN == 3) {
    flux_mlau_out(L, R, bnc, gamma, gammam1i, dv0, dv1, out);
  } else {
    double F[7];
    riemann<RMN>(L, R, bnc, gamma, gammam1i, dv0, dv1, F);
#pragma unroll
    for (int m = 0; m < 7; m++) out(m, F[m]);
  }
}

// CUCT corner weight, common/mhd_func.c:56-76. Arguments are the values at the
// four cells (a-1,b-1),(a,b-1),(a-1,b),(a,b) of the corner's plane, ba at
// (a,b-1),(a,b) and bb at (a-1,b),(a,b).
QAS_HD double cuct_weight(double r0, double r1, double r2, double r3, double va0, double va1,
                                              double va2, double va3, double vb0, double vb1, double vb2, double vb3,
                                              double ba1, double ba3, double bb2, double bb3)
{
  const double eps = 1e-12;
  double roc = 0.25 * (r0 + r1 + r2 + r3);
  roc = 1.0 / sqrt(roc);
  double vac = 0.25 * (va0 + va1 + va2 + va3);
  double vbc = 0.25 * (vb0 + vb1 + vb2 + vb3);
  double bac = 0.5 * (ba1 + ba3);
  double bbc = 0.5 * (bb2 + bb3);
  vac = fabs(vac) + fabs(bac * roc);
  vbc = fabs(vbc) + fabs(bbc * roc);
  return (vac + 0.5 * eps) / (vac + vbc + eps);
}

// SSP-RK combine, common/common_func.h:28-31
QAS_HD double rk_combine(double f1, double f0, double df, double c0, double c1)
{
  return c0 * f0 + c1 * (f1 + df);
}

}  // namespace qas
