// Device-side building blocks of the B200 self-consistency path: complex
// arithmetic, the midpoint Riccati step, the local Green functions and the
// bilinear lookups into the reference grid.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace scb {

constexpr int MAX_COMP = 4;

template <typename R>
struct Cx {
  R re, im;
};

// Per-angle constants of one trajectory frame.
struct AngleParams {
  double cD, sD;  // order parameter into the frame (float trig, promoted)
  double cA, sA;  // induced vector potential into the frame
  double cB, sB;  // frame back to the reference grid
  double cE, sE;  // external vector potential coordinates (double trig)
  double vx, vy;  // Fermi velocity
  double w;       // Fermi-surface integrand factor
  double hs;      // Riccati step h / |v_F| (RiccatiSolverConfined.h:525-527)
  double sx, sy;  // vx * w, vy * w
  double eta[MAX_COMP];  // basis function of every component at this angle
};

template <typename R>
__device__ __forceinline__ Cx<R> cmul(Cx<R> a, Cx<R> b) {
  return Cx<R>{a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re};
}

// Precision-specific primitives: IEEE-rounded reciprocal and accurate
// reciprocal square root in FP64; the fast MUFU approximations in FP32.
// FP64 reciprocal: the hardware approximation r (relative error about 2^-20)
// refined by one third-order step of the series 1/x = r / (1 - e) with
// e = 1 - x r, truncated after e^2: r (1 + e + e^2), error O(e^3) (measured on
// B200: within 2 ulp of IEEE 1/x; the arguments here are finite and nonzero).
__device__ __forceinline__ double rcp_(double x) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  const double e = fma(-x, r, 1.0);
  return fma(r, fma(e, e, e), r);
}
__device__ __forceinline__ float rcp_(float x) { return __fdividef(1.0f, x); }
// FP64 reciprocal square root of a positive normal argument: the hardware
// approximation r refined by one third-order step of the binomial series
// 1/sqrt(x) = r (1 - e)^(-1/2) with e = 1 - x r^2, truncated after e^2:
// r (1 + e/2 + 3 e^2/8), error O(e^3) (measured on B200: within 3 ulp).
__device__ __forceinline__ double rsqrt_(double x) {
  double r;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  const double e = fma(-x * r, r, 1.0);
  return fma(r, e * fma(0.375, e, 0.5), r);
}
__device__ __forceinline__ float rsqrt_(float x) { return rsqrtf(x); }
// FP64 square root of a non-negative argument as x / sqrt(x); the estimate is
// taken of max(x, smallest normal), which gives 0 for x = 0 with no branch and
// leaves every normal argument unchanged.
__device__ __forceinline__ double sqrt_(double x) {
  return x * rsqrt_(fmax(x, 2.2250738585072014e-308));
}
// FP32 square root of a non-negative argument: the hardware approximation
// (sqrt.approx; 0 for 0), one instruction.
__device__ __forceinline__ float sqrt_(float x) {
  float r;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// Principal square root, branch cut on the negative real axis, through one
// square root and one reciprocal square root:
//   u = (|z| + |x|)/2, t = sqrt(u), v = |y| / (2 t);
//   sqrt(z) = (t, sign(y) v) for x >= 0 and (v, sign(y) t) otherwise.
// u = 0 only for z = 0, where the estimate of max(u, smallest normal) is
// finite and t = v = 0: the root 0 with no branch.
template <typename R>
__device__ __forceinline__ Cx<R> csqrt_dev(R x, R y) {
  const R m = sqrt_(x * x + y * y);
  const R u = R(0.5) * (m + fabs(x));
  const R r = rsqrt_(fmax(u, R(sizeof(R) == 8 ? 2.2250738585072014e-308 : 1.17549435e-38)));
  const R t = u * r;
  const R v = R(0.5) * fabs(y) * r;
  const bool pos = x >= R(0);
  return Cx<R>{pos ? t : v, copysign(pos ? v : t, y)};
}

// Midpoint Riccati step, riccati::computeStep (RiccatiSolutions.h:65-94):
//   a = i h/4 conj(D), b = 2 a g0 + i h e - 1, c = (a g0 + i h e + 1) g0 + i h D,
//   g1 = 2 c / (-b + sqrt(b^2 - 4 a c)).
// The products with the purely imaginary step are written out (they are exact).
// With u = a g0 and B = i h e the discriminant reduces to
//   b^2 - 4 a c = (B - 1)^2 + h^2 |D|^2 - 8 u,
// because a (i h D) = -(h^2 / 4) |D|^2 is real; that form skips two complex
// products and avoids the cancellation of b^2 against 4 a c.
template <typename R>
__device__ __forceinline__ Cx<R> riccati_step(R dre, R dim, R ere, R eim, Cx<R> g, R h) {
  const R q = R(0.25) * h;
  const Cx<R> a{q * dim, q * dre};
  const R ser = -h * eim, sei = h * ere;  // (i h) * e
  const Cx<R> ag = cmul(a, g);
  const Cx<R> b{R(2) * ag.re + ser - R(1), R(2) * ag.im + sei};
  const Cx<R> t{ag.re + ser + R(1), ag.im + sei};
  const Cx<R> tg = cmul(t, g);
  const Cx<R> c{tg.re - h * dim, tg.im + h * dre};
  const R bm = ser - R(1);
  const R s0 = h * h * (dre * dre + dim * dim) - sei * sei;  // the site's part: shared by all energies
  const Cx<R> disc = csqrt_dev<R>((bm * bm + s0) - R(8) * ag.re, (R(2) * bm) * sei - R(8) * ag.im);
  const R den_re = disc.re - b.re, den_im = disc.im - b.im;
  const R inv = rcp_(den_re * den_re + den_im * den_im);
  const R c2r = R(2) * c.re, c2i = R(2) * c.im;
  return Cx<R>{(c2r * den_re + c2i * den_im) * inv, (c2i * den_re - c2r * den_im) * inv};
}

// Whether the fields of a site allow step_fast for every energy: with
// |gamma| <= 1 the discriminant's real part (over 4) is at least
// 1/4 - (h e_re / 2)^2 - 2 (h/4) |D| (the imaginary energies are positive, so
// (1 + h e_im) / 2 >= 1/2); the factor 2.5 instead of 2 leaves room for
// rounding.  False for NaN.  At 20 lattice points per xi0 the left side is
// 0.25 and the right side 0.01.
__device__ __forceinline__ bool fields_allow_fast(float dre, float dim, float es, float h, float e_re_max) {
  const float s = 0.5f * h * (fabsf(es) + e_re_max);
  return 0.25f - s * s > 0.625f * h * (fabsf(dre) + fabsf(dim));
}

// The midpoint step in the interior of the grain, where fields_allow_fast
// holds on both sites, in fewer operations than riccati_step: everything is
// kept at half scale (b/2, the discriminant/4, its real part/8), so that
//   g1 = c / (sqrt(w) - b/2),  w = (b^2 - 4 a c) / 4,
//   xh = Re w / 2 = ((1/2 + d)^2 + s0)/2 - Re(a g0),
//   u = Im w / 2 = -(1/2 + d) sh - Im(a g0),
//   sqrt(w) = (t, u / t),  t = sqrt(|w|/2 + xh),
// with d = h e_im / 2 of the energy and sh = h e_re / 2,
// s0 = (h |D| / 2)^2 - sh^2 of the site.  Re w > 0, so the root has no branch
// and no sign to choose, and the smallest normal number added to |w|^2 keeps
// every estimate finite with no guard.
// The small numbers (d, a g0, s0, sh) are added up before a term of order one
// is: a rounded -(1/2 + d) in their place is an error of the energy that all
// steps share, so that it grows with the 1 / (h e_im) sites that a column
// remembers, not with their square root.  Columns of 60 to 260 sites at
// h = 0.07 to 0.13 xi0 against 128 bits, relative: e_im = 0.3 2e-15 with the
// rounded sum, 4e-16 here, 6e-16 in riccati_step; real energies with broadening
// 0.008 10e-15, 0.9e-15 and 2.3e-15.  46 FP64 operations instead of 59 (43 with
// the rounded sum).
template <typename R>
struct SiteConst {
  R ar, ai, hdr, hdi, s0h, sh;  // a, h D, s0 / 2 + sh^2 / 2, h e_re / 2 (without the energy's own real part)
};
template <typename R>
__device__ __forceinline__ SiteConst<R> site_const(R dre, R dim, R es, R h) {
  SiteConst<R> c;
  const R q = R(0.25) * h;
  c.ar = q * dim;
  c.ai = q * dre;
  c.hdr = R(4) * c.ai;
  c.hdi = R(4) * c.ar;
  c.sh = R(0.5) * h * es;
  c.s0h = R(2) * (c.ar * c.ar + c.ai * c.ai);  // sh^2 / 2 is subtracted where sh is final
  return c;
}
// x / sqrt(x) and 1 / sqrt(x) for the step: the estimate refined as in rsqrt_.
__device__ __forceinline__ double sqrt_pos(double x) {
  double r;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  const double p = x * r;
  const double e = fma(-p, r, 1.0);
  return fma(p, e * fma(0.375, e, 0.5), p);
}
// Reciprocal and reciprocal square root of arguments of order one: in FP32 the
// hardware estimates without the scaling that subnormal arguments need.
__device__ __forceinline__ double rsqrt_pos(double x) { return rsqrt_(x); }
__device__ __forceinline__ float rsqrt_pos(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ double rcp_pos(double x) { return rcp_(x); }
__device__ __forceinline__ float rcp_pos(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
// s0 and sh: the energy's own real part included.
__device__ __forceinline__ Cx<double> step_fast(const SiteConst<double> &S, double s0, double sh, double d,
                                                Cx<double> g) {
  const double agd = S.ar * g.re - (S.ai * g.im + d), agim = S.ar * g.im + S.ai * g.re;  // a g0 - d
  const double br = agd - 0.5, bi = agim + sh;  // b / 2
  const double tr = (agd - d) + 1.0, ti = bi + sh;
  const double cre = tr * g.re - (ti * g.im + S.hdi), cim = tr * g.im + (ti * g.re + S.hdr);
  const double xh = (0.5 * ((d * d + s0) - d) - agd) + 0.125, u = -(d * sh + (0.5 * sh + agim));
  const double m = sqrt_pos(xh * xh + (u * u + 1e-300));
  const double U = m + xh;
  const double rho = rsqrt_pos(U);
  const double dr = U * rho - br, di = u * rho - bi;
  const double inv = rcp_pos(dr * dr + di * di);
  return Cx<double>{(cre * dr + cim * di) * inv, (cim * dr - cre * di) * inv};
}

// Two energies of one thread, lane by lane in FP32 pairs:
// re = (Re z_j, Re z_j+1), im = (Im z_j, Im z_j+1).  sm_100 executes one
// FFMA2 / FMUL2 / FADD2 instruction for both lanes, so the FP32 arithmetic of
// the mixed-precision sweep takes half the issue slots; the square roots and
// reciprocals stay one instruction per lane.  Each lane is rounded as the
// scalar FP32 operation would be.
struct Cx2 {
  float2 re, im;
};
__device__ __forceinline__ float2 bc2(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
// The interior step of the FP32 sweep, two energies at a time.  The step is
// close to the identity, and its terms of order one (1 + h e, the root near
// 1/2) round off the small numbers that make up the change: in their place it
// is written for the change itself,
//   g1 = g0 + (k g0 + i h D) / den,  k = 2 a g0 - 3 d - sg + 3 i sh,
//   den = 1 + d + sg - a g0 - i sh,  d = h e_im / 2,  sh = h e_re / 2,
// with the root sqrt(w) = 1/2 + sg of w = 1/4 + om,
//   om = d + d^2 + (h |D| / 2)^2 - sh^2 - 2 a g0 - i (1 + 2 d) sh,
// whose small part sg is taken once through sg = om - sg^2 (from
// sg (1 + sg) = om), which leaves 2 |sg| of the error that sg has as the
// root's estimate minus 1/2.  Then k, i h D and the change carry relative FP32
// errors, and only the last addition rounds at the size of g0.
// Negated quantities (nx = -x) are carried where that saves a sign change:
// the packed instructions have no operand negation, and a change of sign costs
// one more.  39 packed operations (a step on the values themselves: 42).
struct SiteConst2 {
  float2 ai, nar, nai, hdi, nhdr;
};
struct EnergyConst2 {
  float2 nbh, c1, d2h, d3;  // 1/2 + d, 1 + d, (d + d^2) / 2, 3 d
};
__device__ __forceinline__ Cx2 step_fast2(const SiteConst2 &S, float2 s0h, float2 nsh, float2 n3sh,
                                          const EnergyConst2 &E, Cx2 g) {
  const float2 m1 = bc2(-1.0f), two = bc2(2.0f);
  const float2 nur = fma2(S.ai, g.im, mul2(S.nar, g.re)), nui = fma2(S.nar, g.im, mul2(S.nai, g.re));  // -a g0
  const float2 omr = add2(add2(E.d2h, s0h), nur), y = fma2(E.nbh, nsh, nui);                           // om / 2
  const float2 xh = add2(omr, bc2(0.125f));
  const float2 xx = fma2(xh, xh, fma2(y, y, bc2(1e-37f)));
  const float2 U = add2(make_float2(sqrt_(xx.x), sqrt_(xx.y)), xh);
  const float2 rho = make_float2(rsqrt_pos(U.x), rsqrt_pos(U.y));
  const float2 sgr = fma2(U, rho, bc2(-0.5f)), sgi = mul2(y, rho);
  const float2 dr = add2(add2(nur, E.c1), sgr), di = add2(add2(nui, nsh), sgi);
  const float2 nsgr = mul2(sgr, m1);
  const float2 nkr = fma2(sgi, sgi, fma2(nsgr, sgr, fma2(two, add2(omr, nur), E.d3)));
  const float2 nki = fma2(two, add2(nui, fma2(nsgr, sgi, y)), n3sh);
  const float2 ngi = mul2(g.im, m1);
  const float2 nnr = fma2(nkr, g.re, fma2(nki, ngi, S.hdi)), nni = fma2(nkr, g.im, fma2(nki, g.re, S.nhdr));
  const float2 s = fma2(dr, dr, mul2(di, di));
  const float2 ninv = make_float2(-rcp_pos(s.x), -rcp_pos(s.y));
  const float2 ndi = mul2(di, m1);
  return Cx2{fma2(fma2(nnr, dr, mul2(nni, di)), ninv, g.re), fma2(fma2(nni, dr, mul2(nnr, ndi)), ninv, g.im)};
}
// The same for one energy.
__device__ __forceinline__ Cx<float> step_fast_f32(const SiteConst<float> &S, float s0h, float sh, float d,
                                                   Cx<float> g) {
  const float nur = S.ai * g.im - S.ar * g.re, nui = -(S.ar * g.im + S.ai * g.re);
  const float omr = ((0.5f * d) * (1.0f + d) + s0h) + nur, y = nui - (0.5f + d) * sh;
  const float xh = omr + 0.125f;
  const float U = sqrt_(xh * xh + (y * y + 1e-37f)) + xh;
  const float rho = rsqrt_pos(U);
  const float sgr = fmaf(U, rho, -0.5f), sgi = y * rho;
  const float dr = (nur + (1.0f + d)) + sgr, di = (nui - sh) + sgi;
  const float nkr = fmaf(sgi, sgi, fmaf(-sgr, sgr, fmaf(2.0f, omr + nur, 3.0f * d)));
  const float nki = fmaf(2.0f, nui + fmaf(-sgr, sgi, y), -3.0f * sh);
  const float nnr = fmaf(nkr, g.re, fmaf(-nki, g.im, S.hdi)), nni = fmaf(nkr, g.im, fmaf(nki, g.re, -S.hdr));
  const float ninv = -rcp_pos(dr * dr + di * di);
  return Cx<float>{fmaf(nnr * dr + nni * di, ninv, g.re), fmaf(nni * dr - nnr * di, ninv, g.im)};
}

// greens_g_im<float> of two real energies: Im g = -[(1 - Re p)(1 + Re p) - (Im p)^2] / |1 + p|^2.
__device__ __forceinline__ float2 greens_g_im2(Cx2 g, Cx2 gt) {
  const float2 one = bc2(1.0f), m1 = bc2(-1.0f);
  const float2 ngi = mul2(g.im, m1);
  const float2 pre = fma2(g.re, gt.re, mul2(ngi, gt.im));
  const float2 pim = fma2(g.re, gt.im, mul2(g.im, gt.re));
  const float2 den_re = add2(one, pre), nnr = add2(pre, m1);  // nnr = -(1 - Re p)
  const float2 pim2 = mul2(pim, pim);
  const float2 s = fma2(den_re, den_re, pim2);
  const float2 inv = make_float2(rcp_pos(s.x), rcp_pos(s.y));
  return mul2(fma2(nnr, den_re, pim2), inv);
}

// Homogeneous solutions, riccati::computeHomogeneous (RiccatiSolutions.h:36-54).
template <typename R>
__device__ __forceinline__ void riccati_homogeneous(R dre, R dim, R ere, R eim, Cx<R> &g,
                                                    Cx<R> &gt) {
  const R nd = dre * dre + dim * dim;
  const R e2re = ere * ere - eim * eim, e2im = ere * eim + eim * ere;
  const Cx<R> om = csqrt_dev<R>(nd - e2re, -e2im);
  const R dr = ere - om.im, di = eim + om.re;  // energy + i * Omega
  const R inv = rcp_(dr * dr + di * di);
  const Cx<R> invd{dr * inv, -di * inv};
  g = cmul(Cx<R>{-dre, -dim}, invd);
  gt = cmul(Cx<R>{dre, -dim}, invd);
}

// Im g of one real energy, g = -i (1 - g gt) / (1 + g gt) (LocalGreens.h:32-43).
template <typename R>
__device__ __forceinline__ R greens_g_im(Cx<R> g, Cx<R> gt) {
  const Cx<R> p = cmul(g, gt);
  const R den_re = R(1) + p.re, den_im = p.im;
  const R inv = rcp_(den_re * den_re + den_im * den_im);
  const R nr = R(1) - p.re, ni = -p.im;
  return -(nr * den_re + ni * den_im) * inv;
}

// Bilinear lookup of insertRotatedGrid(_Additive)_kernel
// (GridFunctions_GPU.h:436-546): coordinates of site (x, y) of an n_out grid in
// an n_in grid rotated by the angle whose (cos, sin) of minus the angle are
// (c, s).  Returns false when the reference leaves the site untouched.
struct Bilinear {
  int i00;  // index of the lower-left corner in the input grid
  double xf, yf;
};
// (int)v and v - (int)v of |v| < 2^31 through the low word of v + 3 * 2^51
// rounded down: two additions where the conversions to an integer and back are
// quarter-rate instructions.  Rounding down differs from truncation only for
// v < 0, of which only -1 < v is ever used.
__device__ __forceinline__ int split(double v, double &frac) {
  const double magic = 6755399441055744.0;  // 3 * 2^51
  const double t = __dadd_rd(v, magic);
  int i = __double2loint(t);
  frac = v - (t - magic);
  if (i == -1 && v > -1.0) {
    i = 0;
    frac = v;
  }
  return i;
}
__device__ __forceinline__ bool rotated_lookup(int x, int y, int n_out, int n_in, double c,
                                               double s, Bilinear &b) {
  const double xt = (double)(n_in - n_out) / 2.0;
  const double sh = (double)(n_in - 1) / 2.0;
  const double X = (double)x + xt - sh, Y = (double)y + xt - sh;
  const double xr = X * c - Y * s + sh;
  const double yr = X * s + Y * c + sh;
  const int xi = split(xr, b.xf), yi = split(yr, b.yf);
  if (xi >= 0 && xi + 1 < n_in && yi >= 0 && yi + 1 < n_in) {
    b.i00 = yi * n_in + xi;
    return true;
  }
  return false;
}
// The four corner weights of a lookup: a field then costs four fused
// multiply-adds (against nine operations as three interpolations).
struct Corners {
  double w00, w01, w10, w11;
};
__device__ __forceinline__ Corners corners(const Bilinear &b, double scale = 1.0) {
  const double y1 = b.yf * scale, y0 = scale - y1;
  const double w01 = b.xf * y0, w11 = b.xf * y1;
  return Corners{y0 - w01, w01, y1 - w11, w11};
}
__device__ __forceinline__ double weigh(const Corners &w, double v00, double v01, double v10, double v11) {
  return fma(w.w11, v11, fma(w.w10, v10, fma(w.w01, v01, w.w00 * v00)));
}

}  // namespace scb
