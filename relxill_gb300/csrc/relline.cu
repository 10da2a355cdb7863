// relline.cu -- line profile kernel: transfer-function interpolation, g*
// integration of every (radius, energy bin) pair and binning into radial zones
// and the emission-angle histogram (Relprofile.cpp:39-80, 141-303, 489-958).
//
// line_table_kernel writes each set's (a, mu0)-interpolated transfer functions on
// all table radii once (two float2 planes: trff1/trff2, cosne1/cosne2), read by the line
// profile and the histogram.
//
// Line profile: the profile of a zone is summed per bin in eight classes (radius index in the
// zone modulo 8), each in the order of its radii, and the classes in order: every sum has one
// order, whatever kernel, tile or batch it is formed in.
//  * A warp integrates a group of eight consecutive radii side by side, one of each class, four
//    lanes per radius (line_group).  Bound: instruction issue (FP32 and integer); neighbouring
//    radii reach nearly the same bins and need the same rule (midpoint below 0.95 keV, Romberg
//    with the reference's prec 0.02 / itermax 5 above, sqrt edge terms within 5e-3 of g* = 0
//    and 1), so the lanes stay together (28 of 32 active in the loops over the runs of bins).  A
//    warp per radius with its lanes on 32 consecutive bins used 20 of 32 and set every radius
//    up alone: 5.22 ms per 4096 relxilllp sets of 10 zones, now 2.36 ms; instructions per set
//    1.17 M, now 0.54 M.
//  * Many sets: relline_solo_kernel, a warp per (set, zone, tile of 128 bins), no synchronisation
//    between warps.  Few sets: relline_team_kernel, a CTA per (set, zone, tile of 32 bins) whose
//    warps take groups in parallel and whose threads then add their values in the classes'
//    order (one relline spectrum of 3000 bins: 540 us, now 54 us).
//  * Arithmetic is FP32.  Bin edges and gmin/gmax enter as float-float so
//    that g* is accurate to an ulp.  Two decisions of the reference are
//    discrete and are taken in higher precision where the FP32 value lies close
//    to the decision point: the side of a transfer-function grid point (the
//    reference's interpolation weights are reversed, so the interpolant jumps
//    there; decided in float-float from the reference's own energy abscissa
//    within 2e-5 grid units of the point), and Romberg's convergence test
//    obtprec > 0.02 (a bin whose FP32 test came within 2e-6 of 0.02 is
//    integrated again with FP64 Romberg: one level more or less changes the bin
//    by up to about 2%).  Such bins are marked and redone by one out-of-line call between
//    groups, so that the loops over bins hold no call.
#include <algorithm>

#include "relx_device.cuh"
#include "relx_kernels.h"

namespace relx {

constexpr int kLineWarps = 8;
constexpr int kLineThreads = kLineWarps * 32;
constexpr float kH = 5e-3f;
constexpr float kSideBand = 2e-5f;  // grid units within which the side of a g* point is taken in float-float
// |obtprec - 0.02| within which a bin is integrated again in FP64: about five times the error of the
// FP32 obtprec (the level sums carry a few ulp each, 2-5e-7 of the integral)
constexpr float kConvBand = 2e-6f;
constexpr int kGroup = 8;         // consecutive radii of a zone that a warp integrates side by side
constexpr int kRadLanes = 32 / kGroup;  // lanes per radius, each with a quarter of the radius's bins
static_assert(kSumBinsH == 32, "a profile-sum block is the bins of one warp's sum");

constexpr float kMagic = 12582912.0f;   // 1.5 2^23: x + kMagic holds x rounded to an integer in its low bits
constexpr int kMagicBits = 0x4b400000;  // its bit pattern
// rsqrtf for arguments that are not denormal (here x (1 - x) with x within [H, 1 - H])
__device__ __forceinline__ float rsqrt_norm(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// 1 / (4^n - 1)
__constant__ float c_inv4m1[7] = {0.f, 1.f / 3.f, 1.f / 15.f, 1.f / 63.f, 1.f / 255.f, 1.f / 1023.f, 1.f / 4095.f};

// constants of the radius a lane works on
struct RadL {
  float2 gmin, gmax;      // float-float
  float dgf, inv_dg;      // gmax - gmin and its inverse
  float edge_lo, edge_hi; // 2 sqrt(H) sum_k F_k(H), same at 1-H (emissivity factored out)
  int limb;               // limb law (read with LIMB only)
};
// constants of the relline table (a kernel parameter: constant-bank operands hold no registers)
struct LineC {
  int ng;
  float inv_dgs;     // (ng-1) / (1-2H)
  float ng2;         // ng - 2
};

// transfer functions at one radius: trff (and cosne for limb laws) at the table g* points
template <bool LIMB> struct TW;
template <> struct TW<false> { float2 t; };
template <> struct TW<true> { float4 t; };

// limb law at one table point (Relprofile.cpp:512-519)
__device__ __forceinline__ float limb_factor(int limb, float mu) {
  if (limb == 1) return __fmaf_rn(2.06f, mu, 1.0f);
  if (limb == 2) return logf(__fadd_rn(1.0f, 1.0f / mu));
  return 1.0f;
}

// The arithmetic of a bin's value is written with explicit roundings (which product of a sum is fused
// is otherwise the compiler's choice, call by call): a bin then has the same value in every kernel
// variant, whichever warps it is spread over.  The roundings are those of the kernel this one took the
// place of (one CTA per 512 bins), so that its results stay what they were.
// a sum of two products, the first one fused
__device__ __forceinline__ float sum2(float f, float a, float g, float b) {
  return __fmaf_rn(f, a, __fmul_rn(g, b));
}
// the integrand of both branches: e3 q_k, kept as products where they enter sums; with a limb law the
// rounded values
template <bool LIMB> struct Fval;
template <> struct Fval<false> {
  float e3, q0, q1;
  __device__ __forceinline__ float both() const { return sum2(e3, q0, e3, q1); }
  __device__ __forceinline__ void add(float &a0, float &a1) const {
    a0 = __fmaf_rn(e3, q0, a0);
    a1 = __fmaf_rn(e3, q1, a1);
  }
  __device__ __forceinline__ float2 value() const { return make_float2(__fmul_rn(e3, q0), __fmul_rn(e3, q1)); }
};
template <> struct Fval<true> {
  float v0, v1;
  __device__ __forceinline__ float both() const { return __fadd_rn(v0, v1); }
  __device__ __forceinline__ void add(float &a0, float &a1) const {
    a0 = __fadd_rn(a0, v0);
    a1 = __fadd_rn(a1, v1);
  }
  __device__ __forceinline__ float2 value() const { return make_float2(v0, v1); }
};

// the interior of a bin in g* and 1 - g*, the sum of its edge terms, and which ends are those at H
struct Interior {
  float ga, ca, gb, cb, flu;
  bool lo_H, hi_H;
};

// position of x among the table's g* points: t, the nearest point tr and the offset dt from it (adding
// 1.5 2^23 rounds without a conversion instruction)
struct GPos { float xh, t, tr, dt; };
__device__ __forceinline__ GPos g_pos(float x, const LineC &lc) {
  GPos g;
  g.xh = __fsub_rn(x, kH);
  g.t = __fmul_rn(g.xh, lc.inv_dgs);
  g.tr = __fsub_rn(__fadd_rn(g.t, kMagic), kMagic);
  g.dt = __fsub_rn(g.t, g.tr);
  return g;
}
// integrand F_k(x) = E^3 trf_k(x) [limb] / sqrt(x (1-x)), k = 0, 1  (relb_func,
// Relprofile.cpp:489-521 times (gmax - gmin) / emis), between the table points fi and fi + 1; y = 1 - x.
// romb: the Romberg abscissae take the interpolation factor in one rounding.
template <bool LIMB>
__device__ __forceinline__ Fval<LIMB> F_at(float x, float y, const GPos &g, float fi, bool romb, const RadL &rc,
                                           const LineC &lc, const TW<LIMB> *__restrict__ tw) {
  fi = fmaxf(0.0f, fminf(fi, lc.ng2));
  const int ind = __float_as_int(__fadd_rn(fi, kMagic)) - kMagicBits;
  const float inte = romb ? __fmaf_rn(g.xh, lc.inv_dgs, -fi) : __fsub_rn(g.t, fi);
  const float inte1 = __fsub_rn(1.0f, inte);
  const float e = __fmaf_rn(x, rc.dgf, rc.gmin.x);
  const float e3 = __fmul_rn(__fmul_rn(__fmul_rn(e, e), e), rsqrt_norm(__fmul_rn(x, y)));
  if constexpr (!LIMB) {
    const float2 A = tw[ind].t, B = tw[ind + 1].t;
    return {e3, sum2(inte, A.x, inte1, B.x), sum2(inte, A.y, inte1, B.y)};
  } else {
    const float4 A = tw[ind].t, B = tw[ind + 1].t;
    float f0 = __fmul_rn(e3, sum2(inte, A.x, inte1, B.x));
    float f1 = __fmul_rn(e3, sum2(inte, A.y, inte1, B.y));
    f0 = __fmul_rn(f0, limb_factor(rc.limb, sum2(inte, A.z, inte1, B.z)));
    f1 = __fmul_rn(f1, limb_factor(rc.limb, sum2(inte, A.w, inte1, B.w)));
    return {f0, f1};
  }
}
// F_k(x) where x is not close to a table point; *off receives the distance to the nearest one (the
// caller passes bins with an abscissa within kSideBand of one on to bin_general)
template <bool LIMB, bool ROMB>
__device__ __forceinline__ Fval<LIMB> eval_F(float x, float y, const RadL &rc, const LineC &lc,
                                             const TW<LIMB> *__restrict__ tw, float *off) {
  const GPos g = g_pos(x, lc);
  *off = fabsf(g.dt);
  return F_at<LIMB>(x, y, g, g.dt < 0.0f ? __fsub_rn(g.tr, 1.0f) : g.tr, ROMB, rc, lc, tw);
}

// the midpoint rule's value of both branches
template <bool LIMB>
__device__ __forceinline__ float mid_F(float2 lo, float2 hi, const RadL &rc, const LineC &lc, const TW<LIMB> *tw,
                                       float *off) {
  return eval_F<LIMB, false>(0.5f * __fadd_rn(lo.x, hi.x), 0.5f * __fadd_rn(lo.y, hi.y), rc, lc, tw, off).both();
}

// Romberg's first refinement (bin_general has them all) between the edges lo and hi with the integrand
// values fa, fb; *val receives the integral where both branches stop there (true); false where a branch
// goes on or its test is close to 0.02
template <bool LIMB>
__device__ __forceinline__ bool romberg_first(float2 lo, float2 hi, const Fval<LIMB> &fa, const Fval<LIMB> &fb,
                                              const RadL &rc, const LineC &lc, const TW<LIMB> *__restrict__ tw,
                                              float *val, float *off) {
  const float pas0 = __fsub_rn(hi.x, lo.x);
  const float2 va = fa.value();
  float ta0 = va.x, ta1 = va.y;
  fb.add(ta0, ta1);
  ta0 = __fmul_rn(ta0, 0.5f);
  ta1 = __fmul_rn(ta1, 0.5f);
  const float p0 = __fmul_rn(ta0, pas0), p1 = __fmul_rn(ta1, pas0);
  const float2 f =
      eval_F<LIMB, true>(__fmaf_rn(pas0, 0.5f, lo.x), __fmaf_rn(-pas0, 0.5f, lo.y), rc, lc, tw, off).value();
  const float pas = __fmul_rn(pas0, 0.5f);
  const float t0 = __fmul_rn(__fmaf_rn(4.0f, __fmul_rn(__fadd_rn(ta0, f.x), pas), -p0), 1.f / 3.f);
  const float t1 = __fmul_rn(__fmaf_rn(4.0f, __fmul_rn(__fadd_rn(ta1, f.y), pas), -p1), 1.f / 3.f);
  *val = __fadd_rn(t0, t1);
  // |t - p| / t below 0.0198 for certain (romberg_on)
  return (fabsf(t0 - p0) < 0.0198f * t0) & (fabsf(t1 - p1) < 0.0198f * t1);
}

// Romberg's first two refinements between the ends of q's interior; *val receives the integral where both
// branches stop within them (true); false where a branch goes on, a test is close to 0.02 or an
// abscissa close to a table point
template <bool LIMB>
__device__ __forceinline__ bool romberg_second(const Interior &q, const RadL &rc, const LineC &lc,
                                               const TW<LIMB> *__restrict__ tw, float *val) {
  const float pas0 = __fsub_rn(q.gb, q.ga);
  float off, offm;
  const float2 va = eval_F<LIMB, true>(q.ga, q.ca, rc, lc, tw, &off).value();
  float ta0 = va.x, ta1 = va.y;
  eval_F<LIMB, true>(q.gb, q.cb, rc, lc, tw, &offm).add(ta0, ta1);
  ta0 = __fmul_rn(ta0, 0.5f);
  ta1 = __fmul_rn(ta1, 0.5f);
  off = fminf(off, offm);
  const float2 f1 =
      eval_F<LIMB, true>(__fmaf_rn(pas0, 0.5f, q.ga), __fmaf_rn(-pas0, 0.5f, q.ca), rc, lc, tw, &offm).value();
  off = fminf(off, offm);
  float a0 = 0.0f, a1 = 0.0f;
#pragma unroll
  for (int i = 0; i < 2; i++) {
    const float c = i ? 0.75f : 0.25f;
    float x = __fmaf_rn(pas0, c, q.ga), y = __fmaf_rn(-pas0, c, q.ca);
    if (LIMB) {
      const float u = __fmul_rn(pas0, c);
      x = __fadd_rn(q.ga, u);
      y = __fsub_rn(q.ca, u);
    }
    const Fval<LIMB> f = eval_F<LIMB, true>(x, y, rc, lc, tw, &offm);
    off = fminf(off, offm);
    if (i == 0) {
      const float2 v = f.value();
      a0 = v.x;
      a1 = v.y;
    } else {
      f.add(a0, a1);
    }
  }
  const float h1 = __fmul_rn(pas0, 0.5f), h2 = __fmul_rn(pas0, 0.25f);
  auto branch = [&](float ta, float f, float a, float *r) {
    const float p = __fmul_rn(ta, pas0);
    const float t1 = __fmul_rn(__fadd_rn(ta, f), h1);
    const float u1 = __fmul_rn(__fmaf_rn(4.0f, t1, -p), 1.f / 3.f);
    const float t2 = __fmul_rn(__fadd_rn(ta, __fadd_rn(f, a)), h2);
    const float u2 = __fmul_rn(__fmaf_rn(4.0f, t2, -t1), 1.f / 3.f);
    const float w2 = __fmul_rn(__fmaf_rn(16.0f, u2, -u1), 1.f / 15.f);
    const float d1 = fabsf(u1 - p), d2 = fabsf(w2 - u1);
    const bool one = d1 < 0.0198f * u1, on = (u1 > 0.0f) & (d1 > 0.0202f * u1);
    *r = one ? u1 : w2;
    return one | (on & (d2 < 0.0198f * w2));
  };
  float r0, r1;
  const bool ok = branch(ta0, f1.x, a0, &r0) & branch(ta1, f1.y, a1, &r1);
  *val = __fadd_rn(r0, r1);
  return ok & (off >= kSideBand);
}

// Romberg's convergence test of one branch: obtprec = |t0 - old| / t0 > 0.02 means another level.
// The quotient is formed only where the products do not decide (also for zero, negative and
// non-finite values); *rare is set when it lies within kConvBand of 0.02.
__device__ __forceinline__ bool romberg_on(float t0, float old, bool *rare) {
  const float d = fabsf(t0 - old);
  if (t0 > 0.0f && d > 0.0202f * t0) return true;
  if (d < 0.0198f * t0) return false;
  const float o = d / t0;
  if (fabsf(o - 0.02f) < kConvBand) *rare = true;
  return o > 0.02f;
}

// sqrt(hi) - sqrt(lo) without cancellation
__device__ __forceinline__ float sqrt_diff(float hi, float lo) {
  float d = hi - lo;
  float sh = sqrtf(hi), sl = sqrtf(lo);
  float den = sh + sl;
  return den > 0.0f ? d / den : 0.0f;
}

// g* and 1 - g* of a bin edge, clamped to [0, 1] (integ_relline_bin, Relprofile.cpp:653-666).
// The side of gmin and gmax is taken from the signs of the float-float differences: the two
// rounded quotients alone can give g <= 1 with 1 - g < 0 for an edge just above gmax.
// (ff_diff: near gmin and gmax the sign is right and the value within about an ulp)
__device__ __forceinline__ float2 edge_gc(float2 E, const RadL &rc) {
  const float dlo = ff_diff(E, rc.gmin), dhi = ff_diff(rc.gmax, E);
  const bool below = dlo <= 0.0f, above = dhi <= 0.0f;
  const float g = fminf(__fmul_rn(dlo, rc.inv_dg), 1.0f), c = fminf(__fmul_rn(dhi, rc.inv_dg), 1.0f);
  return make_float2(below ? 0.0f : above ? 1.0f : g, below ? 1.0f : above ? 0.0f : c);
}

// ---- bins close to Romberg's threshold, in FP64 by a whole warp ----
// gmin or gmax of the radius in FP64, as the set-up kernel computes it (Relprofile.cpp:295-300)
__device__ double gext_fp64(const RelxTables &tab, const RelxSetState &s, int itab, double ifac, bool is_max) {
  const int nr = tab.rel_nr, nm = tab.rel_nmu0;
  const size_t b00 = (size_t) s.ind_a * nm + s.ind_mu0, b10 = (size_t) (s.ind_a + 1) * nm + s.ind_mu0;
  const size_t b01 = b00 + 1, b11 = b10 + 1;
  const float *a = is_max ? tab.rel_gmax : tab.rel_gmin;
  const double fa = s.ifac_a, fm = s.ifac_mu0;
  double v[2];
  for (int q = 0; q < 2; q++) {
    const int i = itab + q;
    v[q] = lerp2(fa, fm, a[b00 * nr + i], a[b10 * nr + i], a[b01 * nr + i], a[b11 * nr + i]);
  }
  return lerp1(ifac, v[1], v[0]);
}

// the radius's transfer functions in FP64 (interp_lin_2d_float, then interp_lin_1d of the two table rows,
// Relprofile.cpp:67-77, 280-293) at table point g: trf1, trf2, cosne1, cosne2
__device__ void trf_fp64(const RelxTables &tab, const RelxSetState &s, int itab, double ifac, int g, double *tf) {
  const int nr = tab.rel_nr, nm = tab.rel_nmu0, ng = tab.rel_ng;
  const size_t b00 = (size_t) s.ind_a * nm + s.ind_mu0, b10 = (size_t) (s.ind_a + 1) * nm + s.ind_mu0;
  const size_t b01 = b00 + 1, b11 = b10 + 1;
  const double fa = s.ifac_a, fm = s.ifac_mu0;
  double v[2][4];
#pragma unroll
  for (int q = 0; q < 2; q++) {  // rows itab and itab + 1
    const size_t row = (size_t) (itab + q) * ng + g;
    const float4 c00 = __ldg(&tab.rel_tc[b00 * nr * ng + row]), c10 = __ldg(&tab.rel_tc[b10 * nr * ng + row]);
    const float4 c01 = __ldg(&tab.rel_tc[b01 * nr * ng + row]), c11 = __ldg(&tab.rel_tc[b11 * nr * ng + row]);
    v[q][0] = lerp2(fa, fm, c00.x, c10.x, c01.x, c11.x);
    v[q][1] = lerp2(fa, fm, c00.y, c10.y, c01.y, c11.y);
    v[q][2] = lerp2(fa, fm, c00.z, c10.z, c01.z, c11.z);
    v[q][3] = lerp2(fa, fm, c00.w, c10.w, c01.w, c11.w);
  }
#pragma unroll
  for (int c = 0; c < 4; c++) tf[c] = lerp1(ifac, v[1][c], v[0][c]);
}

// the table's g* points, and the last one at or below x (binary_search, relutility.c:155-170) from a first
// guess and exact comparisons
__device__ __forceinline__ double gstar_fp64(int ng, int g) {
  return 5e-3 + (1.0 - 2 * 5e-3) / (ng - 1) * (double) (float) g;
}
__device__ __forceinline__ int gstar_index(int ng, double x) {
  int k = (int) ((x - 5e-3) * ((ng - 1) / (1.0 - 2 * 5e-3)));
  k = max(0, min(k, ng - 2));
  if (k < ng - 2 && gstar_fp64(ng, k + 1) <= x) k++;
  if (k > 0 && gstar_fp64(ng, k) > x) k--;
  return k;
}

// relb_func (Relprofile.cpp:489-521) of branch k in FP64 without the emissivity factor (it scales every value
// of one integration alike); point(g, c): transfer function c at table point g, g0 <= g <= g1
template <class Point>
__device__ __forceinline__ double relb_fp64(int ng, int limb, double gmn, double gmx, int g0, int g1, int k, double eg,
                                            Point point) {
  const double del_g = 1.0 / (gmx - gmn);
  const double egstar = (eg - gmn) * del_g;
  const int klo = min(max(gstar_index(ng, egstar), g0), g1 - 1);  // within [g0, g1] up to rounding
  const double x0 = gstar_fp64(ng, klo), x1 = gstar_fp64(ng, klo + 1);
  const double inte = (egstar - x0) / (x1 - x0), inte1 = 1.0 - inte;
  const double ftrf = inte * point(klo, k) + inte1 * point(klo + 1, k);
  double val = eg * eg * eg / ((gmx - gmn) * sqrt(egstar - egstar * egstar)) * ftrf;
  if (limb != 0) {
    const double mu = inte * point(klo, 2 + k) + inte1 * point(klo + 1, 2 + k);
    val *= (limb == 1) ? (1.0 + 2.06 * mu) : log(1.0 + 1.0 / mu);
  }
  return val;
}
// one step of the Romberg table of level n (t[ii] holds t[ii][n-ii] of the last completed level) from the
// trapezoid sum u: updates u to t[n][0] and returns whether another level is due
__device__ __forceinline__ bool romberg_row_fp64(double *t, int n, double &u) {
  double rr = 1.0, old = 0.0;
#pragma unroll
  for (int ii = 1; ii <= 6; ii++) {
    if (ii > n) break;
    rr *= 4.0;
    const double w = (rr * u - t[ii - 1]) / (rr - 1.0);
    old = t[ii - 1];
    t[ii - 1] = u;
    u = w;
  }
#pragma unroll
  for (int ii = 1; ii <= 6; ii++)
    if (ii == n) t[ii] = u;
  return fabs(u - old) / u > 0.02;
}

// Both branches' romberg_integration (Relprofile.cpp:524-579) in FP64 over [a, b] in energy at one radius, the
// emissivity factored out.  By one lane: fewest instructions on the FP64 pipe (GB300: 2 lanes per clock
// and SM), for the solo kernel.
__device__ double romberg_lane_fp64(const RelxTables &tab, const RelxSetState &s, int itab, double ifac, double gmn,
                                    double gmx, double a, double b) {
  const int ng = tab.rel_ng, limb = s.limb;
  const double del_g = 1.0 / (gmx - gmn);
  const int g0 = gstar_index(ng, (a - gmn) * del_g), g1 = gstar_index(ng, (b - gmn) * del_g) + 1;
  double tf[RELX_MAX_NG][4];
  for (int g = g0; g <= g1; g++) trf_fp64(tab, s, itab, ifac, g, tf[g - g0]);
  double total = 0.0;
  for (int k = 0; k < 2; k++) {
    auto func = [&](double eg) {
      return relb_fp64(ng, limb, gmn, gmx, g0, g1, k, eg, [&](int g, int c) { return tf[g - g0][c]; });
    };
    const double ta = (func(a) + func(b)) / 2.0;
    double t[7], pas = b - a, u = 0.0;
    t[0] = ta * pas;
    for (int n = 1; n <= 6; n++) {
      pas = pas / 2.0;
      double sum = ta;
      for (int i = 1; i < (1 << n); i++) sum += func(a + pas * i);
      u = sum * pas;
      if (!romberg_row_fp64(t, n, u)) break;
    }
    total += u;
  }
  return total;
}
// The same by a warp, for the team kernel (a single spectrum waits for its one or two such bins: 50 us by
// one lane): branch 0 on the lower half, 1 on the upper; the abscissae of a level go to the lanes, their
// values are added in order.  Lane l holds the transfer functions at the table points g0 + l, g0 + 32 + l.
// Every lane returns the sum of the branches.
__device__ double romberg_warp_fp64(const RelxTables &tab, const RelxSetState &s, int itab, double ifac, double gmn,
                                    double gmx, double a, double b) {
  constexpr unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31, k = lane >> 4, sub = lane & 15, ng = tab.rel_ng;
  const double del_g = 1.0 / (gmx - gmn);
  const int g0 = gstar_index(ng, (a - gmn) * del_g), g1 = gstar_index(ng, (b - gmn) * del_g) + 1;
  double tf[2][4] = {};
  for (int q = 0; q < 2; q++)
    if (g0 + 32 * q + lane <= g1) trf_fp64(tab, s, itab, ifac, g0 + 32 * q + lane, tf[q]);
  // transfer function c of either branch (c and its neighbour are both fetched: the halves differ in k)
  auto point = [&](int g, int c) {
    const int l = g - g0, c0 = c & 2;
    const double a0 = __shfl_sync(full, tf[0][c0], l & 31), a1 = __shfl_sync(full, tf[0][c0 + 1], l & 31);
    const double b0 = __shfl_sync(full, tf[1][c0], l & 31), b1 = __shfl_sync(full, tf[1][c0 + 1], l & 31);
    return l < 32 ? ((c & 1) ? a1 : a0) : ((c & 1) ? b1 : b0);
  };
  auto func = [&](double eg) { return relb_fp64(ng, s.limb, gmn, gmx, g0, g1, k, eg, point); };
  const double f = func(sub == 1 ? b : a);
  const double ta = (__shfl_sync(full, f, 0, 16) + __shfl_sync(full, f, 1, 16)) / 2.0;
  double t[7], pas = b - a, res = 0.0;
  t[0] = ta * pas;
  bool on = true;
  for (int n = 1; n <= 6; n++) {
    pas = pas / 2.0;
    double sum = ta;
    const int last = (1 << n) - 1;
    for (int i0 = 1; i0 <= last; i0 += 16) {
      const double v = func(a + pas * min(i0 + sub, last));
      const int m = min(16, last + 1 - i0);
      for (int i = 0; i < m; i++) sum += __shfl_sync(full, v, i, 16);
    }
    double u = sum * pas;
    const bool more = romberg_row_fp64(t, n, u);
    if (on) res = u;
    on = on && more;
    if (!__any_sync(full, on)) break;
  }
  return __shfl_sync(full, res, 0) + __shfl_sync(full, res, 16);
}

// edge_gc of an edge between gmin and gmax, by the same products (elsewhere g* comes out at most 0 or at
// least 1 - H, which sends the bin to the general path)
__device__ __forceinline__ float2 edge_in(float2 E, const RadL &rc) {
  return make_float2(__fmul_rn(ff_diff(E, rc.gmin), rc.inv_dg), __fmul_rn(ff_diff(rc.gmax, E), rc.inv_dg));
}
// both edges away from the sqrt terms: the whole bin is interior
__device__ __forceinline__ bool edges_inner(float2 lo, float2 hi) { return (lo.x > kH) & (hi.x < 1.0f - kH); }

// The parts of integ_relline_bin (Relprofile.cpp:650-726) before the interior integration: the sqrt
// edge terms within H of g* = 0 and 1, and the interior's ends in g* and 1 - g*; returns whether the
// bin has an interior.  lo, hi: the clamped g*, 1 - g* of the bin's edges.
__device__ __forceinline__ bool bin_interior(float2 lo, float2 hi, const RadL &rc, Interior &q) {
  q.ga = lo.x;
  q.ca = lo.y;
  q.gb = hi.x;
  q.cb = hi.y;
  q.flu = 0.0f;
  q.lo_H = q.hi_H = false;
  if (lo.x > kH && hi.x < 1.0f - kH) return true;
  if (hi.x == 0.0f) return false;
  bool has_lo = true, has_hi = true;
  if (lo.x <= kH) {
    float hhi = kH;
    q.ga = kH;
    q.ca = 1.0f - kH;
    q.lo_H = true;
    if (hi.x <= kH) { hhi = hi.x; has_lo = false; }
    q.flu = __fmul_rn(rc.edge_lo, sqrt_diff(hhi, lo.x));
  }
  if (hi.x >= 1.0f - kH) {
    float hi_c = kH;  // 1 - hlo
    q.gb = 1.0f - kH;
    q.cb = kH;
    q.hi_H = true;
    if (lo.x >= 1.0f - kH) { hi_c = lo.y; has_hi = false; }
    q.flu = __fmaf_rn(rc.edge_hi, sqrt_diff(hi_c, hi.y), q.flu);
  }
  return has_lo && has_hi;
}

// The interior of any bin: the midpoint rule, or romberg_integration (Relprofile.cpp:524-579), both
// branches in lock step; a level's sum reuses the earlier levels' points, p[ii] holds t[ii][n-ii] of the
// last completed level.  *rare is set when a tested FP32 obtprec lies within kConvBand of 0.02.  One
// place forms every abscissa and its integrand: few bins come here, and their code has to stay out of
// the way of the loops that the others run (instruction cache).
template <bool LIMB>
__device__ __forceinline__ float bin_general(const Interior &q, const float2 *eb, bool romb, const RadL &rc,
                                             const RelxRadRec &rec, const LineC &lc, const float2 *gs,
                                             const TW<LIMB> *__restrict__ tw, bool *rare) {
  const float pas0 = __fsub_rn(q.gb, q.ga);
  float ta0 = 0.0f, ta1 = 0.0f, s0 = 0.0f, s1 = 0.0f, r0 = 0.0f, r1 = 0.0f;
  float p0[7], p1[7];
  bool c0 = false, c1 = false;
#pragma unroll 1
  for (int n = romb ? 0 : -1; n <= 6; n++) {
    // the abscissae of level n: the midpoint (-1), both ends (0), the odd multiples of 2^-n
    const float sc = __int_as_float((127 - n) << 23);
    const int last = n <= 0 ? n + 1 : 1 << n;
    float a0 = 0.0f, a1 = 0.0f;
    Fval<LIMB> f = {};
#pragma unroll 1
    for (int i = n <= 0 ? 0 : 1; n <= 0 ? i <= last : i < last; i += n <= 0 ? 1 : 2) {
      float x, y;
      if (n < 0) {
        x = 0.5f * __fadd_rn(q.ga, q.gb);
        y = 0.5f * __fadd_rn(q.ca, q.cb);
      } else if (n == 0) {
        x = i ? q.gb : q.ga;
        y = i ? q.cb : q.ca;
      } else {
        const float c = (float) i * sc;
        x = __fmaf_rn(pas0, c, q.ga);
        y = __fmaf_rn(-pas0, c, q.ca);
        if (LIMB && n == 2) {
          const float u = __fmul_rn(pas0, c);
          x = __fadd_rn(q.ga, u);
          y = __fsub_rn(q.ca, u);
        }
      }
      const GPos g = g_pos(x, lc);
      float fi = g.dt < 0.0f ? __fsub_rn(g.tr, 1.0f) : g.tr;
      if (fabsf(g.dt) < kSideBand && g.tr >= 1.0f && g.tr <= lc.ng2) {
        // side of grid point k from the reference's abscissa in energy (float-float)
        const int k = (int) g.tr;
        const float2 alo = q.lo_H ? rec.eH : eb[0];
        const float2 ahi = q.hi_H ? rec.e1H : eb[1];
        float2 eg;
        if (n < 0) {
          eg = ff_mulf(ff_add(alo, ahi), 0.5f);
        } else if (i == (1 << n)) {
          eg = ahi;
        } else {
          const float2 w = ff_add(ahi, ff_neg(alo));
          eg = ff_add(alo, ff_mulf(w, (float) i * sc));
        }
        const float2 G = ff_add(rc.gmin, ff_mul(gs[k], rec.dg));
        fi = ff_ge(eg, G) ? g.tr : __fsub_rn(g.tr, 1.0f);
      }
      f = F_at<LIMB>(x, y, g, fi, romb, rc, lc, tw);
      if (n == 0 && i == 0) {
        const float2 v = f.value();
        a0 = v.x;
        a1 = v.y;
      } else {
        f.add(a0, a1);
      }
    }
    if (n < 0) return __fmaf_rn(f.both(), pas0, q.flu);
    if (n == 0) {
      ta0 = __fmul_rn(a0, 0.5f);
      ta1 = __fmul_rn(a1, 0.5f);
      p0[0] = __fmul_rn(ta0, pas0);
      p1[0] = __fmul_rn(ta1, pas0);
      continue;
    }
    s0 = __fadd_rn(s0, a0);
    s1 = __fadd_rn(s1, a1);
    const float pas = __fmul_rn(pas0, sc);
    const float old0 = p0[n - 1], old1 = p1[n - 1];
    float t0 = __fmul_rn(__fadd_rn(ta0, s0), pas), t1 = __fmul_rn(__fadd_rn(ta1, s1), pas);
    float r = 1.0f;
#pragma unroll 1
    for (int ii = 1; ii <= n; ii++) {
      r *= 4.0f;
      const float inv = c_inv4m1[ii];
      const float n0 = __fmul_rn(__fmaf_rn(r, t0, -p0[ii - 1]), inv);
      const float n1 = __fmul_rn(__fmaf_rn(r, t1, -p1[ii - 1]), inv);
      p0[ii - 1] = t0;
      p1[ii - 1] = t1;
      t0 = n0;
      t1 = n1;
    }
    p0[n] = t0;
    p1[n] = t1;
    if (!c0) {
      r0 = t0;
      c0 = !romberg_on(t0, old0, rare);
    }
    if (!c1) {
      r1 = t1;
      c1 = !romberg_on(t1, old1, rare);
    }
    if (c0 && c1) break;
  }
  return __fadd_rn(q.flu, __fadd_rn(r0, r1));
}

// int_edge norms (Relprofile.cpp:585-621) of a radius: trf at g* = H is T[1], at 1 - H is T[ng-2]
template <bool LIMB>
__device__ __forceinline__ void line_edges(RadL &rc, const TW<LIMB> *tw, int ng) {
  const float sH = sqrtf(kH), isq = rsqrtf(kH * (1.0f - kH));
  auto norm = [&](float g, const TW<LIMB> &t) {
    const float e = __fmaf_rn(g, rc.dgf, rc.gmin.x), e3 = __fmul_rn(__fmul_rn(__fmul_rn(e, e), e), isq);
    float f;
    if constexpr (!LIMB) f = __fadd_rn(t.t.x, t.t.y);
    else f = sum2(t.t.y, limb_factor(rc.limb, t.t.w), t.t.x, limb_factor(rc.limb, t.t.z));
    return __fmul_rn(__fmul_rn(__fmul_rn(2.0f, sH), e3), f);
  };
  rc.edge_lo = norm(kH, tw[1]);
  rc.edge_hi = norm(1.0f - kH, tw[ng - 2]);
}
__device__ __forceinline__ void line_rad(RadL &rc, const RelxRadRec &rr) {
  rc.gmin = rr.gmin;
  rc.gmax = rr.gmax;
  rc.dgf = rr.dg.x;
  rc.inv_dg = rr.inv_dg;
}

// The bins of a group that bin_general marked rare (mask: T bits per radius, cleared here): the interior
// integrated again with FP64 Romberg over the reference's interval (the bin's edges, or gstar2ener(H) /
// gstar2ener(1 - H)).  About two bins of a set come here; called between groups, where the caller
// holds few registers (a call among the bins' loops would make the compiler spill theirs).
template <bool LIMB, bool SOLO>
__device__ __noinline__ void rare_bins(const RelxTables &tab, const RelxSetState &s, const double *ge,
                                       const double *ifac, int ng, const RelxRadRec *recs, const TW<LIMB> *twb, int twp,
                                       const float2 *eff, float *rows, int rpitch, int tlo, unsigned *mask, int nword) {
  const int lane = threadIdx.x & 31;
  // solo: the first lane of every radius takes the radius's bins; team: the warp takes them in turn
  for (int c = SOLO ? lane / kRadLanes : 0; c < (SOLO ? lane / kRadLanes + 1 : kGroup); c++) {
    for (int w = 0; w < nword; w++) {
      unsigned m = mask[c * nword + w];
      __syncwarp();
      if (SOLO ? lane % kRadLanes != 0 : false) m = 0u;
      if (SOLO ? lane % kRadLanes == 0 : lane == 0) mask[c * nword + w] = 0u;
      for (; m; m &= m - 1) {
        const RelxRadRec &rr = recs[c];
        RadL rc;
        line_rad(rc, rr);
        rc.limb = s.limb;
        line_edges<LIMB>(rc, twb + c * twp, ng);
        const double gmn = gext_fp64(tab, s, rr.itab, ifac[c], false), gmx = gext_fp64(tab, s, rr.itab, ifac[c], true);
        const int jj = w * 32 + __ffs(m) - 1, j = tlo + jj;
        Interior q;
        bin_interior(edge_gc(eff[jj], rc), edge_gc(eff[jj + 1], rc), rc, q);
        const double a = q.lo_H ? (RELX_GFAC_H * (gmx - gmn) + gmn) : ge[j];
        const double b = q.hi_H ? ((1 - RELX_GFAC_H) * (gmx - gmn) + gmn) : ge[j + 1];
        float *o = &rows[c * rpitch + jj];
        if constexpr (SOLO) {
          *o = __fmaf_rn(q.flu + (float) romberg_lane_fp64(tab, s, rr.itab, ifac[c], gmn, gmx, a, b), rr.ew, *o);
        } else {
          const float v = q.flu + (float) romberg_warp_fp64(tab, s, rr.itab, ifac[c], gmn, gmx, a, b);
          if (lane == 0) *o = v;
        }
      }
    }
  }
  __syncwarp();
}

// pitch of a radius's transfer functions in shared memory (entries): even (16-byte rows of float2) with
// an odd half, so that the eight radii of a group start in different banks
__host__ __device__ inline int line_tw_pitch(int ng) {
  int p = (ng + 1) & ~1;
  return ((p >> 1) & 1) ? p : p + 2;
}
// pitch of a class's row of bins: T + 4 puts the four lanes of the eight radii in different banks
constexpr int line_row_pitch(int T) { return T + 4; }

// copy of a group's radius records (eight 64-byte rows) into shared memory, 16 bytes per lane;
// n: records of the group that exist
__device__ __forceinline__ void group_fetch(RelxRadRec *dst, const RelxRadRec *src, int n) {
  const int lane = threadIdx.x & 31;
  if ((lane >> 2) < n) {
    const uint32_t d = (uint32_t) __cvta_generic_to_shared(reinterpret_cast<unsigned char *>(dst) + lane * 16);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d),
                 "l"(reinterpret_cast<const unsigned char *>(src) + lane * 16)
                 : "memory");
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
}
template <int N>
__device__ __forceinline__ void group_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
  __syncwarp();
}

// One group: the warp integrates the bins [tlo, thi) of kGroup consecutive radii, kRadLanes lanes per
// radius, each lane a run of consecutive bins, first those below 0.95 keV (midpoint rule), then the
// others (Romberg).  Neighbouring radii have nearly the same bins, so the lanes stay together, the
// radius's constants sit in registers, and a bin's upper edge (its g* and, for Romberg, the
// integrand there) is the next bin's lower one.  The radii of a group are the eight summation
// classes of the zone (radius index from the zone's first modulo 8): row[class] has no other
// contributor, so the adds need no order within a group.
// SOLO: rows hold the classes' sums, v ew is added; otherwise rows receive the values v.  Returns
// whether the lane marked a bin in rmask.
template <bool LIMB, bool SOLO>
__device__ __forceinline__ bool line_group(const RelxTables &tab, const RelxSetState *__restrict__ sst,
                                           const float4 *__restrict__ htab, int set, int nrad,
                                           const RelxRadRec *recs, TW<LIMB> *twb, int twp, const float2 *eff,
                                           float *rows, int rpitch, int tlo, int thi, int jred, const LineC &lc,
                                           const float2 *gs, unsigned *rmask, int nword) {
  const int lane = threadIdx.x & 31, c = lane / kRadLanes, sub = lane % kRadLanes;
  const RelxRadRec &rr = recs[c];
  const int ng = lc.ng;
  bool live = false, any = false;
  if (c < nrad) {
    const int ielo = rr.ielo;
    live = ielo >= 0 && ielo < thi && rr.iehi >= tlo;
  }
  TW<LIMB> *tw = twb + c * twp;
  if (live) {
    // trf(g*) at this radius: interp_lin_1d(ifac_r, T[ind+1], T[ind]) (Relprofile.cpp:280-293)
    const int it = rr.itab;
    const float2 *__restrict__ T = reinterpret_cast<const float2 *>(htab + (size_t) set * tab.rel_nr * ng);
    const float fr = rr.ifac, fr1 = __fsub_rn(1.0f, fr);
    if constexpr (!LIMB) {
      if ((ng & 1) == 0) {  // two table points per 16-byte load
        const float4 *hi4 = reinterpret_cast<const float4 *>(T + it * ng);
        const float4 *lo4 = reinterpret_cast<const float4 *>(T + (it + 1) * ng);
        float4 *o4 = reinterpret_cast<float4 *>(tw);
#pragma unroll 5
        for (int g = sub; g < ng >> 1; g += kRadLanes) {
          const float4 lo = __ldg(lo4 + g), hi = __ldg(hi4 + g);
          o4[g] = make_float4(sum2(fr1, lo.x, fr, hi.x), sum2(fr1, lo.y, fr, hi.y),
                              sum2(fr1, lo.z, fr, hi.z), sum2(fr1, lo.w, fr, hi.w));
        }
      } else {
        for (int g = sub; g < ng; g += kRadLanes) {
          const float2 lo = __ldg(&T[(it + 1) * ng + g]), hi = __ldg(&T[it * ng + g]);
          tw[g].t = make_float2(sum2(fr1, lo.x, fr, hi.x), sum2(fr1, lo.y, fr, hi.y));
        }
      }
    } else {
      const float2 *__restrict__ C = T + tab.rel_nr * ng;
      // The points [pa, pb) that the tile's bins reach: an abscissa between its ends reads the point below it, one
      // further down where it lies on a point, and the next; one point more either side than that.  Points 1 and
      // ng - 2 of line_edges are among them where a bin has an edge term.  (All points of four functions cost a tile of 32
      // bins more than its bins: 4096 relline sets, 64 points 6.08 ms so, 5.57 ms with these.)
      int pa = 0, pb = ng;
      {
        RadL q;
        line_rad(q, rr);
        const float xa = edge_gc(eff[0], q).x, xb = edge_gc(eff[thi - tlo], q).x;
        if (xa > kH) pa = max(0, (int) ((xa - kH) * lc.inv_dgs) - 2) & ~1;
        if (xb < 1.0f - kH) pb = min(ng, (int) ((fmaxf(xb, kH) - kH) * lc.inv_dgs) + 4);
      }
      if ((ng & 1) == 0) {
        const float4 *thi4 = reinterpret_cast<const float4 *>(T + it * ng);
        const float4 *tlo4 = reinterpret_cast<const float4 *>(T + (it + 1) * ng);
        const float4 *chi4 = reinterpret_cast<const float4 *>(C + it * ng);
        const float4 *clo4 = reinterpret_cast<const float4 *>(C + (it + 1) * ng);
#pragma unroll 2
        for (int g = (pa >> 1) + sub; 2 * g < pb; g += kRadLanes) {
          const float4 lo = __ldg(tlo4 + g), hi = __ldg(thi4 + g), cl = __ldg(clo4 + g), ch = __ldg(chi4 + g);
          tw[2 * g].t = make_float4(sum2(fr1, lo.x, fr, hi.x), sum2(fr1, lo.y, fr, hi.y), sum2(fr1, cl.x, fr, ch.x),
                                    sum2(fr1, cl.y, fr, ch.y));
          tw[2 * g + 1].t = make_float4(sum2(fr1, lo.z, fr, hi.z), sum2(fr1, lo.w, fr, hi.w),
                                        sum2(fr1, cl.z, fr, ch.z), sum2(fr1, cl.w, fr, ch.w));
        }
      } else {
        for (int g = pa + sub; g < pb; g += kRadLanes) {
          const float2 lo = __ldg(&T[(it + 1) * ng + g]), hi = __ldg(&T[it * ng + g]);
          const float2 cl = __ldg(&C[(it + 1) * ng + g]), ch = __ldg(&C[it * ng + g]);
          tw[g].t = make_float4(sum2(fr1, lo.x, fr, hi.x), sum2(fr1, lo.y, fr, hi.y), sum2(fr1, cl.x, fr, ch.x),
                                sum2(fr1, cl.y, fr, ch.y));
        }
      }
    }
  }
  __syncwarp();
  if (live) {
    RadL rc;
    line_rad(rc, rr);
    if constexpr (LIMB) rc.limb = sst[set].limb;
    line_edges<LIMB>(rc, tw, ng);
    const float ew = rr.ew;
    const int jlo = max(rr.ielo, tlo), jend = min(rr.iehi + 1, thi);
    float *row = rows + c * rpitch;
    auto put = [&](float *o, float v) {
      if constexpr (SOLO) *o = __fmaf_rn(v, ew, *o);
      else *o = v;
    };
    // The radius's bins in sections: its lowest ones, within H of g* = 0 at their lower edge, and its last
    // four are dealt to the lanes one by one (they carry sqrt edge terms, and near gmax most need a
    // second Romberg level); between them the midpoint bins [jh, jm) below 0.95 keV and the Romberg bins
    // [jm, jt) in runs of consecutive bins per lane.  The loops over the runs
    // hold only what nearly all their bins need; the others are marked in resta and restb and go
    // through the last loop, with the lowest and the last ones: two Romberg levels there, and
    // bin_general for what these do not finish.
    int nlow = 0;  // this lane's lowest bins: jlo + sub, jlo + sub + kRadLanes, ...
    for (int j = jlo + sub; j < jend && !(edge_in(eff[j - tlo], rc).x > kH); j += kRadLanes) nlow++;
    int jh = nlow;
#pragma unroll
    for (int o = 1; o < kRadLanes; o <<= 1)
      jh += __shfl_xor_sync(((1u << kRadLanes) - 1u) << (lane & ~(kRadLanes - 1)), jh, o);
    jh += jlo;
    const int jt = min(jend, max(jh, rr.iehi + 1 - kRadLanes));
    const int jm = max(jh, min(jred, jt));
    const int qa = (jm - jh + kRadLanes - 1) / kRadLanes, qb = (jt - jm + kRadLanes - 1) / kRadLanes;
    const int ja = jh + sub * qa, jb = jm + sub * qb;
    unsigned resta = 0, restb = 0;
    {
      const int n = min(jm, ja + qa) - ja;
      const float2 *e = &eff[ja - tlo];
      float *o = &row[ja - tlo];
      if (n > 0) {
        float2 lo = edge_in(*e, rc);
        const float2 *end = e + n;
        for (unsigned bit = 1u; e != end; bit <<= 1, o++) {
          const float2 hi = edge_in(*++e, rc);
          float off;
          const float v = __fmul_rn(mid_F<LIMB>(lo, hi, rc, lc, tw, &off), __fsub_rn(hi.x, lo.x));
          if (edges_inner(lo, hi) & (off >= kSideBand)) put(o, v);
          else resta |= bit;
          lo = hi;
        }
      }
    }
    {
      const int n = min(jt, jb + qb) - jb;
      const float2 *e = &eff[jb - tlo];
      float *o = &row[jb - tlo];
      if (n > 0) {
        float2 lo = edge_in(*e, rc);
        float offa;
        Fval<LIMB> fa = eval_F<LIMB, true>(lo.x, lo.y, rc, lc, tw, &offa);
        const float2 *end = e + n;
        for (unsigned bit = 1u; e != end; bit <<= 1, o++) {
          const float2 hi = edge_in(*++e, rc);
          float v, offb, offm;
          const Fval<LIMB> fb = eval_F<LIMB, true>(hi.x, hi.y, rc, lc, tw, &offb);
          const bool one = romberg_first<LIMB>(lo, hi, fa, fb, rc, lc, tw, &v, &offm);
          if (one & edges_inner(lo, hi) & (fminf(fminf(offa, offb), offm) >= kSideBand)) put(o, v);
          else restb |= bit;
          fa = fb;
          offa = offb;
          lo = hi;
        }
      }
    }
    bool last = jt + sub < jend;
    int jlow = jlo + sub;
    while (last || nlow > 0 || resta || restb) {
      int j;
      if (last) {
        j = jt + sub;
        last = false;
      } else if (nlow > 0) {
        j = jlow;
        jlow += kRadLanes;
        nlow--;
      } else if (resta) {
        j = ja + __ffs(resta) - 1;
        resta &= resta - 1;
      } else {
        j = jb + __ffs(restb) - 1;
        restb &= restb - 1;
      }
      const int jj = j - tlo;
      Interior n;
      if (bin_interior(edge_gc(eff[jj], rc), edge_gc(eff[jj + 1], rc), rc, n)) {
        const bool romb = n.lo_H ? rr.red_H != 0 : j >= jred;
        float v;
        bool done;
        if (romb) {
          done = romberg_second<LIMB>(n, rc, lc, tw, &v);
          v = __fadd_rn(n.flu, v);
        } else {
          float off;
          v = __fmaf_rn(mid_F<LIMB>(make_float2(n.ga, n.ca), make_float2(n.gb, n.cb), rc, lc, tw, &off),
                        __fsub_rn(n.gb, n.ga), n.flu);
          done = off >= kSideBand;
        }
        if (!done) {
          bool rare = false;
          v = bin_general<LIMB>(n, &eff[jj], romb, rc, rr, lc, gs, tw, &rare);
          if (rare) {  // stored by rare_bins before the class's next radius
            atomicOr(&rmask[c * nword + (jj >> 5)], 1u << (jj & 31));
            any = true;
            continue;
          }
        }
        n.flu = v;
      }
      put(&row[jj], n.flu);
    }
  }
  __syncwarp();
  return any;
}

// bins of a zone's tile k: tiles of T bins from the profile-sum block that holds the zone's first bin
struct LineTile {
  int tlo, thi;  // thi: the zone's end at most
};
__device__ __forceinline__ LineTile line_tile(const RelxSetState &s, int z, int k, int T) {
  LineTile t;
  t.tlo = s.win_lo + ((s.zw_lo[z] - s.win_lo) & ~(kSumBinsH - 1)) + k * T;
  t.thi = min(t.tlo + T, s.zw_hi[z]);
  return t;
}
__device__ __forceinline__ int line_ntiles(const RelxSetState &s, int z, int T) {
  if (s.zw_hi[z] <= s.zw_lo[z] || s.zi1[z] < s.zi0[z]) return 0;
  const int t0 = s.win_lo + ((s.zw_lo[z] - s.win_lo) & ~(kSumBinsH - 1));
  return (s.zw_hi[z] - t0 + T - 1) / T;
}
// first entry of zone z's groups in RelxRadial::gr: zones are runs of radii, the outermost first
__device__ __forceinline__ int line_group_base(const RelxSetState &s, int z) {
  return s.zi0[z] / kGroup + (s.nz - 1 - z);
}

// the line-profile grid of a set and where its profile goes
struct LineOut {
  const double *ge;
  size_t pbase, zstride;
  bool prof;  // this zone's profile is stored
};
__device__ __forceinline__ LineOut line_out(const RelxTables &tab, const RelxSetIn *sin, const RelxSetState &s, int set,
                                            int z, int nza, const double *line_e) {
  const bool is_line = (s.model == RELX_RELLINE);
  LineOut o;
  o.ge = is_line ? (line_e + sin[set].e_off) : tab.conv_e;
  o.pbase = is_line ? (size_t) sin[set].e_off : (size_t) set * nza * RELX_NCONV;
  o.zstride = is_line ? 0 : RELX_NCONV;
  o.prof = !is_line || z == s.nz - 1;  // a line model's profile is its last zone's
  return o;
}

// sum of the eight classes in order, divided by the bin centre (renorm_relline_profile,
// Relprofile.cpp:753-762), and the profile sum of the 32 bins of one warp
__device__ __forceinline__ void line_store(const float *rows, int rpitch, const float2 *eff, int tlo, int b,
                                           const RelxSetState &s, int z, const LineOut &o, float *prof, double *tsum,
                                           int set, int nblk, int nza) {
  const int lane = threadIdx.x & 31, jj = b * kSumBinsH + lane, j = tlo + jj;
  double part = 0.0;
  if (j < s.zw_hi[z]) {
    float v = 0.0f;
#pragma unroll
    for (int w = 0; w < kGroup; w++) v += rows[w * rpitch + jj];
    const float emid = 0.5f * (eff[jj].x + eff[jj + 1].x);
    const float pv = v / emid;
    if (o.prof && j >= s.zw_lo[z]) prof[o.pbase + z * o.zstride + j] = pv;
    part = f2d(pv);
  }
#pragma unroll
  for (int m = 16; m > 0; m >>= 1) part += __shfl_xor_sync(0xffffffffu, part, m);
  if (lane == 0) tsum[((size_t) set * nblk + (tlo - s.win_lo) / kSumBinsH + b) * nza + z] = part;
}

static LineC line_const(int ng) {
  return LineC{ng, (float) ((ng - 1) / (1.0 - 2 * 5e-3)), (float) (ng - 2)};
}
__device__ __forceinline__ void line_gstar(float2 *gs, int ng) {  // Relprofile.cpp:104-106
  for (int g = threadIdx.x; g < ng; g += blockDim.x)
    gs[g] = ff_from_double(5e-3 + (1.0 - 2 * 5e-3) / (ng - 1) * ((float) g));
}
// the edges of the bins [tlo, thi) as float-float, by one warp; returns the first bin with a lower edge of at
// least 0.95 keV (thi if none)
__device__ __forceinline__ int line_edge_table(const double *ge, int tlo, int thi, float2 *eff) {
  int low = 0;
  for (int j0 = tlo; j0 <= thi; j0 += 32) {
    const int j = j0 + (threadIdx.x & 31);
    bool below = false;
    if (j <= thi) {
      const double e = ge[j];
      eff[j - tlo] = ff_split(e);
      below = j < thi && !dge(e, 0.95);
    }
    low += __popc(__ballot_sync(0xffffffffu, below));
  }
  return tlo + low;
}
// bit mask of the groups g0 .. g0 + 31 of zone z with a radius that reaches [tlo, thi)
__device__ __forceinline__ unsigned line_groups(const RelxRadial &R, int gb, int ngr, int g0, int tlo, int thi) {
  const int g = g0 + (threadIdx.x & 31);
  bool hit = false;
  if (g < ngr) {
    const int2 r = R.gr[gb + g];
    hit = r.x < thi && r.y >= tlo;
  }
  return __ballot_sync(0xffffffffu, hit);
}

// A warp's shared memory in the line kernels, from the CTA's dynamic shared memory: two groups' records
// (one in the team kernel), a group's transfer functions, the rows of its eight classes, the bin edges
// (solo kernel), and the masks of rare bins
template <bool LIMB, int T, int NRECS, int NROWS, bool EDGES>
struct LineWarp {
  static constexpr int rpitch = line_row_pitch(T), nword = T / 32;
  RelxRadRec *recs;
  TW<LIMB> *tw;
  float *rows;
  float2 *eff;
  unsigned *rmask;
  static __host__ __device__ size_t bytes(int twp) {
    return sizeof(RelxRadRec) * NRECS * kGroup + sizeof(TW<LIMB>) * kGroup * twp +
           sizeof(float) * NROWS * kGroup * rpitch + (EDGES ? sizeof(float2) * (T + 2) : 0) +
           (sizeof(unsigned) * kGroup * nword + 15) / 16 * 16;
  }
  // base: 16-byte aligned
  __device__ __forceinline__ LineWarp(unsigned char *base, int twp, int warp) {
    unsigned char *p = base + (size_t) warp * bytes(twp);
    recs = reinterpret_cast<RelxRadRec *>(p);
    p += sizeof(RelxRadRec) * NRECS * kGroup;
    tw = reinterpret_cast<TW<LIMB> *>(p);
    p += sizeof(TW<LIMB>) * kGroup * twp;
    rows = reinterpret_cast<float *>(p);
    p += sizeof(float) * NROWS * kGroup * rpitch;
    eff = reinterpret_cast<float2 *>(p);
    if (EDGES) p += sizeof(float2) * (T + 2);
    rmask = reinterpret_cast<unsigned *>(p);
  }
};
// Many sets: one warp per (set, zone, tile of T bins), taken from the list that line_table_kernel
// wrote, by persistent warps.  A zone's groups are summed in order by the one warp, so no warp waits
// for another (sets with a limb law run in the team kernel).
constexpr int kSoloWarps = 4;  // warps per CTA
constexpr int kSoloCtas = 6;   // CTAs per SM
template <int T>
__global__ void __launch_bounds__(kSoloWarps * 32, kSoloCtas) relline_solo_kernel(
    RelxTables tab, const RelxSetIn *__restrict__ sin, const RelxSetState *__restrict__ sst,
    const RelxRadial *__restrict__ srad, const double *__restrict__ line_e, const float4 *__restrict__ htab, int nza,
    float *__restrict__ prof, double *__restrict__ tsum, int nblk, const uint2 *__restrict__ list,
    int *cnt, LineC lc) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  static_assert(T % kSumBinsH == 0 && T <= 32 * kRadLanes, "whole sum blocks; a lane's bins fit a 32-bit mask");
  using Warp = LineWarp<false, T, 2, 1, true>;
  constexpr int rpitch = Warp::rpitch, nword = Warp::nword;
  const int ng = lc.ng, twp = line_tw_pitch(ng);
  const int lane = threadIdx.x & 31;
  float2 *gs = reinterpret_cast<float2 *>(smem_raw);  // [RELX_MAX_NG]
  const Warp w(smem_raw + sizeof(float2) * RELX_MAX_NG, twp, threadIdx.x >> 5);
  line_gstar(gs, ng);
  for (int i = lane; i < kGroup * rpitch; i += 32) w.rows[i] = 0.0f;
  for (int i = lane; i < kGroup * nword; i += 32) w.rmask[i] = 0u;
  __syncthreads();
  for (;;) {
    int t = 0;
    if (lane == 0) t = atomicAdd(&cnt[1], 1);
    t = __shfl_sync(0xffffffffu, t, 0);
    if (t >= cnt[0]) break;
    const uint2 task = list[t];
    const int set = (int) task.x, z = (int) (task.y & 255u);
    int tlo, thi, i0, i1, gb, jred;
    {
      const RelxSetState &s = sst[set];
      const LineTile tl = line_tile(s, z, (int) (task.y >> 8), T);
      tlo = tl.tlo;
      thi = tl.thi;
      i0 = s.zi0[z];
      i1 = s.zi1[z];
      gb = line_group_base(s, z);
      const double *ge = line_out(tab, sin, s, set, z, nza, line_e).ge;
      jred = line_edge_table(ge, tlo, thi, w.eff);
    }
    __syncwarp();
    for (int g0 = 0; g0 * kGroup <= i1 - i0; g0 += 32) {
      unsigned mask = line_groups(srad[set], gb, (i1 - i0) / kGroup + 1, g0, tlo, thi);
      int buf = 0;
      if (mask) {
        const int r = i0 + (g0 + __ffs(mask) - 1) * kGroup;
        group_fetch(w.recs, &srad[set].rec[r], min(kGroup, i1 + 1 - r));
      }
      while (mask) {
        const int r0 = i0 + (g0 + __ffs(mask) - 1) * kGroup;
        mask &= mask - 1;
        if (mask) {  // the next group's records arrive while this one is integrated
          const int r = i0 + (g0 + __ffs(mask) - 1) * kGroup;
          group_fetch(w.recs + (buf ^ 1) * kGroup, &srad[set].rec[r], min(kGroup, i1 + 1 - r));
          group_wait<1>();
        } else {
          group_wait<0>();
        }
        const bool any = line_group<false, true>(tab, sst, htab, set, min(kGroup, i1 + 1 - r0), w.recs + buf * kGroup,
                                                w.tw, twp, w.eff, w.rows, rpitch, tlo, thi, jred, lc, gs, w.rmask,
                                                nword);
        if (__any_sync(0xffffffffu, any)) {
          rare_bins<false, true>(tab, sst[set], line_out(tab, sin, sst[set], set, z, nza, line_e).ge,
                                &srad[set].ifac[r0], ng, w.recs + buf * kGroup, w.tw, twp, w.eff, w.rows, rpitch, tlo,
                                w.rmask, nword);
        }
        buf ^= 1;
      }
    }
    {
      const RelxSetState &s = sst[set];
      const LineOut o = line_out(tab, sin, s, set, z, nza, line_e);
      for (int b = 0; b * kSumBinsH < thi - tlo; b++)
        line_store(w.rows, rpitch, w.eff, tlo, b, s, z, o, prof, tsum, set, nblk, nza);
    }
    __syncwarp();
    for (int i = threadIdx.x & 31; i < kGroup * rpitch; i += 32) w.rows[i] = 0.0f;
    __syncwarp();
  }
}

// Few sets: a CTA of NW warps per (set, zone, tile of T bins); grid.x CTAs share a set's tiles.  The
// warps integrate NW groups of a zone at a time into rows of values (a NaN pattern that no arithmetic
// returns marks bins a radius does not reach); after each round one thread per (class, bin) adds the
// round's groups in order, so every sum has the order the solo kernel has.
constexpr unsigned kLineHole = 0xffffffffu;
template <bool LIMB, int T, int NW>
__global__ void __launch_bounds__(NW * 32, 32 / NW) relline_team_kernel(
    RelxTables tab, const RelxSetIn *__restrict__ sin, const RelxSetState *__restrict__ sst,
    const RelxRadial *__restrict__ srad, const double *__restrict__ line_e, const float4 *__restrict__ htab, int nza,
    float *__restrict__ prof, double *__restrict__ tsum, int nblk, LineC lc) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  static_assert(T == kSumBinsH, "one sum block per tile");
  constexpr int rpitch = line_row_pitch(T);
  constexpr int kMaxGroups = RELX_NFRAD / kGroup + 1;
  const int set = blockIdx.y;
  const RelxSetState &s = sst[set];
  if (s.status != RELX_OK || s.cached) return;
  if ((s.limb != 0) != LIMB) return;
  const int ng = tab.rel_ng, twp = line_tw_pitch(ng);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  __shared__ int tstart[RELX_NZMAX + 1];
  __shared__ int nlist, jred_s;
  __shared__ unsigned short glist[kMaxGroups + 31];
  __shared__ float ews[2][NW][kGroup];
  using Warp = LineWarp<LIMB, T, 1, 2, false>;
  constexpr int nword = Warp::nword, vpitch = kGroup * rpitch;  // a warp's two rows of values follow each other
  float2 *gs = reinterpret_cast<float2 *>(smem_raw);  // [RELX_MAX_NG]
  unsigned char *const base = smem_raw + sizeof(float2) * RELX_MAX_NG;
  const Warp w(base, twp, warp);
  float2 *eff = reinterpret_cast<float2 *>(base + NW * Warp::bytes(twp));  // [T + 1]
  if (lane < kGroup * nword) w.rmask[lane] = 0u;
  const int nz = s.nz;
  line_gstar(gs, ng);
  if (warp == 0) {  // the zones' tiles as one list
    int run = 0;
    for (int z0 = 0; z0 < nz; z0 += 32) {
      const int z = z0 + lane;
      const int n = z < nz ? line_ntiles(s, z, T) : 0;
      int inc = n;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += u;
      }
      if (z < nz) tstart[z] = run + inc - n;
      run += __shfl_sync(0xffffffffu, inc, 31);
    }
    if (lane == 0) tstart[nz] = run;
  }
  __syncthreads();
  const RelxRadial &R = srad[set];
  for (int task = blockIdx.x; task < tstart[nz]; task += gridDim.x) {
    int z = 0;
    while (tstart[z + 1] <= task) z++;
    const LineTile tl = line_tile(s, z, task - tstart[z], T);
    const int tlo = tl.tlo, thi = tl.thi;
    const LineOut o = line_out(tab, sin, s, set, z, nza, line_e);
    const int i0 = s.zi0[z], i1 = s.zi1[z], ngr = (i1 - i0) / kGroup + 1, gb = line_group_base(s, z);
    if (warp == 0) {
      const int j = line_edge_table(o.ge, tlo, thi, eff);
      if (lane == 0) jred_s = j;
    }
    if (warp == NW - 1) {  // the groups that reach the tile, in order
      int n = 0;
      for (int g0 = 0; g0 < ngr; g0 += 32) {
        const unsigned mask = line_groups(R, gb, ngr, g0, tlo, thi);
        if (mask >> lane & 1u) glist[n + __popc(mask & ((1u << lane) - 1u))] = (unsigned short) (g0 + lane);
        n += __popc(mask);
      }
      if (lane == 0) nlist = n;
    }
    __syncthreads();
    const int ngl = nlist, jred = jred_s;
    float acc = 0.0f;
    const int ac = tid / T, aj = tid % T;  // the (class, bin) this thread adds
    for (int q0 = 0, buf = 0; q0 < ngl; q0 += NW, buf ^= 1) {
      float *mine = w.rows + buf * vpitch;
      const int nq = min(NW, ngl - q0);
      if (warp < nq) {
        const int r0 = i0 + (int) glist[q0 + warp] * kGroup, nrad = min(kGroup, i1 + 1 - r0);
        group_fetch(w.recs, &R.rec[r0], nrad);
        for (int i = lane; i < kGroup * rpitch; i += 32) mine[i] = __uint_as_float(kLineHole);
        group_wait<0>();
        if (lane < kGroup) ews[buf][warp][lane] = lane < nrad ? w.recs[lane].ew : 0.0f;
        const bool any = line_group<LIMB, false>(tab, sst, htab, set, nrad, w.recs, w.tw, twp, eff, mine, rpitch, tlo,
                                                 thi, jred, lc, gs, w.rmask, nword);
        if (__any_sync(0xffffffffu, any))
          rare_bins<LIMB, false>(tab, s, o.ge, &R.ifac[r0], ng, w.recs, w.tw, twp, eff, mine, rpitch, tlo,
                                 w.rmask, nword);
      }
      __syncthreads();
      if (tid < kGroup * T) {
        const float *v0 = Warp(base, twp, 0).rows + buf * vpitch + ac * rpitch + aj;
#pragma unroll 4
        for (int q = 0; q < nq; q++) {
          const float v = v0[q * (Warp::bytes(twp) / sizeof(float))];
          if (__float_as_uint(v) != kLineHole) acc = __fmaf_rn(v, ews[buf][q][ac], acc);
        }
      }
    }
    __syncthreads();
    float *sums = Warp(base, twp, 0).rows;
    if (tid < kGroup * T) sums[ac * rpitch + aj] = acc;
    __syncthreads();
    if (warp == 0) line_store(sums, rpitch, eff, tlo, 0, s, z, o, prof, tsum, set, nblk, nza);
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// emission-angle distribution per zone (Relprofile.cpp:908-938), one CTA per set (few sets: per zone).  The set's
// (a, mu0)-interpolated transfer functions and emission-angle cosines on all table radii are
// written once per set by line_table_kernel (which the line profile reads as well) and read
// through the read-only cache.
// ---------------------------------------------------------------------------
constexpr int kHistWarps = 8;  // classes of radii of a zone, each summed by itself

// interpol_a_mu0 (Relprofile.cpp:39-80) of (trff1, trff2, cosne1, cosne2) at every (table radius,
// g*) of a set, for the line profile and the histogram: grid (chunks of kLineThreads entries, sets).
// A set's rel_nr x rel_ng float4 slot holds two planes of float2: (trff1, trff2), then (cosne1,
// cosne2), so that the line profile without a limb law reads half the bytes.
// The first CTA of a set also writes the range of bins that every group of radii reaches
// (RelxRadial::gr) and, for the solo line kernel (list not null), the set's (zone, tile) tasks.
__global__ void __launch_bounds__(kLineThreads) line_table_kernel(RelxTables tab, const RelxSetState *__restrict__ sst,
                                                                  float4 *__restrict__ htab,
                                                                  RelxRadial *__restrict__ srad,
                                                                  uint2 *__restrict__ list, int *__restrict__ cnt,
                                                                  int T) {
  const int set = blockIdx.y;
  const RelxSetState &s = sst[set];
  if (s.status != RELX_OK || s.cached) return;
  const int nr = tab.rel_nr, nm = tab.rel_nmu0, ng = tab.rel_ng;
  if (blockIdx.x == 0) {
    RelxRadial &R = srad[set];
    for (int i = threadIdx.x; i < RELX_NFRAD / kGroup + s.nz; i += kLineThreads) {
      // entry i belongs to the zone whose groups start at or before it
      int z = 0;
      while (z < s.nz - 1 && (s.zi1[z] < s.zi0[z] || line_group_base(s, z) > i)) z++;
      const int r0 = s.zi0[z] + (i - line_group_base(s, z)) * kGroup;
      int lo = 1 << 30, hi = -1;
      for (int r = r0; r < r0 + kGroup && r <= s.zi1[z]; r++) {
        const int a = R.rec[r].ielo;
        if (a >= 0) {
          lo = min(lo, a);
          hi = max(hi, R.rec[r].iehi);
        }
      }
      R.gr[i] = make_int2(lo, hi);
    }
    if (list && s.limb == 0 && threadIdx.x < 32) {
      for (int z0 = 0; z0 < s.nz; z0 += 32) {
        const int z = z0 + threadIdx.x;
        const int n = z < s.nz ? line_ntiles(s, z, T) : 0;
        int inc = n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int u = __shfl_up_sync(0xffffffffu, inc, o);
          if ((int) threadIdx.x >= o) inc += u;
        }
        int base = 0;
        if (threadIdx.x == 31) base = atomicAdd(&cnt[0], inc);
        base = __shfl_sync(0xffffffffu, base, 31) + inc - n;
        for (int k = 0; k < n; k++) list[base + k] = make_uint2((unsigned) set, (unsigned) z | (unsigned) k << 8);
      }
    }
  }
  const int q = blockIdx.x * kLineThreads + threadIdx.x;
  if (q >= nr * ng) return;
  const size_t b00 = (size_t) s.ind_a * nm + s.ind_mu0, b10 = (size_t) (s.ind_a + 1) * nm + s.ind_mu0;
  const size_t b01 = b00 + 1, b11 = b10 + 1;
  const float f1 = s.ifac_a, f2 = s.ifac_mu0;
  const float w00 = (1.0f - f1) * (1.0f - f2), w10 = f1 * (1.0f - f2), w01 = (1.0f - f1) * f2, w11 = f1 * f2;
  const float4 a = __ldg(&tab.rel_tc[b00 * nr * ng + q]), b = __ldg(&tab.rel_tc[b10 * nr * ng + q]);
  const float4 c = __ldg(&tab.rel_tc[b01 * nr * ng + q]), d = __ldg(&tab.rel_tc[b11 * nr * ng + q]);
  float2 *ht = reinterpret_cast<float2 *>(htab + (size_t) set * nr * ng);
  ht[q] = make_float2(w00 * a.x + w10 * b.x + w01 * c.x + w11 * d.x, w00 * a.y + w10 * b.y + w01 * c.y + w11 * d.y);
  ht[nr * ng + q] =
      make_float2(w00 * a.z + w10 * b.z + w01 * c.z + w11 * d.z, w00 * a.w + w10 * b.w + w01 * c.w + w11 * d.w);
}

// FP64 emission-angle cosine of one fine radius, table point g, branch k
// (interp_lin_2d_float then interp_lin_1d as Relprofile.cpp:67-77, 287-290)
__device__ double cosne_fp64(const RelxTables &tab, const RelxSetState &s, int itab, double ifac, int g, int k) {
  const int nr = tab.rel_nr, nm = tab.rel_nmu0, ng = tab.rel_ng;
  const size_t b00 = (size_t) s.ind_a * nm + s.ind_mu0, b10 = (size_t) (s.ind_a + 1) * nm + s.ind_mu0;
  const size_t b01 = b00 + 1, b11 = b10 + 1;
  double v[2];
  for (int q = 0; q < 2; q++) {
    int i = itab + 1 - q;  // q=0: lower radius (ind+1), q=1: upper (ind)
    float4 c00 = tab.rel_tc[(b00 * nr + i) * ng + g], c10 = tab.rel_tc[(b10 * nr + i) * ng + g];
    float4 c01 = tab.rel_tc[(b01 * nr + i) * ng + g], c11 = tab.rel_tc[(b11 * nr + i) * ng + g];
    double a = k ? c00.w : c00.z, b = k ? c10.w : c10.z, c = k ? c01.w : c01.z, d = k ? c11.w : c11.z;
    v[q] = lerp2((double) s.ifac_a, (double) s.ifac_mu0, a, b, c, d);
  }
  return lerp1(ifac, v[0], v[1]);
}

// the bin of a cosine so near a bin's edge that FP32 does not decide it (get_cosne_bin, Relprofile.cpp:799-801)
__device__ __noinline__ int cosne_bin_fp64(const RelxTables &tab, const RelxSetState &s, int itab, double ifac, int g, int k) {
  const double mud = cosne_fp64(tab, s, itab, ifac, g, k);
  return ((int) (tab.x_nincl * (1 - mud) + 1)) - 1;
}

// A zone's radii fall into kHistWarps classes: class w the radii 4 w to 4 w + 3 of every 32 from the zone's start.  A
// warp takes four radii at a time, 8 lanes per radius, each lane a block of at most GP consecutive table
// points (gper = (ng + 7) / 8 of them) with both branches.  Consecutive points mostly fall into the same
// angle bin: a lane adds runs and flushes a run on a change of bin into its private histogram.  At the end of
// a class the lanes are added by a shuffle tree, and the classes in order.
// A CTA of kHistWarps warps per zone, a class each (a warp per zone without barriers, eight classes one after
// the other: 771 us against 681 us for 4096 relxilllp sets).  Bound by issue and the latency of the loads.
// 4096 sets took 762 us, 1000 relxilllpCp sets 249 us and 64 relxill sets 72 us by a CTA per set with a loop over the
// points (addresses, integer conversions and a dependent load each, divergent flushes) and records staged in
// shared memory with two barriers per 128 radii; with the points unrolled, a radius's loads in flight together, the
// next radius's record fetched ahead and flushes without branches 681 us, 177 us and 35 us.
constexpr int kHistFull = 5;  // the 40 points of the relline tables, 5 for each of 8 lanes
constexpr int kHistFew = 3;   // tables of up to 24 points

template <int GP>
struct HistLane {
  int g0, np;  // the lane's points
  float gsf[GP], gfac[GP];
};

// class w of zone [i0, i1]; the lane's sums end in lh; FULL: every lane has GP points
template <int GP, bool FULL>
__device__ __forceinline__ void hist_class(const RelxTables &tab, const RelxSetState &s, const RelxRadial &R,
                                           const float2 *__restrict__ T, const HistLane<GP> &L, int i0, int i1, int w,
                                           float *lh) {
  const int lane = threadIdx.x & 31, grp = lane >> 3;
  const int nr = tab.rel_nr, ng = tab.rel_ng, n_incl = tab.x_nincl;
  const float c4pi2 = (float) (4.0 * kPi * kPi);
  const float fn = (float) n_incl;
  int r = i0 + w * 4 + grp;
  int4 q3 = make_int4(0, -1, -1, 0);  // ifac, ielo, iehi, itab
  float gmn = 0.0f, dg = 0.0f, ew = 0.0f, re = 0.0f;
  const auto fetch = [&](int k) {
    const RelxRadRec *rp = &R.rec[k];
    q3 = __ldg(reinterpret_cast<const int4 *>(rp) + 3);
    gmn = __ldg(&rp->gmin.x);
    dg = __ldg(&rp->dg.x);
    ew = __ldg(&rp->ew);
    re = __ldg(&R.re[k]);
  };
  if (r <= i1) fetch(r);
  for (; i0 + w * 4 <= i1 && __any_sync(0xffffffffu, r <= i1); r += kHistWarps * 4) {
    const bool on = r <= i1 && q3.y >= 0 && L.np > 0;  // radius inside the line-profile grid (Relprofile.cpp:863)
    const float fr = __int_as_float(q3.x), fl = 1.0f - fr;
    const int it = (short) (q3.w & 0xffff);
    const float c = re * re * re * c4pi2 * ew, dgr = dg, gmr = gmn;
    const float2 *hi = T + it * ng, *lo = hi + ng, *chi = hi + nr * ng, *clo = lo + nr * ng;
    // the cosines first, then the transfer functions: half the registers
    float2 wh[GP], wl[GP];
#pragma unroll
    for (int e = 0; e < GP; e++) {
      wh[e] = wl[e] = make_float2(0.0f, 0.0f);
      if (on && e < L.np) {
        wh[e] = __ldg(chi + e);
        wl[e] = __ldg(clo + e);
      }
    }
    if (r + kHistWarps * 4 <= i1) fetch(r + kHistWarps * 4);
    // trf(g*) and cosne(g*) at this radius: interp_lin_1d(ifac_r, T[ind+1], T[ind]) (Relprofile.cpp:280-293).  The
    // angle bin is floor(n_incl (1 - cosne)), from the nearest integer to that minus 1/2, by a magic sum whose
    // low bits hold the integer; FP32 decides it unless the fraction is within 1e-5 of an edge
    const float wl_ = -fn * fl, wh_ = -fn * fr;
    int b[GP][2];
    float edge = 0.0f;
#pragma unroll
    for (int e = 0; e < GP; e++) {
#pragma unroll
      for (int k = 0; k < 2; k++) {
        const float x = __fmaf_rn(wh_, k ? wh[e].y : wh[e].x, __fmaf_rn(wl_, k ? wl[e].y : wl[e].x, fn - 0.5f));
        const float q = __fadd_rn(x, kMagic);
        if (FULL || e < L.np) edge = fmaxf(edge, fabsf(__fadd_rn(x, -__fadd_rn(q, -kMagic))));
        b[e][k] = max(kMagicBits, min(__float_as_int(q), kMagicBits + n_incl - 1));
      }
    }
    if (on && edge > 0.5f - 1e-5f) {
#pragma unroll 1
      for (int q = 0; q < 2 * L.np; q++) {
        const int e_ = q >> 1;
        const float2 h = __ldg(chi + e_), l = __ldg(clo + e_);
        const float x = __fmaf_rn(wh_, q & 1 ? h.y : h.x, __fmaf_rn(wl_, q & 1 ? l.y : l.x, fn - 0.5f));
        if (!(fabsf(x - rintf(x)) > 0.5f - 1e-5f)) continue;
        const int v = kMagicBits + max(0, min(cosne_bin_fp64(tab, s, it, R.ifac[r], L.g0 + e_, q & 1), n_incl - 1));
#pragma unroll
        for (int e = 0; e < GP; e++) {
          if (2 * e == q) b[e][0] = v;
          if (2 * e + 1 == q) b[e][1] = v;
        }
      }
    }
    float2 vh[GP], vl[GP];
#pragma unroll
    for (int e = 0; e < GP; e++) {
      vh[e] = vl[e] = make_float2(0.0f, 0.0f);
      if (on && e < L.np) {
        vh[e] = __ldg(hi + e);
        vl[e] = __ldg(lo + e);
      }
    }
    // the runs; a lane that has none to flush adds to the row for nothing, which costs less than a branch.  (The
    // second branch's products are rounded before they are added: the sums are those of the kernel before
    // this one.)
    int cur[2] = {b[0][0], b[0][1]};
    float run[2] = {0.0f, 0.0f};
    const auto flush = [&](bool f0, bool f1) {
      float *a0 = lh + (f0 ? cur[0] - kMagicBits : RELX_MAX_INCL) * 32, *a1 = lh + (f1 ? cur[1] - kMagicBits : RELX_MAX_INCL) * 32;
      const float v0 = *a0 + run[0];
      float v1 = a1 == a0 ? v0 : *a1;
      v1 += run[1];
      *a0 = v0;
      *a1 = v1;
    };
#pragma unroll
    for (int e = 0; e < GP; e++) {
      const float ge_ = __fmaf_rn(L.gsf[e], dgr, gmr);
      const float cg = c * ge_ * ge_ * L.gfac[e];
      const float t0 = __fmaf_rn(fl, vl[e].x, __fmul_rn(fr, vh[e].x)), t1 = __fmaf_rn(fl, vl[e].y, __fmul_rn(fr, vh[e].y));
      if (e == 0) {
        run[0] = __fmul_rn(cg, t0);
        run[1] = __fmul_rn(cg, t1);
      } else {
        const bool in = on && e < L.np;
        const bool f0 = in && b[e][0] != cur[0], f1 = in && b[e][1] != cur[1];
        flush(f0, f1);
        if (!FULL && !in) continue;
        run[0] = __fmaf_rn(cg, t0, f0 ? 0.0f : run[0]);
        run[1] = __fadd_rn(f1 ? 0.0f : run[1], __fmul_rn(cg, t1));
      }
      cur[0] = b[e][0];
      cur[1] = b[e][1];
    }
    flush(on, on);
  }
}

// sums of the lanes' histograms, two bins at a time, one in each half of the warp: lane j returns bin j's
__device__ __forceinline__ float hist_lanes(float (*lh)[32], int n_incl) {
  const int lane = threadIdx.x & 31;
  float h = 0.0f;
  for (int j = 0; j < n_incl; j += 2) {
    const float v0 = lh[j][lane], v1 = lh[j + 1][lane];
    float v = lane < 16 ? v0 : v1;
    v += __shfl_xor_sync(0xffffffffu, lane < 16 ? v1 : v0, 16);
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const float u = __shfl_xor_sync(0xffffffffu, v, 16);
    if (lane == j) h = lane < 16 ? v : u;
    if (lane == j + 1) h = lane < 16 ? u : v;
  }
  return h;
}

template <int GP, bool FULL>
__global__ void __launch_bounds__(kHistWarps * 32, GP <= kHistFew ? 4 : GP <= kHistFull ? 3 : 2)
    hist_kernel(RelxTables tab, const RelxSetState *__restrict__ sst, const RelxRadial *__restrict__ srad, int nza,
                const float4 *__restrict__ htab, float *__restrict__ dist) {
  __shared__ float lhs[kHistWarps][RELX_MAX_INCL + 1][32];  // per-lane histograms, lane fastest (no bank conflicts), and a row for nothing
  __shared__ float hw[kHistWarps][RELX_MAX_INCL];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, z = blockIdx.x, set = blockIdx.y;
  const RelxSetState &s = sst[set];
  if (s.status != RELX_OK || s.model < RELX_RELXILL || s.cached || z >= s.nz) return;
  const int ng = tab.rel_ng, n_incl = tab.x_nincl;
  HistLane<GP> L;
  const int gper = FULL ? GP : (ng + 7) >> 3;
  L.g0 = (lane & 7) * gper;
  L.np = FULL ? GP : max(0, min(gper, ng - L.g0));
#pragma unroll
  for (int e = 0; e < GP; e++) {
    const float2 g = __ldg(&tab.rel_gs[min(L.g0 + e, ng - 1)]);
    L.gsf[e] = g.x;
    L.gfac[e] = g.y;
  }
  // the set's interpolated table: (trff1, trff2) plane, then (cosne1, cosne2)
  const float2 *__restrict__ T = reinterpret_cast<const float2 *>(htab + (size_t) set * tab.rel_nr * ng) + min(L.g0, ng - 1);
  float(*lh)[32] = lhs[warp];
  for (int j = 0; j <= RELX_MAX_INCL; j++) lh[j][lane] = 0.0f;
  hist_class<GP, FULL>(tab, s, srad[set], T, L, s.zi0[z], s.zi1[z], warp, &lh[0][lane]);
  const float h = hist_lanes(lh, n_incl);
  if (lane < n_incl) hw[warp][lane] = h;
  __syncthreads();
  if (tid < n_incl) {
    float v = 0.0f;
    for (int w = 0; w < kHistWarps; w++) v += hw[w][tid];
    dist[((size_t) set * nza + z) * RELX_MAX_INCL + tid] = v;
  }
}

constexpr int kSoloTile = kLineTileH;
template <bool LIMB>
static size_t line_team_smem(int ng, int nw) {
  return sizeof(float2) * RELX_MAX_NG + nw * LineWarp<LIMB, kSumBinsH, 1, 2, false>::bytes(line_tw_pitch(ng)) +
         sizeof(float2) * (kSumBinsH + 1);
}
static size_t line_solo_smem(int ng) {
  return sizeof(float2) * RELX_MAX_NG + kSoloWarps * LineWarp<false, kSoloTile, 2, 1, true>::bytes(line_tw_pitch(ng));
}

size_t line_list_entries(int n_sets, int nza, int nblk) {
  return (size_t) n_sets * nza * ((size_t) (nblk * kSumBinsH + kSumBinsH - 1) / kSoloTile + 1);
}

cudaError_t relline_set_smem(int nr, int ng) {
  cudaError_t e;
#define SET(kern, bytes)                                                                                \
  e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) (bytes));           \
  if (e != cudaSuccess) return e;
  SET(relline_solo_kernel<kSoloTile>, line_solo_smem(ng))
  SET((relline_team_kernel<false, kSumBinsH, 8>), line_team_smem<false>(ng, 8))
  SET((relline_team_kernel<true, kSumBinsH, 8>), line_team_smem<true>(ng, 8))
  SET((relline_team_kernel<false, kSumBinsH, 16>), line_team_smem<false>(ng, 16))
  SET((relline_team_kernel<true, kSumBinsH, 16>), line_team_smem<true>(ng, 16))
  SET((relline_team_kernel<false, kSumBinsH, 32>), line_team_smem<false>(ng, 32))
#undef SET
  return cudaSuccess;
}

// Which line kernel a range of sets without a limb law runs.  A warp of the solo kernel sums a whole
// zone (130 us for a tenth of the 1000 radii, 700 us for all of them), so it pays once its tasks fill
// the GPU several times; up to there the team kernel, which spends about half as much again per bin on
// narrower tiles and its ordered sums, is ahead.  Measured (line profile, us, solo / team): 10 zones
// 128 sets 290 / 190, 256 360 / 370, 512 440 / 620; 25 zones 32 sets 145 / 145, 128 200 / 250; one
// zone 1024 sets 1280 / 1040, 2048 1690 / 2000.  Between few table points the interpolant jumps so far that most bins
// need more than two Romberg levels, which a warp does one after the other: one zone, 20 points, 1600 sets
// 2670 / 1540, 4096 5020 / 3420 (12 points, 8192 sets 6890 / 6730); from 24 points on as above (4096 sets 2860 / 2950).
// A limb law always runs in the team kernel: there is no solo form with the law's twice as many table functions, which
// leave a warp 12 KB.  Line profile of relline with a law, us, now / by a CTA per 512 bins before: 153 sets 430 / 860, 1100
// 1570 / 1900, 4096 5350 / 5540 (64 points 5570 / 5650).
static bool line_solo(int n_sets, int nza, int ng) {
  return nza > 1 ? (int64_t) n_sets * nza >= 2560 : n_sets >= 1536 && ng >= 24;
}

// list: line_list_entries() entries for the solo kernel's tasks, cnt: its two counters (zero); both may be
// null (then the team kernel runs whatever the number of sets)
cudaError_t launch_line_table(int n_sets, int nza, cudaStream_t s, const RelxTables &tab, const RelxSetState *sst,
                              float4 *htab, RelxRadial *srad, uint2 *list, int *cnt) {
  const int nq = tab.rel_nr * tab.rel_ng;
  const bool solo = list && line_solo(n_sets, nza, tab.rel_ng);
  line_table_kernel<<<dim3((nq + kLineThreads - 1) / kLineThreads, n_sets), kLineThreads, 0, s>>>(
      tab, sst, htab, srad, solo ? list : nullptr, cnt, kSoloTile);
  return cudaGetLastError();
}

template <bool LIMB>
static void launch_team(int n_sets, int nblk, cudaStream_t s, const RelxTables &tab, const RelxSetIn *sin,
                        const RelxSetState *sst, const RelxRadial *srad, const double *line_e, int nza, float *prof,
                        double *tsum, const float4 *htab) {
  const int ng = tab.rel_ng;
  // warps per CTA: as many as the zone has groups of radii for (125, 13 with 10 zones) while the CTAs of
  // all tiles still find room, else 8 (four CTAs per SM).  One zone, us with 8 / 16 / 32 warps: 2 sets
  // 85 / 66 / 60, 32 158 / 129 / 116, 128 216 / 205 / 253, 512 570 / 640 / 870; 10 zones: 2 sets
  // 39 / 36 / 31, 8 54 / 47 / 54, 32 86 / 89 / 110.  (A limb law doubles the transfer functions: 16 at most.)
  const int nw = nza > 1 ? (n_sets * nza <= 160 ? 16 : 8) : LIMB ? (n_sets <= 64 ? 16 : 8)
                 : n_sets <= 32 ? 32 : n_sets <= 128 ? 16 : 8;
  const int gx = std::max(1, std::min(nblk + nza, 4 * kSMs * 32 / (nw * n_sets)));
  const dim3 grid(gx, n_sets);
#define TEAM(NW)                                                                                             \
  if (nw == NW)                                                                                              \
    relline_team_kernel<LIMB, kSumBinsH, NW><<<grid, NW * 32, line_team_smem<LIMB>(ng, NW), s>>>(             \
        tab, sin, sst, srad, line_e, htab, nza, prof, tsum, nblk, line_const(ng));
  TEAM(8) TEAM(16)
  if constexpr (!LIMB) { TEAM(32) }
#undef TEAM
}

// launches the line profile (both variants where a limb law may occur: a set runs in the one matching
// its law); htab, srad->gr, list and cnt: written by launch_line_table with the same n_sets, nza
cudaError_t launch_relline(int n_sets, int nblk, cudaStream_t s, const RelxTables &tab, const RelxSetIn *sin,
                           const RelxSetState *sst, const RelxRadial *srad, const double *line_e, int nza, float *prof,
                           double *tsum, bool any_limb, const float4 *htab, const uint2 *list, int *cnt) {
  if (list && line_solo(n_sets, nza, tab.rel_ng)) {
    const int64_t most = (int64_t) line_list_entries(n_sets, nza, nblk);
    const int grid = (int) std::min<int64_t>(kSMs * kSoloCtas, (most + kSoloWarps - 1) / kSoloWarps);
    relline_solo_kernel<kSoloTile><<<grid, kSoloWarps * 32, line_solo_smem(tab.rel_ng), s>>>(
        tab, sin, sst, srad, line_e, htab, nza, prof, tsum, nblk, list, cnt, line_const(tab.rel_ng));
  } else {
    launch_team<false>(n_sets, nblk, s, tab, sin, sst, srad, line_e, nza, prof, tsum, htab);
  }
  if (any_limb) launch_team<true>(n_sets, nblk, s, tab, sin, sst, srad, line_e, nza, prof, tsum, htab);
  return cudaGetLastError();
}

// The instance by the points of a lane: with fewer unrolled points than eight more CTAs fit an SM.  4096 relxilllp sets,
// histograms, us: tables of 20 points 2280 by the instance of eight points whose missing points all counted as near an
// edge, so 479 (a loop over the points before that 587); 33 points 2618, so 755 (774); 64 points 2339 at one CTA per SM,
// so 1500 at two (1467).
cudaError_t launch_hist(int n_sets, cudaStream_t s, const RelxTables &tab, const RelxSetState *sst,
                        const RelxRadial *srad, int nza, float *dist, const float4 *htab) {
  const dim3 grid(nza, n_sets);
  if (tab.rel_ng == 8 * kHistFull)
    hist_kernel<kHistFull, true><<<grid, kHistWarps * 32, 0, s>>>(tab, sst, srad, nza, htab, dist);
  else if (tab.rel_ng <= 8 * kHistFew)
    hist_kernel<kHistFew, false><<<grid, kHistWarps * 32, 0, s>>>(tab, sst, srad, nza, htab, dist);
  else if (tab.rel_ng < 8 * kHistFull)
    hist_kernel<kHistFull, false><<<grid, kHistWarps * 32, 0, s>>>(tab, sst, srad, nza, htab, dist);
  else
    hist_kernel<RELX_MAX_NG / 8, false><<<grid, kHistWarps * 32, 0, s>>>(tab, sst, srad, nza, htab, dist);
  return cudaGetLastError();
}

}  // namespace relx
