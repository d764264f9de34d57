// swe_math.cuh -- per-face and per-cell FP64 arithmetic of the shallow-water step.
//
// Every expression keeps the operand order of the reference (src/swe.mjs of
// Syntaxswine/water-simulator); the library is built with -fmad=false so no
// multiply-add is fused, which makes +, -, *, /, sqrt round exactly as the
// JavaScript engine's do.  Math.max / Math.min keep their JavaScript meaning
// (NaN in, NaN out; +0 above -0) so a blow-up propagates instead of being
// clipped away by IEEE maxNum.
#pragma once

#define SWE_G 9.80665                    // src/swe.mjs:85
#define SWE_SQRT2 1.4142135623730951     // Math.SQRT2

namespace swe {

__host__ __device__ __forceinline__ double jmax(double a, double b) {
  if (a != a) return a;
  if (b != b) return b;
  if (a > b) return a;
  if (b > a) return b;
  return signbit(a) ? b : a;
}
__host__ __device__ __forceinline__ double jmin(double a, double b) {
  if (a != a) return a;
  if (b != b) return b;
  if (a < b) return a;
  if (b < a) return b;
  return signbit(a) ? a : b;
}
// Math.max(0, x)
__host__ __device__ __forceinline__ double jmax0(double x) { return x > 0 ? x : (x == x ? 0.0 : x); }

// x / y correctly rounded (the operator's own PTX division), as an opaque
// operation: the compiler cannot see through it to rewrite its operands.
__device__ __forceinline__ double div_rn(double x, double y) {
  double q;
  asm("div.rn.f64 %0, %1, %2;" : "=d"(q) : "d"(x), "d"(y));
  return q;
}

// x / y, bit for bit, for a dividend that is often +-0 (the momentum of
// water at rest).  A zero dividend takes the division's slow path on B200
// (measured: 3.4x the time of a nonzero one).  +-0 / y with y finite and
// nonzero is the zero whose sign is the product of the signs, formed here
// from the bits; the division then gets the dividend 1 instead, so that lanes
// holding zeros stay on the fast path.  Every other case is the plain
// division.  The division is opaque because the compiler otherwise folds
// the substituted dividend back to x under the select.
// The tests are on the bit patterns (integer work, off the FP64 pipe).
__device__ __forceinline__ double qdiv(double x, double y) {
  const unsigned long long xb = __double_as_longlong(x), yb = __double_as_longlong(y);
  const bool z = (xb << 1) == 0 && (yb << 1) != 0 && ((yb >> 52) & 0x7ff) != 0x7ff;
  const double q = div_rn(z ? 1.0 : x, y);
  return z ? __longlong_as_double(xb ^ (yb & 0x8000000000000000ull)) : q;
}

// h^(4/3) of Manning friction (src/swe.mjs:683, 699: Math.pow(hk, 4 / 3)) as
// h * cbrt(h): within about 2 ulp of the power, as CUDA's pow is (the
// reference's Math.pow is not correctly rounded either, so friction is held
// to a tolerance rather than to the bits), at a fraction of pow's cost.
// Callers pass h > minDepth >= 0.
__device__ __forceinline__ double pow43(double h) { return h * cbrt(h); }

// Limiters, src/swe.mjs:88-141.  lim: 0 mc (default), 1 minmod, 2 central.
__device__ __forceinline__ double limiter(int lim, double a, double b) {
  if (lim == 0) {                                   // mc, src/swe.mjs:133-138
    const double p = a * b;
    if (p > 0) {
      // a, b are then non-NaN and nonzero of one sign, so c is too and the
      // three candidates are non-NaN and > +0: IEEE minNum is Math.min here.
      const double c = 0.5 * (a + b);
      const double m = fmin(fmin(fabs(c), 2 * fabs(a)), 2 * fabs(b));
      return a > 0 ? m : -m;
    }
    if (p <= 0) return 0;
    // a * b is NaN: Math.min's NaN rule decides
    const double c = 0.5 * (a + b);
    const double m = jmin(jmin(fabs(c), 2 * fabs(a)), 2 * fabs(b));
    return a > 0 ? m : -m;
  }
  if (lim == 1) {                                   // minmod, src/swe.mjs:88-92
    if (a > 0 && b > 0) return a < b ? a : b;
    if (a < 0 && b < 0) return a > b ? a : b;
    return 0;
  }
  return 0.5 * (a + b);                             // central, src/swe.mjs:141
}

// Desingularised velocity, src/swe.mjs:282-285.  The denominator depends on
// h only, so callers that need u and v of one cell share it (same double).
__device__ __forceinline__ double vel_den(double h, double eps4) {
  const double h4 = h * h * h * h;
  // h4 is +0, positive or NaN; for a NaN h4 the sum is NaN whichever maximum
  // is taken, so IEEE maxNum gives Math.max's result unless eps4 itself is
  // NaN (a NaN minDepth), where Math.max is NaN.
  return sqrt(h4 + (eps4 == eps4 ? fmax(h4, eps4) : eps4));
}
__device__ __forceinline__ double vel_num(double hq, double h) { return SWE_SQRT2 * h * hq; }
__device__ __forceinline__ double vel(double hq, double h, double eps4) {
  return qdiv(vel_num(hq, h), vel_den(h, eps4));
}

// HLLC with Einfeldt speeds and Toro's dry-state speeds, src/swe.mjs:975-1018.
// out = (mass, normal momentum, transverse momentum) flux.
__device__ __forceinline__ void hllc(double& o0, double& o1, double& o2,
                                     double hL, double huL, double hvL,
                                     double hR, double huR, double hvR, double dry) {
  const bool wetL = hL > dry, wetR = hR > dry;
  if (!wetL && !wetR) { o0 = 0; o1 = 0; o2 = 0; return; }
  const double uL = wetL ? qdiv(huL, hL) : 0, vL = wetL ? qdiv(hvL, hL) : 0;
  const double uR = wetR ? qdiv(huR, hR) : 0, vR = wetR ? qdiv(hvR, hR) : 0;
  const double cL = sqrt(SWE_G * jmax(hL, 0)), cR = sqrt(SWE_G * jmax(hR, 0));
  double sL, sR;
  if (!wetL) { sL = uR - 2 * cR; sR = uR + cR; }
  else if (!wetR) { sL = uL - cL; sR = uL + 2 * cL; }
  else {
    const double a = (cL + cR) / 2 + (uL - uR) / 4;
    const double hStar = a * a / SWE_G;
    const double qL = hStar > hL ? sqrt(0.5 * (hStar + hL) * hStar / (hL * hL)) : 1;
    const double qR = hStar > hR ? sqrt(0.5 * (hStar + hR) * hStar / (hR * hR)) : 1;
    sL = uL - cL * qL;
    sR = uR + cR * qR;
  }
  if (sL >= 0) {                                      // flux1D(left)
    o0 = huL; o1 = huL * uL + 0.5 * SWE_G * hL * hL; o2 = hvL * uL; return;
  }
  if (sR <= 0) {                                      // flux1D(right)
    o0 = huR; o1 = huR * uR + 0.5 * SWE_G * hR * hR; o2 = hvR * uR; return;
  }
  const double num = sL * hR * (uR - sR) - sR * hL * (uL - sL);
  const double den = hR * (uR - sR) - hL * (uL - sL);
  const double sM = fabs(den) > 1e-30 ? qdiv(num, den) : 0.5 * (sL + sR);
  const double FL0 = huL, FL1 = huL * uL + 0.5 * SWE_G * hL * hL;
  const double FR0 = huR, FR1 = huR * uR + 0.5 * SWE_G * hR * hR;
  const double inv = 1 / (sR - sL);
  o0 = (sR * FL0 - sL * FR0 + sL * sR * (hR - hL)) * inv;
  o1 = (sR * FL1 - sL * FR1 + sL * sR * (huR - huL)) * inv;
  o2 = o0 * (sM >= 0 ? vL : vR);
}

// One interface: MUSCL reconstruction from the two cells' slopes along the
// face normal, Audusse hydrostatic reconstruction against the higher bed,
// HLLC, and the two interface-local pressure corrections
// (src/swe.mjs:415-445 for x faces, :448-475 for y faces).  For a y face the
// caller passes (v, u) as (normal, transverse).
struct Face { double M, N, T, pL, pR; };

__device__ __forceinline__ Face face_flux(
    double bL_c, double hL_c, double nL_c, double tL_c,        // left cell b, h, normal vel, transverse vel
    double sEL, double sBL, double sNL, double sTL,            // left slopes along the normal
    double bR_c, double hR_c, double nR_c, double tR_c,
    double sER, double sBR, double sNR, double sTR, double dry) {
  const double etaL = bL_c + hL_c + 0.5 * sEL;
  const double etaR = bR_c + hR_c - 0.5 * sER;
  const double bL = bL_c + 0.5 * sBL;
  const double bR = bR_c - 0.5 * sBR;
  const double hLf = jmax0(etaL - bL);
  const double hRf = jmax0(etaR - bR);
  const double nL = nL_c + 0.5 * sNL;
  const double nR = nR_c - 0.5 * sNR;
  const double tL = tL_c + 0.5 * sTL;
  const double tR = tR_c - 0.5 * sTR;
  const double bStar = jmax(bL, bR);
  const double hsL = jmax0(etaL - bStar);
  const double hsR = jmax0(etaR - bStar);
  Face f;
  hllc(f.M, f.N, f.T, hsL, hsL * nL, hsL * tL, hsR, hsR * nR, hsR * tR, dry);
  f.pL = 0.5 * SWE_G * (hLf * hLf - hsL * hsL);
  f.pR = 0.5 * SWE_G * (hRf * hRf - hsR * hsR);
  return f;
}

// ---- the same arithmetic for operands in a known range --------------------------
// A division or square root compiled from the operator carries, besides its
// arithmetic, the handling of every exponent: tests, a branch and a call per
// operation, which also keeps the compiler from interleaving independent ones.
// Of the face kernel's 2270 instructions per cell on an all-wet grid, 33% were
// FP64.  The functions below are correctly rounded for operands whose
// exponents are known to be moderate ("tame", below), have no branch, and
// share what several quotients have in common; the face kernel takes them for
// tiles all of whose cells are tame and keeps the operators for the others.
//
// Reciprocal: Newton-Raphson with the fused multiply-add from the hardware's
// approximation (20 bits), and Markstein's theorem for the last step (P.
// Markstein, Computation of elementary functions on the IBM RISC System/6000
// processor, 1990): an approximation within an ulp of 1/b, corrected once by
// its exact residual, is 1/b correctly rounded unless every bit of b's
// significand is 1.  Callers test for those b (ones_lo) and use the operator.
// Quotient: by the same author's theorem, with y = 1/b correctly rounded, q
// within an ulp of a/b and r = a - b q exact, q + r y is a/b correctly rounded.
// Square root: Goldschmidt's iteration with a final residual step (P.
// Markstein, Software division and square root using Goldschmidt's algorithms,
// 2004).  Its result is within 2^-51 ulp of the root before the last rounding;
// the 24 significands whose root lies that near a rounding boundary are
// checked one by one by a test.
//
// The residual of an exact quotient is a sum of opposite equals; rounded down
// it is -0, which leaves the sign of a zero quotient as it is.
constexpr double INV_G = 1 / SWE_G;      // 0.015 ulp from 1/G: a * INV_G is within 0.52 ulp of a / G

__device__ __forceinline__ double rcp_seed(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  return y;
}
__device__ __forceinline__ double rsqrt_seed(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  return y;
}
// One correction of y towards 1/b.
__device__ __forceinline__ double rcp_refine(double b, double y) { return fma(y, fma(-b, y, 1.0), y); }
__device__ __forceinline__ double rcp_tame(double b) {
  return rcp_refine(b, rcp_refine(b, rcp_refine(b, rcp_seed(b))));
}
// Whether the low word of x is all ones, as it is when the significand is.
__device__ __forceinline__ bool ones_lo(double x) { return __double2loint(x) == -1; }
// a / b, y = 1/b correctly rounded.
__device__ __forceinline__ double div_tame(double a, double b, double y) {
  double q = a * y;                             // within 1.5 ulp
  q = fma(__fma_rd(-b, q, a), y, q);            // within 1
  return fma(__fma_rd(-b, q, a), y, q);
}
// p / h where p is n * h rounded: n itself is within an ulp of the quotient.
__device__ __forceinline__ double div_product(double p, double h, double n, double y) {
  return fma(__fma_rd(-h, n, p), y, n);
}
__device__ __forceinline__ double div_g(double a) {
  const double q = a * INV_G;
  return fma(__fma_rd(-SWE_G, q, a), INV_G, q);
}
// sqrt(x), and through half_r about 1 / (2 sqrt(x)).
__device__ __forceinline__ double sqrt_tame(double x, double& half_r) {
  const double y = rsqrt_seed(x);
  double g = x * y, h = 0.5 * y;
  double r = fma(-g, h, 0.5);
  g = fma(g, r, g); h = fma(h, r, h);
  r = fma(-g, h, 0.5);
  g = fma(g, r, g); h = fma(h, r, h);
  half_r = h;
  return fma(fma(-g, g, x), h, g);
}
__device__ __forceinline__ double sqrt_tame(double x) { double h; return sqrt_tame(x, h); }

// x is +-0 or 2^lo <= |x| < 2^hi (false for a NaN).
template <int LO, int HI>
__device__ __forceinline__ bool tame_value(double x) {
  const unsigned u = __double2hiint(x) & 0x7fffffff;
  return u - ((unsigned)(1023 + LO) << 20) < ((unsigned)(HI - LO) << 20) || x == 0;
}
// A cell whose face arithmetic stays clear of underflow and overflow in every
// product whose rounding error is formed: depths, momenta and bed in metres
// leave these ranges only in a field that has blown up, or below 1e-30 (h)
// and 1e-210 (momentum).  minDepth is at least 2^-60 then (StageArgs::tame),
// so wet depths are too.
__device__ __forceinline__ bool tame_cell(double b, double h, double hu, double hv) {
  return tame_value<-700, 60>(b) && tame_value<-100, 40>(h) && tame_value<-700, 100>(hu) &&
         tame_value<-700, 100>(hv);
}
// The velocities' denominator of a tame cell and its reciprocal; false when
// the operators must be used.
__device__ __forceinline__ bool vel_den_tame(double h, double eps4, double& den, double& y) {
  const double h4 = h * h * h * h;
  double hr;
  den = sqrt_tame(h4 + (h4 > eps4 ? h4 : eps4), hr);
  y = rcp_refine(den, rcp_refine(den, 2 * hr));
  return !ones_lo(den);
}
__device__ __forceinline__ bool vel_tame(double hu, double hv, double h, double eps4, double& u, double& v) {
  double den, y;
  const bool ok = vel_den_tame(h, eps4, den, y);
  u = div_tame(vel_num(hu, h), den, y);
  v = div_tame(vel_num(hv, h), den, y);
  return ok;
}

// The MC limiter of non-NaN arguments: of one sign, the least in magnitude of
// (a + b) / 2 and twice the smaller of a and b, which carries their sign.
__device__ __forceinline__ double limiter_mc_tame(double a, double b) {
  const double s = fabs(a) < fabs(b) ? a : b;
  const double c = 0.5 * (a + b), t = s + s;
  const double m = fabs(c) < fabs(t) ? c : t;
  return a * b > 0 ? m : 0;
}

// face_flux for tame cells, without a branch on the common path (a solve that
// branches per operation ran its warps' left and right sides one after the
// other).  0.5 x and 0.25 x are exact, so adding them by a fused multiply-add
// rounds as the two operations do.  A velocity is hn / h for the momentum hn
// just formed as h * n, so n is the quotient's first approximation.  Of
// the contact speed num / den only the sign is used.  redo: a divisor whose
// reciprocal is not covered; the caller then uses face_flux.
struct FaceSums { double M, T, NpL, NpR; };     // N + pL, N + pR
__device__ __forceinline__ double pos(double x) { return x > 0 ? x : 0; }
// The solve of two reconstructed states of which one is wet.  BOTH: both are, in
// every lane of the warp, and the selects of a dry side go (the face kernel of an
// all-wet 2048 x 2048 grid 239 -> 231 us).
template <bool BOTH>
__device__ __forceinline__ FaceSums solve_tame(double hL, double hR, double nL, double nR, double tL, double tR,
                                               double pL, double pR, bool wetL, bool wetR, bool& redo) {
  if (BOTH) wetL = wetR = true;
  const double huL = hL * nL, hvL = hL * tL, huR = hR * nR, hvR = hR * tR;
  const double DL = hL * hL, DR = hR * hR;
  FaceSums f;
  // a dry side's quotients are not used (its depth may be 0)
  const double yL = rcp_tame(hL), yR = rcp_tame(hR);
  const double uL = wetL ? div_product(huL, hL, nL, yL) : 0, vL = wetL ? div_product(hvL, hL, tL, yL) : 0;
  const double uR = wetR ? div_product(huR, hR, nR, yR) : 0, vR = wetR ? div_product(hvR, hR, tR, yR) : 0;
  const double cL = sqrt_tame(SWE_G * hL), cR = sqrt_tame(SWE_G * hR);
  const double a = fma(0.5, cL + cR, 0.25 * (uL - uR));
  const double hStar = div_g(a * a);
  const bool both = wetL && wetR, needL = both && hStar > hL, needR = both && hStar > hR;
  const double half = 0.5 * hStar;
  const double yDL = rcp_refine(DL, rcp_refine(DL, yL * yL)), yDR = rcp_refine(DR, rcp_refine(DR, yR * yR));
  const double qL = sqrt_tame(div_tame((hStar + hL) * half, DL, yDL));
  const double qR = sqrt_tame(div_tame((hStar + hR) * half, DR, yDR));
  const double sL = wetL ? uL - cL * (needL ? qL : 1.0) : fma(-2.0, cR, uR);
  const double sR = wetR ? uR + cR * (needR ? qR : 1.0) : fma(2.0, cL, uL);
  const double dL = uL - sL, dR = uR - sR;
  const double num = sL * hR * dR - sR * hL * dL;
  const double den = hR * dR - hL * dL;
  const bool left = fabs(den) > 1e-30 ? (num == 0 || (__double2hiint(num) ^ __double2hiint(den)) >= 0)
                                      : sL + sR >= 0;
  const double FL1 = huL * uL + 0.5 * SWE_G * hL * hL, FR1 = huR * uR + 0.5 * SWE_G * hR * hR;
  const double w = sR - sL, inv = rcp_tame(w), ss = sL * sR;
  f.M = (sR * huL - sL * huR + ss * (hR - hL)) * inv;
  double N = (sR * FL1 - sL * FR1 + ss * (huR - huL)) * inv;
  f.T = f.M * (left ? vL : vR);
  redo = (wetL && ones_lo(hL)) || (wetR && ones_lo(hR)) || (needL && ones_lo(DL)) || (needR && ones_lo(DR)) ||
         ones_lo(w);
  if (sL >= 0) { f.M = huL; N = FL1; f.T = hvL * uL; }
  else if (sR <= 0) { f.M = huR; N = FR1; f.T = hvR * uR; }
  f.NpL = N + pL;
  f.NpR = N + pR;
  return f;
}
// lanes: the lanes of the warp that make this call together, for the vote on BOTH.
__device__ __forceinline__ FaceSums face_flux_tame(
    double bL_c, double hL_c, double nL_c, double tL_c, double sEL, double sBL, double sNL, double sTL,
    double bR_c, double hR_c, double nR_c, double tR_c, double sER, double sBR, double sNR, double sTR, double dry,
    bool& redo, unsigned lanes = __activemask()) {
  const double etaL = fma(0.5, sEL, bL_c + hL_c), etaR = fma(-0.5, sER, bR_c + hR_c);
  const double bL = fma(0.5, sBL, bL_c), bR = fma(-0.5, sBR, bR_c);
  const double hLf = pos(etaL - bL), hRf = pos(etaR - bR);
  const double nL = fma(0.5, sNL, nL_c), nR = fma(-0.5, sNR, nR_c);
  const double tL = fma(0.5, sTL, tL_c), tR = fma(-0.5, sTR, tR_c);
  const double bStar = bL > bR ? bL : bR;
  const double hL = pos(etaL - bStar), hR = pos(etaR - bStar);
  const double pL = 0.5 * SWE_G * (hLf * hLf - hL * hL), pR = 0.5 * SWE_G * (hRf * hRf - hR * hR);
  const bool wetL = hL > dry, wetR = hR > dry;
  redo = false;
  if (__all_sync(lanes, wetL && wetR))
    return solve_tame<true>(hL, hR, nL, nR, tL, tR, pL, pR, true, true, redo);
  if (!wetL && !wetR) return {0, 0, 0 + pL, 0 + pR};
  return solve_tame<false>(hL, hR, nL, nR, tL, tR, pL, pR, wetL, wetR, redo);
}

}  // namespace swe
