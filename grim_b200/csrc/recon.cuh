// recon.cuh -- face reconstruction of one variable from its 5-point stencil
// (templated on the scalar so the op-counting build can run the same code)
// y0..y4 = v[i-2..i+2] along one direction.  Returns the value on the left
// face (i-1/2) and the right face (i+1/2) of zone i, as primLeft / primRight
// of the reference's reconstruct (reconstruction.cpp:3-36).
#pragma once
#include "common.cuh"

namespace grim {

// minmod.cpp:3-19; ArrayFire's sign() is 1 for x < 0 and 0 otherwise
template <class S>
GRIM_D S af_sgn(S x) { return (x < S(0.)) ? S(1.) : S(0.); }
template <class S>
GRIM_D S minmod3(S x, S y, S z) {
  S m = fmin(fmin(fabs(x), fabs(y)), fabs(z));
  S sx = 1. - 2. * af_sgn(x), sy = 1. - 2. * af_sgn(y), sz = 1. - 2. * af_sgn(z);
  return 0.25 * fabs(sx + sy) * (sx + sz) * m;
}
// minmod.cpp:21-71 with dX
template <class S>
GRIM_D S slope_mm(S y1, S y2, S y3, double dX, double theta) {
  S fwd = (y3 - y2) / dX;
  S bwd = (y2 - y1) / dX;
  S cen = bwd + fwd;
  return minmod3(theta * bwd, 0.5 * cen, theta * fwd);
}
// weno5.cpp:39-65 (the live code: centred 5-point derivative)
template <class S>
GRIM_D S slope_5pt(S y0, S y1, S y3, S y4, double dX) {
  return (-y4 + 8. * y3 - 8. * y1 + y0) / 12. / dX;
}
// ppm.cpp:41-75 / :120-159
template <class S>
GRIM_D void ppm_faces(S y0, S y1, S y2, S y3, S y4, S& leftV, S& rightV) {
  S d0 = 2. * (y1 - y0), d1 = 2. * (y2 - y1), d2 = 2. * (y3 - y2), d3 = 2. * (y4 - y3);
  S D1 = 0.5 * (y2 - y0), D2 = 0.5 * (y3 - y1), D3 = 0.5 * (y4 - y2);
  S DQ1 = (d1 * d0 <= 0.) ? 0. : ((D1 > 0.) ? 1. : -1.) * fmin(fabs(D1), fmin(fabs(d0), fabs(d1)));
  S DQ2 = (d2 * d1 <= 0.) ? 0. : ((D2 > 0.) ? 1. : -1.) * fmin(fabs(D2), fmin(fabs(d1), fabs(d2)));
  S DQ3 = (d3 * d2 <= 0.) ? 0. : ((D3 > 0.) ? 1. : -1.) * fmin(fabs(D3), fmin(fabs(d2), fabs(d3)));
  S l = 0.5 * (y2 + y1) - 1. / 6. * (DQ2 - DQ1);
  S r = 0.5 * (y3 + y2) - 1. / 6. * (DQ3 - DQ2);
  bool corr1 = ((r - y2) * (y2 - l) <= 0.);
  S qd = r - l;
  S qe = 6. * (y2 - 0.5 * (r + l));
  bool corr2 = (qd * (qd - qe) < 0.);
  bool corr3 = (qd * (qd + qe) < 0.);
  if (corr1) { l = y2; r = y2; }
  if (corr2) l = 3. * y2 - 2. * r;
  if (!corr2 && corr3) r = 3. * y2 - 2. * l;
  leftV = l;
  rightV = r;
}
template <class S>
GRIM_D S slope_ppm(S y0, S y1, S y2, S y3, S y4, double dX) {
  S l, r;
  ppm_faces(y0, y1, y2, y3, y4, l, r);
  return (r - l) / dX;
}
// WENO5 (weno5.cpp:111-257)
template <class S>
GRIM_D void weno5_faces(S y0, S y1, S y2, S y3, S y4, S& lo, S& ro) {
  const S eps2 = 1.0e-17;
  S beta1 = ((4.0 / 3.0) * y0 * y0 - (19.0 / 3.0) * y0 * y1 + (25.0 / 3.0) * y1 * y1 +
                  (11.0 / 3.0) * y0 * y2 - (31.0 / 3.0) * y1 * y2 + (10.0 / 3.0) * y2 * y2) +
                 eps2 * (1.0 + fabs(y0) + fabs(y1) + fabs(y2));
  S beta2 = ((4.0 / 3.0) * y1 * y1 - (13.0 / 3.0) * y1 * y2 + (13.0 / 3.0) * y2 * y2 +
                  (5.0 / 3.0) * y1 * y3 - (13.0 / 3.0) * y2 * y3 + (4.0 / 3.0) * y3 * y3) +
                 eps2 * (1.0 + fabs(y1) + fabs(y2) + fabs(y3));
  S beta3 = ((10.0 / 3.0) * y2 * y2 - (31.0 / 3.0) * y2 * y3 + (25.0 / 3.0) * y3 * y3 +
                  (11.0 / 3.0) * y2 * y4 - (19.0 / 3.0) * y3 * y4 + (4.0 / 3.0) * y4 * y4) +
                 eps2 * (1.0 + fabs(y2) + fabs(y3) + fabs(y4));
  S w1r = 1.0 / (16.0 * beta1 * beta1);
  S w2r = 5.0 / (8.0 * beta2 * beta2);
  S w3r = 5.0 / (16.0 * beta3 * beta3);
  S w1l = 5.0 / (16.0 * beta1 * beta1);
  S w2l = 5.0 / (8.0 * beta2 * beta2);
  S w3l = 1.0 / (16.0 * beta3 * beta3);
  S denl = w1l + w2l + w3l;
  S denr = w1r + w2r + w3r;
  S u1r = 0.375 * y0 - 1.25 * y1 + 1.875 * y2;
  S u2r = -0.125 * y1 + 0.75 * y2 + 0.375 * y3;
  S u3r = 0.375 * y2 + 0.75 * y3 - 0.125 * y4;
  S u1l = -0.125 * y0 + 0.75 * y1 + 0.375 * y2;
  S u2l = 0.375 * y1 + 0.75 * y2 - 0.125 * y3;
  S u3l = 1.875 * y2 - 1.25 * y3 + 0.375 * y4;
  lo = (w1l * u1l + w2l * u2l + w3l * u3l) / denl;
  ro = (w1r * u1r + w2r * u2r + w3r * u3r) / denr;
}
// MP5 (Suresh & Huynh 1997, alpha = 4): interface value at i+1/2 from the
// left-biased stencil.  No counterpart in the reference.
template <class S>
GRIM_D S mm2(S a, S b) {
  return 0.5 * (copysign(1., a) + copysign(1., b)) * fmin(fabs(a), fabs(b));
}
template <class S>
GRIM_D S mm4(S a, S b, S c, S d) {
  S s = 0.125 * (copysign(1., a) + copysign(1., b)) *
             fabs((copysign(1., a) + copysign(1., c)) * (copysign(1., a) + copysign(1., d)));
  return s * fmin(fmin(fabs(a), fabs(b)), fmin(fabs(c), fabs(d)));
}
template <class S>
GRIM_D S mp5(S vm2, S vm1, S v0, S vp1, S vp2) {
  const S alpha = 4.;
  S f = (2. * vm2 - 13. * vm1 + 47. * v0 + 27. * vp1 - 3. * vp2) / 60.;
  S vmp = v0 + mm2(vp1 - v0, alpha * (v0 - vm1));
  if ((f - v0) * (f - vmp) <= 0.) return f;
  S djm1 = vm2 - 2. * vm1 + v0;
  S dj = vm1 - 2. * v0 + vp1;
  S djp1 = v0 - 2. * vp1 + vp2;
  S dm4jph = mm4(4. * dj - djp1, 4. * djp1 - dj, dj, djp1);
  S dm4jmh = mm4(4. * dj - djm1, 4. * djm1 - dj, dj, djm1);
  S vul = v0 + alpha * (v0 - vm1);
  S vav = 0.5 * (v0 + vp1);
  S vmd = vav - 0.5 * dm4jph;
  S vlc = v0 + 0.5 * (v0 - vm1) + 4. / 3. * dm4jmh;
  S vmin = fmax(fmin(fmin(v0, vp1), vmd), fmin(fmin(v0, vul), vlc));
  S vmax = fmin(fmax(fmax(v0, vp1), vmd), fmax(fmax(v0, vul), vlc));
  return f + mm2(vmin - f, vmax - f);
}

// ---- the fast path's forms: the same schemes in fewer FP64 operations, as
// offsets from the zone's value built from the four first differences.  Equal
// to the forms above to a few ulp of the stencil's largest value (WENO5: to
// what the weights' rounding allows; the differences form its smoothness
// measures without the cancellation of the expanded squares).  FP64-pipe
// operations per variable (adds, products, compares): PPM 58 -> 33, WENO5
// about 130 -> 85, minmod 20 -> 10; the reconstruction was over half of a
// face kernel's work.
// The limiters below keep a NaN of their differences, where the plain forms
// drop it from a minimum and take it for positive, and so do with an infinity
// what the plain forms do or make it a NaN.  A zone where one shows is done again
// in the plain form: `top` keeps the largest exponent word among the variables'
// last products, kNonFinite and above says so.
constexpr int kNonFinite = 0x7ff00000;
GRIM_D void note_exponent(int& top, double x) { top = max(top, __double2hiint(x) & 0x7fffffff); }
template <class S>
GRIM_D void note_exponent(int&, S) {}
// the smaller of the two, x if x is a NaN (a compare and a select: fewer
// instructions than fmin, which drops it)
template <class S>
GRIM_D S min_keep(S x, S y) { return x >= y ? y : x; }
// +-1, a's sign, where the two finite numbers' signs agree, else 0 (a zero
// counts as either; the callers' result is zero then)
GRIM_D double common_sign(double a, double b) {
  const int ha = __double2hiint(a);
  return __hiloint2double((ha ^ __double2hiint(b)) >= 0 ? (ha & 0x80000000) | 0x3ff00000 : 0, 0);
}
template <class S>
GRIM_D S common_sign(S a, S b) { return (a < S(0.)) == (b < S(0.)) ? copysign(S(1.), a) : S(0.); }

// PPM: with the differences e = y[k+1] - y[k], a limited slope is twice
// h = sgn min(|e0 + e1| / 4, |e0|, |e1|) (zero at an extremum) and the zone's
// offsets to its faces are al = y2 - l, ar = r - y2.  The three corrections
// become: offsets of opposite sign vanish, neither exceeds twice the other.
template <class S>
GRIM_D S ppm_half_slope(S a, S b) {
  return common_sign(a, b) * min_keep(S(0.25) * fabs(a + b), min_keep(fabs(a), fabs(b)));
}
template <class S>
GRIM_D void ppm_offsets(S y0, S y1, S y2, S y3, S y4, S& al, S& ar, int& top) {
  const S e0 = y1 - y0, e1 = y2 - y1, e2 = y3 - y2, e3 = y4 - y3;
  const S h1 = ppm_half_slope(e0, e1), h2 = ppm_half_slope(e1, e2), h3 = ppm_half_slope(e2, e3);
  const S l = S(0.5) * e1 + S(1. / 3.) * (h2 - h1);
  const S r = S(0.5) * e2 - S(1. / 3.) * (h3 - h2);
  const S l2 = l + l, r2 = r + r;
  const S lr = l * r;
  note_exponent(top, lr);
  const bool flat = lr <= S(0.);
  al = (fabs(l) > fabs(r2)) ? r2 : l;
  ar = (fabs(r) > fabs(l2)) ? l2 : r;
  if (flat) al = ar = S(0.);
}
template <class S>
GRIM_D void ppm_faces_fast(S y0, S y1, S y2, S y3, S y4, S& leftV, S& rightV, int& top) {
  S al, ar;
  ppm_offsets(y0, y1, y2, y3, y4, al, ar, top);
  leftV = y2 - al;
  rightV = y2 + ar;
}

// WENO5: the smoothness measures in differences (4 p^2 - 11 p q + 10 q^2
// towards the edge, 4 p^2 - 5 p q + 4 q^2 centred; the factor 1/3 scales the
// small terms instead), one division per face value (the weights over their
// common denominator beta1^2 beta2^2 beta3^2), candidates as offsets from y2.
template <class S>
GRIM_D void weno5_faces_fast(S y0, S y1, S y2, S y3, S y4, S& lo, S& ro) {
  const S eps = 3.0e-17;
  const S e0 = y1 - y0, e1 = y2 - y1, e2 = y3 - y2, e3 = y4 - y3;
  const S a1 = fabs(y1), a3 = fabs(y3), m = S(1.) + fabs(y2);
  const S beta1 = e0 * (S(4.) * e0 - S(11.) * e1) + S(10.) * (e1 * e1) + eps * (m + (fabs(y0) + a1));
  const S beta2 = e1 * (S(4.) * e1 - S(5.) * e2) + S(4.) * (e2 * e2) + eps * (m + (a1 + a3));
  const S beta3 = e3 * (S(4.) * e3 - S(11.) * e2) + S(10.) * (e2 * e2) + eps * (m + (a3 + fabs(y4)));
  const S b1 = beta1 * beta1, b2 = beta2 * beta2, b3 = beta3 * beta3;
  // w1 ~ 1/b1 -> b2 b3, w2 ~ 1/b2 -> b1 b3, w3 ~ 1/b3 -> b1 b2 (x 1, 10, 5 / 5, 10, 1)
  const S p23 = b2 * b3, p13 = S(10.) * (b1 * b3), p12 = b1 * b2;
  const S q23 = S(5.) * p23, q12 = S(5.) * p12;
  // right: u1 = y2 + 0.875 e1 - 0.375 e0, u2 = y2 + 0.125 e1 + 0.375 e2, u3 = y2 + 0.625 e2 - 0.125 e3
  // left:  u1 = y2 - 0.625 e1 + 0.125 e0, u2 = y2 - 0.375 e1 - 0.125 e2, u3 = y2 - 0.875 e2 + 0.375 e3
  const S r1 = S(0.875) * e1 - S(0.375) * e0, r2 = S(0.125) * e1 + S(0.375) * e2, r3 = S(0.625) * e2 - S(0.125) * e3;
  const S l1 = S(0.125) * e0 - S(0.625) * e1, l2 = -(S(0.375) * e1 + S(0.125) * e2), l3 = S(0.375) * e3 - S(0.875) * e2;
  ro = y2 + (p23 * r1 + p13 * r2 + q12 * r3) / (p23 + p13 + q12);
  lo = y2 + (q23 * l1 + p13 * l2 + p12 * l3) / (q23 + p13 + p12);
}

// minmod: the limited slope is the smallest of the three where all signs agree
template <class S>
GRIM_D S slope_mm_fast(S bwd, S fwd, double theta, int& top) {
  const S slope = common_sign(bwd, fwd) *
                  min_keep(S(0.5) * fabs(bwd + fwd), S(theta) * min_keep(fabs(bwd), fabs(fwd)));
  note_exponent(top, slope);
  return slope;
}

// face values of zone i
template <class S>
GRIM_D void recon_faces(int scheme, double theta, S y0, S y1, S y2, S y3, S y4,
                        S& lo, S& ro) {
  switch (scheme) {
    case GRIM_WENO5: weno5_faces(y0, y1, y2, y3, y4, lo, ro); return;
    case GRIM_PPM: ppm_faces(y0, y1, y2, y3, y4, lo, ro); return;
    case GRIM_MP5:
      ro = mp5(y0, y1, y2, y3, y4);
      lo = mp5(y4, y3, y2, y1, y0);
      return;
    default: {
      // minmod.cpp:73-95 (dX = 1)
      S s = slope_mm(y1, y2, y3, 1., theta);
      lo = y2 - 0.5 * s;
      ro = y2 + 0.5 * s;
      return;
    }
  }
}
template <class S>
GRIM_D void recon_faces_fast(int scheme, double theta, S y0, S y1, S y2, S y3, S y4,
                             S& lo, S& ro, int& top) {
  if (scheme == GRIM_WENO5) {
    weno5_faces_fast(y0, y1, y2, y3, y4, lo, ro);
  } else if (scheme == GRIM_PPM) {
    ppm_faces_fast(y0, y1, y2, y3, y4, lo, ro, top);
  } else if (scheme == GRIM_MINMOD) {
    const S s = slope_mm_fast(y2 - y1, y3 - y2, theta, top);
    lo = y2 - S(0.5) * s;
    ro = y2 + S(0.5) * s;
  } else {
    recon_faces(scheme, theta, y0, y1, y2, y3, y4, lo, ro);
  }
}

// face values of DOF variables, get(v, m) their stencils' points, with the
// scheme fixed at compile time (RS >= 0: one scheme's code in the kernel) or
// read at run time (RS < 0); FAST selects the fast path's forms.  The second
// pass, hardly ever taken, is a loop of one variable's code with loads of its
// own: unrolled, or on the values of the first pass, its code and registers
// slowed every face (PPM vortex 301x187 127 -> 148 us).
template <int DOF, int RS, bool FAST, class Get>
GRIM_D void recon_vars(int scheme, double theta, const Get& get, double* lo, double* ro) {
  const int rs = RS < 0 ? scheme : RS;  // a constant scheme folds the choice
  [[maybe_unused]] int top = 0;
#pragma unroll
  for (int v = 0; v < DOF; v++) {
    const double y0 = get(v, 0), y1 = get(v, 1), y2 = get(v, 2), y3 = get(v, 3), y4 = get(v, 4);
    if constexpr (FAST)
      recon_faces_fast(rs, theta, y0, y1, y2, y3, y4, lo[v], ro[v], top);
    else
      recon_faces(rs, theta, y0, y1, y2, y3, y4, lo[v], ro[v]);
  }
  if constexpr (FAST) {
    if (__builtin_expect((rs == GRIM_PPM || rs == GRIM_MINMOD) && top >= kNonFinite, 0)) {
#pragma unroll 1
      for (int v = 0; v < DOF; v++) {
        double l, r;
        recon_faces(rs, theta, get(v, 0), get(v, 1), get(v, 2), get(v, 3), get(v, 4), l, r);
#pragma unroll
        for (int u = 0; u < DOF; u++)
          if (u == v) { lo[u] = l; ro[u] = r; }
      }
    }
  }
}

// the slope() used by the EMHD gradients (reconstruction.cpp:39-64); MP5
// uses the centred 5-point derivative
template <class S>
GRIM_D S recon_slope(int scheme, double theta, S y0, S y1, S y2, S y3,
                          S y4, double dX) {
  switch (scheme) {
    case GRIM_WENO5: return slope_5pt(y0, y1, y3, y4, dX);
    case GRIM_PPM: return slope_ppm(y0, y1, y2, y3, y4, dX);
    case GRIM_MP5: return slope_5pt(y0, y1, y3, y4, dX);
    default: return slope_mm(y1, y2, y3, dX, theta);
  }
}
// the same in the fast path's forms, idX = 1 / dX; top as for the faces
template <class S>
GRIM_D S recon_slope_fast(int scheme, double theta, S y0, S y1, S y2, S y3, S y4, double idX, int& top) {
  if (scheme == GRIM_PPM) {
    S al, ar;
    ppm_offsets(y0, y1, y2, y3, y4, al, ar, top);
    return (al + ar) * idX;
  }
  if (scheme == GRIM_MINMOD) return slope_mm_fast((y2 - y1) * idX, (y3 - y2) * idX, theta, top);
  return (S(8.) * (y3 - y1) - (y4 - y0)) * (S(1. / 12.) * idX);
}

}  // namespace grim
