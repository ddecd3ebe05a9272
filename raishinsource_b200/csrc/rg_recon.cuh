// rg_recon.cuh -- face reconstruction of rec.f90 (MP5, WENO5, PPM) as device
// functions templated on the arithmetic type T (see rg_device.cuh).
#pragma once

namespace rg {

// rec.f90:2346-2370.  dmm = 0.5*(sign(1,x)+sign(1,y))*min(|x|,|y|) and
// dm4 = 0.125*(sw+sx)*|sw+sy|*(sw+sz)*min(|w|,|x|,|y|,|z|) (s = sign(1,.);
// note the reference's abs covers only the middle factor, so dm4 is +min
// when all four signs agree, whatever that sign).  The sign factors are
// +-1 or a signed zero, so the products are evaluated here as selects on the
// sign bits: the same values bit for bit (signed zeros and NaN included) with
// the FP64 arithmetic reduced to the min and one multiply.
template <typename T>
__device__ __forceinline__ T dmm(T xx, T yy) {
  const T mn = dmin2(mabs(xx), mabs(yy));
  // same signs: 0.5*(+-2)*mn = +-mn; otherwise 0.5*(+0)*mn = +0 (or NaN)
  return (signbit(xx) == signbit(yy)) ? copysign(mn, xx) : T(0) * mn;
}
template <typename T>
__device__ __forceinline__ T dm4(T ww, T xx, T yy, T zz) {
  T mn = mabs(ww);
  if (mabs(xx) < mn) mn = mabs(xx);
  if (mabs(yy) < mn) mn = mabs(yy);
  if (mabs(zz) < mn) mn = mabs(zz);
  const bool nw = signbit(ww);
  const bool az = nw != signbit(xx), bz = nw != signbit(yy), cz = nw != signbit(zz);
  if (!az && !bz && !cz) return mn;  // 0.125 * (2 sw) * 2 * (2 sw) = +1
  // a zero factor: the product ((0.125*A)*B)*C*mn is a zero with the sign of
  // A times the sign of C, where A = sw+sx and C = sw+sz are +0 when their
  // signs differ and 2 sw otherwise (B = |sw+sy| >= 0 keeps the sign)
  const bool neg = (!az && nw) != (!cz && nw);
  return (neg ? T(-0.0) : T(0)) * mn;
}

// rec.f90:2095-2178: MP5 face state of cell 0 from u(-2..+2) given in the
// order (a2, a1, u0, b1, b2): the left state at +1/2 takes
// (u-2, u-1, u0, u+1, u+2) and sg = +1; the right state at -1/2 takes the
// mirrored stencil (u+2, u+1, u0, u-1, u-2) and sg = -1, because the
// reference's right state flips the signs of the dm4 terms of md and lc
// (rec.f90:2172-2176).  Negation is exact, so both equal the reference's
// separate formulas bit for bit, and the two lanes of a face run one code path.
// The second differences are the exception: the reference evaluates them once
// per cell in stencil order, (u-2 - 2 u-1) + u0, (u-1 - 2 u0) + u+1 and
// (u0 - 2 u+1) + u+2, for both states, and a sum taken in the mirrored order
// can round differently; the right state therefore picks its operands so
// that each difference is summed as the reference sums it.
//
// mp_monotone: the test that lets the unlimited value ul1 stand
// (rec.f90:2092); mp_limit_to: the limited value otherwise.
template <typename T>
__device__ __forceinline__ bool mp_monotone(T ul1, T a1, T u0, T b1) {
  const T alpha = T(4.0), eps1 = T(1.0e-10);
  const T ulmp = u0 + dmm(b1 - u0, alpha * (u0 - a1));
  const T t = (ul1 - u0) * (ul1 - ulmp);
  return t <= eps1;
}
template <typename T>
__device__ __forceinline__ T mp_limit_to(T ul1, T a2, T a1, T u0, T b1, T b2, T sg) {
  const T tmp2 = T(4.0) / T(3.0), alpha = T(4.0);
  const bool right = sg < T(0);
  // left: dim1 = (a2 - 2 a1) + u0, di1 = (a1 - 2 u0) + b1, dip1 = (u0 - 2 b1) + b2;
  // right (a = u+, b = u-): dim1 = (u0 - 2 a1) + a2, di1 = (b1 - 2 u0) + a1, dip1 = (b2 - 2 b1) + u0
  const T dim1 = (right ? u0 : a2) - T(2.) * a1 + (right ? a2 : u0);
  const T di1 = (right ? b1 : a1) - T(2.) * u0 + (right ? a1 : b1);
  const T dip1 = (right ? b2 : u0) - T(2.) * b1 + (right ? u0 : b2);
  const T dm4p = dm4(T(4.) * di1 - dip1, T(4.) * dip1 - di1, di1, dip1);
  const T dm4m = dm4(T(4.) * di1 - dim1, T(4.) * dim1 - di1, di1, dim1);
  const T ul = u0 + alpha * (u0 - a1);
  const T av = T(0.5) * (u0 + b1);
  const T md = av - (sg * T(0.5)) * dm4p;
  const T lc = u0 + T(0.5) * (u0 - a1) + (sg * tmp2) * dm4m;
  const T m1 = fmin3(u0, b1, md), m2 = fmin3(u0, ul, lc);
  const T m3 = fmax3(u0, b1, md), m4 = fmax3(u0, ul, lc);
  const T umax = dmax2(m1, m2), umin = dmin2(m3, m4);
  return ul1 + dmm(umin - ul1, umax - ul1);
}
template <typename T>
__device__ __forceinline__ T mp_limit(T ul1, T a2, T a1, T u0, T b1, T b2, T sg) {
  return mp_monotone(ul1, a1, u0, b1) ? ul1 : mp_limit_to(ul1, a2, a1, u0, b1, b2, sg);
}
// The unlimited value.  Its roundings are spelled out (in the uncontracted
// build they are the reference's), so that every pass and kernel that forms it
// gets the same bits whatever it goes on to do with it.
template <typename T>
__device__ __forceinline__ T mp5_value(T a2, T a1, T u0, T b1, T b2) {
  const T tmp1 = T(1.0) / T(60.0);
#ifdef RG_EXACT_ARITH
  return tmp1 * (T(2.) * a2 - T(13.) * a1 + T(47.) * u0 + T(27.) * b1 - T(3.) * b2);
#else
  return mul_rn(tmp1, fma(T(-3.), b2, fma(T(27.), b1, fma(T(47.), u0, fma(T(2.), a2, -mul_rn(T(13.), a1))))));
#endif
}

// The convex combination of the three candidates with the weights n_m / d_m
// as the reference forms it: six quotients.
template <typename T>
__device__ __forceinline__ T weno_quot(T n0, T d0, T n1, T d1, T n2, T d2, T q0, T q1, T q2) {
  const T w0 = n0 / d0, w1 = n1 / d1, w2 = n2 / d2;
  const T wt = w0 + w1 + w2;
  const T o0 = w0 / wt, o1 = w1 / wt, o2 = w2 / wt;
  return o0 * q0 + o1 * q1 + o2 * q2;
}
// Out of line, for FP64 states that hardly ever take it.
__device__ __noinline__ double weno_quot_rare(double n0, double d0, double n1, double d1, double n2, double d2,
                                              double q0, double q1, double q2) {
  return weno_quot(n0, d0, n1, d1, n2, d2, q0, q1, q2);
}
// The same in FP64 with weights already multiplied by their common denominator,
// which leaves one reciprocal.  Where the products leave the range in which
// they and the reciprocal are exact to rounding (fields beyond about 1e37,
// non-finite values), `quot` forms the quotients instead.  FP32 states always
// form them: the products of six small weights keep too little of FP32's range.
template <typename F>
__device__ __forceinline__ double weno_mean(double w0, double w1, double w2, double q0, double q1, double q2,
                                            const F& quot) {
  const double wt = w0 + w1 + w2;
  if (!(wt < 0x1p500 && wt > 0x1p-500)) return quot();
  return (w0 * q0 + w1 * q1 + w2 * q2) * rcp_newton(wt);
}
#ifdef RG_EXACT_ARITH
template <typename T>
constexpr bool kWenoMean = false;
#else
template <typename T>
constexpr bool kWenoMean = sizeof(T) == 8;
#endif

// rec.f90:2373-2643 (WENO5-JS); the left state at +1/2 takes
// (u-2, u-1, u0, u+1, u+2), the right state at -1/2 the mirrored stencil.
// (13./12.) is a single-precision literal in the reference.
// b1s is the value the smoothness indicator beta_1 reads in place of b1: b1
// itself, except in mpweno5's radial right state (rec.f90:2757, see face_lane).
template <typename T>
__device__ __forceinline__ T weno5_js(T a2, T a1, T u0, T b1, T b2, T b1s) {
  const T cd0 = T(1.0 / 10.0), cd1 = T(6.0 / 10.0), cd2 = T(3.0 / 10.0);
  const T c00 = T(2.0 / 6.0), c01 = T(-7.0 / 6.0), c02 = T(11.0 / 6.0);
  const T c10 = T(-1.0 / 6.0), c11 = T(5.0 / 6.0), c12 = T(2.0 / 6.0);
  const T c20 = T(2.0 / 6.0), c21 = T(5.0 / 6.0), c22 = T(-1.0 / 6.0);
  const T epsi = T(1.0e-6), c1312 = T((double)(13.0f / 12.0f)), c14 = T(0.25);
  const T s0 = a2 - T(2.) * a1 + u0, t0 = a2 - T(4.) * a1 + T(3.) * u0;
  const T s1 = a1 - T(2.) * u0 + b1s, t1 = a1 - b1;
  const T s2 = u0 - T(2.) * b1 + b2, t2 = T(3.) * u0 - T(4.) * b1 + b2;
  const T be0 = c1312 * (s0 * s0) + c14 * (t0 * t0) + epsi;
  const T be1 = c1312 * (s1 * s1) + c14 * (t1 * t1) + epsi;
  const T be2 = c1312 * (s2 * s2) + c14 * (t2 * t2) + epsi;
  const T q0 = c00 * a2 + c01 * a1 + c02 * u0;
  const T q1 = c10 * a1 + c11 * u0 + c12 * b1;
  const T q2 = c20 * u0 + c21 * b1 + c22 * b2;
  if constexpr (kWenoMean<T>) {
    // the weights cd_m / beta_m^2 times (beta_0 beta_1 beta_2)^2
    const T p0 = be1 * be2, p1 = be0 * be2, p2 = be0 * be1;
    return weno_mean(cd0 * (p0 * p0), cd1 * (p1 * p1), cd2 * (p2 * p2), q0, q1, q2, [&] {
      return weno_quot_rare(cd0, be0 * be0, cd1, be1 * be1, cd2, be2 * be2, q0, q1, q2);
    });
  } else {
    return weno_quot(cd0, be0 * be0, cd1, be1 * be1, cd2, be2 * be2, q0, q1, q2);
  }
}
template <typename T>
__device__ __forceinline__ T weno5_state(T a2, T a1, T u0, T b1, T b2) {
  return weno5_js(a2, a1, u0, b1, b2, b1);
}

// rec.f90:3161-3436 (WENO-Z, Borges et al. 2008): WENO5 with the weights
// cd_m (1 + tau / (beta_m + eps)), tau = |beta_0 - beta_2|, the smoothness
// indicators without eps; p0 = 1 makes (beta + eps)**p0 the plain sum.
template <typename T>
__device__ __forceinline__ T weno5z_state(T a2, T a1, T u0, T b1, T b2) {
  const T cd0 = T(1.0 / 10.0), cd1 = T(6.0 / 10.0), cd2 = T(3.0 / 10.0);
  const T c00 = T(2.0 / 6.0), c01 = T(-7.0 / 6.0), c02 = T(11.0 / 6.0);
  const T c10 = T(-1.0 / 6.0), c11 = T(5.0 / 6.0), c12 = T(2.0 / 6.0);
  const T c20 = T(2.0 / 6.0), c21 = T(5.0 / 6.0), c22 = T(-1.0 / 6.0);
  const T epsi = T(1.0e-6), c1312 = T((double)(13.0f / 12.0f)), c14 = T(0.25);
  const T s0 = a2 - T(2.) * a1 + u0, t0 = a2 - T(4.) * a1 + T(3.) * u0;
  const T s1 = a1 - T(2.) * u0 + b1, t1 = a1 - b1;
  const T s2 = u0 - T(2.) * b1 + b2, t2 = T(3.) * u0 - T(4.) * b1 + b2;
  const T be0 = c1312 * (s0 * s0) + c14 * (t0 * t0);
  const T be1 = c1312 * (s1 * s1) + c14 * (t1 * t1);
  const T be2 = c1312 * (s2 * s2) + c14 * (t2 * t2);
  const T tau = mabs(be0 - be2);
  const T q0 = c00 * a2 + c01 * a1 + c02 * u0;
  const T q1 = c10 * a1 + c11 * u0 + c12 * b1;
  const T q2 = c20 * u0 + c21 * b1 + c22 * b2;
  auto quot = [&] {
    const T w0 = cd0 * (T(1.0) + tau / (be0 + epsi));
    const T w1 = cd1 * (T(1.0) + tau / (be1 + epsi));
    const T w2 = cd2 * (T(1.0) + tau / (be2 + epsi));
    const T wt = w0 + w1 + w2;
    const T o0 = w0 / wt, o1 = w1 / wt, o2 = w2 / wt;
    return o0 * q0 + o1 * q1 + o2 * q2;
  };
  if constexpr (kWenoMean<T>) {
    // the weights times the product of the beta_m + eps
    const T e0 = be0 + epsi, e1 = be1 + epsi, e2 = be2 + epsi;
    return weno_mean(cd0 * (e0 + tau) * (e1 * e2), cd1 * (e1 + tau) * (e0 * e2), cd2 * (e2 + tau) * (e0 * e1), q0, q1,
                     q2, quot);
  } else {
    return quot();
  }
}

// rec.f90:3439-3793 (mapped WENO5, Henrick et al. 2005): the JS weights
// cd_m / (beta_m + eps)^2 with eps = 1e-40, normalised, mapped by
// g_m(w) = w (cd_m + cd_m^2 - 3 cd_m w + w^2) / (cd_m^2 + w (1 - 2 cd_m)) and
// normalised again.
template <typename T>
__device__ __forceinline__ T weno5m_state(T a2, T a1, T u0, T b1, T b2) {
  const T cd[3] = {T(1.0 / 10.0), T(6.0 / 10.0), T(3.0 / 10.0)};
  const T c00 = T(2.0 / 6.0), c01 = T(-7.0 / 6.0), c02 = T(11.0 / 6.0);
  const T c10 = T(-1.0 / 6.0), c11 = T(5.0 / 6.0), c12 = T(2.0 / 6.0);
  const T c20 = T(2.0 / 6.0), c21 = T(5.0 / 6.0), c22 = T(-1.0 / 6.0);
  const T epsi = T(1.0e-40), c1312 = T((double)(13.0f / 12.0f)), c14 = T(0.25);
  const T s0 = a2 - T(2.) * a1 + u0, t0 = a2 - T(4.) * a1 + T(3.) * u0;
  const T s1 = a1 - T(2.) * u0 + b1, t1 = a1 - b1;
  const T s2 = u0 - T(2.) * b1 + b2, t2 = T(3.) * u0 - T(4.) * b1 + b2;
  const T be[3] = {c1312 * (s0 * s0) + c14 * (t0 * t0), c1312 * (s1 * s1) + c14 * (t1 * t1),
                   c1312 * (s2 * s2) + c14 * (t2 * t2)};
  const T q0 = c00 * a2 + c01 * a1 + c02 * u0;
  const T q1 = c10 * a1 + c11 * u0 + c12 * b1;
  const T q2 = c20 * u0 + c21 * b1 + c22 * b2;
  auto quot = [&] {
    T wa[3], g[3];
#pragma unroll
    for (int m = 0; m < 3; ++m) wa[m] = cd[m] / ((be[m] + epsi) * (be[m] + epsi));
    const T wat = wa[0] + wa[1] + wa[2];
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      const T w = wa[m] / wat;
      g[m] = w * (cd[m] + cd[m] * cd[m] - T(3.) * cd[m] * w + w * w) / (cd[m] * cd[m] + w * (T(1.) - T(2.) * cd[m]));
    }
    const T gt = g[0] + g[1] + g[2];
    const T o0 = g[0] / gt, o1 = g[1] / gt, o2 = g[2] / gt;
    return o0 * q0 + o1 * q1 + o2 * q2;
  };
  if constexpr (kWenoMean<T>) {
    // the weights times (beta_0 + eps)^2 (beta_1 + eps)^2 (beta_2 + eps)^2, the
    // beta_m + eps (at least 1e-40) scaled by 2^60 to keep the products from
    // underflowing; the mapped weights over their common denominator
    const T sc = T(0x1p60);
    const T e0 = sc * (be[0] + epsi), e1 = sc * (be[1] + epsi), e2 = sc * (be[2] + epsi);
    const T p0 = e1 * e2, p1 = e0 * e2, p2 = e0 * e1;
    const T w[3] = {cd[0] * (p0 * p0), cd[1] * (p1 * p1), cd[2] * (p2 * p2)};
    const T wt = w[0] + w[1] + w[2];
    if (!(wt < T(0x1p500) && wt > T(0x1p-500))) return quot();
    const T iw = rcp_newton(wt);
    T num[3], den[3];
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      const T o = w[m] * iw;
      num[m] = o * (cd[m] + cd[m] * cd[m] - T(3.) * cd[m] * o + o * o);
      den[m] = cd[m] * cd[m] + o * (T(1.) - T(2.) * cd[m]);
    }
    return weno_mean(num[0] * (den[1] * den[2]), num[1] * (den[0] * den[2]), num[2] * (den[0] * den[1]), q0, q1, q2,
                     quot);
  } else {
    return quot();
  }
}

// The second-order limiters of rec.f90 on nonuniform coordinates: mclim
// (irec 1, rec.f90:208-367), minlim (2, 568-739), lim03a (11, 4037-4267),
// mvllim (12, 4269-4477) and koren (13, 4480-4697).  One cell's state on the
// side `side` (0: left state at its +1/2 face, 1: right state at its -1/2
// face) from its neighbours um, up and the per-index coefficients co[6] of
// its coordinate (small = 1e-12, a = x_p - x_c + small, b = x_c - x_m + small,
// c = xa_p - x_c + small, d = x_c - xa_m + small):
//   irec 1, 2, 11: (1/a, 1/b, -, -, xa_p - x_c, x_c - xa_m)
//   irec 13:       (1/a, 1/b, a (1/c), b (1/d), xa_p - x_c, x_c - xa_m)
//   irec 12:       (a, b, a/c, b/d, c, d)
// MAX/MIN follow Fortran's order (the first argument seeds the result).
// tmp_b is the sign used in koren's backward slope: the reference takes the
// i-direction sign there in its j sweep (rec.f90:4628), else the cell's own.
template <int IREC, typename T>
__device__ __forceinline__ T limiter_state(T um, T u0, T up, const T co[6], int side, T tmp_b) {
  const T s3 = T(1.0 / 3.0);
  if (IREC == 12) {
    const T sp = (up - u0) / co[0], sm = (u0 - um) / co[1];
    T dk = T(0);
    if (!(sp * sm <= T(0))) {
      const T t = sm * sm + (co[2] + co[3] - T(2)) * sm * sp + sp * sp;
      dk = (sm * sp * (co[2] * sm + co[3] * sp)) / (t + T(1.0e-12));
    }
    return side ? u0 - dk * co[5] : u0 + dk * co[4];
  }
  const T sp = (up - u0) * co[0], sm = (u0 - um) * co[1];
  const T tmp = (sp < T(0)) ? T(-1) : T(1);
  T dk;
  if (IREC == 1) {
    dk = tmp * dmax2(T(0), fmin3(T(2) * mabs(sp), tmp * T(2) * sm, tmp * T(0.5) * (sp + sm)));
  } else if (IREC == 2) {
    dk = tmp * dmax2(T(0), dmin2(mabs(sp), tmp * sm));
  } else if (IREC == 11) {
    const T al = T(0.5), be = T(2), ga = T(1.6);
    if (side) {
      const T e = (T(2) * mabs(sp) + tmp * sm) * s3;
      dk = dmax2(T(0), dmin2(e, dmax2(-al * sm * tmp, fmin3(be * sm * tmp, e, ga * mabs(sp)))));
    } else {
      const T e = (mabs(sp) + tmp * T(2) * sm) * s3;
      dk = dmax2(T(0), dmin2(e, dmax2(-al * mabs(sp), fmin3(be * mabs(sp), e, ga * tmp * sm))));
    }
  } else {  // 13
    const T e = side ? (mabs(sp) + T(2) * tmp_b * sm) * s3 : (T(2) * mabs(sp) + tmp * sm) * s3;
    dk = tmp * dmax2(T(0), fmin3(mabs(co[2] * sp), tmp * co[3] * sm, e));
  }
  return side ? u0 - dk * co[5] : u0 + dk * co[4];
}

// rec.f90:742-1258 (ceno, irec 4, convex ENO): one cell's state on side
// `side` from u(-2..+2) along the direction and the per-index coefficients
// co[10] of its physical coordinate x (rg_capi.cu, ceno_coefs): the minmod
// state u1, three quadratic candidates (centred at the cell before, at and
// after it), their deviations from u1 weighted by (1, 0.7, 1), and the
// candidate of smallest deviation when all three deviate the same way.
// kquirk drops the third candidate from the negative branch, as the
// reference's theta sweep compares |dklp| with itself there (rec.f90:1211).
template <typename T>
__device__ __forceinline__ T ceno_state(T um2, T um, T u0, T up, T up2, const T co[10], int side, bool kquirk) {
  const T sp = (up - u0) / co[0], sm = (u0 - um) / co[1];
  T dk = T(0);
  if (!(sp * sm <= T(0))) {
    const T tmp = (sp < T(0)) ? T(-1) : T(1);
    dk = tmp * dmin2(mabs(sp), mabs(sm));
  }
  const T u1 = side ? u0 - dk * co[3] : u0 + dk * co[2];
  const T d2m = T(0.5) * (u0 - um2), d20 = T(0.5) * (up - um), d2p = T(0.5) * (up2 - u0);
  const T d3m = u0 - T(2.0) * um + um2, d30 = up - T(2.0) * u0 + um, d3p = up2 - T(2.0) * up + u0;
  const T tm = side ? co[7] : co[4], t0 = side ? co[8] : co[5], tp = side ? co[9] : co[6];
  const T cm = u0 + d2m * tm + T(0.5) * d3m * (tm * tm);
  const T c0 = u0 + d20 * t0 + T(0.5) * d30 * (t0 * t0);
  const T cp = u0 + d2p * tp + T(0.5) * d3p * (tp * tp);
  const T dm = T(1.0) * (cm - u1), d0 = T(0.7) * (c0 - u1), dp = T(1.0) * (cp - u1);
  T out = u1;
  if (dp > T(0) && d0 > T(0) && dm > T(0)) {
    out = cm;
    if (mabs(d0) < mabs(dm) && mabs(d0) < mabs(dp)) out = c0;
    if (mabs(dp) < mabs(dm) && mabs(dp) < mabs(d0)) out = cp;
  }
  if (dm < T(0) && d0 < T(0) && dp < T(0)) {
    out = cm;
    if (mabs(d0) < mabs(dm) && mabs(d0) < mabs(dp)) out = c0;
    if (!kquirk && mabs(dp) < mabs(dm) && mabs(dp) < mabs(d0)) out = cp;
  }
  return out;
}

// rec.f90:145-205 (muscl, irec 3, beta = 1/3, no limiter): the left state of
// a cell at its +1/2 face (side 0) and its right state at its -1/2 face
// (side 1; the reference stores it as uriir of the face's left cell).
template <typename T>
__device__ __forceinline__ T muscl_state(T um, T u0, T up, int side) {
  const T beta = T(1.0 / 3.0);
  if (side) return u0 - T(0.25) * ((T(1.0) + beta) * (u0 - um) + (T(1.0) - beta) * (up - u0));
  return u0 + T(0.25) * ((T(1.0) + beta) * (up - u0) + (T(1.0) - beta) * (u0 - um));
}

// ------------------------------------------------------------------- PPM
// rPPM of Marti & Muller (1996) as restated by rec.f90:1261-2058.  The four
// passes (interp, detect, flaten, monoto) touch only the two face states of
// one cell each, so both states of cell c follow from the cells c-3..c+3:
// L = state at c-1/2 (the reference's uriir(c-1)), R = state at c+1/2
// (uriil(c)).  dx is rec2's shifted dx?b (dummy dx?b(m) = actual dx?b(m-1),
// rec.f90:58), x the cell centres (contact detection).

// The coefficients of the spacings are the run's (PpmCoef planes of
// DevRun::ppm, rg_capi.cu): each is the reference's expression in its order,
// evaluated once per index instead of once per cell, variable and face (about
// 40 divisions a cell and variable), so the values are the same.  FP32 faces
// have planes of their own, evaluated in FP32 from the rounded spacings.
// Planes at 0-based index m-1, with dx(m) the shifted spacing:
enum PpmCoef {
  PC_A = 0,  // dx(m) / (dx(m-1) + dx(m) + dx(m+1))
  PC_B,      // (2 dx(m-1) + dx(m)) / (dx(m+1) + dx(m))
  PC_C,      // (dx(m) + 2 dx(m+1)) / (dx(m-1) + dx(m))
  PC_T2,     // interface m+1/2: dx(m) / (dx(m) + dx(m+1))
  PC_T3, PC_T4, PC_T5,
  PC_D,      // contact: 1 / (dx(m-1) + dx(m) + dx(m+1))
  PC_S, PC_RS,   // dx(m) + dx(m+1) and its reciprocal
  PC_X,      // x(m+1) - x(m-1)
  PC_X3,     // (x(m) - x(m-1))^3 + (x(m+1) - x(m))^3
  kPpmCoef
};
static_assert(kPpmCoef == kPpmPlanes, "one plane of the tables per coefficient");

// interp Eq. (60)-(61) (rec.f90:1346-1418); the theta direction lacks the
// factor 2 of r and phi (rec.f90:1414).
template <typename T>
__device__ __forceinline__ T ppm_dma(T um, T u0, T up, T ca, T cb, T cc, bool kdir) {
  const T sp1 = up - u0, sm1 = u0 - um;
  const T spm1 = sp1 * sm1;
  const T da = ca * (cb * sp1 + cc * sm1);
  if (spm1 <= T(0)) return T(0);
  const T t1 = (da < T(0)) ? T(-1) : T(1);
  const T t1d = dmin2(mabs(sm1), mabs(sp1));
  return kdir ? t1 * dmin2(mabs(da), t1d) : t1 * dmin2(mabs(da), T(2.0) * t1d);
}

// interp Eq. (51) (rec.f90:1422-1468): interface value at c+1/2.
template <typename T>
__device__ __forceinline__ T ppm_face(T u0, T u1, T dma0, T dma1, T t2c, T t3c, T t4, T t5) {
  const T d = u1 - u0;
  const T t2 = t2c * d;
  const T t3 = t3c * d;
  return u0 + t2 + t3 - t4 * dma1 + t5 * dma0;
}

// a / b for a spacing b > 0 with its correctly rounded reciprocal rb
__device__ __forceinline__ double ppm_over(double a, double b, double rb) {
#ifdef RG_EXACT_ARITH
  return a / b;
#else
  return div_by_rcp(a, b, rb);
#endif
}
__device__ __forceinline__ float ppm_over(float a, float b, float) { return a / b; }

// The contact steepening factor (detect, rec.f90:1479-1686) and the shock
// flattening factor f2a (flaten, rec.f90:1689-1884) of the cell `o` cells above
// the view's cell: U(v, o) the primitives, C(plane, o) the coefficients.
// Quotients whose value cannot matter are not formed: the contact's pressure
// test only where eta is not zero already (eta is never NaN), and a
// flattening ratio only where its weight omg1 is one or the ratio could
// overflow (0 * inf).
template <int D, typename T, typename FU, typename FC>
__device__ __forceinline__ void ppm_factors(const FU& U, const FC& C, int o, T gam, T& eta, T& f2a) {
  const T pp = U(4, o + 1), pm = U(4, o - 1);
  {
    const T eta1 = T(5.0), eta2 = T(0.05), eps1 = T(0.1), ak0 = T(1.0);
    auto dda = [&](int c) {
      const T t0b = ppm_over(U(0, c + 1) - U(0, c), C(PC_S, c), C(PC_RS, c));
      const T t0c = ppm_over(U(0, c) - U(0, c - 1), C(PC_S, c - 1), C(PC_RS, c - 1));
      return C(PC_D, c) * (t0b - t0c);
    };
    const T ddp = dda(o + 1), ddm = dda(o - 1);
    const T rp = U(0, o + 1), rm = U(0, o - 1);
    const T t1 = ddp * ddm;
    const T t2 = mabs(rp - rm) - eps1 * dmin2(mabs(rp), mabs(rm));
    T etatil;
    if (t1 >= T(0) && t2 <= T(0)) {
      etatil = T(0);
    } else {
      const T t2a = -(ddp - ddm) / C(PC_X, o);
      const T t2b = C(PC_X3, o) / (rp - rm);
      etatil = t2a * t2b;
    }
    eta = dmax2(T(0), dmin2(eta1 * (etatil - eta2), T(1)));
    if (eta > T(0)) {
      const T t3 = mabs(rp - rm) / dmin2(rp, rm);
      const T t4 = mabs(pp - pm) / dmin2(pp, pm);
      if (gam * ak0 * t3 < t4) eta = T(0);
    }
  }
  {
    const T eps2 = T(1.0), omg2 = T(0.52), omg3 = T(10.0);
    const T tiny = sizeof(T) == 8 ? T(0x1p-1000) : T(0x1p-120f);
    auto f1a = [&](int c) {
      const T pp1 = U(4, c + 1), pm1 = U(4, c - 1);
      const T t3a = mabs(pp1 - pm1);
      const T t1 = eps2 * dmin2(pp1, pm1) - t3a;
      const T t2 = U(D, c + 1) - U(D, c - 1);
      const T omg1 = (t1 < T(0) && t2 < T(0)) ? T(1) : T(0);
      const T t3b = U(4, c + 2) - U(4, c - 2);
      if (omg1 == T(0) && !(mabs(t3b) < t3a * tiny)) return T(0);
      T t4;
      if (t3b == T(0)) t4 = (t3a == T(0)) ? -omg2 : T(1.0) - omg2;
      else t4 = (t3a / t3b) - omg2;
      return dmin2(T(1), omg1 * dmax2(T(0), t4 * omg3));
    };
    const T f1b = (pp - pm < T(0)) ? f1a(o + 1) : f1a(o - 1);
    f2a = dmax2(f1a(o), f1b);
  }
}

// r (1 - w) + x w, its roundings spelled out: it sums two products, and a face
// gets the same bits whichever kernel forms it.
template <typename T>
__device__ __forceinline__ T ppm_blend(T r, T x, T w) {
  return mad(x, w, mul_rn(r, T(1.0) - w));
}

// flaten's blend and monoto (rec.f90:1887-2056) of one cell's states.
template <typename T>
__device__ __forceinline__ void ppm_monoto(T u0, T f2a, T& l, T& r) {
  r = ppm_blend(r, u0, f2a);
  l = ppm_blend(l, u0, f2a);
  if ((r - u0) * (l - u0) >= T(0)) { r = u0; l = u0; }
  const T t3 = T(6.0) * (r - l) * (u0 - T(0.5) * (r + l));
  const T t4 = (r - l) * (r - l);
  if (t3 > t4) l = T(3.0) * u0 - T(2.0) * r;
  if (-t3 > t4) r = T(3.0) * u0 - T(2.0) * l;
}

// State of the cell at p (primitive v at p[v*N], storage type S), stride st
// along direction D, at its upper (side 0) or lower (side 1) face; pc: the
// coefficient planes at the cell's index, n apart.  gam enters the contact
// test (rec.f90:1623).  ALL: also the sixth variable (the per-routine rec2
// outputs every face state).
template <int D, typename T, typename S, bool ALL>
__device__ __forceinline__ void ppm_cell(const S* __restrict__ p, size_t N, long long st, const T* __restrict__ pc,
                                         int n, T gam, int side, T q[9]) {
  auto U = [&](int v, int o) { return T(p[(size_t)v * N + o * st]); };
  auto C = [&](int a, int o) { return __ldg(pc + a * n + o); };
  T eta, f2a;
  ppm_factors<D, T>(U, C, 0, gam, eta, f2a);
#pragma unroll 1
  for (int v = 0; v < 9; ++v) {
    T o = T(0);
    if (v != 5 || ALL) {  // var 6 faces are never read downstream
      const T um2 = U(v, -2), um1 = U(v, -1), u0 = U(v, 0), up1 = U(v, 1), up2 = U(v, 2);
      const T dm = ppm_dma(um2, um1, u0, C(PC_A, -1), C(PC_B, -1), C(PC_C, -1), D == 3);
      const T d0 = ppm_dma(um1, u0, up1, C(PC_A, 0), C(PC_B, 0), C(PC_C, 0), D == 3);
      const T dp = ppm_dma(u0, up1, up2, C(PC_A, 1), C(PC_B, 1), C(PC_C, 1), D == 3);
      T l = ppm_face(um1, u0, dm, d0, C(PC_T2, -1), C(PC_T3, -1), C(PC_T4, -1), C(PC_T5, -1));
      T r = ppm_face(u0, up1, d0, dp, C(PC_T2, 0), C(PC_T3, 0), C(PC_T4, 0), C(PC_T5, 0));
      if (v == 0) {
        r = ppm_blend(r, up1 - T(0.5) * dp, eta);
        l = ppm_blend(l, um1 + T(0.5) * dm, eta);
      }
      ppm_monoto(u0, f2a, l, r);
      o = side ? l : r;
    }
#pragma unroll
    for (int w = 0; w < 9; ++w)
      if (w == v) q[w] = o;
  }
}

// Both states of one face by one thread: the upper state of the cell at p (L)
// and the lower state of the next (R), which share two of their slopes and
// the interface value between them.  PACK: p holds the eight variables other
// than the sixth one after another.  put(v, L, R) receives each variable's
// states; ROLL keeps the loop over the variables rolled (the 24 coefficients
// then leave room in the registers; put must take a run-time v).
template <int D, typename T, typename S, bool PACK, bool ROLL, typename Put>
__device__ __forceinline__ void ppm_face_pair(const S* __restrict__ p, size_t N, long long st,
                                              const T* __restrict__ pc, int n, T gam, const Put& put) {
  auto U = [&](int v, int o) { return T(p[(size_t)(PACK && v > 5 ? v - 1 : v) * N + o * st]); };
  auto C = [&](int a, int o) { return __ldg(pc + a * n + o); };
  T etaL, fL, etaR, fR;
  ppm_factors<D, T>(U, C, 0, gam, etaL, fL);
  ppm_factors<D, T>(U, C, 1, gam, etaR, fR);
  T ca[4], cb[4], cc[4], t2[3], t3[3], t4[3], t5[3];
#pragma unroll
  for (int o = 0; o < 4; ++o) { ca[o] = C(PC_A, o - 1); cb[o] = C(PC_B, o - 1); cc[o] = C(PC_C, o - 1); }
#pragma unroll
  for (int o = 0; o < 3; ++o) { t2[o] = C(PC_T2, o - 1); t3[o] = C(PC_T3, o - 1); t4[o] = C(PC_T4, o - 1); t5[o] = C(PC_T5, o - 1); }
  auto one = [&](int v) {
    T u[6], d[4], f[3];
#pragma unroll
    for (int o = 0; o < 6; ++o) u[o] = U(v, o - 2);
#pragma unroll
    for (int o = 0; o < 4; ++o) d[o] = ppm_dma(u[o], u[o + 1], u[o + 2], ca[o], cb[o], cc[o], D == 3);
#pragma unroll
    for (int o = 0; o < 3; ++o) f[o] = ppm_face(u[o + 1], u[o + 2], d[o], d[o + 1], t2[o], t3[o], t4[o], t5[o]);
    T l0 = f[0], r0 = f[1], l1 = f[1], r1 = f[2];
    if (v == 0) {
      r0 = ppm_blend(r0, u[3] - T(0.5) * d[2], etaL);
      l0 = ppm_blend(l0, u[1] + T(0.5) * d[0], etaL);
      r1 = ppm_blend(r1, u[4] - T(0.5) * d[3], etaR);
      l1 = ppm_blend(l1, u[2] + T(0.5) * d[1], etaR);
    }
    ppm_monoto(u[2], fL, l0, r0);
    ppm_monoto(u[3], fR, l1, r1);
    put(v, r0, l1);
  };
  if constexpr (ROLL) {
#pragma unroll 1
    for (int v = 0; v < 9; ++v)
      if (v != 5) one(v);  // var 6 faces are never read downstream
  } else {
#pragma unroll
    for (int v = 0; v < 9; ++v)
      if (v != 5) one(v);
  }
}

}  // namespace rg
