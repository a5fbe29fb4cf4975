// Derivatives of the hair BSDF (f * cos and the lobe-mixture pdf) with
// respect to the material: sigma_a (3), beta_m, beta_n, alpha (radians).
//
// Forward-mode differentiation with dual numbers: every quantity carries its
// value and its partials, and each operation applies the chain rule.  Which
// partials a quantity has is part of its type (a bit mask): the attenuations
// depend on one absorption each, M_p on beta_m and alpha, N_p on beta_n, and
// only their products on several, so the terms that are zero by structure are
// neither computed nor held (with all six partials everywhere the kernel took
// 180 registers and 5,750 instructions per warp, 302 us for 1,000,003
// queries against 145 now).  Every partial is
// the same sum of products as with all six.  The formulas and statement order
// are those of hair_eval
// (disney_hair.cuh:186-266) and setupHairShading (:26-41), with the
// material-only terms (v[k], s, sin/cos 2^k alpha, the trimmed-logistic
// normaliser) differentiated too, since they depend on the parameters.
// The branches (log-space M_p for v <= 0.1, LogI0 for x > 12, the wrap of
// delta phi, |cos theta'|) follow the value, as in the primal.  The M_p
// branch runs in FP32 here for every beta_m (the primal's FP64 branch for
// beta_m < 0.1 only changes rounding).
#pragma once
#include "hm_hair_bsdf.cuh"

namespace hm {

constexpr int kNd = 6;  // sigma_a r, g, b, beta_m, beta_n, alpha
constexpr unsigned kBm = 8u, kBn = 16u, kAl = 32u;  // masks: bits 0 to 2 are sigma_a

template <unsigned M>
struct DualT {  // partials outside M are not set
  float v;
  float d[kNd];
};
using Dual = DualT<63u>;

// Loops over the partials with compile-time bounds; the body is kept where
// the mask has the bit.
#define HM_FOR_D(i, mask)            \
  _Pragma("unroll") for (int i = 0; i < kNd; ++i) if (((mask) >> i) & 1u)

template <unsigned M>
HM_D DualT<M> dvar(float x) {  // M: one bit
  DualT<M> r;
  r.v = x;
  HM_FOR_D(i, M) r.d[i] = 1.f;
  return r;
}
// r = value with partials scaled by g (the derivative of a unary function)
template <unsigned M>
HM_D DualT<M> dmap(const DualT<M>& a, float value, float g) {
  DualT<M> r;
  r.v = value;
  HM_FOR_D(i, M) r.d[i] = g * a.d[i];
  return r;
}
template <unsigned A, unsigned B>
HM_D DualT<(A | B)> operator+(const DualT<A>& a, const DualT<B>& b) {
  DualT<(A | B)> r;
  r.v = a.v + b.v;
  HM_FOR_D(i, A | B) {
    if (((A & B) >> i) & 1u)
      r.d[i] = a.d[i] + b.d[i];
    else
      r.d[i] = (A >> i) & 1u ? a.d[i] : b.d[i];
  }
  return r;
}
template <unsigned A, unsigned B>
HM_D DualT<(A | B)> operator-(const DualT<A>& a, const DualT<B>& b) {
  DualT<(A | B)> r;
  r.v = a.v - b.v;
  HM_FOR_D(i, A | B) {
    if (((A & B) >> i) & 1u)
      r.d[i] = a.d[i] - b.d[i];
    else
      r.d[i] = (A >> i) & 1u ? a.d[i] : -b.d[i];
  }
  return r;
}
template <unsigned M>
HM_D DualT<M> operator-(const DualT<M>& a) { return dmap(a, -a.v, -1.f); }
template <unsigned A, unsigned B>
HM_D DualT<(A | B)> operator*(const DualT<A>& a, const DualT<B>& b) {
  DualT<(A | B)> r;
  r.v = a.v * b.v;
  HM_FOR_D(i, A | B) {
    if (((A & B) >> i) & 1u)
      r.d[i] = a.d[i] * b.v + a.v * b.d[i];
    else
      r.d[i] = (A >> i) & 1u ? a.d[i] * b.v : a.v * b.d[i];
  }
  return r;
}
template <unsigned A, unsigned B>
HM_D DualT<(A | B)> operator/(const DualT<A>& a, const DualT<B>& b) {
  DualT<(A | B)> r;
  r.v = a.v / b.v;
  const float ib = 1.f / b.v;
  HM_FOR_D(i, A | B) {
    if (((A & B) >> i) & 1u)
      r.d[i] = (a.d[i] - r.v * b.d[i]) * ib;
    else
      r.d[i] = ((A >> i) & 1u ? a.d[i] : -(r.v * b.d[i])) * ib;
  }
  return r;
}
template <unsigned M> HM_D DualT<M> operator+(const DualT<M>& a, float b) { DualT<M> r = a; r.v += b; return r; }
template <unsigned M> HM_D DualT<M> operator+(float a, const DualT<M>& b) { return b + a; }
template <unsigned M> HM_D DualT<M> operator-(const DualT<M>& a, float b) { DualT<M> r = a; r.v -= b; return r; }
template <unsigned M> HM_D DualT<M> operator-(float a, const DualT<M>& b) { return dmap(b, a - b.v, -1.f); }
template <unsigned M> HM_D DualT<M> operator*(const DualT<M>& a, float b) { return dmap(a, a.v * b, b); }
template <unsigned M> HM_D DualT<M> operator*(float a, const DualT<M>& b) { return dmap(b, a * b.v, a); }
template <unsigned M> HM_D DualT<M> operator/(const DualT<M>& a, float b) { return dmap(a, a.v / b, 1.f / b); }
template <unsigned M> HM_D DualT<M> operator/(float a, const DualT<M>& b) { return dmap(b, a / b.v, -a / (b.v * b.v)); }

template <unsigned M> HM_D DualT<M> dsqr(const DualT<M>& a) { return a * a; }
template <unsigned M> HM_D DualT<M> dexp(const DualT<M>& a) { const float e = expf(a.v); return dmap(a, e, e); }
template <unsigned M> HM_D DualT<M> dlog(const DualT<M>& a) { return dmap(a, logf(a.v), 1.f / a.v); }
template <unsigned M>
HM_D DualT<M> dsqrt_safe(const DualT<M>& a) {
  const float s = a.v <= 0.f ? 0.f : sqrtf(a.v);
  DualT<M> r = dmap(a, s, 0.5f / s);
  if (a.v <= 0.f) HM_FOR_D(i, M) r.d[i] = 0.f;
  return r;
}
template <unsigned M> HM_D DualT<M> dsin(const DualT<M>& a) { return dmap(a, sinf(a.v), cosf(a.v)); }
template <unsigned M> HM_D DualT<M> dsinh(const DualT<M>& a) { return dmap(a, sinhf(a.v), coshf(a.v)); }
template <unsigned M> HM_D DualT<M> dabs(const DualT<M>& a) { return a.v < 0.f ? -a : a; }
template <unsigned M>
HM_D DualT<M> dpow_int(const DualT<M>& a, int n) {  // a^n, n >= 1
  const float p = powf(a.v, (float)n);
  return dmap(a, p, (float)n * powf(a.v, (float)(n - 1)));
}
template <unsigned M>
struct DMask {
  static constexpr unsigned value = M;
};
// All six partials, zero where a has none.
template <unsigned M>
HM_D Dual dfull(const DualT<M>& a) {
  Dual r;
  r.v = a.v;
#pragma unroll
  for (int i = 0; i < kNd; ++i) r.d[i] = (M >> i) & 1u ? a.d[i] : 0.f;
  return r;
}

struct HairConstsD {
  DualT<kBm> v[3];
  DualT<kBn> s;
  DualT<kAl> sin2k[3], cos2k[3];
  float sigma_a[3];
  float gain[4];
  DualT<kBn> trim_den;
};

// setupHairShading (disney_hair.cuh:26-41) with the parameters as variables.
HM_D HairConstsD hair_consts_dual(const float sigma_a[3], float beta_m, float beta_n, float alpha,
                                  const float gain[4]) {
  HairConstsD hc;
  const DualT<kBm> bm = dvar<kBm>(beta_m);
  const DualT<kBn> bn = dvar<kBn>(beta_n);
  const DualT<kAl> al = dvar<kAl>(alpha);
  hc.v[0] = dsqr(0.726f * bm + 0.812f * dsqr(bm) + 3.7f * dpow_int(bm, 20));
  hc.v[1] = 0.25f * hc.v[0];
  hc.v[2] = 4.f * hc.v[0];
  hc.s = kSqrtPiOver8 * (0.265f * bn + 1.194f * dsqr(bn) + 5.372f * dpow_int(bn, 22));
  hc.sin2k[0] = dsin(al);
  hc.cos2k[0] = dsqrt_safe(1.f - dsqr(hc.sin2k[0]));
  for (int i = 1; i < 3; ++i) {
    hc.sin2k[i] = 2.f * hc.cos2k[i - 1] * hc.sin2k[i - 1];
    hc.cos2k[i] = dsqr(hc.cos2k[i - 1]) - dsqr(hc.sin2k[i - 1]);
  }
  for (int c = 0; c < 3; ++c) hc.sigma_a[c] = sigma_a[c];
  for (int k = 0; k < 4; ++k) hc.gain[k] = gain[k];
  auto cdf = [&](float x) { return 1.f / (1.f + dexp(-x / hc.s)); };  // LogisticCDF :123-125
  hc.trim_den = cdf(kPi) - cdf(-kPi);
  return hc;
}

template <unsigned M>
HM_D DualT<M> bessel_i0_dual(const DualT<M>& x) {  // disney_hair.cuh:54-67
  DualT<M> val = dmap(x, 0.f, 0.f), x2i = dmap(x, 1.f, 0.f);
  float ifact = 1.f, i4 = 1.f;
  const DualT<M> xx = x * x;
  for (int i = 0; i < 10; ++i) {
    if (i > 1) ifact *= (float)i;
    val = val + x2i / (i4 * ifact * ifact);
    x2i = x2i * xx;
    i4 *= 4.f;
  }
  return val;
}

template <unsigned M>
HM_D DualT<M> log_i0_dual(const DualT<M>& x) {  // disney_hair.cuh:70-75
  if (x.v > 12.f) return x + 0.5f * ((-logf(2.f * kPi)) + dlog(1.f / x) + 1.f / (8.f * x));
  return dlog(bessel_i0_dual(x));
}

// M_p (disney_hair.cuh:78-88); cto, sto carry alpha's partial or none.
template <unsigned M>
HM_D DualT<(M | kBm)> mp_dual(float cti, const DualT<M>& cto, float sti, const DualT<M>& sto, const DualT<kBm>& v) {
  const DualT<(M | kBm)> a = (cti * cto) / v;
  const DualT<(M | kBm)> b = (sti * sto) / v;
  if (v.v <= 0.1f) return dexp(log_i0_dual(a) - b - 1.f / v + 0.6931f + dlog(1.f / (2.f * v)));
  return (dexp(-b) * bessel_i0_dual(a)) / (dsinh(1.f / v) * 2.f * v);
}

HM_D DualT<kBn> np_dual(float phi, int p, float gamma_o, float gamma_t, const HairConstsD& hc) {
  float dphi = phi - phi_p(p, gamma_o, gamma_t);
  while (dphi > kPi) dphi -= 2.f * kPi;
  while (dphi < -kPi) dphi += 2.f * kPi;
  const DualT<kBn> e = dexp(-fabsf(dphi) / hc.s);
  return (e / (hc.s * dsqr(1.f + e))) / hc.trim_den;
}

struct HairEvalD {
  Dual f[3];
  Dual pdf;
};

// hair_eval with derivatives; wo, wi in the hair frame, h = dot(Y, n).
HM_D HairEvalD hair_eval_dual(f3 wo, f3 wi, float h, const HairConstsD& hc) {
  const float sin_to = wo.x;
  const float cos_to = safe_sqrt(1.f - sqr(sin_to));
  const float phi_o = atan2f(wo.z, wo.y);
  const float sin_ti = wi.x;
  const float cos_ti = safe_sqrt(1.f - sqr(sin_ti));
  const float phi_i = atan2f(wi.z, wi.y);
  const float sin_tt = sin_to / kEta;
  const float cos_tt = safe_sqrt(1.f - sqr(sin_tt));
  const float gamma_o = asinf(h);
  const float cos_go = cosf(gamma_o);
  const float etap = sqrtf(kEta * kEta - sqr(sin_to)) / cos_to;
  const float sin_gt = h / etap;
  const float cos_gt = safe_sqrt(1.f - sqr(sin_gt));
  const float gamma_t = safe_asin(sin_gt);
  const float fac = (2.f * cos_gt / cos_tt);
  const float F0 = sqr(1.f - kEta) / sqr(1.f + kEta);
  const float xd = 1.f - cos_to * cos_go;
  const float fr = F0 + (1.f - F0) * xd * xd * xd * xd * xd;
  const float phi = phi_i - phi_o;

  // M_p and N_p of the lobes.  alpha's terms of each tilted lobe, then one
  // loop body for all four M_p (TRRT's tilt has no partial: zero ones)
  DualT<(kBm | kAl)> mp[4];
  DualT<kBn> np[3];
#pragma unroll 1
  for (int p = 0; p < 4; ++p) {
    DualT<kAl> sop, cop;
    sop.v = sin_to;
    cop.v = cos_to;
    sop.d[5] = cop.d[5] = 0.f;
    if (p == 0) {
      sop = sin_to * hc.cos2k[1] - cos_to * hc.sin2k[1];
      cop = dabs(cos_to * hc.cos2k[1] + sin_to * hc.sin2k[1]);
    } else if (p < 3) {
      const int k = p == 1 ? 0 : 2;
      sop = sin_to * hc.cos2k[k] + cos_to * hc.sin2k[k];
      cop = dabs(cos_to * hc.cos2k[k] - sin_to * hc.sin2k[k]);
    }
    mp[p] = mp_dual(cos_ti, cop, sin_ti, sop, hc.v[p < 3 ? p : 2]);
    if (p < 3) np[p] = np_dual(phi, p, gamma_o, gamma_t, hc);
  }
  const float npm = 1.f / (2.f * kPi);

  // attenuations of one colour channel: value and its own absorption's partial
  auto channel = [&](auto mask, auto& f, auto& a1, auto& a2, auto& a3) {
    constexpr unsigned M = decltype(mask)::value;
    constexpr int c = M == 1u ? 0 : (M == 2u ? 1 : 2);
    const DualT<M> sig = dvar<M>(hc.sigma_a[c]);
    const DualT<M> T = dexp(-sig * fac);
    a1 = sqr(1.f - fr) * T;
    a2 = sqr(1.f - fr) * T * T * fr;
    a3 = a2 * fr * T / (1.f - T * fr);
    f = dfull(hc.gain[0] * mp[0] * fr * np[0] + hc.gain[1] * mp[1] * a1 * np[1] + hc.gain[2] * mp[2] * a2 * np[2] +
              hc.gain[3] * mp[3] * a3 * npm);
  };
  HairEvalD out;
  DualT<1u> a1x, a2x, a3x;
  DualT<2u> a1y, a2y, a3y;
  DualT<4u> a1z, a2z, a3z;
  channel(DMask<1u>{}, out.f[0], a1x, a2x, a3x);
  channel(DMask<2u>{}, out.f[1], a1y, a2y, a3y);
  channel(DMask<4u>{}, out.f[2], a1z, a2z, a3z);
  DualT<0u> ap0;  // no partials
  ap0.v = (fr + fr + fr) / 3.f;
  const DualT<7u> ap1 = (a1x + a1y + a1z) / 3.f;
  const DualT<7u> ap2 = (a2x + a2y + a2z) / 3.f;
  const DualT<7u> ap3 = (a3x + a3y + a3z) / 3.f;
  const DualT<7u> sum = ap0 + ap1 + ap2 + ap3;
  out.pdf = mp[0] * (ap0 / sum) * np[0] + mp[1] * (ap1 / sum) * np[1] + mp[2] * (ap2 / sum) * np[2] +
            mp[3] * (ap3 / sum) * npm;
  return out;
}

}  // namespace hm
