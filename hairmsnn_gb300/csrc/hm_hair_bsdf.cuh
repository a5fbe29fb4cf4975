// Chiang 2016 / d'Eon hair BSDF ("disney_hair") for sm_103a.
//
// Same formulas, statement order and lobe layout as the reference's
// cuda_headers/disney_hair.cuh; what changes is where the work happens:
//  * everything that depends only on the material (setupHairShading
//    disney_hair.cuh:26-41, the trimmed-logistic normaliser, the per-lobe
//    1/v, log(1/2v), sinh(1/v)*2v and exp(-2/v) terms) is computed once on the
//    host into HairConsts (kernel-parameter / constant memory) instead of at
//    every closest hit;
//  * callers pass wo/wi already in the hair frame and h = dot(Y, n), not a
//    ~300-byte Interaction by value;
//  * for beta_m < 0.1 the log-space M_p branch (disney_hair.cuh:82-83) runs in
//    FP64, where the FP32 cancellation between LogI0(a) and 1/v loses digits.
#pragma once
#include "hm_common.cuh"

namespace hm {

struct HairConsts {
  float v[4];         // v[0..2] as setupHairShading; v[3] == s (see sample_disney_hair)
  float s;            // logistic scale
  float sin2k[3], cos2k[3];
  float sigma_a[3];
  float gain[4];      // R, TT, TRT, TRRT
  float trim_den;     // LogisticCDF(pi, s) - LogisticCDF(-pi, s)
  float cdf_lo;       // LogisticCDF(-pi, s)
  float inv_v[3];     // 1 / v[k]
  float mp_logc[3];   // log(1 / (2 v[k]))
  float mp_den[3];    // sinh(1 / v[k]) * 2 * v[k]
  float exp_m2v[4];   // exp(-2 / v[p]), p = 0..3
  int fp64_mp;        // beta_m < 0.1
  double mp_inv_d[3], mp_logc_d[3];  // then: 1 / v[k] and log(1 / (2 v[k])) in FP64
};

HM_HD float logistic_cdf_s(float x, float s) { return 1.f / (1.f + expf(-x / s)); }  // LogisticCDF :123-125

// setupHairShading (disney_hair.cuh:26-41) and every other material-only
// term, in the reference's single-precision order.  The library evaluates it
// once per material on the host (hair_consts_from_params); code that
// includes include/hairmsnn_device.cuh may also call it on the device.
HM_HD HairConsts hair_consts(const hm_hair_params& p) {
  HairConsts hc;
  const float bm = p.beta_m, bn = p.beta_n;
  hc.v[0] = sqr(0.726f * bm + 0.812f * sqr(bm) + 3.7f * powf(bm, 20.f));
  hc.v[1] = (float)(.25 * (double)hc.v[0]);
  hc.v[2] = 4.f * hc.v[0];
  hc.s = kSqrtPiOver8 * (0.265f * bn + 1.194f * sqr(bn) + 5.372f * powf(bn, 22.f));
  hc.v[3] = hc.s;
  hc.sin2k[0] = sinf(p.alpha);
  hc.cos2k[0] = safe_sqrt(1.f - sqr(hc.sin2k[0]));
  for (int i = 1; i < 3; ++i) {
    hc.sin2k[i] = 2.f * hc.cos2k[i - 1] * hc.sin2k[i - 1];
    hc.cos2k[i] = sqr(hc.cos2k[i - 1]) - sqr(hc.sin2k[i - 1]);
  }
  for (int i = 0; i < 3; ++i) hc.sigma_a[i] = p.sigma_a[i];
  hc.gain[0] = p.gain_r;
  hc.gain[1] = p.gain_tt;
  hc.gain[2] = p.gain_trt;
  hc.gain[3] = p.gain_trrt;
  hc.trim_den = logistic_cdf_s(kPi, hc.s) - logistic_cdf_s(-kPi, hc.s);
  hc.cdf_lo = logistic_cdf_s(-kPi, hc.s);
  for (int k = 0; k < 3; ++k) {
    hc.inv_v[k] = 1.f / hc.v[k];
    hc.mp_logc[k] = logf(1.f / (2.f * hc.v[k]));
    hc.mp_den[k] = sinhf(1.f / hc.v[k]) * 2.f * hc.v[k];
  }
  for (int k = 0; k < 4; ++k) hc.exp_m2v[k] = expf(-2.f / hc.v[k]);
  hc.fp64_mp = bm < 0.1f ? 1 : 0;
  for (int k = 0; k < 3; ++k) {
    hc.mp_inv_d[k] = hc.fp64_mp ? 1.0 / (double)hc.v[k] : 0.0;
    hc.mp_logc_d[k] = hc.fp64_mp ? log(1.0 / (2.0 * (double)hc.v[k])) : 0.0;
  }
  return hc;
}

// Host-side precompute of hair_consts (see hm_bsdf.cu).
HairConsts hair_consts_from_params(const hm_hair_params& p);

// a / c for a positive constant c whose reciprocal is a compile-time constant:
// the quotient estimate, its exact remainder and one correction (Markstein,
// IBM J. Res. Dev. 34, 1990).  For every c used here this is the correctly rounded quotient of every
// normal a (checked over all mantissas, tests/test_div_const_header.py), so
// results keep their bits; a must not be infinite.
HM_HD float div_const(float a, float c) {
  const float y = 1.f / c;
#ifdef __CUDA_ARCH__
  const float q = __fmul_rn(a, y);
  return __fmaf_rn(__fmaf_rn(-c, q, a), y, q);
#else
  const float q = a * y;
  return fmaf(fmaf(-c, q, a), y, q);
#endif
}

HM_D float bessel_i0(float x) {  // disney_hair.cuh:54-67
  float val = 0.f, x2i = 1.f;
  float ifact = 1.f;  // i! for i <= 9 is exact in float (int64 in the reference)
  float i4 = 1.f;
#pragma unroll
  for (int i = 0; i < 10; ++i) {
    if (i > 1) ifact *= (float)i;
    val += div_const(x2i, i4 * sqr(ifact));
    x2i *= x * x;
    i4 *= 4.f;
  }
  return val;
}

// disney_hair.cuh:70-75.  The reference forms x + 0.5 * g in FP64 and rounds
// to float; that FP64 sum is exact (x in (12, 1 / v], v > 0.0015 where this
// branch runs, and |g| > 4 span at most 50 bits), so one fused multiply-add
// gives the same float without the FP64 units.
HM_D float log_i0(float x) {
  if (x > 12.f) return __fmaf_rn(0.5f, -logf(2.f * kPi) + logf(1.f / x) + 1.f / (8.f * x), x);
  return logf(bessel_i0(x));
}

HM_D double bessel_i0_d(double x) {
  double val = 0.0, x2i = 1.0, ifact = 1.0, i4 = 1.0;
#pragma unroll
  for (int i = 0; i < 10; ++i) {
    if (i > 1) ifact *= i;
    val += x2i / (i4 * ifact * ifact);
    x2i *= x * x;
    i4 *= 4.0;
  }
  return val;
}

// The log-space branch of M_p in FP64.  One copy of the code, called: inlined
// into every lobe of every evaluation its logarithms and exponential made the
// kernels larger than the instruction caches: five to eight issue slots lost
// to fetching for each instruction of the shading kernel, and bsdf_eval_kernel
// took 36 us for 262,144 queries instead of 22.  Where it runs it is bound by
// the FP64 units; the material's two terms come with the constants (2,000,003
// queries at beta_m 0.09: 3203 us inlined with those terms in every lobe, 3324
// called, 2721 now).
static __device__ __noinline__ float mp_lobe_fp64(float cti, float cto, float sti, float sto, float v, double inv_v,
                                                  double logc) {
  double dv = v;
  double a = (double)cti * (double)cto / dv;
  double b = (double)sti * (double)sto / dv;
  double li = a > 12.0 ? a + 0.5 * (-log(2.0 * (double)kPi) + log(1.0 / a) + 1.0 / (8.0 * a))
                       : log(bessel_i0_d(a));
  return (float)exp(li - b - inv_v + 0.6931 + logc);
}

// M_p (disney_hair.cuh:78-88) for lobe constants k; v = v[k].
HM_D float mp_lobe(float cti, float cto, float sti, float sto, const HairConsts& hc, int k) {
  const float v = hc.v[k];
  if (hc.fp64_mp && v <= 0.1f) return mp_lobe_fp64(cti, cto, sti, sto, v, hc.mp_inv_d[k], hc.mp_logc_d[k]);
  float a = cti * cto / v;
  float b = sti * sto / v;
  if (v <= 0.1f) return expf(log_i0(a) - b - hc.inv_v[k] + 0.6931f + hc.mp_logc[k]);
  return (expf(-b) * bessel_i0(a)) / hc.mp_den[k];
}

HM_D float phi_p(int p, float gamma_o, float gamma_t) {  // disney_hair.cuh:112-114
  return (float)(2 * p) * gamma_t - 2.f * gamma_o + (float)p * kPi;
}

// TrimmedLogistic(dphi, s, -pi, pi) after wrapping dphi to [-pi, pi] (:117-139)
HM_D float np_lobe(float phi, int p, float gamma_o, float gamma_t, const HairConsts& hc) {
  float dphi = phi - phi_p(p, gamma_o, gamma_t);
  while (dphi > kPi) dphi -= 2.f * kPi;
  while (dphi < -kPi) dphi += 2.f * kPi;
  const float s = hc.s;
  float e = expf(-fabsf(dphi) / s);
  return (e / (s * sqr(1.f + e))) / hc.trim_den;
}

struct HairEval {
  f3 f;       // f * cos (the reference's disney_hair return value)
  float pdf;  // full 4-lobe mixture pdf
};

// What an evaluation or a sample needs of (wo, h, material) alone: computed
// once for a vertex and shared by its light sample, BSDF sample and next
// direction (each once computed it again).
struct HairGeom {
  float sin_to, cos_to, phi_o, gamma_o, gamma_t;
  float fr;       // Fresnel, the R lobe's attenuation
  f3 a1, a2, a3;  // TT, TRT, TRRT attenuations
  float ap[4];    // lobe pmf
};

// disney_hair.cuh:186-218 and computeApPdf (:143-182; with eta = Eta it reuses
// the T and Fresnel of the evaluation).  wo: hair-frame unit vector (x along
// the fibre); h = dot(Y, n) in [-1, 1].
HM_D HairGeom hair_geom(f3 wo, float h, const HairConsts& hc) {
  HairGeom g;
  const float sin_to = wo.x;
  const float cos_to = safe_sqrt(1.f - sqr(sin_to));
  g.sin_to = sin_to;
  g.cos_to = cos_to;
  g.phi_o = atan2f(wo.z, wo.y);
  const float sin_tt = div_const(sin_to, kEta);
  const float cos_tt = safe_sqrt(1.f - sqr(sin_tt));
  g.gamma_o = asinf(h);
  const float cos_go = cosf(g.gamma_o);
  const float etap = sqrtf(kEta * kEta - sqr(sin_to)) / cos_to;
  const float sin_gt = h / etap;
  const float cos_gt = safe_sqrt(1.f - sqr(sin_gt));
  g.gamma_t = safe_asin(sin_gt);
  const float fac = (2.f * cos_gt / cos_tt);
  const f3 T = mk(expf(-hc.sigma_a[0] * fac), expf(-hc.sigma_a[1] * fac), expf(-hc.sigma_a[2] * fac));
  // Fresnel(Eta, cos_to * cos_go), disney_hair.cuh:46-51
  const float F0 = sqr(1.f - kEta) / sqr(1.f + kEta);
  const float xd = 1.f - cos_to * cos_go;
  const float fr = F0 + (1.f - F0) * xd * xd * xd * xd * xd;
  g.fr = fr;
  // A_p, :91-109
  g.a1 = sqr(1.f - fr) * T;
  g.a2 = sqr(1.f - fr) * T * T * fr;
  g.a3 = g.a2 * fr * T / (splat(1.f) - T * fr);
  const float ap[4] = {(fr + fr + fr) / 3.f, (g.a1.x + g.a1.y + g.a1.z) / 3.f, (g.a2.x + g.a2.y + g.a2.z) / 3.f,
                       (g.a3.x + g.a3.y + g.a3.z) / 3.f};
  const float sum = ap[0] + ap[1] + ap[2] + ap[3];
#pragma unroll
  for (int p = 0; p < 4; ++p) g.ap[p] = ap[p] / sum;
  return g;
}

// disney_hair(si, &pdf), disney_hair.cuh:186-266, for the geometry of (wo, h).
// wi: hair-frame unit vector.
HM_D HairEval hair_eval(const HairGeom& g, f3 wi, const HairConsts& hc) {
  const float sin_to = g.sin_to, cos_to = g.cos_to;
  const float sin_ti = wi.x;
  const float cos_ti = safe_sqrt(1.f - sqr(sin_ti));
  const float phi_i = atan2f(wi.z, wi.y);
  const float phi = phi_i - g.phi_o;

  // M_p and N_p of the lobes R, TT, TRT, TRRT.  R tilts by -2^1 alpha, TT by
  // 2^0, TRT by 2^2, TRRT not (the sine's sign carries the direction exactly).
  // A loop, not unrolled: the four copies of a lobe's code overran the
  // instruction caches.  bsdf_sample_kernel, 8,000,003 queries: 502 us unrolled,
  // 470 as a loop; its sums f and pdf stay outside the loop (494 inside it,
  // with the values they keep alive).
  float mp[4], np[3];
#pragma unroll 1
  for (int p = 0; p < 4; ++p) {
    float sop = sin_to, cop = cos_to;
    if (p < 3) {
      const int k = p == 0 ? 1 : (p == 1 ? 0 : 2);
      const float sk = p == 0 ? -hc.sin2k[k] : hc.sin2k[k], ck = hc.cos2k[k];
      sop = sin_to * ck + cos_to * sk;
      cop = fabsf(cos_to * ck - sin_to * sk);
      np[p] = np_lobe(phi, p, g.gamma_o, g.gamma_t, hc);
    }
    mp[p] = mp_lobe(cos_ti, cop, sin_ti, sop, hc, p < 3 ? p : 2);
  }
  const float npm = 1.f / (2.f * kPi);
  f3 f = hc.gain[0] * mp[0] * splat(g.fr) * np[0];
  f = f + hc.gain[1] * mp[1] * g.a1 * np[1];
  f = f + hc.gain[2] * mp[2] * g.a2 * np[2];
  f = f + hc.gain[3] * mp[3] * g.a3 * npm;
  float pdf = 0.f;
  pdf = pdf + mp[0] * g.ap[0] * np[0];
  pdf = pdf + mp[1] * g.ap[1] * np[1];
  pdf = pdf + mp[2] * g.ap[2] * np[2];
  pdf = pdf + mp[3] * g.ap[3] * npm;
  return HairEval{f, pdf};
}

HM_D HairEval hair_eval(f3 wo, f3 wi, float h, const HairConsts& hc) { return hair_eval(hair_geom(wo, h, hc), wi, hc); }

// The direction of sample_disney_hair (hair frame).  The TRRT lobe (p = 3)
// uses v[3] == s: in the reference's HairInteraction the element after v[2]
// is s.
HM_D f3 hair_sample_dir(const HairGeom& g, float u0, float u1, float u2, float u3, const HairConsts& hc) {
  const float sin_to = g.sin_to, cos_to = g.cos_to;
  int p = 0;
  float eps1 = u0;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    if (p == k && !(eps1 < g.ap[k])) {
      eps1 -= g.ap[k];
      p = k + 1;
    }
  }
  float sop, cop;
  if (p == 0) {
    sop = sin_to * hc.cos2k[1] - cos_to * hc.sin2k[1];
    cop = cos_to * hc.cos2k[1] + sin_to * hc.sin2k[1];
  } else if (p == 1) {
    sop = sin_to * hc.cos2k[0] + cos_to * hc.sin2k[0];
    cop = cos_to * hc.cos2k[0] - sin_to * hc.sin2k[0];
  } else if (p == 2) {
    sop = sin_to * hc.cos2k[2] + cos_to * hc.sin2k[2];
    cop = cos_to * hc.cos2k[2] - sin_to * hc.sin2k[2];
  } else {
    sop = sin_to;
    cop = cos_to;
  }
  const float eps2 = fmaxf(u1, 1e-5f);
  const float vp = hc.v[p];
  const float cos_theta = 1.f + vp * logf(eps2 + (1.f - eps2) * hc.exp_m2v[p]);
  const float sin_theta = safe_sqrt(1.f - sqr(cos_theta));
  const float cos_phi = cosf(2.f * kPi * u2);
  const float sin_ti = -cos_theta * sop + sin_theta * cos_phi * cop;
  const float cos_ti = safe_sqrt(1.f - sqr(sin_ti));
  float dphi;
  if (p < 3) {
    // SampleTrimmedLogistic(u3, s, -pi, pi), :269-274
    float x = -hc.s * logf(1.f / (u3 * hc.trim_den + hc.cdf_lo) - 1.f);
    dphi = phi_p(p, g.gamma_o, g.gamma_t) + fminf(fmaxf(x, -kPi), kPi);
  } else {
    dphi = 2.f * kPi * u3;
  }
  const float phi_i = g.phi_o + dphi;
  return normalize(mk(sin_ti, cos_ti * cosf(phi_i), cos_ti * sinf(phi_i)));
}

// sample_disney_hair(si, rand, &pdf), disney_hair.cuh:277-386.  Returns the
// hair-frame wi and the full eval at it.
HM_D HairEval hair_sample(f3 wo, float h, float u0, float u1, float u2, float u3,
                          const HairConsts& hc, f3* wi_out) {
  const HairGeom g = hair_geom(wo, h, hc);
  *wi_out = hair_sample_dir(g, u0, u1, u2, u3, hc);
  return hair_eval(g, *wi_out, hc);
}

// Hair shading frame of the reference's closest-hit program
// (optix_common.cuh:571-583): X = tangent, Y = normalize(wo x X), Z = X x Y.
HM_D Frame hair_frame(f3 wo, f3 t) {
  Frame fr;
  fr.r0 = t;
  fr.r1 = normalize(cross(wo, t));
  fr.r2 = normalize(cross(t, fr.r1));
  return fr;
}

}  // namespace hm
