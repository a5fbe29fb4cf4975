// Radiance-cache network forward on the 5th-generation tensor cores.
//
// One persistent CTA of 128 threads per SM slot; each CTA keeps every layer's
// weights in shared memory (loaded once) and walks 128-query tiles:
//   encode   thread t computes the encoded input row of query t of the tile
//            (same per-feature arithmetic as the FP32 encode kernel) and
//            stores it, rounded to FP16 / BF16 / E4M3, as the A operand
//   layers   thread 0 issues tcgen05.mma (M=128, N=width or 16, K=16/32 per
//            instruction) with A and B in shared memory and the FP32
//            accumulator in tensor memory, then tcgen05.commit to an mbarrier
//   epilogue every thread reads its row of the accumulator (tcgen05.ld
//            32x32b), applies ReLU and stores it as the next layer's A
//   output   the 16-column accumulator of the last layer -> out (FP32)
// Layer 0 is split along K into chunks when the encoded row does not fit
// next to the weights.
//
// Operand layout (both A and B, K-major, no swizzle): 8-row x 16-byte core
// matrices; for an R-row operand the byte at (row, kb) sits at
//   ((kb / 16) * (R / 8) + row / 8) * 128 + (row % 8) * 16 + kb % 16,
// so core matrices adjacent in K are 16*R bytes apart (leading byte offset)
// and those adjacent in M/N 128 bytes apart (stride byte offset).
//
// E4M3: weights carry one scale per layer (448 / amax of the layer), the
// activations one scale per query row (448 / amax of the row; for the
// encoded input an upper bound: 1 for Frequency/OneBlob/padding, |x| for
// Identity inputs, the table amax for hash grids).  Scaling rows of A scales
// rows of D, so the epilogue owning the row undoes it exactly.
//
// Every wait on the mbarrier is bounded; on expiry the kernel records the
// fact in a host-mapped flag, stops issuing work, frees its tensor memory
// and returns.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>

#include <string.h>

#include <algorithm>
#include <string>

#include "hm_mlp.cuh"
#include "hm_tc.cuh"

namespace hm {

enum { TC_FP16 = 1, TC_BF16 = 2, TC_E4M3 = 3 };
constexpr int kTcThreads = 256;
constexpr float kE4M3Max = 448.f;

// ------------------------------------------------------------ quantisation
template <int PREC>
HM_D uint32_t pack2(float a, float b) {
  if (PREC == TC_BF16) {
    __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&h);
  } else {
    __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&h);
  }
}
HM_D uint32_t pack4_e4m3(float a, float b, float c, float d) {
  const uint32_t lo = __nv_cvt_float2_to_fp8x2(make_float2(a, b), __NV_SATFINITE, __NV_E4M3);
  const uint32_t hi = __nv_cvt_float2_to_fp8x2(make_float2(c, d), __NV_SATFINITE, __NV_E4M3);
  return (lo & 0xFFFFu) | (hi << 16);
}

// ---------------------------------------------------------------- encoding
// Features are produced in increasing order and packed through a 128-bit
// shift register into 16-byte groups, one conflict-free store per group
// (the 32 rows of a warp are 32 consecutive 16-byte core-matrix rows);
// 16-bit operands take consecutive features in pairs where they can.
template <int PREC>
struct RowPacker {
  static constexpr int kPer = PREC == TC_E4M3 ? 16 : 8;  // values per 16 bytes
  uint32_t w0 = 0, w1 = 0, w2 = 0, w3 = 0;
  int cnt = 0, group;
  uint8_t* A;
  int row;
  float scale;
  uint8_t* mirror = nullptr;  // training: the row's operand bytes also go here
  // training with E4M3 operands: the row's features, unscaled, as FP16 (the
  // backward pass runs on FP16 operands)
  uint16_t* mirror16 = nullptr;
  HM_D RowPacker(uint8_t* a, int r, int first_group, float sc) : group(first_group), A(a), row(r), scale(sc) {}
  HM_D void push(float v) {
    constexpr int SH = PREC == TC_E4M3 ? 8 : 16;
    if (PREC == TC_E4M3 && mirror16) mirror16[group * kPer + cnt] = __half_as_ushort(__float2half_rn(v));
    uint32_t h;
    if (PREC == TC_E4M3)
      h = (uint32_t)__nv_cvt_float_to_fp8(v * scale, __NV_SATFINITE, __NV_E4M3);
    else if (PREC == TC_BF16)
      h = (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(v));
    else
      h = (uint32_t)__half_as_ushort(__float2half_rn(v));
    w0 = __funnelshift_r(w0, w1, SH);
    w1 = __funnelshift_r(w1, w2, SH);
    w2 = __funnelshift_r(w2, w3, SH);
    w3 = (w3 >> SH) | (h << (32 - SH));
    if (++cnt == kPer) flush();
  }
  // Two consecutive features: for 16-bit operands at an even fill, one
  // paired conversion (the same round-to-nearest of each value) and one
  // 32-bit step of the register; otherwise two pushes.
  HM_D void push2(float a, float b) {
    if (PREC == TC_E4M3 || (cnt & 1)) {
      push(a);
      push(b);
      return;
    }
    w0 = w1;
    w1 = w2;
    w2 = w3;
    w3 = pack2<PREC>(a, b);
    cnt += 2;
    if (cnt == kPer) flush();
  }
  HM_D void flush() {
    *reinterpret_cast<uint4*>(A + op_offset(kTcRows, row, group * 16)) = make_uint4(w0, w1, w2, w3);
    if (mirror) *reinterpret_cast<uint4*>(mirror + group * 16) = make_uint4(w0, w1, w2, w3);
    ++group;
    cnt = 0;
  }
};

// Encoded features [kb, ke) of one row (k >= n_enc: padding 1; k >= in_pad:
// 0, the extra K columns of the E4M3 layout carry zero weights).
// Identity / OneBlob / hash grid values use the arithmetic of encode_kernel;
// the Frequency pair (sin, cos) of 2^f * pi * x comes from sincospif, whose
// reduction is exact (encode_kernel forms the phase 2^f * x * 3.1415926 in
// FP32 and adds pi/2 for the cosine: at most ~5e-4 apart at 2^11, below the
// 16-bit operand rounding).  OneBlob bins more than two
// bins away from x (circularly) are exactly 0 in encode_kernel's formula and
// are not evaluated.
template <int PREC>
HM_D void enc_range(const MlpDims& d, const float* __restrict__ xin, const float* __restrict__ enc_params, int kb,
                    int ke, RowPacker<PREC>& pk) {
  for (int si = 0; si < d.n_segs; ++si) {
    const EncSeg& s = d.segs[si];
    const int lo = max(kb, s.out_off), hi = min(ke, s.out_off + s.n_out);
    if (lo >= hi) continue;
    const int j0 = lo - s.out_off, j1 = hi - s.out_off;
    if (s.type == ENC_IDENTITY) {
      int j = j0;
      for (; j + 1 < j1; j += 2) pk.push2(xin[s.in_off + j], xin[s.in_off + j + 1]);
      if (j < j1) pk.push(xin[s.in_off + j]);
    } else if (s.type == ENC_FREQUENCY) {
      int u = j0 >> 1;
      int dim = u / s.n_freq, f = u - dim * s.n_freq;
      for (int j = j0; j < j1;) {
        float sn, cs;
        sincospif(scale_pow2(xin[s.in_off + dim], f), &sn, &cs);
        if (!(j & 1) && j + 1 < j1) {
          pk.push2(sn, cs);
          j += 2;
        } else {
          if (!(j & 1)) {
            pk.push(sn);
            ++j;
          }
          if (j < j1) {
            pk.push(cs);
            ++j;
          }
        }
        if (++f == s.n_freq) {
          f = 0;
          ++dim;
        }
      }
    } else if (s.type == ENC_ONEBLOB) {
      // the five bins around x (circularly) are evaluated once per input
      // dimension, without branches that would diverge across the rows of
      // a warp; every other bin is 0
      const float nb = (float)s.n_bins;
      int dim = j0 / s.n_bins, b = j0 - dim * s.n_bins;
      int b0 = 0;
      float wv[5];
      auto window = [&](int dm) {
        const float x = xin[s.in_off + dm];
        // bin of x on the period [0, 1) (x itself may lie outside it)
        b0 = (((int)floorf(x * nb)) % s.n_bins + s.n_bins) % s.n_bins;
        const float c0 = oneblob_cdf(0.f, x, nb);
        // mass of window bin t = right edge - left edge; bin t's right edge
        // is bin t+1's left edge (+1 where bin t is the last bin: the edge
        // wraps to 0), so six edge evaluations give the five masses
        float left[5];
        int wb[5];
#pragma unroll
        for (int t = 0; t < 5; ++t) {
          // (b0 - 2 + t) mod n_bins: b0 is in [0, n_bins), so with two or
          // more bins one correction lands in range (one bin: always 0)
          int w = b0 - 2 + t;
          w += w < 0 ? s.n_bins : 0;
          w -= w >= s.n_bins ? s.n_bins : 0;
          wb[t] = s.n_bins == 1 ? 0 : w;
          left[t] = wb[t] == 0 ? c0 : oneblob_cdf((float)wb[t] / nb, x, nb);
        }
        const float right4 = (wb[4] == s.n_bins - 1) ? c0 + 1.f : oneblob_cdf((float)(wb[4] + 1) / nb, x, nb);
#pragma unroll
        for (int t = 0; t < 5; ++t) {
          const float right = t < 4 ? ((wb[t] == s.n_bins - 1) ? left[t + 1] + 1.f : left[t + 1]) : right4;
          wv[t] = right - left[t];
        }
      };
      window(dim);
      auto bin_value = [&](int bb) {
        int dd = bb - b0;
        if (dd > (s.n_bins >> 1)) dd -= s.n_bins;
        if (dd < -(s.n_bins >> 1)) dd += s.n_bins;
        float v = 0.f;
        v = dd == -2 ? wv[0] : v;
        v = dd == -1 ? wv[1] : v;
        v = dd == 0 ? wv[2] : v;
        v = dd == 1 ? wv[3] : v;
        v = dd == 2 ? wv[4] : v;
        return v;
      };
      for (int j = j0; j < j1;) {
        if (b + 1 < s.n_bins && j + 1 < j1) {  // two bins of the same dimension
          pk.push2(bin_value(b), bin_value(b + 1));
          b += 2;
          j += 2;
        } else {
          pk.push(bin_value(b));
          ++b;
          ++j;
        }
        if (b == s.n_bins && j < j1) {
          b = 0;
          ++dim;
          window(dim);
        }
      }
    } else {  // hash grid
      const float* table = enc_params + s.param_off;
      const bool pair_table = s.n_feat == 2 && (reinterpret_cast<uintptr_t>(table) & 7) == 0;
      const float px = xin[s.in_off], py = xin[s.in_off + 1], pz = xin[s.in_off + 2];
      int l = j0 / s.n_feat, f0 = j0 - l * s.n_feat;
      for (int j = j0; j < j1; ++l) {
        const float sc = s.level_scale[l];
        const float fx = fmaf(sc, px, 0.5f), fy = fmaf(sc, py, 0.5f), fz = fmaf(sc, pz, 0.5f);
        const float gx = floorf(fx), gy = floorf(fy), gz = floorf(fz);
        const float wx = fx - gx, wy = fy - gy, wz = fz - gz;
        const uint32_t ix = (uint32_t)(int)gx, iy = (uint32_t)(int)gy, iz = (uint32_t)(int)gz;
        float acc[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) acc[q] = 0.f;
        uint32_t e[8];
        grid_entries(s, l, ix, iy, iz, e);
        if (pair_table) {
          // two features per entry: the eight corners' entries are loaded
          // first (eight 8-byte gathers in flight), then accumulated in
          // corner order as below
          float2 tv[8];
#pragma unroll
          for (int c = 0; c < 8; ++c) tv[c] = __ldg(reinterpret_cast<const float2*>(table) + e[c]);
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            const float w = ((c & 1) ? wx : 1.f - wx) * (((c >> 1) & 1) ? wy : 1.f - wy) *
                            (((c >> 2) & 1) ? wz : 1.f - wz);
            acc[0] += w * tv[c].x;
            acc[1] += w * tv[c].y;
          }
        } else {
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            const float w = ((c & 1) ? wx : 1.f - wx) * (((c >> 1) & 1) ? wy : 1.f - wy) *
                            (((c >> 2) & 1) ? wz : 1.f - wz);
            const float* tv = table + (int64_t)e[c] * s.n_feat;
#pragma unroll
            for (int q = 0; q < 8; ++q)
              if (q < s.n_feat) acc[q] += w * __ldg(tv + q);
          }
        }
#pragma unroll
        for (int q = 0; q < 8; q += 2) {
          const bool ok0 = q >= f0 && q < s.n_feat && j < j1;
          const bool ok1 = q + 1 >= f0 && q + 1 < s.n_feat && j + (ok0 ? 1 : 0) < j1;
          if (ok0 && ok1) {
            pk.push2(acc[q], acc[q + 1]);
            j += 2;
          } else {
            if (ok0) {
              pk.push(acc[q]);
              ++j;
            }
            if (ok1) {
              pk.push(acc[q + 1]);
              ++j;
            }
          }
        }
        f0 = 0;
      }
    }
  }
  int k = max(kb, d.n_enc);
  for (; k + 1 < ke; k += 2) pk.push2(k < d.in_pad ? 1.f : 0.f, k + 1 < d.in_pad ? 1.f : 0.f);
  if (k < ke) pk.push(k < d.in_pad ? 1.f : 0.f);
}

// ---- encodings whose segments are made of whole 8-feature units
// (enc_units_ok): every Frequency, OneBlob and hash-grid segment starts and
// ends on a multiple of 8 features, and what follows the last one is identity
// inputs and padding.  The same values as enc_range, built a unit at a time
// in registers and stored to the unit's address: no packing register, no
// per-feature bookkeeping.  A OneBlob input's bins are all zero but five
// consecutive ones (circularly): its units are stored as zeros and the two or
// three words that hold the five masses are stored over them, where the
// mass-by-mass selection cost about eleven instructions per bin.
// The kernels that encode are bound by instruction issue.  Feature by feature
// through the packing register of enc_range -> by units: tc_encode_kernel<E4M3>,
// 300,007 queries of the 5 x 128 network 104 -> 41 us; mlp_tc_fused_kernel<FP16,
// 64>, 2^20 queries 498 -> 240 us.
//
// The caller's row: operand bytes of feature k at
//   a + (k * bytes / 16) * 2048 + k * bytes % 16    (128-row core-matrix layout)
// and, in a training forward, copies of it for the backward pass: `mirror`
// (16-bit operands as they are) or `mirror16` (FP16 of an E4M3 row's unscaled
// features), with unit u at + u * mirror_unit bytes.
struct EncRow {
  uint8_t* a;
  uint8_t* mirror;
  uint32_t mirror_unit;
  float scale;
};

HM_HD bool enc_units_ok(const MlpDims& d) {
  for (int si = 0; si < d.n_segs; ++si) {
    const EncSeg& s = d.segs[si];
    if (s.out_off % 8 != 0) return false;
    if (s.type == ENC_IDENTITY) return si == d.n_segs - 1;
    if (s.n_out % 8 != 0) return false;
    if (s.type == ENC_FREQUENCY && s.n_freq > 120) return false;
    if (s.type == ENC_ONEBLOB && s.n_bins % 8 != 0 && s.n_bins != 4) return false;
    if (s.type == ENC_HASHGRID && s.n_feat != 2) return false;
  }
  return true;
}

template <int PREC>
HM_D void enc_store8(const EncRow& r, int k, const float (&v)[8]) {
  if (PREC == TC_E4M3) {
    if (r.mirror) {
      uint4 h;
      h.x = pack2<TC_FP16>(v[0], v[1]);
      h.y = pack2<TC_FP16>(v[2], v[3]);
      h.z = pack2<TC_FP16>(v[4], v[5]);
      h.w = pack2<TC_FP16>(v[6], v[7]);
      *reinterpret_cast<uint4*>(r.mirror + (uint32_t)(k >> 3) * r.mirror_unit) = h;
    }
    uint2 w;
    w.x = pack4_e4m3(v[0] * r.scale, v[1] * r.scale, v[2] * r.scale, v[3] * r.scale);
    w.y = pack4_e4m3(v[4] * r.scale, v[5] * r.scale, v[6] * r.scale, v[7] * r.scale);
    *reinterpret_cast<uint2*>(r.a + (uint32_t)(k >> 4) * 2048u + (uint32_t)(k & 8)) = w;
  } else {
    constexpr int P16 = PREC == TC_E4M3 ? TC_FP16 : PREC;
    uint4 w;
    w.x = pack2<P16>(v[0], v[1]);
    w.y = pack2<P16>(v[2], v[3]);
    w.z = pack2<P16>(v[4], v[5]);
    w.w = pack2<P16>(v[6], v[7]);
    *reinterpret_cast<uint4*>(r.a + (uint32_t)(k >> 3) * 2048u) = w;
    if (r.mirror) *reinterpret_cast<uint4*>(r.mirror + (uint32_t)(k >> 3) * r.mirror_unit) = w;
  }
}

// The masses m of bins first .. first + 4 (mod n_bins) of the OneBlob input
// whose features start at k0, as the words that hold them; only words of
// features [lo, hi) (multiples of 8) are stored.
template <int PREC>
HM_D void enc_store_window(const EncRow& r, int k0, int n_bins, int first, const float (&m)[5], int lo, int hi) {
  if (PREC == TC_E4M3) {  // four lanes per word, two words
    const uint64_t b = (uint64_t)pack4_e4m3(m[0] * r.scale, m[1] * r.scale, m[2] * r.scale, m[3] * r.scale) |
                       (uint64_t)(pack4_e4m3(m[4] * r.scale, 0.f, 0.f, 0.f) & 0xFFu) << 32;
    const uint64_t v = b << (8 * (first & 3));
    int w = first & ~3;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int k = k0 + w;
      if (k >= lo && k < hi)
        *reinterpret_cast<uint32_t*>(r.a + (uint32_t)(k >> 4) * 2048u + (uint32_t)(k & 15)) =
            i ? (uint32_t)(v >> 32) : (uint32_t)v;
      w += 4;
      w -= w >= n_bins ? n_bins : 0;
    }
    if (!r.mirror) return;
  }
  constexpr int P16 = PREC == TC_E4M3 ? TC_FP16 : PREC;
  const bool odd = first & 1;
  const uint32_t v[3] = {odd ? pack2<P16>(0.f, m[0]) : pack2<P16>(m[0], m[1]),
                         odd ? pack2<P16>(m[1], m[2]) : pack2<P16>(m[2], m[3]),
                         odd ? pack2<P16>(m[3], m[4]) : pack2<P16>(m[4], 0.f)};
  int w = first & ~1;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const int k = k0 + w;
    if (k >= lo && k < hi) {
      const uint32_t u = (uint32_t)(k >> 3), byte = (uint32_t)(k & 7) * 2u;
      if (PREC != TC_E4M3) *reinterpret_cast<uint32_t*>(r.a + u * 2048u + byte) = v[i];
      if (r.mirror) *reinterpret_cast<uint32_t*>(r.mirror + u * r.mirror_unit + byte) = v[i];
    }
    w += 2;
    w -= w >= n_bins ? n_bins : 0;
  }
}

// Features [kb, ke) (multiples of 8) of one row.
template <int PREC>
HM_D void enc_units(const MlpDims& d, const float* __restrict__ xin, const float* __restrict__ enc_params, int kb,
                    int ke, const EncRow& r) {
  int done = kb;  // features before it are stored
  for (int si = 0; si < d.n_segs; ++si) {
    const EncSeg& s = d.segs[si];
    if (s.type == ENC_IDENTITY) break;  // the last segment, with the padding below
    const int lo = max(kb, s.out_off), hi = min(ke, s.out_off + s.n_out);
    if (lo >= hi) continue;
    done = hi;
    const float* x = xin + s.in_off;
    if (s.type == ENC_FREQUENCY) {
      const int u = (lo - s.out_off) >> 1;
      int dim = u / s.n_freq, f = u - dim * s.n_freq;
      float xs = x[dim], p2 = scale_pow2(1.f, f);
      for (int k = lo; k < hi; k += 8) {
        float v[8];
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          sincospif(xs * p2, &v[2 * t], &v[2 * t + 1]);
          p2 += p2;
          if (++f == s.n_freq) {
            f = 0;
            p2 = 1.f;
            xs = x[min(++dim, s.n_dims - 1)];
          }
        }
        enc_store8<PREC>(r, k, v);
      }
    } else if (s.type == ENC_ONEBLOB) {
      const int nb_i = s.n_bins;
      const float nb = (float)nb_i, inv_nb = 1.f / nb;
      const bool pow2 = (nb_i & (nb_i - 1)) == 0;  // then e * inv_nb is e / nb exactly
      auto edge = [&](int e) { return pow2 ? (float)e * inv_nb : (float)e / nb; };
      if (nb_i == 4) {  // two inputs per unit, every bin evaluated
        for (int k = lo; k < hi; k += 8) {
          const int dim = (k - s.out_off) >> 2;
          float v[8];
#pragma unroll
          for (int t = 0; t < 2; ++t) {
            const float c0 = oneblob_cdf(0.f, x[dim + t], nb);
            float left = c0;
#pragma unroll
            for (int b = 0; b < 4; ++b) {
              const float right = b == 3 ? c0 + 1.f : oneblob_cdf((float)(b + 1) * 0.25f, x[dim + t], nb);
              v[4 * t + b] = right - left;
              left = right;
            }
          }
          enc_store8<PREC>(r, k, v);
        }
        continue;
      }
      int dim = (lo - s.out_off) / nb_i;
      for (int k0 = s.out_off + dim * nb_i; k0 < hi; k0 += nb_i, ++dim) {
        const int klo = max(lo, k0), khi = min(hi, k0 + nb_i);
        const float zero[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        for (int k = klo; k < khi; k += 8) enc_store8<PREC>(r, k, zero);
        const float xv = x[dim];
        // bin of x on the period [0, 1) (x itself may lie outside it)
        int b0 = (int)floorf(xv * nb);
        b0 = pow2 ? b0 & (nb_i - 1) : (b0 % nb_i + nb_i) % nb_i;
        int first = b0 - 2;
        first += first < 0 ? nb_i : 0;
        // five masses from six edges; the edge after the last bin is edge 0
        // of the next period, one full mass on
        float m[5], left = oneblob_cdf(edge(first), xv, nb);
        int e = first;
#pragma unroll
        for (int t = 0; t < 5; ++t) {
          e = e + 1 == nb_i ? 0 : e + 1;
          const float c = oneblob_cdf(edge(e), xv, nb);
          m[t] = (e == 0 ? c + 1.f : c) - left;
          left = c;
        }
        enc_store_window<PREC>(r, k0, nb_i, first, m, klo, khi);
      }
    } else {  // hash grid, two features per entry, four levels per unit
      const float2* table = reinterpret_cast<const float2*>(enc_params + s.param_off);
      const float px = x[0], py = x[1], pz = x[2];
      for (int k = lo; k < hi; k += 8) {
        float v[8];
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          const int l = ((k - s.out_off) >> 1) + t;
          const float sc = s.level_scale[l];
          const float fx = fmaf(sc, px, 0.5f), fy = fmaf(sc, py, 0.5f), fz = fmaf(sc, pz, 0.5f);
          const float gx = floorf(fx), gy = floorf(fy), gz = floorf(fz);
          const float wx = fx - gx, wy = fy - gy, wz = fz - gz;
          uint32_t e[8];
          grid_entries(s, l, (uint32_t)(int)gx, (uint32_t)(int)gy, (uint32_t)(int)gz, e);
          float2 tv[8];  // eight gathers in flight
#pragma unroll
          for (int c = 0; c < 8; ++c) tv[c] = __ldg(table + e[c]);
          float a0 = 0.f, a1 = 0.f;
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            const float w = ((c & 1) ? wx : 1.f - wx) * (((c >> 1) & 1) ? wy : 1.f - wy) *
                            (((c >> 2) & 1) ? wz : 1.f - wz);
            a0 += w * tv[c].x;
            a1 += w * tv[c].y;
          }
          v[2 * t] = a0;
          v[2 * t + 1] = a1;
        }
        enc_store8<PREC>(r, k, v);
      }
    }
  }
  // identity inputs, then padding: 1 up to in_pad, 0 past it
  const EncSeg& s = d.segs[d.n_segs - 1];
  for (int k = done; k < ke; k += 8) {
    float v[8];
#pragma unroll
    for (int t = 0; t < 8; ++t) {
      const int f = k + t;
      v[t] = f < d.n_enc ? xin[s.in_off + f - s.out_off] : (f < d.in_pad ? 1.f : 0.f);
    }
    enc_store8<PREC>(r, k, v);
  }
}

// Upper bound of |feature| over the row (E4M3 input scale).
HM_D float enc_row_bound(const MlpDims& d, const float* __restrict__ xin, float grid_amax) {
  float m = 1.f;
  for (int si = 0; si < d.n_segs; ++si) {
    const EncSeg& s = d.segs[si];
    if (s.type == ENC_IDENTITY)
      for (int k = 0; k < s.n_dims; ++k) m = fmaxf(m, fabsf(xin[s.in_off + k]));
    else if (s.type == ENC_HASHGRID)
      m = fmaxf(m, grid_amax);
  }
  return m;
}

// --------------------------------------------------------------- the kernel
struct TcArgs {
  MlpDims d;
  const uint8_t* blob;
  int64_t blob_bytes;
  int64_t boff[16];
  int N[16], K[16];
  int n_layers;
  int kc0;  // layer-0 K chunk (elements)
  const float* scales;
  const float* enc_params;
  const float* in;
  float* out;
  int out_stride;
  int64_t n;
  int* err;  // host-mapped
  int a_bytes;
  int ncols;
  // training forward (STORE): operands kept for the backward pass
  uint16_t* x16;  // [n][K0]
  uint16_t* h16;  // [L][n][W]
  float* pred;    // [n][16]
  // inference with the encoding done beforehand by tc_encode_kernel: the
  // layer-0 operand of tile t is the tile_bytes at a_pre + t * tile_bytes, in
  // the MMA layout; E4M3 rows carry their activation scale in row_inv_pre
  const uint8_t* a_pre;
  const float* row_inv_pre;
  int64_t tile_bytes;
  // warp-specialised inference: shared-memory bytes of the weights, of one
  // layer-0 operand stage and of one hidden operand; number of stages
  int fz_w, fz_a0, fz_h, fz_stages;
  int units;  // enc_units_ok and the hash tables 8-byte aligned
};

// Encoding of every row into the layer-0 operand, in the MMA's shared-memory
// layout one tile after another, so the forward kernel loads a tile (or a K
// chunk of it) with one bulk copy.  One thread per row, 128 rows (one tile)
// per block: the 32 rows of a warp write each 16-byte group as four 128-byte
// runs.  Same arithmetic as the fused encoding (enc_range).
template <int PREC>
__global__ void __launch_bounds__(kTcRows) tc_encode_kernel(const __grid_constant__ TcArgs p, uint8_t* __restrict__ a_out,
                                                            float* __restrict__ row_inv_out) {
  const int row = threadIdx.x;
  const int64_t tile = blockIdx.x;
  const int64_t q = tile * kTcRows + row;
  const bool valid = q < p.n;
  const MlpDims& d = p.d;
  const float* xin = p.in + (valid ? q : 0) * d.in_ch;
  float row_scale = 1.f;
  if (PREC == TC_E4M3) {
    const float bound = valid ? enc_row_bound(d, xin, p.scales[15]) : 1.f;
    row_scale = kE4M3Max / bound;
    if (valid) row_inv_out[q] = bound / kE4M3Max;
  }
  const int K0 = p.K[0];
  if (valid && p.units) {
    enc_units<PREC>(d, xin, p.enc_params, 0, K0,
                    EncRow{a_out + tile * p.tile_bytes + op_offset(kTcRows, row, 0), nullptr, 0, row_scale});
    return;
  }
  RowPacker<PREC> pk(a_out + tile * p.tile_bytes, row, 0, row_scale);
  if (valid) {
    enc_range<PREC>(d, xin, p.enc_params, 0, K0, pk);
  } else {
    for (int k = 0; k < K0; ++k) pk.push(0.f);
  }
}

// 256 threads: thread (warp w, lane i) owns row 32 * (w % 4) + i of the tile
// (tensor-memory lanes are split by warp quadrant) and half h = w / 4 of the
// work on that row: every other 16-byte feature group when encoding, and
// accumulator columns [h * W/2, (h + 1) * W/2) in the epilogues.
template <int PREC, int W, bool STORE>
__global__ void __launch_bounds__(kTcThreads, 2) mlp_tc_fwd_kernel(const __grid_constant__ TcArgs p) {
  constexpr bool F8 = PREC == TC_E4M3;
  constexpr int EB = F8 ? 1 : 2;       // bytes per element
  constexpr int KI = 32 / EB;          // K per MMA instruction
  constexpr int CK = 16 / EB;          // elements per 16-byte core-matrix row
  constexpr int FMT = PREC == TC_BF16 ? 1 : 0;
  constexpr int HW = W / 2;            // accumulator columns per half
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* A = smem;
  uint8_t* Wt = smem + p.a_bytes;
  uint64_t* bar = reinterpret_cast<uint64_t*>(Wt + ((p.blob_bytes + 127) & ~(int64_t)127));
  uint64_t* bar_a = bar + 1;  // bulk copies of pre-encoded operands
  uint32_t* holder = reinterpret_cast<uint32_t*>(bar + 2);
  float* amax_x = reinterpret_cast<float*>(holder + 4);  // [2][128] E4M3 row maxima

  const int tid = threadIdx.x, warp = tid >> 5;
  const int row = ((warp & 3) << 5) | (tid & 31);
  const int half = warp >> 2;
  const MlpDims& d = p.d;
  const int L = p.n_layers - 1;  // index of the output layer

  for (int64_t i = tid; i < p.blob_bytes / 16; i += kTcThreads)
    reinterpret_cast<uint4*>(Wt)[i] = __ldg(reinterpret_cast<const uint4*>(p.blob) + i);
  if (tid == 0) {
    mbar_init(bar, 1);
    mbar_init(bar_a, 1);
    fence_mbar_init();
  }
  if (warp == 0) tmem_alloc(holder, p.ncols);
  fence_proxy_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *holder;
  const uint32_t row_taddr = tmem + ((uint32_t)((warp & 3) * 32) << 16);
  const uint32_t a_base = smem_u32(A), w_base = smem_u32(Wt);
  const uint32_t a_lbo = 16 * kTcRows;
  uint32_t phase = 0, phase_a = 0;
  bool failed = false;
  auto w_inv = [&](int l) { return F8 ? __ldg(p.scales + l) : 1.f; };
  const float grid_amax = F8 ? p.scales[15] : 0.f;

  // issue the MMAs of one layer (or layer-0 chunk) and wait for them
  auto run_layer = [&](int l, int k_begin, int k_count, bool accumulate_first) -> bool {
    if (tid == 0) {
      tc_fence_after();
      const uint32_t idesc = tc_idesc(kTcRows, p.N[l], FMT);
      const uint32_t b_lbo = 16 * p.N[l];
      const uint32_t b_base = w_base + (uint32_t)p.boff[l];
      for (int ks = 0; ks < k_count / KI; ++ks) {
        const uint64_t ad = tc_sdesc(a_base + (uint32_t)ks * 2 * a_lbo, a_lbo, 128);
        const uint64_t bd = tc_sdesc(b_base + (uint32_t)((k_begin / KI) + ks) * 2 * b_lbo, b_lbo, 128);
        tc_mma<F8>(tmem, ad, bd, idesc, (accumulate_first || ks > 0) ? 1u : 0u);
      }
      tc_commit(bar);
    }
    // thread 0 (which committed) polls the barrier; the others sleep in the
    // block barrier instead of spinning
    const bool ok = threadIdx.x == 0 ? mbar_wait_bounded(bar, phase) : true;
    phase ^= 1u;
    const bool bad = __syncthreads_or(!ok);
    tc_fence_after();
    return !bad;
  };

  const int64_t n_tiles = (p.n + kTcRows - 1) / kTcRows;
  for (int64_t tile = blockIdx.x; tile < n_tiles && !failed; tile += gridDim.x) {
    const int64_t q = tile * kTcRows + row;
    const bool valid = q < p.n;
    const float* xin = p.in + (valid ? q : 0) * d.in_ch;
    float row_inv = 1.f;  // 1 / activation scale of this row of A
    float row_scale = 1.f;
    if (F8) {
      if (p.a_pre) {
        row_inv = valid ? __ldg(p.row_inv_pre + q) : 1.f;
      } else {
        const float bound = valid ? enc_row_bound(d, xin, grid_amax) : 1.f;
        row_scale = kE4M3Max / bound;
        row_inv = bound / kE4M3Max;
      }
    }
    // ---- layer 0, in K chunks
    const int K0 = p.K[0];
    for (int kc = 0; kc < K0 && !failed; kc += p.kc0) {
      const int kn = min(p.kc0, K0 - kc);
      if (p.a_pre) {
        // the chunk's K range is one contiguous run of the tile in the MMA layout
        if (tid == 0) {
          fence_proxy_async_smem();  // the previous tile's epilogue wrote A through the generic proxy
          const uint32_t bytes = (uint32_t)(kn * EB * kTcRows);
          mbar_arrive_expect_tx(bar_a, bytes);
          bulk_copy_g2s(A, p.a_pre + tile * p.tile_bytes + (int64_t)kc * EB * kTcRows, bytes, bar_a);
        }
        const bool ok = tid == 0 ? mbar_wait_bounded(bar_a, phase_a) : true;
        phase_a ^= 1u;
        if (__syncthreads_or(!ok)) {
          failed = true;
          break;
        }
      } else {
        // the two halves of the row: groups [0, G/2) and [G/2, G) of the chunk
        const int G = kn / CK, gsplit = (G + 1) >> 1;
        const int g0 = half ? gsplit : 0, g1 = half ? G : gsplit;
        RowPacker<PREC> pk(A, row, g0, row_scale);
        if (STORE && valid) {
          if (F8)
            pk.mirror16 = p.x16 + q * K0 + kc;
          else
            pk.mirror = reinterpret_cast<uint8_t*>(p.x16 + q * K0 + kc);
        }
        if (valid && p.units) {
          EncRow r{A + op_offset(kTcRows, row, 0) - (size_t)(kc / CK) * 2048, nullptr, 16, row_scale};
          if (STORE) r.mirror = reinterpret_cast<uint8_t*>(p.x16 + q * K0);
          enc_units<PREC>(d, xin, p.enc_params, kc + g0 * CK, kc + g1 * CK, r);
        } else if (valid) {
          enc_range<PREC>(d, xin, p.enc_params, kc + g0 * CK, kc + g1 * CK, pk);
        } else {
          for (int k = g0 * CK; k < g1 * CK; ++k) pk.push(0.f);
        }
        fence_proxy_async_smem();
        __syncthreads();
      }
      if (!run_layer(0, kc, kn, kc > 0)) failed = true;
    }
    // ---- hidden epilogues and the following layers
    for (int l = 1; l <= L && !failed; ++l) {
      const float sc = row_inv * w_inv(l - 1);
      float v[HW];
#pragma unroll
      for (int c = 0; c < HW / 16; ++c) {
        float t[16];
        tmem_ld16(row_taddr + half * HW + c * 16, t);
#pragma unroll
        for (int e = 0; e < 16; ++e) v[c * 16 + e] = fmaxf(F8 ? t[e] * sc : t[e], 0.f);
      }
      if constexpr (HW == 8) {  // width 16: eight columns of one load each
        float t[16];
        tmem_ld16(row_taddr, t);
#pragma unroll
        for (int e = 0; e < 8; ++e) v[e] = fmaxf(half ? t[8 + e] : t[e], 0.f);
      }
      if (F8) {
        float amax = 0.f;
#pragma unroll
        for (int e = 0; e < HW; ++e) amax = fmaxf(amax, v[e]);
        amax_x[half * kTcRows + row] = amax;
        __syncthreads();
        amax = fmaxf(amax_x[row], amax_x[kTcRows + row]);
        const float s = amax > 0.f ? kE4M3Max / amax : 1.f;
        row_inv = amax > 0.f ? amax / kE4M3Max : 1.f;
#pragma unroll
        for (int g = 0; g < HW / 16; ++g) {
          uint32_t word[4];
#pragma unroll
          for (int w4 = 0; w4 < 4; ++w4)
            word[w4] = pack4_e4m3(v[g * 16 + 4 * w4] * s, v[g * 16 + 4 * w4 + 1] * s, v[g * 16 + 4 * w4 + 2] * s,
                                  v[g * 16 + 4 * w4 + 3] * s);
          *reinterpret_cast<uint4*>(A + op_offset(kTcRows, row, half * HW + g * 16)) =
              make_uint4(word[0], word[1], word[2], word[3]);
        }
        if (STORE && valid) {  // the backward pass's FP16 copy of the activations
#pragma unroll
          for (int g = 0; g < HW / 8; ++g) {
            uint32_t word[4];
#pragma unroll
            for (int w2 = 0; w2 < 4; ++w2) word[w2] = pack2<TC_FP16>(v[g * 8 + 2 * w2], v[g * 8 + 2 * w2 + 1]);
            *reinterpret_cast<uint4*>(p.h16 + ((int64_t)(l - 1) * p.n + q) * W + half * HW + g * 8) =
                make_uint4(word[0], word[1], word[2], word[3]);
          }
        }
      } else {
#pragma unroll
        for (int g = 0; g < HW / 8; ++g) {
          uint32_t word[4];
#pragma unroll
          for (int w2 = 0; w2 < 4; ++w2) word[w2] = pack2<PREC>(v[g * 8 + 2 * w2], v[g * 8 + 2 * w2 + 1]);
          *reinterpret_cast<uint4*>(A + op_offset(kTcRows, row, (half * HW + g * 8) * 2)) =
              make_uint4(word[0], word[1], word[2], word[3]);
          if (STORE && valid)
            *reinterpret_cast<uint4*>(p.h16 + ((int64_t)(l - 1) * p.n + q) * W + half * HW + g * 8) =
                make_uint4(word[0], word[1], word[2], word[3]);
        }
      }
      tc_fence_before();
      fence_proxy_async_smem();
      __syncthreads();
      if (!run_layer(l, 0, p.K[l], false)) failed = true;
    }
    if (failed) break;
    // ---- output layer accumulator -> out (columns 0..15, first half of the warps)
    if (half == 0) {
      float t[16];
      tmem_ld16(row_taddr, t);
      const float sc = row_inv * w_inv(L);
      if (valid) {
        if (STORE) {
#pragma unroll
          for (int o = 0; o < 16; ++o) p.pred[q * 16 + o] = t[o] * sc;
        } else {
#pragma unroll
          for (int o = 0; o < 16; ++o)
            if (o < d.out_ch && o < p.out_stride) p.out[q * p.out_stride + o] = t[o] * sc;
        }
      }
    }
    tc_fence_before();
    __syncthreads();
  }
  if (failed && tid == 0) atomicOr(p.err, 1);
  __syncthreads();
  tc_fence_after();
  if (warp == 0) tmem_dealloc(tmem, p.ncols);
}

// ---------------------------------------------- warp-specialised inference
// Encoding and layers overlapped inside one persistent CTA per SM (16-bit
// operands).  24 encoder warps write layer-0 operands into a ring of NS
// stages (each the whole K of one 128-row tile): they form NS teams of
// 4 * P warps, team t encoding the CTA's tiles k = t (mod NS) into stage t
// with P threads per row (each an equal contiguous range of the row's
// 16-byte feature groups; P = 6 / NS with NS 6 or 2, the most stages that
// fit next to the weights, so small operands get one thread per row as in
// tc_encode_kernel).  Two lanes of 4 layer warps walk the layers: lane s
// takes the tiles k = s (mod 2) (with NS even, stage t always feeds lane
// t % 2), with its own hidden operand H[s] (128 x W) and W columns of
// tensor memory; warp w reads tensor-memory lanes 32 * (w % 4) .. (one
// thread per row) and the lane's first thread issues the MMAs.  A team refills its stage as soon as the layer-0 MMAs of its
// previous tile have read it, so encoding runs while the layer warps walk
// layers 1..L, and the two lanes fill each other's waits.  Hand-offs:
// full[t] (team -> layer lane, one arrival after the team's named barrier),
// empty[t] (layer-0 MMAs done -> team), mma[s] (tcgen05.commit).  Every
// mbarrier wait is bounded; an expired wait is reduced over the waiting
// group through its named barrier, the group stops and the waits of the
// groups that depend on it then expire too.  The encoded operands, the MMAs
// and the epilogue arithmetic are those of mlp_tc_fwd_kernel, so the
// outputs are the same bits.
constexpr int kFzLanes = 2;
constexpr int kFzLayWarps = 4;   // per lane
constexpr int kFzEncWarps = 24;  // in all
constexpr int kFzLayThreads = kFzLanes * kFzLayWarps * 32;
constexpr int kFzThreads = kFzLayThreads + kFzEncWarps * 32;
constexpr int kFzMaxStages = kFzEncWarps / 4;
constexpr int kFzMisc = 128;  // 2 * kFzMaxStages + 2 mbarriers + the tensor-memory address

template <int PREC, int W>
__global__ void __launch_bounds__(kFzThreads, 1) mlp_tc_fused_kernel(const __grid_constant__ TcArgs p) {
  static_assert(PREC != TC_E4M3, "16-bit operands only");
  static_assert(8 * (2 * kFzMaxStages + 2) + 4 <= kFzMisc, "barrier area");
  constexpr int CK = 8;  // elements per 16-byte core-matrix row
  constexpr int FMT = PREC == TC_BF16 ? 1 : 0;
  extern __shared__ __align__(1024) uint8_t smem[];
  const int NS = p.fz_stages, P = kFzMaxStages / NS;
  uint8_t* Wt = smem;
  uint8_t* A0 = smem + p.fz_w;
  uint8_t* Hb = A0 + NS * p.fz_a0;
  uint64_t* bars = reinterpret_cast<uint64_t*>(Hb + kFzLanes * p.fz_h);
  uint64_t* full = bars;                 // [NS]
  uint64_t* empty = bars + kFzMaxStages;  // [NS]
  uint64_t* mma = bars + 2 * kFzMaxStages;  // [2]
  uint32_t* holder = reinterpret_cast<uint32_t*>(bars + 2 * kFzMaxStages + 2);

  const int tid = threadIdx.x, warp = tid >> 5, lane_id = tid & 31;
  const MlpDims& d = p.d;
  const int L = p.n_layers - 1;
  const int K0 = p.K[0];
  const int64_t n_tiles = (p.n + kTcRows - 1) / kTcRows;

  for (int64_t i = tid; i < p.blob_bytes / 16; i += kFzThreads)
    reinterpret_cast<uint4*>(Wt)[i] = __ldg(reinterpret_cast<const uint4*>(p.blob) + i);
  if (tid == 0) {
    for (int b = 0; b < 2 * kFzMaxStages + 2; ++b) mbar_init(bars + b, 1);
    fence_mbar_init();
  }
  if (warp == 0) tmem_alloc(holder, p.ncols);
  fence_proxy_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *holder;
  bool failed = false;

  if (tid < kFzLayThreads) {
    // ---------------- layer warps of lane s
    const int s = warp / kFzLayWarps, quad = warp % 4, row = quad * 32 + lane_id;
    const int bar_id = 1 + s;
    const bool leader = (warp % kFzLayWarps) == 0 && lane_id == 0;
    const uint32_t tm = tmem + (uint32_t)(s * W);
    const uint32_t row_taddr = tm + ((uint32_t)(quad * 32) << 16);
    uint8_t* Hs = Hb + s * p.fz_h;
    uint64_t* mma_s = mma + s;
    const uint32_t a_lbo = 16 * kTcRows;
    const uint32_t h_base = smem_u32(Hs), w_base = smem_u32(Wt);
    uint32_t ph_mma = 0;
    // the MMAs of layer l over A (k_count elements of K), committed to mma_s
    auto issue = [&](int l, uint32_t a_base, int k_count) {
      tc_fence_after();
      const uint32_t idesc = tc_idesc(kTcRows, p.N[l], FMT);
      const uint32_t b_lbo = 16 * p.N[l];
      uint64_t ad = tc_sdesc(a_base, a_lbo, 128);
      uint64_t bd = tc_sdesc(w_base + (uint32_t)p.boff[l], b_lbo, 128);
      for (int ks = 0; ks < k_count / 16; ++ks) {
        tc_mma<false>(tm, ad, bd, idesc, ks > 0 ? 1u : 0u);
        ad += 2 * a_lbo >> 4;  // the descriptors' start addresses, in 16-byte units
        bd += 2 * b_lbo >> 4;
      }
      tc_commit(mma_s);
    };
    for (int64_t k = s;; k += kFzLanes) {
      const int64_t tile = blockIdx.x + k * (int64_t)gridDim.x;
      if (tile >= n_tiles) break;
      const int st = (int)(k % NS);
      // every warp waits for the MMAs itself (a leader polling for the group
      // costs one more barrier per layer: 300 against 120 cycles).  A warp
      // whose wait expired goes on to the group's barriers without waiting
      // again, the leader's without issuing, and the group stops at the tile's
      // end.  ok is the same in all lanes of a warp.
      bool ok = true;
      if (leader) {
        ok = mbar_wait_bounded(full + st, (uint32_t)((k / NS) & 1));
        if (ok) issue(0, smem_u32(A0 + st * p.fz_a0), K0);
      }
      ok = __all_sync(0xffffffffu, ok) && mbar_wait_warp(mma_s, ph_mma);
      if (leader && ok) mbar_arrive(empty + st);  // the stage has been read
      ph_mma ^= 1u;
      tc_fence_after();
      for (int l = 1; l <= L; ++l) {
        // epilogue of layer l - 1: ReLU, rounded to the operand type, as the A of layer l
#pragma unroll
        for (int c = 0; c < W / 16; ++c) {
          float t[16];
          tmem_ld16(row_taddr + c * 16, t);
#pragma unroll
          for (int g = 0; g < 2; ++g) {
            uint32_t word[4];
#pragma unroll
            for (int w2 = 0; w2 < 4; ++w2)
              word[w2] = pack2<PREC>(fmaxf(t[g * 8 + 2 * w2], 0.f), fmaxf(t[g * 8 + 2 * w2 + 1], 0.f));
            *reinterpret_cast<uint4*>(Hs + op_offset(kTcRows, row, (c * 16 + g * 8) * 2)) =
                make_uint4(word[0], word[1], word[2], word[3]);
          }
        }
        tc_fence_before();
        fence_proxy_async_smem();
        group_sync(bar_id, kFzLayWarps * 32);
        if (leader && ok) issue(l, h_base, p.K[l]);
        __syncwarp();
        ok = ok && mbar_wait_warp(mma_s, ph_mma);
        ph_mma ^= 1u;
        tc_fence_after();
      }
      // output layer accumulator -> out
      float t[16];
      tmem_ld16(row_taddr, t);
      const int64_t q = tile * kTcRows + row;
      if (q < p.n && ok)
        for (int o = 0; o < d.out_ch && o < p.out_stride; ++o) p.out[q * p.out_stride + o] = t[o];
      // the next tile's layer-0 MMAs overwrite these columns
      tc_fence_before();
      if (group_sync_or(bar_id, kFzLayWarps * 32, !ok)) {
        failed = true;
        break;
      }
    }
  } else {
    // ---------------- encoder team t (4 * P warps)
    const int e = tid - kFzLayThreads;
    const int team = e / (kTcRows * P), et = e % (kTcRows * P);
    const int row = et % kTcRows, part = et / kTcRows;
    const int bar_id = 3 + team;
    const bool leader = et == 0;
    uint8_t* As = A0 + team * p.fz_a0;
    const int G = K0 / CK;
    const int g0 = part * G / P, g1 = (part + 1) * G / P;
    uint32_t ph_empty = 0;
    for (int64_t k = team;; k += NS) {
      const int64_t tile = blockIdx.x + k * (int64_t)gridDim.x;
      if (tile >= n_tiles) break;
      if (k >= NS) {  // wait until the layer-0 MMAs of the team's previous tile have read the stage
        const bool ok = leader ? mbar_wait_bounded(empty + team, ph_empty) : true;
        ph_empty ^= 1u;
        if (group_sync_or(bar_id, kTcRows * P, !ok)) {
          failed = true;
          break;
        }
      }
      const int64_t q = tile * kTcRows + row;
      RowPacker<PREC> pk(As, row, g0, 1.f);
      if (q < p.n && p.units) {
        enc_units<PREC>(d, p.in + q * d.in_ch, p.enc_params, g0 * CK, g1 * CK,
                        EncRow{As + op_offset(kTcRows, row, 0), nullptr, 0, 1.f});
      } else if (q < p.n) {
        enc_range<PREC>(d, p.in + q * d.in_ch, p.enc_params, g0 * CK, g1 * CK, pk);
      } else {
        for (int kk = g0 * CK; kk < g1 * CK; ++kk) pk.push(0.f);
      }
      fence_proxy_async_smem();
      group_sync(bar_id, kTcRows * P);
      if (leader) mbar_arrive(full + team);
    }
  }
  if (failed && lane_id == 0) atomicOr(p.err, 1);
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 0) tmem_dealloc(tmem, p.ncols);
}

// ------------------------------------------------------------ weight packing
// All layers in one launch: blockIdx.y the layer, blockIdx.z 0 for the
// forward operand, 1 for the transposed one of the backward pass (a launch
// per layer and direction cost 36 us before every training step of the
// 5 x 64 network, one costs 4).
struct TcPackArgs {
  MlpDims d;
  const float* params;
  int n_layers;
  int N[16], K[16], NT[16], KT[16];
  int64_t boff[16], boff_t[16];
  uint8_t* blob;
  uint8_t* blob_t;  // W_l^T: element (n = input, k = output) of layer l
  float* scales;    // [16] weight scales (E4M3; [15]: hash-grid amax)
  const uint32_t* amax;  // [16] largest |weight| as float bits, from tc_amax_kernel
};

// E4M3: amax of layer blockIdx.y's weights, blockIdx.y == n_layers: of the
// encoding parameters (as integers: the bits of non-negative floats order as
// the floats do, so the result does not depend on the blocks' order).
__global__ void __launch_bounds__(256) tc_amax_kernel(const __grid_constant__ MlpDims d,
                                                      const float* __restrict__ params, int n_layers,
                                                      uint32_t* __restrict__ amax) {
  __shared__ float red[8];
  const int l = blockIdx.y;
  int64_t begin, count;
  if (l < n_layers) {
    const int fan_in = l == 0 ? d.in_pad : d.width;
    const int fan_out = l == n_layers - 1 ? d.out_pad : d.width;
    begin = d.layer_off[l];
    count = (int64_t)fan_in * fan_out;
  } else {
    begin = d.n_net_params;
    count = d.n_enc_params;
  }
  float m = 0.f;
  for (int64_t i = blockIdx.x * 256 + threadIdx.x; i < count; i += (int64_t)gridDim.x * 256)
    m = fmaxf(m, fabsf(params[begin + i]));
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; ++w) m = fmaxf(m, red[w]);
    if (m > 0.f) atomicMax(amax + (l < n_layers ? l : 15), __float_as_uint(m));
  }
}

template <int PREC>
__global__ void __launch_bounds__(256) tc_pack_kernel(const __grid_constant__ TcPackArgs p) {
  const int l = blockIdx.y;
  const int64_t i = blockIdx.x * 256 + threadIdx.x;
  const int fan_in = l == 0 ? p.d.in_pad : p.d.width;
  const float* W = p.params + p.d.layer_off[l];
  if (blockIdx.z == 1) {  // transposed, FP16 / BF16
    if (i >= (int64_t)p.NT[l] * p.KT[l]) return;
    const int n = (int)(i / p.KT[l]), k = (int)(i % p.KT[l]);
    const float w = n < fan_in ? W[(int64_t)k * fan_in + n] : 0.f;
    uint8_t* dst = p.blob_t + p.boff_t[l] + op_offset(p.NT[l], n, 2 * k);
    if (PREC == TC_BF16)
      *reinterpret_cast<__nv_bfloat16*>(dst) = __float2bfloat16_rn(w);
    else
      *reinterpret_cast<__half*>(dst) = __float2half_rn(w);
    return;
  }
  const int N = p.N[l], K = p.K[l];
  float scale = 1.f;
  if (PREC == TC_E4M3) {
    const float m = __uint_as_float(p.amax[l]);
    scale = m > 0.f ? m / kE4M3Max : 1.f;
    if (i == 0) p.scales[l] = scale;
    if (i == 0 && l == 0) p.scales[15] = __uint_as_float(p.amax[15]);
  }
  if (i >= (int64_t)N * K) return;
  const int n = (int)(i / K), k = (int)(i % K);
  const float w = k < fan_in ? W[(int64_t)n * fan_in + k] : 0.f;
  uint8_t* blob = p.blob + p.boff[l];
  if (PREC == TC_E4M3) {
    const float s = 1.f / scale;
    const uint32_t v = __nv_cvt_float2_to_fp8x2(make_float2(w * s, 0.f), __NV_SATFINITE, __NV_E4M3);
    blob[op_offset(N, n, k)] = (uint8_t)(v & 0xFF);
  } else if (PREC == TC_BF16) {
    *reinterpret_cast<__nv_bfloat16*>(blob + op_offset(N, n, 2 * k)) = __float2bfloat16_rn(w);
  } else {
    *reinterpret_cast<__half*>(blob + op_offset(N, n, 2 * k)) = __float2half_rn(w);
  }
}

// ------------------------------------------------------------------ host API
static int tc_kinst(int precision) { return precision == HM_PREC_FP8_E4M3 ? 32 : 16; }
static int round_up(int x, int m) { return (x + m - 1) / m * m; }

bool tc_supported(const MlpDims& d, int precision, std::string* why) {
  if (precision != HM_PREC_FP16 && precision != HM_PREC_BF16 && precision != HM_PREC_FP8_E4M3) {
    if (why) *why = "unknown precision";
    return false;
  }
  if (precision == HM_PREC_FP8_E4M3 && d.width < 32) {
    if (why) *why = "E4M3 needs n_neurons >= 32 (K of one MMA is 32)";
    return false;
  }
  if (d.n_hidden + 1 > 15) {
    if (why) *why = "too many layers";
    return false;
  }
  TcPack pk;
  pk.precision = precision;
  pk.elem_bytes = precision == HM_PREC_FP8_E4M3 ? 1 : 2;
  const int KI = tc_kinst(precision);
  int64_t blob = 0;
  for (int l = 0; l <= d.n_hidden; ++l) {
    const int N = l == d.n_hidden ? d.out_pad : d.width;
    const int K = round_up(l == 0 ? d.in_pad : d.width, KI);
    blob += (int64_t)N * K * pk.elem_bytes;
  }
  const int64_t a_min = (int64_t)kTcRows * std::max(KI, d.width) * pk.elem_bytes;
  if (((blob + 127) & ~127) + a_min + 1152 > kTcSmemMax) {
    if (why) *why = "weights do not fit in shared memory";
    return false;
  }
  return true;
}

int tc_pack_alloc(const MlpDims& d, int precision, TcPack* pk) {
  pk->precision = precision;
  pk->elem_bytes = precision == HM_PREC_FP8_E4M3 ? 1 : 2;
  pk->kinst = tc_kinst(precision);
  pk->n_layers = d.n_hidden + 1;
  int64_t off = 0;
  for (int l = 0; l < pk->n_layers; ++l) {
    pk->N[l] = l == d.n_hidden ? d.out_pad : d.width;
    pk->K[l] = round_up(l == 0 ? d.in_pad : d.width, pk->kinst);
    pk->boff[l] = off;
    off += (int64_t)pk->N[l] * pk->K[l] * pk->elem_bytes;
  }
  pk->bytes = off;
  cudaError_t e = cudaMalloc(&pk->blob, (size_t)off);
  if (e == cudaSuccess) e = cudaMalloc(&pk->scales, 32 * sizeof(float));  // [16..31]: amax bits
  if (e == cudaSuccess && tc_trainable(d, precision)) {
    int64_t ot = 0;
    for (int l = 0; l < pk->n_layers; ++l) {
      pk->NT[l] = pk->K[l];  // the layer's inputs
      pk->KT[l] = pk->N[l];  // the layer's outputs
      pk->boff_t[l] = ot;
      ot += (int64_t)pk->NT[l] * pk->KT[l] * 2;
    }
    pk->bytes_t = ot;
    e = cudaMalloc(&pk->blob_t, (size_t)ot);
  }
  if (e != cudaSuccess) return hm_cuda_status(e, "tensor-core weight blob");
  cudaMemset(pk->scales, 0, 32 * sizeof(float));
  return HM_OK;
}

void tc_pack_free(TcPack* pk) {
  cudaFree(pk->blob);
  cudaFree(pk->scales);
  cudaFree(pk->blob_t);
  pk->blob = nullptr;
  pk->scales = nullptr;
  pk->blob_t = nullptr;
}

int tc_pack(const MlpDims& d, const float* params, TcPack& pk, cudaStream_t st) {
  TcPackArgs a;
  memset(&a, 0, sizeof(a));
  a.d = d;
  a.params = params;
  a.n_layers = pk.n_layers;
  a.blob = pk.blob;
  a.blob_t = pk.blob_t;
  a.scales = pk.scales;
  uint32_t* amax = reinterpret_cast<uint32_t*>(pk.scales + 16);
  a.amax = amax;
  int64_t most = 1;
  for (int l = 0; l < pk.n_layers; ++l) {
    a.N[l] = pk.N[l];
    a.K[l] = pk.K[l];
    a.boff[l] = pk.boff[l];
    a.NT[l] = pk.NT[l];
    a.KT[l] = pk.KT[l];
    a.boff_t[l] = pk.boff_t[l];
    most = std::max(most, (int64_t)pk.N[l] * pk.K[l]);
  }
  if (pk.precision == HM_PREC_FP8_E4M3) {
    cudaError_t e = cudaMemsetAsync(amax, 0, 16 * sizeof(uint32_t), st);
    if (e != cudaSuccess) return hm_cuda_status(e, "weight scales");
    // encoding parameters: 64 blocks (one block of 256 threads took 0.3 ms for
    // the renderer's million)
    tc_amax_kernel<<<dim3(64, pk.n_layers + (d.n_enc_params > 0 ? 1 : 0)), 256, 0, st>>>(d, params, pk.n_layers, amax);
    HM_CHECK_LAUNCH("tc_amax_kernel");
  }
  const dim3 grid((unsigned)((most + 255) / 256), (unsigned)pk.n_layers, pk.blob_t ? 2 : 1);
  if (pk.precision == HM_PREC_FP8_E4M3)
    tc_pack_kernel<TC_E4M3><<<grid, 256, 0, st>>>(a);
  else if (pk.precision == HM_PREC_BF16)
    tc_pack_kernel<TC_BF16><<<grid, 256, 0, st>>>(a);
  else
    tc_pack_kernel<TC_FP16><<<grid, 256, 0, st>>>(a);
  HM_CHECK_LAUNCH("tc_pack_kernel");
  return HM_OK;
}

template <int PREC, int W, bool STORE = false>
static int tc_launch(const TcArgs& a, size_t smem, cudaStream_t st) {
  auto kern = mlp_tc_fwd_kernel<PREC, W, STORE>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, (int)cudaSharedmemCarveoutMaxShared);
  if (e != cudaSuccess) return hm_cuda_status(e, "mlp_tc_fwd_kernel smem");
  int dev = 0, sms = 0, smem_sm = 0, smem_res = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev);
  cudaDeviceGetAttribute(&smem_res, cudaDevAttrReservedSharedMemoryPerBlock, dev);
  cudaFuncAttributes fa;
  cudaFuncGetAttributes(&fa, kern);
  int per_sm = smem_sm / (int)(smem + smem_res);
  per_sm = std::min(per_sm, 65536 / std::max(1, fa.numRegs * kTcThreads));
  per_sm = std::max(1, std::min(per_sm, 512 / a.ncols));  // tensor-memory columns per SM
  const int64_t tiles = (a.n + kTcRows - 1) / kTcRows;
  const int blocks = (int)std::min<int64_t>(tiles, (int64_t)sms * per_sm);
  kern<<<blocks, kTcThreads, smem, st>>>(a);
  HM_CHECK_LAUNCH("mlp_tc_fwd_kernel");
  return HM_OK;
}

static int tc_args(const MlpDims& d, const TcPack& pk, const float* enc_params, const float* in, float* out,
                   int out_stride, int64_t n, int* err_flag, TcArgs* ap, size_t* smem_out) {
  TcArgs& a = *ap;
  memset(&a, 0, sizeof(a));
  a.d = d;
  a.blob = pk.blob;
  a.blob_bytes = pk.bytes;
  for (int l = 0; l < 16; ++l) {
    a.boff[l] = l < pk.n_layers ? pk.boff[l] : 0;
    a.N[l] = l < pk.n_layers ? pk.N[l] : 0;
    a.K[l] = l < pk.n_layers ? pk.K[l] : 0;
  }
  a.n_layers = pk.n_layers;
  a.units = enc_units_ok(d) && (reinterpret_cast<uintptr_t>(enc_params) & 7) == 0;
  for (int si = 0; si < d.n_segs; ++si)
    if (d.segs[si].type == ENC_HASHGRID && d.segs[si].param_off % 2 != 0) a.units = 0;
  a.scales = pk.scales;
  a.enc_params = enc_params;
  a.in = in;
  a.out = out;
  a.out_stride = out_stride;
  a.n = n;
  a.err = err_flag;
  int ncols = 32;
  while (ncols < std::max(d.width, 16)) ncols *= 2;
  a.ncols = ncols;
  // shared memory: A tile + weights + barrier
  const int eb = pk.elem_bytes;
  const int64_t wbytes = (pk.bytes + 127) & ~(int64_t)127;
  const int64_t misc = 1152;  // barrier, tensor-memory address, E4M3 row maxima
  auto a_bytes_for = [&](int kc) { return (int64_t)kTcRows * std::max(kc, d.width) * eb; };
  auto total = [&](int kc) { return a_bytes_for(kc) + wbytes + misc; };
  // prefer a layer-0 chunk that leaves room for two CTAs per SM
  const int64_t two_per_sm = 113 * 1024;
  int kc0 = pk.K[0];
  while (total(kc0) > two_per_sm && kc0 > pk.kinst) kc0 -= pk.kinst;
  if (total(kc0) > two_per_sm) {
    kc0 = pk.K[0];
    while (total(kc0) > kTcSmemMax && kc0 > pk.kinst) kc0 -= pk.kinst;
  }
  if (total(kc0) > kTcSmemMax) return hm_set_error("mlp: tensor-core tile does not fit"), HM_EUNSUPPORTED;
  a.kc0 = kc0;
  a.a_bytes = (int)a_bytes_for(kc0);
  *smem_out = (size_t)(a.a_bytes + wbytes + misc);
  return HM_OK;
}

int64_t tc_encode_bytes(const MlpDims& d, const TcPack& pk, int64_t n) {
  const int64_t tiles = (n + kTcRows - 1) / kTcRows;
  const int64_t tile_bytes = (int64_t)kTcRows * pk.K[0] * pk.elem_bytes;
  return tiles * tile_bytes + (pk.precision == HM_PREC_FP8_E4M3 ? ((n * 4 + 255) & ~(int64_t)255) : 0);
}

// Form of the 16-bit inferences: 0 automatic (below), 1 never the
// warp-specialised kernel, 2 only it (HM_EUNSUPPORTED where it does not
// fit).  Set by hm_debug_tc_path.
static int g_tc_path = 0;

// Shared memory of mlp_tc_fused_kernel (0: the network does not fit it).
static int64_t tc_fused_smem(const MlpDims& d, const TcPack& pk, TcArgs* a) {
  if (pk.precision == HM_PREC_FP8_E4M3 || (d.width != 32 && d.width != 64) || pk.N[pk.n_layers - 1] > d.width)
    return 0;
  const int64_t w = (pk.bytes + 1023) & ~(int64_t)1023;
  const int64_t a0 = (int64_t)kTcRows * pk.K[0] * 2;
  const int64_t h = (int64_t)kTcRows * d.width * 2;
  // the most stages (the fewest encoder threads per row) that fit; an even
  // count, so that each stage is read by one layer lane only and every
  // parity wait on it is for the phase after the one that lane last saw
  for (int ns : {6, 2}) {
    const int64_t total = w + ns * a0 + kFzLanes * h + kFzMisc;
    if (total > kTcSmemMax) continue;
    if (a) {
      a->fz_w = (int)w;
      a->fz_a0 = (int)a0;
      a->fz_h = (int)h;
      a->fz_stages = ns;
    }
    return total;
  }
  return 0;
}

template <int PREC, int W>
static int tc_fused_launch(const TcArgs& a, size_t smem, cudaStream_t st) {
  auto kern = mlp_tc_fused_kernel<PREC, W>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return hm_cuda_status(e, "mlp_tc_fused_kernel smem");
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int64_t tiles = (a.n + kTcRows - 1) / kTcRows;
  const int blocks = (int)std::min<int64_t>(tiles, (int64_t)sms);
  kern<<<blocks, kFzThreads, smem, st>>>(a);
  HM_CHECK_LAUNCH("mlp_tc_fused_kernel");
  return HM_OK;
}

bool tc_wants_workspace(const MlpDims& d, const TcPack& pk) {
  return g_tc_path != 2 && (g_tc_path == 1 || tc_fused_smem(d, pk, nullptr) == 0);
}

int tc_forward(const MlpDims& d, const TcPack& pk, const float* enc_params, const float* in, float* out,
               int out_stride, int64_t n, int* err_flag, cudaStream_t st, uint8_t* work, int64_t work_bytes) {
  if (n <= 0) return HM_OK;
  TcArgs a;
  size_t smem = 0;
  if (int e = tc_args(d, pk, enc_params, in, out, out_stride, n, err_flag, &a, &smem)) return e;
  const bool have_work = work && work_bytes >= tc_encode_bytes(d, pk, n);
  // The warp-specialised kernel wherever it fits, from the measured times
  // (FP16, width 64; 517 / 65,536 / 2^20 queries): 16 / 26 / 240 us on the
  // Frequency / OneBlob network and 17 / 35 / 347 us on the hash grid, against
  // 23 / 34 / 308 and 18 / 38 / 404 us for the encode kernel + layer kernel
  // and 18 / 32 / 335 and 18 / 61 / 666 us for the layer kernel encoding its
  // own tiles.
  const bool want_fz = g_tc_path != 1;
  if (want_fz) {
    const int64_t fz = tc_fused_smem(d, pk, &a);
    if (fz > 0) {
      // both lanes' accumulators
      int ncols = 32;
      while (ncols < 2 * d.width) ncols *= 2;
      a.ncols = ncols;
      if (pk.precision == HM_PREC_BF16)
        return d.width == 32 ? tc_fused_launch<TC_BF16, 32>(a, (size_t)fz, st)
                             : tc_fused_launch<TC_BF16, 64>(a, (size_t)fz, st);
      return d.width == 32 ? tc_fused_launch<TC_FP16, 32>(a, (size_t)fz, st)
                           : tc_fused_launch<TC_FP16, 64>(a, (size_t)fz, st);
    }
    if (g_tc_path == 2) return hm_set_error("mlp: the warp-specialised kernel does not fit this network"), HM_EUNSUPPORTED;
  }
  if (have_work) {
    // encode every row first (high occupancy, no tensor work), then the
    // layers with the layer-0 operand loaded by bulk copies
    const int64_t tiles = (n + kTcRows - 1) / kTcRows;
    a.tile_bytes = (int64_t)kTcRows * pk.K[0] * pk.elem_bytes;
    float* row_inv = pk.precision == HM_PREC_FP8_E4M3 ? reinterpret_cast<float*>(work + tiles * a.tile_bytes)
                                                      : nullptr;
    if (pk.precision == HM_PREC_BF16)
      tc_encode_kernel<TC_BF16><<<(unsigned)tiles, kTcRows, 0, st>>>(a, work, row_inv);
    else if (pk.precision == HM_PREC_FP16)
      tc_encode_kernel<TC_FP16><<<(unsigned)tiles, kTcRows, 0, st>>>(a, work, row_inv);
    else
      tc_encode_kernel<TC_E4M3><<<(unsigned)tiles, kTcRows, 0, st>>>(a, work, row_inv);
    HM_CHECK_LAUNCH("tc_encode_kernel");
    a.a_pre = work;
    a.row_inv_pre = row_inv;
  }
  const int W = d.width;
  switch (pk.precision) {
    case HM_PREC_BF16:
      return W == 16 ? tc_launch<TC_BF16, 16>(a, smem, st) : W == 32 ? tc_launch<TC_BF16, 32>(a, smem, st)
             : W == 64 ? tc_launch<TC_BF16, 64>(a, smem, st) : tc_launch<TC_BF16, 128>(a, smem, st);
    case HM_PREC_FP16:
      return W == 16 ? tc_launch<TC_FP16, 16>(a, smem, st) : W == 32 ? tc_launch<TC_FP16, 32>(a, smem, st)
             : W == 64 ? tc_launch<TC_FP16, 64>(a, smem, st) : tc_launch<TC_FP16, 128>(a, smem, st);
    default:
      return W == 32 ? tc_launch<TC_E4M3, 32>(a, smem, st) : W == 64 ? tc_launch<TC_E4M3, 64>(a, smem, st)
             : tc_launch<TC_E4M3, 128>(a, smem, st);
  }
}

// =================================================================== training
// E4M3 handles train with the E4M3 forward (the operands inference uses)
// and the FP16 backward (dgrad chain and weight gradients on FP16 operands:
// the activations and encoded inputs kept as FP16, W^T packed as FP16).
bool tc_trainable(const MlpDims& d, int precision) {
  return ((precision == HM_PREC_FP16 || precision == HM_PREC_BF16) && d.width >= 16) ||
         (precision == HM_PREC_FP8_E4M3 && d.width >= 32);
}

int tc_train_alloc(const MlpDims& d, int64_t cap, bool need_dx, TcTrainBufs* b) {
  tc_train_free(b);
  const int L = d.n_hidden;
  const int wz = std::max(d.width, 16);
  // encoded inputs at the widest layer-0 pitch (E4M3 pads K to 32)
  cudaError_t e = cudaMalloc(&b->x16, (size_t)cap * round_up(d.in_pad, 32) * 2);
  if (e == cudaSuccess) e = cudaMalloc(&b->h16, (size_t)L * cap * d.width * 2);
  if (e == cudaSuccess) e = cudaMalloc(&b->dz16, (size_t)(L + 1) * cap * wz * 2);
  if (e == cudaSuccess) e = cudaMalloc(&b->pred, (size_t)cap * 16 * sizeof(float));
  if (e == cudaSuccess && need_dx) e = cudaMalloc(&b->dX, (size_t)cap * d.in_pad * sizeof(float));
  if (e == cudaSuccess) e = cudaMalloc(&b->loss_part, 4096 * sizeof(float));
  if (e != cudaSuccess) {
    tc_train_free(b);
    return hm_cuda_status(e, "tensor-core training buffers");
  }
  b->cap = cap;
  return HM_OK;
}

void tc_train_free(TcTrainBufs* b) {
  cudaFree(b->x16);
  cudaFree(b->h16);
  cudaFree(b->dz16);
  cudaFree(b->pred);
  cudaFree(b->dX);
  cudaFree(b->loss_part);
  *b = TcTrainBufs{};
}

int tc_train_forward(const MlpDims& d, const TcPack& pk, const float* enc_params, const float* in, int64_t n,
                     const TcTrainBufs& b, int* err_flag, cudaStream_t st) {
  if (n <= 0) return HM_OK;
  TcArgs a;
  size_t smem = 0;
  if (int e = tc_args(d, pk, enc_params, in, nullptr, 16, n, err_flag, &a, &smem)) return e;
  a.x16 = b.x16;
  a.h16 = b.h16;
  a.pred = b.pred;
  const int W = d.width;
  if (pk.precision == HM_PREC_FP8_E4M3)
    return W == 32 ? tc_launch<TC_E4M3, 32, true>(a, smem, st) : W == 64 ? tc_launch<TC_E4M3, 64, true>(a, smem, st)
           : tc_launch<TC_E4M3, 128, true>(a, smem, st);
  if (pk.precision == HM_PREC_BF16)
    return W == 16 ? tc_launch<TC_BF16, 16, true>(a, smem, st) : W == 32 ? tc_launch<TC_BF16, 32, true>(a, smem, st)
           : W == 64 ? tc_launch<TC_BF16, 64, true>(a, smem, st) : tc_launch<TC_BF16, 128, true>(a, smem, st);
  return W == 16 ? tc_launch<TC_FP16, 16, true>(a, smem, st) : W == 32 ? tc_launch<TC_FP16, 32, true>(a, smem, st)
         : W == 64 ? tc_launch<TC_FP16, 64, true>(a, smem, st) : tc_launch<TC_FP16, 128, true>(a, smem, st);
}

// ---- backward: loss gradient and the dgrad chain, one 128-row tile at a time
// dZ_{L+1} = loss gradient x loss_scale (16 columns); for j = L .. 1:
// dH_j = dZ_{j+1} W_j (A = dZ_{j+1}, B = W_j^T, accumulator in tensor memory),
// dZ_j = dH_j where h_j > 0; and dX = dZ_1 W_0 when the encoding has
// parameters.  Every dZ is rounded to the operand type, kept in shared memory
// as the next A operand and written out for the weight gradients.
struct TcBwdArgs {
  MlpDims d;
  const uint8_t* blob_t;
  int64_t blob_bytes;
  int64_t boff_t[16];
  int NT[16], KT[16];
  int L;
  const uint16_t* h16;
  uint16_t* dz16;
  const float* pred;
  const float* target;
  float* dX;
  float* loss_part;
  int loss;
  float inv_total, loss_scale;
  int64_t n;
  int* err;
  int a_bytes;
  int ncols;
  int wz;  // row pitch of dz16 (max(W, 16))
};

constexpr int kTcMaxN = 256;  // columns of one MMA

template <int PREC, int W>
__global__ void __launch_bounds__(kTcThreads, 1) mlp_tc_bwd_kernel(const __grid_constant__ TcBwdArgs p) {
  constexpr int FMT = PREC == TC_BF16 ? 1 : 0;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* A = smem;
  uint8_t* Wt = smem + p.a_bytes;
  uint64_t* bar = reinterpret_cast<uint64_t*>(Wt + ((p.blob_bytes + 127) & ~(int64_t)127));
  uint32_t* holder = reinterpret_cast<uint32_t*>(bar + 1);
  float* red = reinterpret_cast<float*>(holder + 4);  // [256] loss partials

  const int tid = threadIdx.x, warp = tid >> 5;
  const int row = ((warp & 3) << 5) | (tid & 31);
  const int half = warp >> 2;
  const MlpDims& d = p.d;
  const int L = p.L;
  for (int64_t i = tid; i < p.blob_bytes / 16; i += kTcThreads)
    reinterpret_cast<uint4*>(Wt)[i] = __ldg(reinterpret_cast<const uint4*>(p.blob_t) + i);
  if (tid == 0) {
    mbar_init(bar, 1);
    fence_mbar_init();
  }
  if (warp == 0) tmem_alloc(holder, p.ncols);
  fence_proxy_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *holder;
  const uint32_t row_taddr = tmem + ((uint32_t)((warp & 3) * 32) << 16);
  const uint32_t a_base = smem_u32(A), w_base = smem_u32(Wt);
  const uint32_t a_lbo = 16 * kTcRows;
  uint32_t phase = 0;
  bool failed = false;
  float loss_acc = 0.f;

  // MMAs of columns [n0, n0 + n_count) of dH_j = dZ_{j+1} W_j
  auto run = [&](int j, int k_count, int n0, int n_count) -> bool {
    if (tid == 0) {
      tc_fence_after();
      const uint32_t idesc = tc_idesc(kTcRows, n_count, FMT);
      const uint32_t b_lbo = 16 * p.NT[j];
      const uint32_t b_base = w_base + (uint32_t)p.boff_t[j] + (uint32_t)op_offset(p.NT[j], n0, 0);
      for (int ks = 0; ks < k_count / 16; ++ks) {
        const uint64_t ad = tc_sdesc(a_base + (uint32_t)ks * 2 * a_lbo, a_lbo, 128);
        const uint64_t bd = tc_sdesc(b_base + (uint32_t)ks * 2 * b_lbo, b_lbo, 128);
        tc_mma<false>(tmem, ad, bd, idesc, ks > 0 ? 1u : 0u);
      }
      tc_commit(bar);
    }
    // thread 0 (which committed) polls the barrier; the others sleep in the
    // block barrier instead of spinning
    const bool ok = threadIdx.x == 0 ? mbar_wait_bounded(bar, phase) : true;
    phase ^= 1u;
    const bool bad = __syncthreads_or(!ok);
    tc_fence_after();
    return !bad;
  };

  const int64_t n_tiles = (p.n + kTcRows - 1) / kTcRows;
  for (int64_t tile = blockIdx.x; tile < n_tiles && !failed; tile += gridDim.x) {
    const int64_t q = tile * kTcRows + row;
    const bool valid = q < p.n;
    // ---- loss gradient (half 0 of each row): dZ_{L+1}, 16 columns
    if (half == 0) {
      float g[16], pr[16];
#pragma unroll
      for (int o = 0; o < 16; ++o) {
        g[o] = 0.f;
        pr[o] = valid ? p.pred[q * 16 + o] : 0.f;
      }
      if (valid) {
        float tg[16];
        for (int o = 0; o < d.out_ch; ++o) tg[o] = __ldg(p.target + q * d.out_ch + o);
        float v = 0.f;
        loss_grad(p.loss, pr, tg, d.out_ch, p.inv_total, g, &v);
        loss_acc += v;
      }
      uint32_t word[8];
#pragma unroll
      for (int w2 = 0; w2 < 8; ++w2) word[w2] = pack2<PREC>(g[2 * w2] * p.loss_scale, g[2 * w2 + 1] * p.loss_scale);
      *reinterpret_cast<uint4*>(A + op_offset(kTcRows, row, 0)) = make_uint4(word[0], word[1], word[2], word[3]);
      *reinterpret_cast<uint4*>(A + op_offset(kTcRows, row, 16)) = make_uint4(word[4], word[5], word[6], word[7]);
      if (valid) {
        uint4* dst = reinterpret_cast<uint4*>(p.dz16 + ((int64_t)L * p.n + q) * p.wz);
        dst[0] = make_uint4(word[0], word[1], word[2], word[3]);
        dst[1] = make_uint4(word[4], word[5], word[6], word[7]);
      }
    }
    fence_proxy_async_smem();
    __syncthreads();
    int kk = 16;  // K of the next MMA: columns of the dZ in A
    for (int j = L; j >= 0 && !failed; --j) {
      if (j == 0) {
        // dX (loss-scaled, FP32) for the hash-grid backward, 256 columns (the
        // widest MMA) at a time
        if (!p.dX) break;
        for (int n0 = 0; n0 < p.NT[0] && !failed; n0 += kTcMaxN) {
          const int nt = min(kTcMaxN, p.NT[0] - n0);
          if (!run(0, kk, n0, nt)) {
            failed = true;
            break;
          }
          for (int c = half * 16; c < nt; c += 32) {
            float t[16];
            tmem_ld16(row_taddr + c, t);
            if (valid)
              for (int e = 0; e < 16 && n0 + c + e < d.in_pad; ++e) p.dX[q * d.in_pad + n0 + c + e] = t[e];
          }
          tc_fence_before();
          __syncthreads();
        }
      } else {
        if (!run(j, kk, 0, W)) {
          failed = true;
          break;
        }
        constexpr int HW = W / 2;
        const uint16_t* hrow = p.h16 + ((int64_t)(j - 1) * p.n + (valid ? q : 0)) * W + half * HW;
        if constexpr (HW == 8) {  // width 16: eight columns of one load each
          float t[16];
          tmem_ld16(row_taddr, t);
          const uint4 hv = valid ? __ldg(reinterpret_cast<const uint4*>(hrow)) : make_uint4(0, 0, 0, 0);
          const uint16_t* hs = reinterpret_cast<const uint16_t*>(&hv);
          float g[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            const float te = half ? t[8 + e] : t[e];
            g[e] = hs[e] != 0 && !(hs[e] & 0x8000) ? te : 0.f;
          }
          const uint4 word = make_uint4(pack2<PREC>(g[0], g[1]), pack2<PREC>(g[2], g[3]), pack2<PREC>(g[4], g[5]),
                                        pack2<PREC>(g[6], g[7]));
          *reinterpret_cast<uint4*>(A + op_offset(kTcRows, row, half * 16)) = word;
          if (valid) *reinterpret_cast<uint4*>(p.dz16 + ((int64_t)(j - 1) * p.n + q) * p.wz + half * 8) = word;
        }
#pragma unroll
        for (int c = 0; c < HW / 16; ++c) {
          float t[16];
          tmem_ld16(row_taddr + half * HW + c * 16, t);
          uint4 hv[2];
          hv[0] = valid ? __ldg(reinterpret_cast<const uint4*>(hrow + c * 16)) : make_uint4(0, 0, 0, 0);
          hv[1] = valid ? __ldg(reinterpret_cast<const uint4*>(hrow + c * 16 + 8)) : make_uint4(0, 0, 0, 0);
          const uint16_t* hs = reinterpret_cast<const uint16_t*>(hv);
          uint32_t word[8];
#pragma unroll
          for (int w2 = 0; w2 < 8; ++w2) {
            const float a0 = hs[2 * w2] != 0 && !(hs[2 * w2] & 0x8000) ? t[2 * w2] : 0.f;
            const float a1 = hs[2 * w2 + 1] != 0 && !(hs[2 * w2 + 1] & 0x8000) ? t[2 * w2 + 1] : 0.f;
            word[w2] = pack2<PREC>(a0, a1);
          }
          const int col = half * HW + c * 16;
          *reinterpret_cast<uint4*>(A + op_offset(kTcRows, row, col * 2)) =
              make_uint4(word[0], word[1], word[2], word[3]);
          *reinterpret_cast<uint4*>(A + op_offset(kTcRows, row, col * 2 + 16)) =
              make_uint4(word[4], word[5], word[6], word[7]);
          if (valid) {
            uint4* dst = reinterpret_cast<uint4*>(p.dz16 + ((int64_t)(j - 1) * p.n + q) * p.wz + col);
            dst[0] = make_uint4(word[0], word[1], word[2], word[3]);
            dst[1] = make_uint4(word[4], word[5], word[6], word[7]);
          }
        }
        kk = W;
      }
      tc_fence_before();
      fence_proxy_async_smem();
      __syncthreads();
    }
  }
  // per-CTA loss partial, fixed order
  red[tid] = loss_acc;
  __syncthreads();
  if (tid == 0) {
    float s = 0.f;
    for (int i = 0; i < kTcThreads; ++i) s += red[i];
    p.loss_part[blockIdx.x] = s;
  }
  if (failed && tid == 0) atomicOr(p.err, 1);
  __syncthreads();
  tc_fence_after();
  if (warp == 0) tmem_dealloc(tmem, p.ncols);
}

// ---- weight gradients of every layer: dW[o][i] = sum over rows dZ[row][o] h[row][i]
// One launch: blockIdx.y is a job (a layer's outputs x a tile of its
// inputs), blockIdx.x a chunk of 2048 rows.  A CTA accumulates its chunk in
// tensor memory (A = dZ^T, padded to 128 outputs, B = h^T, K = the rows) and
// writes an FP32 partial; wgrad_sum_kernel sums the partials in chunk
// order.  The tensor cores truncate when they accumulate, so the chunk fixes
// the sums' last digits; what fills the GPU is the tile of inputs (see
// tc_backward), which changes no bit.
//
// dZ and h lie row by row in memory, so both operands are read as MN-major
// (the feature index contiguous): core matrices of 8 rows (k) x 8 features
// (16 bytes per row), element (feature f, row k) of a stage at
//   (f / 8) * kWgGroup + (k / 8) * 128 + (k % 8) * 16 + (f % 8) * 2.
// A 16-byte piece of a row is copied as it is (cp.async), without the 2-byte
// transposes a K-major operand needs.  A feature group is padded by 16 bytes
// so that the pieces of one row fall into different banks.
// Bound by the serial chain over a chunk (32 stages of 64 rows); a ring of
// four stages keeps three stages' copies in flight under the MMAs.  With a
// launch and a reduction per layer, 32 CTAs each and 2-byte transposing stores
// a FP16 step on 65,536 rows of the 5 x 64 network, gradients read back, took
// 958 us, with this 319 (and 232 with the weights packed in one launch as well).
constexpr int kWgRows = 64;                            // rows of a stage
constexpr int kWgGroup = kWgRows / 8 * 128 + 16;       // bytes of one 8-feature group of a stage
constexpr int kWgStages = 4;
constexpr int kWgMaxJobs = 128;
constexpr int64_t kWgChunk = 2048;                     // rows summed in tensor memory

struct TcWgradJob {
  const uint16_t* dz;  // [n][dz_pitch], columns = outputs
  const uint16_t* h;   // [n][h_pitch], from the job's first input column
  int h_pitch;
  int n_out, n_in;     // n_in: multiple of 16, <= 256
  int ld;              // row pitch of the layer's partial
  int64_t part;        // the job's first element inside a chunk's partial
};
struct TcWgradArgs {
  TcWgradJob job[kWgMaxJobs];
  int dz_pitch;
  int64_t n, chunk;
  float* part;         // [chunks][part_stride]
  int64_t part_stride;
  int* err;
  int ncols, stage_bytes;
};

template <int PREC>
__global__ void __launch_bounds__(kTcThreads) mlp_tc_wgrad_kernel(const __grid_constant__ TcWgradArgs p) {
  constexpr int FMT = PREC == TC_BF16 ? 1 : 0;
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ __align__(8) uint64_t bar[kWgStages];
  __shared__ uint32_t holder;
  const TcWgradJob& J = p.job[blockIdx.y];
  const int tid = threadIdx.x, warp = tid >> 5;
  const int ga = J.n_out / 8, gb = J.n_in / 8;  // 16-byte pieces of a row of dZ and of h
  constexpr int kAGroups = kTcRows / 8;
  // A's feature groups beyond the layer's outputs stay zero
  for (int st = 0; st < kWgStages; ++st) {
    uint4* z = reinterpret_cast<uint4*>(smem + st * p.stage_bytes + ga * kWgGroup);
    for (int i = tid; i < (kAGroups - ga) * (kWgGroup / 16); i += kTcThreads) z[i] = make_uint4(0, 0, 0, 0);
  }
  if (tid == 0) {
    for (int st = 0; st < kWgStages; ++st) mbar_init(bar + st, 1);
    fence_mbar_init();
  }
  if (warp == 0) tmem_alloc(&holder, p.ncols);
  fence_proxy_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = holder;
  const uint32_t s_base = smem_u32(smem);
  const int64_t r0 = blockIdx.x * p.chunk, r1 = min(p.n, r0 + p.chunk);
  const int iters = (int)((r1 - r0 + kWgRows - 1) / kWgRows);  // >= 1: the grid has no empty chunk
  auto load = [&](int it) {
    const uint32_t a = s_base + (uint32_t)((it % kWgStages) * p.stage_bytes), b = a + kAGroups * kWgGroup;
    const int64_t q0 = r0 + (int64_t)it * kWgRows;
    for (int i = tid; i < kWgRows * ga; i += kTcThreads) {
      const int k = i / ga, g = i - k * ga;
      const bool ok = q0 + k < r1;
      cp_async16(a + g * kWgGroup + k * 16, J.dz + (ok ? q0 + k : r0) * p.dz_pitch + g * 8, ok);
    }
    for (int i = tid; i < kWgRows * gb; i += kTcThreads) {
      const int k = i / gb, g = i - k * gb;
      const bool ok = q0 + k < r1;
      cp_async16(b + g * kWgGroup + k * 16, J.h + (ok ? q0 + k : r0) * J.h_pitch + g * 8, ok);
    }
  };
  const uint32_t idesc = tc_idesc(kTcRows, J.n_in, FMT) | (1u << 15) | (1u << 16);  // A and B MN-major
  bool failed = false;
  // one cp.async group per step, empty past the end, so that the group to
  // wait for is always the third newest
  for (int it = 0; it < kWgStages - 1; ++it) {
    if (it < iters) load(it);
    cp_async_commit();
  }
  for (int it = 0; it < iters; ++it) {
    const int st = it % kWgStages;
    cp_async_wait<kWgStages - 2>();
    fence_proxy_async_smem();
    __syncthreads();
    bool ok = true;
    if (tid == 0) {
      tc_fence_after();
      const uint32_t a = s_base + (uint32_t)(st * p.stage_bytes), b = a + kAGroups * kWgGroup;
      for (int ks = 0; ks < kWgRows / 16; ++ks)
        tc_mma<false>(tmem, tc_sdesc(a + ks * 256, 128, kWgGroup), tc_sdesc(b + ks * 256, 128, kWgGroup), idesc,
                      (it > 0 || ks > 0) ? 1u : 0u);
      tc_commit(bar + st);
      // the stage to refill was read by the MMAs of step it - 1
      if (it >= 1) ok = mbar_wait_bounded(bar + (it - 1) % kWgStages, (uint32_t)(((it - 1) / kWgStages) & 1));
    }
    if (__syncthreads_or(!ok)) {
      failed = true;
      break;
    }
    if (it + kWgStages - 1 < iters) load(it + kWgStages - 1);
    cp_async_commit();
  }
  if (!failed) {  // the last step's MMAs (a commit covers all earlier ones)
    const int last = iters - 1;
    const bool ok =
        tid == 0 ? mbar_wait_bounded(bar + last % kWgStages, (uint32_t)((last / kWgStages) & 1)) : true;
    failed = __syncthreads_or(!ok);
  }
  cp_async_wait<0>();
  tc_fence_after();
  // row o of the accumulator (tensor-memory lane o) -> the partial; the two
  // halves of the block take alternate 16-column pieces
  if (!failed) {
    const int o = (warp & 3) * 32 + (tid & 31);
    const uint32_t taddr = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    float* dst = p.part + blockIdx.x * p.part_stride + J.part + (int64_t)o * J.ld;
    for (int c = (warp >> 2) * 16; c < J.n_in; c += 32) {
      float t[16];
      tmem_ld16(taddr + c, t);
      if (o < J.n_out)
#pragma unroll
        for (int e = 0; e < 16; e += 4)
          *reinterpret_cast<float4*>(dst + c + e) = make_float4(t[e], t[e + 1], t[e + 2], t[e + 3]);
    }
  }
  if (failed && tid == 0) atomicOr(p.err, 1);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 0) tmem_dealloc(tmem, p.ncols);
}

// Sums the chunks' partials in chunk order into the matrix gradients of
// every layer.  A partial's rows are ld[l] wide, the parameters' fan_in wide
// (they differ in the E4M3 layer 0, whose K is padded).  One block more than
// the gradients need sums the blocks' losses, in block order (a launch of one
// thread reading them from memory took 6 us).
__global__ void __launch_bounds__(128) wgrad_sum_kernel(const __grid_constant__ WgradSum p,
                                                        const float* __restrict__ part, float* __restrict__ out,
                                                        const float* __restrict__ loss_part, int n_loss,
                                                        float* __restrict__ loss_out) {
  if (blockIdx.x == gridDim.x - 1) {
    __shared__ float v[1024];
    float s = 0.f;
    for (int base = 0; base < n_loss; base += 1024) {
      const int m = min(1024, n_loss - base);
      for (int i = threadIdx.x; i < m; i += 128) v[i] = loss_part[base + i];
      __syncthreads();
      if (threadIdx.x == 0)
        for (int i = 0; i < m; ++i) s += v[i];
      __syncthreads();
    }
    if (threadIdx.x == 0) *loss_out = s;
    return;
  }
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= p.goff[p.n_layers]) return;
  int l = 0;
  while (l + 1 < p.n_layers && i >= p.goff[l + 1]) ++l;
  const int64_t j = i - p.goff[l];
  const float* src = part + p.poff[l] + (j / p.fan_in[l]) * p.ld[l] + j % p.fan_in[l];
  float s = 0.f;
#pragma unroll 16
  for (int k = 0; k < p.chunks; ++k) s += __ldg(src + k * p.stride);
  out[i] = s;
}

int wgrad_sum(const WgradSum& r, const float* part, float* grads, const float* loss_part, int n_loss, float* loss_out,
              cudaStream_t st) {
  wgrad_sum_kernel<<<(unsigned)((r.goff[r.n_layers] + 127) / 128 + 1), 128, 0, st>>>(r, part, grads, loss_part, n_loss,
                                                                                    loss_out);
  HM_CHECK_LAUNCH("wgrad_sum_kernel");
  return HM_OK;
}

template <int PREC, int W>
static int tc_bwd_launch(const TcBwdArgs& a, size_t smem, cudaStream_t st, int* blocks_out) {
  auto kern = mlp_tc_bwd_kernel<PREC, W>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return hm_cuda_status(e, "mlp_tc_bwd_kernel smem");
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int64_t tiles = (a.n + kTcRows - 1) / kTcRows;
  const int blocks = (int)std::min<int64_t>(std::min<int64_t>(tiles, sms), 4096);
  kern<<<blocks, kTcThreads, smem, st>>>(a);
  HM_CHECK_LAUNCH("mlp_tc_bwd_kernel");
  *blocks_out = blocks;
  return HM_OK;
}

int tc_backward(const MlpDims& d, const TcPack& pk, const TcTrainBufs& b, const float* target, int loss,
                float loss_scale, int64_t n, float* loss_out, float* grads, float** dw_part, int64_t* dw_cap,
                int* err_flag, cudaStream_t st) {
  if (n <= 0) return HM_OK;
  const int L = d.n_hidden;
  const int W = d.width;
  TcBwdArgs a;
  memset(&a, 0, sizeof(a));
  a.d = d;
  a.blob_t = pk.blob_t;
  // layer 0's transposed block (dX) is only loaded when the encoding needs it
  const bool need_dx = b.dX != nullptr;
  a.blob_bytes = need_dx ? pk.bytes_t : pk.bytes_t;
  for (int l = 0; l < 16; ++l) {
    a.boff_t[l] = l < pk.n_layers ? pk.boff_t[l] : 0;
    a.NT[l] = l < pk.n_layers ? pk.NT[l] : 0;
    a.KT[l] = l < pk.n_layers ? pk.KT[l] : 0;
  }
  a.L = L;
  a.h16 = b.h16;
  a.dz16 = b.dz16;
  a.pred = b.pred;
  a.target = target;
  a.dX = b.dX;
  a.loss_part = b.loss_part;
  a.loss = loss;
  a.inv_total = 1.f / ((float)n * (float)d.out_ch);
  a.loss_scale = loss_scale;
  a.n = n;
  a.err = err_flag;
  a.wz = std::max(W, 16);
  int ncols = 32;
  while (ncols < std::max(W, need_dx ? std::min(pk.NT[0], kTcMaxN) : 16)) ncols *= 2;
  a.ncols = ncols;
  a.a_bytes = kTcRows * std::max(W, 16) * 2;
  const size_t smem = (size_t)a.a_bytes + ((pk.bytes_t + 127) & ~(int64_t)127) + 64 + 1024 + 64;
  if (smem > (size_t)kTcSmemMax) return hm_set_error("mlp: backward tile does not fit"), HM_EUNSUPPORTED;
  int blocks = 0;
  int s = HM_OK;
  if (pk.precision == HM_PREC_BF16)
    s = W == 16 ? tc_bwd_launch<TC_BF16, 16>(a, smem, st, &blocks) : W == 32 ? tc_bwd_launch<TC_BF16, 32>(a, smem, st, &blocks)
        : W == 64 ? tc_bwd_launch<TC_BF16, 64>(a, smem, st, &blocks) : tc_bwd_launch<TC_BF16, 128>(a, smem, st, &blocks);
  else
    s = W == 16 ? tc_bwd_launch<TC_FP16, 16>(a, smem, st, &blocks) : W == 32 ? tc_bwd_launch<TC_FP16, 32>(a, smem, st, &blocks)
        : W == 64 ? tc_bwd_launch<TC_FP16, 64>(a, smem, st, &blocks) : tc_bwd_launch<TC_FP16, 128>(a, smem, st, &blocks);
  if (s) return s;
  // weight gradients: jobs of one layer x a tile of its inputs.  64 inputs
  // per tile; 32 while that still gives at most one CTA per SM.  A whole
  // step, FP16, tiles of 256 / 128 / 64 / 32 inputs: 5 x 64 network, 65,536
  // rows 207 / 206 / 189 / 223 us, 16,384 rows 125 / 113 / 101 / 96 us, 2,048
  // rows 123 / 111 / 101 / 96 us; 5 x 128, 16,384 rows 160 / 144 / 134 / 152 us.
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int chunks = (int)((n + kWgChunk - 1) / kWgChunk);
  auto count_jobs = [&](int t) {
    int c = 0;
    for (int l = 0; l <= L; ++l) c += (pk.K[l] + t - 1) / t;
    return c;
  };
  int tile = chunks * (int64_t)count_jobs(32) <= sms ? 32 : 64;
  while (count_jobs(tile) > kWgMaxJobs && tile < 256) tile *= 2;
  const int wz = std::max(W, 16);
  for (int l0 = 0, l1; l0 <= L; l0 = l1) {
    // layers l0 .. l1 - 1: as many as the partials' limit takes
    auto part = [&](int l) { return (int64_t)pk.N[l] * pk.K[l]; };
    int64_t stride = part(l0);
    for (l1 = l0 + 1; l1 <= L && chunks * (stride + part(l1)) <= kDwPartMax; ++l1) stride += part(l1);
    TcWgradArgs g;
    memset(&g, 0, sizeof(g));
    WgradSum r{};
    int jobs = 0, max_in = 0;
    int64_t poff = 0;
    for (int l = l0; l < l1; ++l) {
      const int N = pk.N[l], K = pk.K[l];
      for (int c = 0; c < K; c += tile) {
        if (jobs == kWgMaxJobs) return hm_set_error("mlp: too many weight-gradient tiles"), HM_EUNSUPPORTED;
        TcWgradJob& j = g.job[jobs++];
        j.dz = b.dz16 + (int64_t)l * n * wz;
        j.h = (l == 0 ? b.x16 : b.h16 + (int64_t)(l - 1) * n * W) + c;
        j.h_pitch = l == 0 ? K : W;
        j.n_out = N;
        j.n_in = std::min(tile, K - c);
        j.ld = K;
        j.part = poff + c;
        max_in = std::max(max_in, j.n_in);
      }
      // the layer's weights are [out][fan_in] with fan_in <= K[l]
      r.goff[l - l0] = d.layer_off[l] - d.layer_off[l0];
      r.poff[l - l0] = poff;
      r.fan_in[l - l0] = l == 0 ? d.in_pad : W;
      r.ld[l - l0] = K;
      poff += part(l);
    }
    r.n_layers = l1 - l0;
    r.goff[l1 - l0] = (l1 <= L ? d.layer_off[l1] : d.n_net_params) - d.layer_off[l0];
    r.stride = stride;
    r.chunks = chunks;
    const int64_t need = (int64_t)chunks * stride;
    if (need > *dw_cap) {
      cudaFree(*dw_part);
      *dw_part = nullptr;
      *dw_cap = 0;
      cudaError_t e = cudaMalloc(dw_part, need * sizeof(float));
      if (e != cudaSuccess) return hm_cuda_status(e, "tensor-core dW partials");
      *dw_cap = need;
    }
    g.dz_pitch = wz;
    g.n = n;
    g.chunk = kWgChunk;
    g.part = *dw_part;
    g.part_stride = stride;
    g.err = err_flag;
    g.ncols = 32;
    while (g.ncols < max_in) g.ncols *= 2;
    g.stage_bytes = (kTcRows / 8 + max_in / 8) * kWgGroup;
    const size_t sm = (size_t)kWgStages * g.stage_bytes;
    auto kern = pk.precision == HM_PREC_BF16 ? mlp_tc_wgrad_kernel<TC_BF16> : mlp_tc_wgrad_kernel<TC_FP16>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (e != cudaSuccess) return hm_cuda_status(e, "mlp_tc_wgrad_kernel smem");
    kern<<<dim3((unsigned)chunks, (unsigned)jobs), kTcThreads, sm, st>>>(g);
    HM_CHECK_LAUNCH("mlp_tc_wgrad_kernel");
    if (int s = wgrad_sum(r, *dw_part, grads + d.layer_off[l0], b.loss_part, blocks, loss_out, st)) return s;
  }
  return HM_OK;
}

// ---- the bounded wait's expiry, exercised on purpose (tests)
// One block: thread 0 sets up an mbarrier that expects one arrival, which
// never comes, and waits on it with the kernels' bounded wait, `limit`
// tries; the expiry is recorded in err and the kernel returns.  Any other
// outcome (the wait completing) is recorded as 2.
__global__ void tc_wait_expiry_kernel(uint32_t limit, int* err) {
  __shared__ __align__(8) uint64_t bar;
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    fence_mbar_init();
    *err = mbar_wait_bounded(&bar, 0u, limit) ? 2 : 1;
  }
}

}  // namespace hm

extern "C" int hm_debug_tc_path(int path) {
  if (path < 0 || path > 2) return hm_set_error("hm_debug_tc_path: path out of range"), HM_EINVAL;
  hm::g_tc_path = path;
  return HM_OK;
}

extern "C" int hm_debug_wait_expiry(int tries, void* stream) {
  if (tries < 1 || tries > (1 << 20)) return hm_set_error("hm_debug_wait_expiry: tries out of range"), HM_EINVAL;
  int* d = nullptr;
  cudaError_t e = cudaMalloc(&d, sizeof(int));
  if (e != cudaSuccess) return hm_cuda_status(e, "hm_debug_wait_expiry");
  cudaMemsetAsync(d, 0, sizeof(int), (cudaStream_t)stream);
  hm::tc_wait_expiry_kernel<<<1, 32, 0, (cudaStream_t)stream>>>((uint32_t)tries, d);
  int h = 0;
  e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaMemcpyAsync(&h, d, sizeof(int), cudaMemcpyDeviceToHost, (cudaStream_t)stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize((cudaStream_t)stream);
  cudaFree(d);
  if (e != cudaSuccess) return hm_cuda_status(e, "hm_debug_wait_expiry");
  if (h == 1) return hm_set_error("hm_debug_wait_expiry: the bounded wait expired"), HM_ETIMEOUT;
  return hm_set_error("hm_debug_wait_expiry: the wait did not expire (%d)", h), HM_EINVAL;
}
