// The matrices of an FP32 network as three BF16 planes (hm_mlp_x3.cu): where a
// weight's planes lie, for the kernels that write weights.
#pragma once
#include <cuda_bf16.h>

#include "hm_mlp.cuh"
#include "hm_tc.cuh"

namespace hm {

struct X3Planes {
  uint8_t* blob;  // NULL: no planes to keep
  int64_t layer_off[16];
  int64_t n_net_params;
  int n_hidden, in_pad, width, out_pad;
};

inline X3Planes x3_planes(const MlpDims& d, uint8_t* blob) {
  X3Planes p{};
  p.blob = blob;
  for (int l = 0; l <= d.n_hidden; ++l) p.layer_off[l] = d.layer_off[l];
  p.n_net_params = d.n_net_params;
  p.n_hidden = d.n_hidden;
  p.in_pad = d.in_pad;
  p.width = d.width;
  p.out_pad = d.out_pad;
  return p;
}

// Matrix parameter i = v.  K step after K step of a layer: [w0 | w1 | w2] rows
// of one 16-wide step as core matrices.
HM_D void x3_store(const X3Planes& p, int64_t i, float v) {
  int l = 0;
  while (l < p.n_hidden && i >= p.layer_off[l + 1]) ++l;
  const int K = l == 0 ? p.in_pad : p.width, N = l == p.n_hidden ? p.out_pad : p.width;
  const int64_t j = i - p.layer_off[l];
  const int o = (int)(j / K), k = (int)(j % K);
  uint8_t* step = p.blob + 6 * p.layer_off[l] + (int64_t)(k / 16) * (3 * N * 32);
#pragma unroll
  for (int pl = 0; pl < 3; ++pl) {
    const __nv_bfloat16 h = __float2bfloat16_rn(v);
    *reinterpret_cast<__nv_bfloat16*>(step + op_offset(3 * N, pl * N + o, (k % 16) * 2)) = h;
    v -= __bfloat162float(h);
  }
}

}  // namespace hm
