// FP32 inference of the radiance-cache network on the tensor cores.
//
// An FP32 value is the exact sum of three BF16 values (8 significand bits
// each, FP32's exponent range): v = b0 + b1 + b2 with b0 = bf16(v), b1 =
// bf16(v - b0), b2 = bf16(v - b0 - b1), each difference exact (the split of
// Henry, Tang and Heinecke, ARITH 2019).  A layer's product is formed from the
// six partial products whose weight is at least 2^-16 of the first, in three
// FP32 accumulators:
//   D0 = a0 w0,   D1 = a0 w1 + a1 w0,   D2 = a0 w2 + a1 w1 + a2 w0
// and h = D0 + (D1 + D2).  What is left out, a1 w2 and a2 w1 above all, is below
// 2^-24 of |a||w|.  The tensor cores truncate when they accumulate, so D0 is
// kept as two sums, of the even and of the odd 16-wide K steps: half the
// truncations in each.  With the planes of W side by side as rows of one B
// operand, a K step is
//   a0 x [w0 | w1 | w2] -> [D0 | D1 | D2]         (even steps)
//   a0 x w0 -> D0', a0 x [w1 | w2] -> [D1 | D2]   (odd steps)
//   a1 x [w0 | w1] -> [D1 | D2],  a2 x w0 -> D2.
// Error against 64 bits on the same encoded inputs, rms over the outputs' rms
// (FP32 multiply-adds in input order -> here): 5 x 64 network 2.1e-7 ->
// 1.3e-7, 5 x 128 3.2e-7 -> 2.0e-7, the renderer's grid network 2.2e-7 ->
// 1.7e-7, 1 x 16 8.2e-8 -> 5.2e-8, 14 x 64 7.0e-7 -> 3.3e-7.  With one sum D0
// the 5 x 128 network was at 3.7e-7.
//
// One CTA walks 128-query tiles.  Its eight compute warps (two threads per
// row) write A (a K chunk of the encoded input, then each hidden layer's
// activations, split into planes), warp 8 streams the packed weights through a
// ring of shared-memory slots by bulk copies, warp 9 issues the MMAs.  The
// weights of one tile come from L2 again for every tile (190 KB for the 5 x 64
// network do not fit next to A).  Hand-offs: a_ready (eight warps -> issuer),
// d_done (tcgen05.commit -> compute), w_full / w_empty per slot.  The compute
// warps and the issuer alternate, so every parity wait is for the phase after
// the one last seen; two CTAs per SM (width <= 64) fill each other's waits.
// Every wait is bounded; an expired one ends its role, the others' waits then
// expire too, and the block reports it and returns.
//
// Bound by the chain of a tile (A written, MMAs, accumulators read) with two
// CTAs to fill it: 39% of the issue slots and 20% of the tensor pipe used.  The
// renderer's network, 262,144 queries: 246 us with FP32 multiply-adds -> 64;
// whole calls, 200,003 queries: 5 x 64 network 1344 -> 220 us, 5 x 128 3025 ->
// 388.
#include <cuda_bf16.h>

#include <string.h>

#include <algorithm>

#include "hm_mlp.cuh"
#include "hm_tc.cuh"
#include "hm_x3.cuh"

namespace hm {

constexpr int kX3Compute = 256;               // compute threads
constexpr int kX3Threads = kX3Compute + 64;   // + the weight warp and the MMA warp
constexpr int kX3Slots = 4;                   // weight slots of 32 K each

struct X3Args {
  MlpDims d;
  const float* params;
  const uint8_t* blob;
  const float* X;  // [n][in_pad] encoded inputs
  float* out;
  int out_stride, out_ch;
  int in_pad, L;  // L: index of the output layer
  int64_t n;
  int* err;
  int ka;          // K of the A buffer
  int slot_bytes, a_plane;
};

// The MMAs of K step `step` of a layer: a = first byte of plane 0's step, b =
// the step's B block ([w0 | w1 | w2], N rows each).  Columns: D0, D1, D2, D0'.
template <int N>
HM_D void x3_mma(uint32_t tmem, uint32_t a, uint32_t a_plane, uint32_t b, int step) {
  constexpr uint32_t kALbo = 16 * kTcRows, kBLbo = 16 * 3 * N, kPlane = 16 * N;  // bytes between B's planes
  const uint64_t a0 = tc_sdesc(a, kALbo, 128), a1 = tc_sdesc(a + a_plane, kALbo, 128),
                 a2 = tc_sdesc(a + 2 * a_plane, kALbo, 128);
  const uint64_t b0 = tc_sdesc(b, kBLbo, 128);
  if (step & 1) {
    tc_mma<false>(tmem + 3 * N, a0, b0, tc_idesc(kTcRows, N, 1), step > 1 ? 1u : 0u);
    tc_mma<false>(tmem + N, a0, tc_sdesc(b + kPlane, kBLbo, 128), tc_idesc(kTcRows, 2 * N, 1), 1u);
  } else if constexpr (3 * N <= 256) {
    tc_mma<false>(tmem, a0, b0, tc_idesc(kTcRows, 3 * N, 1), step > 0 ? 1u : 0u);
  } else {
    tc_mma<false>(tmem, a0, b0, tc_idesc(kTcRows, 2 * N, 1), step > 0 ? 1u : 0u);
    tc_mma<false>(tmem + 2 * N, a0, tc_sdesc(b + 2 * kPlane, kBLbo, 128), tc_idesc(kTcRows, N, 1),
                  step > 0 ? 1u : 0u);
  }
  tc_mma<false>(tmem + N, a1, b0, tc_idesc(kTcRows, 2 * N, 1), 1u);
  tc_mma<false>(tmem + 2 * N, a2, b0, tc_idesc(kTcRows, N, 1), 1u);
}

// 16 columns of a layer of N outputs from column col on; two: the layer has
// odd K steps.
template <int N>
HM_D void x3_sum16(uint32_t row_taddr, int col, bool two, float (&v)[16]) {
  float t[16], u[16];
  tmem_ld16(row_taddr + N + col, t);
  tmem_ld16(row_taddr + 2 * N + col, u);
#pragma unroll
  for (int e = 0; e < 16; ++e) t[e] += u[e];
  tmem_ld16(row_taddr + col, v);
  if (two) {
    tmem_ld16(row_taddr + 3 * N + col, u);
#pragma unroll
    for (int e = 0; e < 16; ++e) v[e] += u[e];
  }
#pragma unroll
  for (int e = 0; e < 16; ++e) v[e] += t[e];
}

// Rows that the planes cannot carry are computed again with multiply-adds
// (x3_plain_row): those with an input of at least kX3Huge, and those with a sum
// that is not finite.  An infinity or NaN among a row's inputs, activations or
// weights, a value that rounds to infinity in BF16 (inf - inf in the next
// plane) and a partial sum that overflows all leave such a sum; the
// multiply-adds may have a number or an infinity there.
constexpr float kX3Huge = 1e30f;
// Their first output until then: a NaN that arithmetic does not produce.
constexpr uint32_t kX3Mark = 0x7fc05a5au;

// Eight values as three planes' 16-byte groups at dst + plane * a_plane.
HM_D void x3_split8(const float (&v)[8], uint8_t* dst, uint32_t a_plane) {
  uint32_t w[3][4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float x = v[2 * i], y = v[2 * i + 1];
#pragma unroll
    for (int p = 0; p < 3; ++p) {
      const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
      const uint32_t bits = *reinterpret_cast<const uint32_t*>(&h);
      w[p][i] = bits;
      x -= __uint_as_float(bits << 16);
      y -= __uint_as_float(bits & 0xffff0000u);
    }
  }
#pragma unroll
  for (int p = 0; p < 3; ++p)
    *reinterpret_cast<uint4*>(dst + p * a_plane) = make_uint4(w[p][0], w[p][1], w[p][2], w[p][3]);
}

// One query layer by layer with FP32 multiply-adds in input order, by one warp
// (a lane has every 32nd output of a layer); h: 2 * 128 floats of the warp's.
static __device__ __noinline__ void x3_plain_row(const MlpDims& d, const float* __restrict__ params,
                                                 const float* __restrict__ x, float* h, float* __restrict__ out,
                                                 int out_ch) {
  const int lane = threadIdx.x & 31;
  for (int l = 0; l <= d.n_hidden; ++l) {
    const int K = l == 0 ? d.in_pad : d.width, N = l == d.n_hidden ? out_ch : d.width;
    const float* src = l == 0 ? x : h + (l & 1) * 128;
    for (int o = lane; o < N; o += 32) {
      const float* w = params + d.layer_off[l] + (int64_t)o * K;
      float acc = 0.f;
      for (int k = 0; k < K; ++k) acc = fmaf(src[k], w[k], acc);
      if (l == d.n_hidden)
        out[o] = acc;
      else
        h[((l + 1) & 1) * 128 + o] = fmaxf(acc, 0.f);
    }
    __syncwarp();
  }
}

template <int W>
__global__ void __launch_bounds__(kX3Threads, W <= 64 ? 2 : 1) mlp_x3_kernel(const __grid_constant__ X3Args p) {
  constexpr int kCols = 4 * W;  // a power of two, 64 to 512
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ __align__(8) uint64_t w_full[kX3Slots], w_empty[kX3Slots], a_ready, d_done;
  __shared__ uint32_t holder;
  __shared__ uint8_t huge[2][kTcRows];  // rows for x3_plain_row, by tile parity
  __shared__ int any_huge;
  uint8_t* A = smem;
  uint8_t* ring = smem + 3 * p.a_plane;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    for (int i = 0; i < kX3Slots; ++i) {
      mbar_init(w_full + i, 1);
      mbar_init(w_empty + i, 1);
    }
    mbar_init(&a_ready, kX3Compute / 32);
    mbar_init(&d_done, 1);
    fence_mbar_init();
  }
  if (warp == 0) tmem_alloc(&holder, kCols);
  if (tid < 2 * kTcRows) huge[tid / kTcRows][tid % kTcRows] = 0;
  if (tid == 0) any_huge = 0;
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = holder;
  const int64_t n_tiles = (p.n + kTcRows - 1) / kTcRows;
  const int L = p.L;
  bool ok = true;

  if (warp == kX3Compute / 32) {
    // ---------------- weights: the layers' 32-wide K chunks, tile after tile
    if (lane == 0) {
      uint32_t k = 0;  // chunks issued
      for (int64_t tile = blockIdx.x; tile < n_tiles && ok; tile += gridDim.x) {
        const uint8_t* src = p.blob;
        for (int l = 0; l <= L && ok; ++l) {
          const int K = l == 0 ? p.in_pad : W, rows = 3 * (l == L ? 16 : W);
          for (int kc = 0; kc < K; kc += 32, ++k) {
            const uint32_t slot = k % kX3Slots, bytes = (uint32_t)(rows * min(32, K - kc) * 2);
            if (k >= kX3Slots && !(ok = mbar_wait_bounded(w_empty + slot, (k / kX3Slots - 1) & 1))) break;
            mbar_arrive_expect_tx(w_full + slot, bytes);
            bulk_copy_g2s(ring + slot * p.slot_bytes, src, bytes, w_full + slot);
            src += bytes;
          }
        }
      }
      // every copy issued has landed before the block may end
      for (uint32_t j = k > kX3Slots ? k - kX3Slots : 0; j < k; ++j)
        ok = mbar_wait_bounded(w_full + j % kX3Slots, (j / kX3Slots) & 1) && ok;
    }
  } else if (warp == kX3Compute / 32 + 1) {
    // ---------------- MMAs
    if (lane == 0) {
      const uint32_t a_base = smem_u32(A), ring_base = smem_u32(ring);
      uint32_t k = 0, ev = 0;  // weight chunks consumed; A hand-offs
      for (int64_t tile = blockIdx.x; tile < n_tiles && ok; tile += gridDim.x) {
        for (int l = 0; l <= L && ok; ++l) {
          const int K = l == 0 ? p.in_pad : W;
          for (int k0 = 0; k0 < K && ok; k0 += p.ka, ++ev) {
            if (!(ok = mbar_wait_bounded(&a_ready, ev & 1))) break;
            tc_fence_after();
            const int kn = min(p.ka, K - k0);
            for (int kc = 0; kc < kn; kc += 32, ++k) {
              const uint32_t slot = k % kX3Slots;
              if (!(ok = mbar_wait_bounded(w_full + slot, (k / kX3Slots) & 1))) break;
              const uint32_t b = ring_base + slot * p.slot_bytes;
              const uint32_t a = a_base + (uint32_t)(kc / 16) * (32 * kTcRows);
              for (int ks = 0; ks < min(2, (kn - kc) / 16); ++ks) {
                const int step = (k0 + kc) / 16 + ks;
                if (l == L)
                  x3_mma<16>(tmem, a + ks * 32 * kTcRows, p.a_plane, b + ks * (3 * 16 * 32), step);
                else
                  x3_mma<W>(tmem, a + ks * 32 * kTcRows, p.a_plane, b + ks * (3 * W * 32), step);
              }
              tc_commit(w_empty + slot);
            }
            if (ok) tc_commit(&d_done);
          }
        }
      }
    }
  } else {
    // ---------------- compute warps: thread (row, half)
    const int row = ((warp & 3) << 5) | lane, half = warp >> 2;
    const uint32_t row_taddr = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    uint8_t* a_row = A + op_offset(kTcRows, row, 0);
    uint32_t ev = 0, parity = 0;
    auto publish = [&]() {  // this warp's part of A is written (and D read)
      tc_fence_before();
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&a_ready);
    };
    for (int64_t tile = blockIdx.x; tile < n_tiles; tile += gridDim.x, parity ^= 1) {
      float amax = 0.f;
      float zero = 0.f;  // NaN once a sum is not finite
      const int64_t q = tile * kTcRows + row;
      const bool valid = q < p.n;
      const float* x = p.X + (valid ? q : 0) * p.in_pad;
      for (int k0 = 0; k0 < p.in_pad && ok; k0 += p.ka) {
        const int groups = min(p.ka, p.in_pad - k0) / 8;
        for (int g0 = half; g0 < groups; g0 += 8) {  // four groups' loads in flight
          float4 u[4][2];
#pragma unroll
          for (int i = 0; i < 4; ++i)
            if (g0 + 2 * i < groups) {
              const float4* src = reinterpret_cast<const float4*>(x + k0 + (g0 + 2 * i) * 8);
              u[i][0] = __ldg(src);
              u[i][1] = __ldg(src + 1);
            }
#pragma unroll
          for (int i = 0; i < 4; ++i)
            if (g0 + 2 * i < groups) {
              const float v[8] = {u[i][0].x, u[i][0].y, u[i][0].z, u[i][0].w,
                                  u[i][1].x, u[i][1].y, u[i][1].z, u[i][1].w};
#pragma unroll
              for (int e = 0; e < 8; ++e) amax = fmaxf(amax, fabsf(v[e]));
              x3_split8(v, a_row + (g0 + 2 * i) * (16 * kTcRows), p.a_plane);
            }
        }
        publish();
        ok = mbar_wait_warp(&d_done, ev & 1);
        ++ev;
      }
      tc_fence_after();
      for (int l = 1; l <= L && ok; ++l) {
        // h = ReLU of the sums, half of the columns each, as the next A
#pragma unroll
        for (int c = 0; c < (W >= 32 ? W / 32 : 1); ++c) {
          const int col = W >= 32 ? half * (W / 2) + c * 16 : 0;
          float h[16];
          x3_sum16<W>(row_taddr, col, (l == 1 ? p.in_pad : W) > 16, h);
#pragma unroll
          for (int g = 0; g < 2; ++g) {
            if (W < 32 && g != half) continue;  // W = 16: eight columns each
            float v[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) {
              zero = __fmaf_rn(h[g * 8 + e], 0.f, zero);
              v[e] = fmaxf(h[g * 8 + e], 0.f);
            }
            x3_split8(v, a_row + (col / 8 + g) * (16 * kTcRows), p.a_plane);
          }
        }
        publish();
        ok = mbar_wait_warp(&d_done, ev & 1);
        ++ev;
        tc_fence_after();
      }
      // both halves of a row have marked it; a role that failed stops the group
      if (amax >= kX3Huge || zero != 0.f) huge[parity][row] = 1;
      if (group_sync_or(1, kX3Compute, !ok)) {
        ok = false;
        break;
      }
      if (half == 0) {
        float y[16];
        x3_sum16<16>(row_taddr, 0, W > 16, y);
        zero = huge[parity][row];
        huge[parity][row] = 0;
        if (valid) {
          float* out = p.out + q * p.out_stride;
#pragma unroll
          for (int o = 0; o < 16; ++o)
            if (o < p.out_ch) {
              out[o] = y[o];
              zero = __fmaf_rn(y[o], 0.f, zero);
            }
          if (zero != 0.f) {
            out[0] = __uint_as_float(kX3Mark);
            any_huge = 1;
          }
        }
      }
    }
  }
  if (!ok) atomicOr(p.err, 1);
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 0) tmem_dealloc(tmem, kCols);
  // The marked rows last, when no other warp waits with a limit: a deep
  // network's takes 0.1 ms.  The operands' memory is free by now.
  if (any_huge == 0) return;
  float* h = reinterpret_cast<float*>(smem) + warp * 256;
  for (int64_t j = warp;; j += kX3Threads / 32) {  // 32 rows of the block's tiles each
    const int64_t q0 = (blockIdx.x + j / 4 * gridDim.x) * kTcRows + j % 4 * 32;
    if (q0 >= p.n) break;
    unsigned marked = __ballot_sync(0xffffffffu, q0 + lane < p.n &&
                                                     __float_as_uint(p.out[(q0 + lane) * p.out_stride]) == kX3Mark);
    for (; marked; marked &= marked - 1) {
      const int64_t q = q0 + __ffs(marked) - 1;
      x3_plain_row(p.d, p.params, p.X + q * p.in_pad, h, p.out + q * p.out_stride, p.out_ch);
    }
  }
}

// The planes of every matrix (adam_kernel keeps them up to date afterwards).
__global__ void __launch_bounds__(256) x3_pack_kernel(const __grid_constant__ X3Planes p,
                                                      const float* __restrict__ params) {
  const int64_t i = blockIdx.x * (int64_t)256 + threadIdx.x;  // element of the matrix parameters
  if (i < p.n_net_params) x3_store(p, i, params[i]);
}

int64_t x3_pack_bytes(const MlpDims& d) { return 6 * d.n_net_params; }

int x3_pack(const MlpDims& d, const float* params, uint8_t* blob, cudaStream_t st) {
  x3_pack_kernel<<<(unsigned)((d.n_net_params + 255) / 256), 256, 0, st>>>(x3_planes(d, blob), params);
  HM_CHECK_LAUNCH("x3_pack_kernel");
  return HM_OK;
}

template <int W>
static int x3_launch(const X3Args& a, size_t smem, cudaStream_t st) {
  cudaError_t e = cudaFuncSetAttribute(mlp_x3_kernel<W>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return hm_cuda_status(e, "mlp_x3_kernel smem");
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int64_t tiles = (a.n + kTcRows - 1) / kTcRows;
  const int64_t most = (int64_t)sms * (W <= 64 ? 2 : 1);
  mlp_x3_kernel<W><<<(unsigned)std::min(tiles, most), kX3Threads, smem, st>>>(a);
  HM_CHECK_LAUNCH("mlp_x3_kernel");
  return HM_OK;
}

int x3_forward(const MlpDims& d, const float* params, const uint8_t* blob, const float* X, float* out, int out_stride,
               int64_t n, int* err_flag, cudaStream_t st) {
  X3Args a;
  memset(&a, 0, sizeof(a));
  a.d = d;
  a.params = params;
  a.blob = blob;
  a.X = X;
  a.out = out;
  a.out_stride = out_stride;
  a.out_ch = std::min(d.out_ch, out_stride);
  a.in_pad = d.in_pad;
  a.L = d.n_hidden;
  a.n = n;
  a.err = err_flag;
  a.ka = std::max(d.width, 64);
  a.a_plane = kTcRows * a.ka * 2;
  a.slot_bytes = 3 * d.width * 64;
  a.slot_bytes = std::max(a.slot_bytes, 3 * 16 * 64);
  const size_t smem = (size_t)3 * a.a_plane + (size_t)kX3Slots * a.slot_bytes;
  switch (d.width) {
    case 16: return x3_launch<16>(a, smem, st);
    case 32: return x3_launch<32>(a, smem, st);
    case 64: return x3_launch<64>(a, smem, st);
    default: return x3_launch<128>(a, smem, st);
  }
}

}  // namespace hm
