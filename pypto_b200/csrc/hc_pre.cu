// DeepSeek-V4 hyper-connection pre-mix ("hc_pre").
// Follows models/deepseek_v4/hc_pre_impl.py:23-206 (golden gen_hc_pre, models/deepseek_v4/test_hc_pre.py:26-118).
// Per token, with x [4 streams, 4096] bf16 read as one 16384-vector:
//   mix[24]  = (x . hc_fn[m, :]) / sqrt(mean(x^2) + norm_eps)                       (fp32)
//   pre[4]   = sigmoid(mix[0:4]  * scale[0] + base[0:4])  + hc_eps
//   post[4]  = 2 * sigmoid(mix[4:8] * scale[1] + base[4:8])
//   comb[4,4]= Sinkhorn(mix[8:24] * scale[2] + base[8:24]): row softmax + hc_eps, column normalisation, then
//              (iters - 1) x (row normalisation, column normalisation), every divisor with + hc_eps
//   y[4096]  = bf16( sum_h pre[h] * x[h, :] )
// Few tokens (up to 64): hc_pre_dots_kernel splits the 16384-long reduction into 128 slices of 128 columns: a CTA holds
// the 24 x 128 slice of hc_fn in shared memory and applies it to a tile of up to 64 tokens; a lane owns 6 outputs x
// 2 tokens, so every lane works and there are no shuffles in the loop.  Partial sums go to a workspace [group][token][24].
// hc_pre_finish_kernel (one CTA per token, launched dependent) reads the token's x with 16-byte loads before the dots have
// ended, takes its sum of squares, adds the partials in a fixed order, runs the 4x4 Sinkhorn on 16 lanes of a warp (row /
// column sums by shuffles) and writes y from the x values it holds.
// More tokens: the products run on tensor cores (hc_pre_tc.cu), which also leave the sums of squares, and
// hc_pre_finish_rows_kernel takes up to eight tokens per CTA: a warp each for the mixing factors, then all warps stream x to y.
// A CTA per token held its 512 threads through the Sinkhorn's serial chain (2 us of 40 divisions): 92 us at 4096 tokens
// against 38 now, the time of reading x once more and writing y.
#include "kernels.cuh"
#include "tc_common.cuh"

namespace dsv32 {

namespace {
constexpr int kHc = 4, kHcD = 4096, kHcK = kHc * kHcD, kHcMix = (2 + kHc) * kHc, kHcOut = kHcMix + 1;
constexpr int kHcSlice = 128, kHcSlices = kHcK / kHcSlice;   // 128 slices of 128 columns
constexpr int kHcTokTile = 64, kHcDotThreads = 256, kHcFinThreads = 512;
constexpr int kHcPad = kHcSlice + 4;                          // padded row stride of the shared-memory tiles
constexpr size_t kHcDotSmem = static_cast<size_t>(kHcMix + kHcTokTile) * kHcPad * sizeof(float);   // 46,464 bytes

__device__ __forceinline__ float hc_sigmoid(float v) { return __fdiv_rn(1.0f, 1.0f + expf(-v)); }

// Sinkhorn on lanes 0..15: lane = 4 * row + col; sums over a row = lanes differing in bits 0..1, over a column = lanes
// differing in bits 2..3.  Lanes 16..31 run the same code on copies.
__device__ __forceinline__ float hc_sinkhorn(float c, int iters, float eps) {
  float rmax = fmaxf(c, __shfl_xor_sync(0xffffffffu, c, 1));
  rmax = fmaxf(rmax, __shfl_xor_sync(0xffffffffu, rmax, 2));
  c = expf(c - rmax);
  auto row_sum = [](float v) {
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    return v + __shfl_xor_sync(0xffffffffu, v, 2);
  };
  auto col_sum = [](float v) {
    v += __shfl_xor_sync(0xffffffffu, v, 4);
    return v + __shfl_xor_sync(0xffffffffu, v, 8);
  };
  c = __fdiv_rn(c, row_sum(c)) + eps;
  c = __fdiv_rn(c, col_sum(c) + eps);
  for (int it = 1; it < iters; ++it) {
    c = __fdiv_rn(c, row_sum(c) + eps);
    c = __fdiv_rn(c, col_sum(c) + eps);
  }
  return c;
}

// y = bf16( sum_h pre[h] * x[h] ) of eight columns
__device__ __forceinline__ uint4 hc_mix8(const uint4 (&x)[4], const float (&pre)[4]) {
  uint32_t out[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    float s0 = 0.f, s1 = 0.f;
#pragma unroll
    for (int h = 0; h < 4; ++h) {
      const uint32_t w = reinterpret_cast<const uint32_t*>(&x[h])[j];
      const float a = __fmul_rn(pre[h], __uint_as_float(w << 16)), b = __fmul_rn(pre[h], __uint_as_float(w & 0xffff0000u));
      s0 = h == 0 ? a : __fadd_rn(s0, a);
      s1 = h == 0 ? b : __fadd_rn(s1, b);
    }
    out[j] = pack_bf16x2(s0, s1);
  }
  return make_uint4(out[0], out[1], out[2], out[3]);
}
}  // namespace

// One CTA per slice; all eight warps load, one per 16 tokens multiplies (with four warps the loads of 64 tokens were what the kernel
// waited for: 18.5 us for the operator inside a graph, 14.0 now).  Dynamic shared memory:
// w_s[24][132] (a slice of hc_fn, row stride padded so that the four output groups of a warp hit different banks)
// and x_s[64][132] (the token tile's slice of x as floats, padded so that the eight token groups do).
// Lane = (output group og = lane / 8: outputs 6 og .. 6 og + 5) x (token group tg = lane % 8: tokens tg, tg + 8 of
// the warp's 16): per four columns 6 + 2 sixteen-byte shared-memory loads (broadcast within a group) feed 48 FMAs.
__global__ void __launch_bounds__(kHcDotThreads) hc_pre_dots_kernel(HcPreParams p) {
  pdl_wait();     // (first kernel of an operator: everything it reads may come from the kernel before)
  pdl_trigger();
  extern __shared__ __align__(16) float hc_smem[];
  float* w_s = hc_smem;                               // [kHcMix][kHcPad]
  float* x_s = hc_smem + kHcMix * kHcPad;             // [kHcTokTile][kHcPad]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int group = blockIdx.x, ntok = p.t, k0 = group * kHcSlice;
  const int og = lane >> 3, tg = lane & 7;
  const int tok_a = warp * 16 + tg, tok_b = tok_a + 8;
  float acc_a[6], acc_b[6];
#pragma unroll
  for (int i = 0; i < 6; ++i) acc_a[i] = acc_b[i] = 0.f;
  for (int i = tid; i < kHcMix * (kHcSlice / 4); i += kHcDotThreads) {
    const int m = i / (kHcSlice / 4), c4 = i % (kHcSlice / 4);
    *reinterpret_cast<float4*>(&w_s[m * kHcPad + 4 * c4]) =
        __ldg(reinterpret_cast<const float4*>(p.hc_fn + static_cast<size_t>(m) * kHcK + k0 + 4 * c4));
  }
  for (int i = tid; i < (ntok + 15) / 16 * 16 * (kHcSlice / 4); i += kHcDotThreads) {
    const int tok = i / (kHcSlice / 4), c4 = i % (kHcSlice / 4);
    float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
    if (tok < ntok) {
      const uint2 v = __ldg(reinterpret_cast<const uint2*>(p.x + static_cast<size_t>(tok) * kHcK + k0 + 4 * c4));
      f = make_float4(__uint_as_float(v.x << 16), __uint_as_float(v.x & 0xffff0000u), __uint_as_float(v.y << 16),
                      __uint_as_float(v.y & 0xffff0000u));
    }
    *reinterpret_cast<float4*>(&x_s[tok * kHcPad + 4 * c4]) = f;
  }
  __syncthreads();
  if (warp * 16 < ntok) {
    const float* wl = w_s + og * 6 * kHcPad;
    const float* xa = x_s + tok_a * kHcPad;
    const float* xb = x_s + tok_b * kHcPad;
#pragma unroll 2
    for (int col = 0; col < kHcSlice; col += 4) {
      const float4 va = *reinterpret_cast<const float4*>(xa + col);
      const float4 vb = *reinterpret_cast<const float4*>(xb + col);
#pragma unroll
      for (int i = 0; i < 6; ++i) {
        const float4 w = *reinterpret_cast<const float4*>(wl + i * kHcPad + col);
        acc_a[i] = fmaf(va.x, w.x, acc_a[i]);
        acc_a[i] = fmaf(va.y, w.y, acc_a[i]);
        acc_a[i] = fmaf(va.z, w.z, acc_a[i]);
        acc_a[i] = fmaf(va.w, w.w, acc_a[i]);
        acc_b[i] = fmaf(vb.x, w.x, acc_b[i]);
        acc_b[i] = fmaf(vb.y, w.y, acc_b[i]);
        acc_b[i] = fmaf(vb.z, w.z, acc_b[i]);
        acc_b[i] = fmaf(vb.w, w.w, acc_b[i]);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 6; ++i) {
    if (tok_a < ntok) p.partial[(static_cast<size_t>(group) * p.t + tok_a) * kHcMix + og * 6 + i] = acc_a[i];
    if (tok_b < ntok) p.partial[(static_cast<size_t>(group) * p.t + tok_b) * kHcMix + og * 6 + i] = acc_b[i];
  }
}

__global__ void __launch_bounds__(kHcFinThreads) hc_pre_finish_kernel(HcPreParams p, int groups) {
  __shared__ float red_s[kHcFinThreads / 32][32];
  __shared__ float mix_s[kHcOut];
  __shared__ float pre_s[kHc];
  const int tok = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // this thread's 32 values of x: columns 8 tid .. 8 tid + 7 of the four streams, one 16-byte load per stream
  const __nv_bfloat16* xrow = p.x + static_cast<size_t>(tok) * kHcK;
  pdl_trigger();
  uint4 x[kHc];
  float sq = 0.f;
#pragma unroll
  for (int h = 0; h < kHc; ++h) {
    x[h] = __ldg(reinterpret_cast<const uint4*>(xrow + h * kHcD + 8 * tid));
    const uint32_t w[4] = {x[h].x, x[h].y, x[h].z, x[h].w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float a = __uint_as_float(w[j] << 16), b = __uint_as_float(w[j] & 0xffff0000u);
      sq = fmaf(a, a, sq);
      sq = fmaf(b, b, sq);
    }
  }
  pdl_wait();
  // partial dot products: lane = output m, warp w adds the groups w, w + 16, ...; then the 16 warps in order
  float part = 0.f;
  if (lane < kHcMix)
    for (int g = warp; g < groups; g += kHcFinThreads / 32) part += p.partial[(static_cast<size_t>(g) * p.t + tok) * kHcMix + lane];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
  red_s[warp][lane] = (lane == kHcMix) ? sq : part;   // column 24 carries the sum of squares
  __syncthreads();
  if (tid < kHcOut) {
    float s = 0.f;
#pragma unroll
    for (int w = 0; w < kHcFinThreads / 32; ++w) s += red_s[w][tid];
    mix_s[tid] = s;
  }
  __syncthreads();
  if (warp == 0) {
    const float denom = sqrtf(__fdiv_rn(mix_s[kHcMix], static_cast<float>(kHcK)) + p.norm_eps);
    if (lane < kHc) {
      const float v = __fdiv_rn(mix_s[lane], denom);
      pre_s[lane] = hc_sigmoid(fmaf(v, p.hc_scale[0], p.hc_base[lane])) + p.hc_eps;
    } else if (lane < 2 * kHc) {
      const float v = __fdiv_rn(mix_s[lane], denom);
      p.post[static_cast<size_t>(tok) * kHc + (lane - kHc)] = 2.0f * hc_sigmoid(fmaf(v, p.hc_scale[1], p.hc_base[lane]));
    }
    const int e = lane & 15;
    const float c = hc_sinkhorn(fmaf(__fdiv_rn(mix_s[2 * kHc + e], denom), p.hc_scale[2], p.hc_base[2 * kHc + e]), p.iters, p.hc_eps);
    if (lane < kHc * kHc) p.comb[static_cast<size_t>(tok) * (kHc * kHc) + lane] = c;
  }
  __syncthreads();
  const float pre[kHc] = {pre_s[0], pre_s[1], pre_s[2], pre_s[3]};
  *reinterpret_cast<uint4*>(p.y + static_cast<size_t>(tok) * kHcD + 8 * tid) = hc_mix8(x, pre);
}

// `per` <= 8 tokens per CTA.  CTAs walk the tokens backwards: what the dots kernel read last is still in L2.
__global__ void __launch_bounds__(256) hc_pre_finish_rows_kernel(HcPreParams p, int splits, int per) {
  __shared__ float pre_s[8][kHc];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int t0 = (gridDim.x - 1 - blockIdx.x) * per, ntok = min(per, p.t - t0);
  pdl_trigger();
  pdl_wait();
  if (warp < ntok) {
    const int tok = t0 + warp;
    float v = 0.f;   // lane = output, 24 = sum of squares
    if (lane < kHcOut)
#pragma unroll 16
      for (int g = 0; g < splits; ++g) v += p.partial[(static_cast<size_t>(g) * p.t + tok) * kHcPartLd + lane];
    const float denom = sqrtf(__fdiv_rn(__shfl_sync(0xffffffffu, v, kHcMix), static_cast<float>(kHcK)) + p.norm_eps);
    v = __fdiv_rn(v, denom);
    if (lane < kHc) pre_s[warp][lane] = hc_sigmoid(fmaf(v, p.hc_scale[0], p.hc_base[lane])) + p.hc_eps;
    else if (lane < 2 * kHc)
      p.post[static_cast<size_t>(tok) * kHc + (lane - kHc)] = 2.0f * hc_sigmoid(fmaf(v, p.hc_scale[1], p.hc_base[lane]));
    const int e = lane & 15;
    const float m = __shfl_sync(0xffffffffu, v, 2 * kHc + e);
    const float c = hc_sinkhorn(fmaf(m, p.hc_scale[2], p.hc_base[2 * kHc + e]), p.iters, p.hc_eps);
    if (lane < kHc * kHc) p.comb[static_cast<size_t>(tok) * (kHc * kHc) + lane] = c;
  }
  __syncthreads();
  for (int i = 0; i < ntok; ++i) {
    const __nv_bfloat16* xrow = p.x + static_cast<size_t>(t0 + i) * kHcK;
    const float pre[kHc] = {pre_s[i][0], pre_s[i][1], pre_s[i][2], pre_s[i][3]};
    uint4 x[2][kHc];
#pragma unroll
    for (int k = 0; k < 2; ++k)
#pragma unroll
      for (int h = 0; h < kHc; ++h) x[k][h] = __ldcs(reinterpret_cast<const uint4*>(xrow + h * kHcD + 8 * (tid + 256 * k)));
#pragma unroll
    for (int k = 0; k < 2; ++k)
      __stcs(reinterpret_cast<uint4*>(p.y + static_cast<size_t>(t0 + i) * kHcD + 8 * (tid + 256 * k)), hc_mix8(x[k], pre));
  }
}

// Tensor cores from 65 tokens on: the CUDA-core kernel's work grows with the 16 tokens of its warps and passes the time of
// the other's fixed parts (tensor memory, pipeline fill, 40 % of the tile idle) there.
static bool hc_pre_tc(int t) { return t > 64; }

size_t hc_pre_workspace_bytes(int t) {
  if (t <= 0) return 0;
  return (hc_pre_tc(t) ? static_cast<size_t>(hc_pre_tc_splits(t)) * kHcPartLd : static_cast<size_t>(kHcSlices) * kHcMix) * t * sizeof(float);
}

int launch_hc_pre(const HcPreParams& p, cudaStream_t stream) {
  if (p.t <= 0) return DSV32_OK;
  int rc;
  if (hc_pre_tc(p.t)) {
    rc = launch_hc_pre_dots_tc(p, stream);
    if (rc != DSV32_OK) return rc;
    int per = p.t / (2 * sm_count());   // two CTAs per SM or more
    per = per < 1 ? 1 : (per > 8 ? 8 : per);
    launch_ex(hc_pre_finish_rows_kernel, dim3((p.t + per - 1) / per), 256, 0, stream, true, 1, p, hc_pre_tc_splits(p.t), per);
  } else {
    cudaFuncSetAttribute(hc_pre_dots_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kHcDotSmem));
    launch_ex(hc_pre_dots_kernel, dim3(kHcSlices), kHcDotThreads, kHcDotSmem, stream, true, 1, p);
    count_launch();
    rc = check_launch("hc_pre_dots_kernel");
    if (rc != DSV32_OK) return rc;
    launch_ex(hc_pre_finish_kernel, dim3(p.t), kHcFinThreads, 0, stream, true, 1, p, kHcSlices);
  }
  count_launch();
  return check_launch("hc_pre_finish_kernel");
}

}  // namespace dsv32
