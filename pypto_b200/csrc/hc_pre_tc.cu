// x . hc_fn^T and the sum of squares of the hyper-connection pre-mix (hc_pre.cu) for more than a few tokens, on tcgen05.
//
// hc_fn is fp32, and the 24 outputs steer a Sinkhorn iteration, so the product keeps fp32 weights: each is split into three
// bf16 pieces that add up to it (8 significant bits each), the pieces are 3 x 32 columns of one N = 96 product, and products of
// bf16 numbers are exact in the fp32 accumulator.  Sums run over 1024 elements in tensor memory and over those segments in
// fp32 registers, in order.  What bounds the kernel is reading x once: 32 KB per token.
//
// A CTA takes a tile of 128 tokens and a range of the 256 reduction chunks.  Warp 0 streams x and hc_fn with TMA, warp 1 issues
// the products, warps 2..9 split a chunk of hc_fn into the B tile, add up the squares of the x tile in shared memory and
// take the finished segments.  4096 tokens: 165 us on CUDA cores (FMA and shared-memory bound) -> 37 us, 134 MB.
#include "kernels.cuh"
#include "tc_common.cuh"

namespace dsv32 {

namespace {
constexpr int kHtThreads = 320;
constexpr int kHtStages = 6;
constexpr int kHtABytes = 128 * 128, kHtBBytes = 96 * 128, kHtWBox = 24 * 128;
constexpr int kHtOffW = kHtABytes + kHtBBytes;      // two boxes of 24 rows x 32 fp32
constexpr int kHtStageBytes = kHtOffW + 2 * kHtWBox;   // 34,816
constexpr int kHtOffBars = kHtStages * kHtStageBytes;
constexpr int kHtNumBars = 3 * kHtStages + 4;      // full (x), bfull (pieces), empty, dfull[2], dempty[2]
constexpr int kHtOffTmem = kHtOffBars + kHtNumBars * 8;
constexpr size_t kHtSmemBytes = kHtOffTmem + 16;
static_assert(kHtSmemBytes <= 232448, "shared memory of one CTA");
constexpr int kHtK = 16384, kHtChunks = kHtK / 64, kHtMix = 24;
constexpr int kHtSeg = 16;                         // chunks per segment
constexpr int kHtDrainLag = 3;                     // chunks after a segment's last before its sums are taken
}  // namespace

__global__ void __launch_bounds__(kHtThreads, 1)
hc_pre_dots_tc_kernel(const __grid_constant__ CUtensorMap x_map, const __grid_constant__ CUtensorMap w_map, HcPreParams p, int splits) {
  extern __shared__ __align__(1024) unsigned char smem[];
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + kHtOffBars);
  uint64_t* bfull_bar = full_bar + kHtStages;
  uint64_t* empty_bar = bfull_bar + kHtStages;
  uint64_t* dfull_bar = empty_bar + kHtStages;    // [2]
  uint64_t* dempty_bar = dfull_bar + 2;           // [2]
  uint32_t* tmem_ptr_s = reinterpret_cast<uint32_t*>(smem + kHtOffTmem);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int split = blockIdx.x, t0 = blockIdx.y * 128;
  const int c0 = kHtChunks * split / splits, nchunks = kHtChunks * (split + 1) / splits - c0;
  if (warp == 0) {
    if (lane == 0) {
      tma_prefetch_desc(&x_map);
      tma_prefetch_desc(&w_map);
      for (int i = 0; i < kHtStages; ++i) {
        mbar_init(&full_bar[i], 1);
        mbar_init(&bfull_bar[i], 8);
        mbar_init(&empty_bar[i], 1);   // (the products are issued after all eight warps have read the stage)
      }
      for (int i = 0; i < 2; ++i) {
        mbar_init(&dfull_bar[i], 1);
        mbar_init(&dempty_bar[i], 8);
      }
      mbar_fence_init();
    }
  } else if (warp == 1) {
    tmem_alloc(tmem_ptr_s, 256);
    tmem_relinquish();
  } else {
    // rows 24..31 of every piece stay zero
    const int e = tid - 64;
    for (int i = e; i < kHtStages * 3 * 8 * 8; i += 256) {
      const int st = i / 192, r = i % 192;
      *reinterpret_cast<uint4*>(smem + st * kHtStageBytes + kHtABytes + ((r / 64) * 32 + 24 + (r % 64) / 8) * 128 + (r % 8) * 16) =
          make_uint4(0u, 0u, 0u, 0u);
    }
    fence_proxy_async_smem();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_ptr_s;
  pdl_wait();     // (first kernel of an operator: everything it reads may come from the kernel before)
  pdl_trigger();

  if (warp == 0) {
    if (lane == 0) {
      int s = 0, ph = 1;
      for (int c = 0; c < nchunks; ++c) {
        if (!mbar_wait(&empty_bar[s], ph, p.status, 101)) break;
        unsigned char* st = smem + s * kHtStageBytes;
        mbar_arrive_expect_tx(&full_bar[s], kHtABytes + 2 * kHtWBox);
        tma_load_2d(st, &x_map, (c0 + c) * 128, t0, &full_bar[s]);
        tma_load_2d(st + kHtOffW, &w_map, (c0 + c) * 256, 0, &full_bar[s]);
        tma_load_2d(st + kHtOffW + kHtWBox, &w_map, (c0 + c) * 256 + 128, 0, &full_bar[s]);
        if (++s == kHtStages) { s = 0; ph ^= 1; }
      }
    }
  } else if (warp == 1) {
    constexpr uint32_t idesc = umma_idesc_bf16(128, 96, false, false);
    const uint32_t tbase = __shfl_sync(0xffffffffu, tmem_base, 0);
    bool ok = true;
    int s = 0, ph = 0;
    for (int c = 0; ok && c < nchunks; ++c) {
      const int g = c / kHtSeg, b = g & 1;
      if (c % kHtSeg == 0) ok = __all_sync(0xffffffffu, mbar_wait(&dempty_bar[b], ((g >> 1) & 1) ^ 1, p.status, 102));
      if (ok) ok = __all_sync(0xffffffffu, mbar_wait(&full_bar[s], ph, p.status, 103) && mbar_wait(&bfull_bar[s], ph, p.status, 104));
      if (!ok) break;
      tc_fence_after();
      const uint32_t st = smem_u32(smem + s * kHtStageBytes);
      const uint64_t ad = umma_smem_desc_sw128(st, 16, 1024), bd = umma_smem_desc_sw128(st + kHtABytes, 16, 1024);
      if (elect_one()) {
#pragma unroll
        for (int ks = 0; ks < 4; ++ks)
          umma_f16_ss(tbase + b * 128, ad + 2 * ks, bd + 2 * ks, idesc, (c % kHtSeg > 0 || ks > 0) ? 1u : 0u);
        umma_commit(&empty_bar[s]);
        if (c % kHtSeg == kHtSeg - 1 || c == nchunks - 1) umma_commit(&dfull_bar[b]);
      }
      __syncwarp();
      if (++s == kHtStages) { s = 0; ph ^= 1; }
    }
  } else {
    const int e = tid - 64;                               // 0 .. 255
    const int quarter = warp & 3, half = (warp - 2) >> 2; // tensor-memory lanes; outputs 16 half ..
    // hc_fn: threads 0..191 take eight consecutive columns of an output's row
    const bool conv = e < kHtMix * 8;
    const int m = e >> 3, u = e & 7;
    const uint32_t woff = static_cast<uint32_t>(kHtOffW + (u >> 2) * kHtWBox + m * 128);
    const uint32_t wsw0 = static_cast<uint32_t>((((u & 3) * 2) ^ (m & 7)) << 4), wsw1 = static_cast<uint32_t>((((u & 3) * 2 + 1) ^ (m & 7)) << 4);
    const uint32_t boff = static_cast<uint32_t>(kHtABytes + m * 128 + ((u ^ (m & 7)) << 4));   // (32 rows a piece: same swizzle)
    // squares: half a row of the x tile per thread
    const int xr = e >> 1;
    const uint32_t xoff = static_cast<uint32_t>(xr * 128);
    float sq0 = 0.f, sq1 = 0.f, acc[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) acc[j] = 0.f;
    const int segs = (nchunks + kHtSeg - 1) / kHtSeg;
    int drained = 0;
    bool ok = true;
    auto drain = [&]() {                                  // segment `drained`: hi + (mid + lo) of this thread's 16 outputs
      const int b = drained & 1;
      ok = __all_sync(0xffffffffu, mbar_wait(&dfull_bar[b], (drained >> 1) & 1, p.status, 105));
      if (!ok) return;
      tc_fence_after();
      const uint32_t ta = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + b * 128 + half * 16;
      uint32_t r0[16], r1[16], r2[16];
      tmem_ld_32x32b_x16(ta, r0);
      tmem_ld_32x32b_x16(ta + 32, r1);
      tmem_ld_32x32b_x16(ta + 64, r2);
      tmem_ld_wait();
#pragma unroll
      for (int j = 0; j < 16; ++j)
        acc[j] += __uint_as_float(r0[j]) + (__uint_as_float(r1[j]) + __uint_as_float(r2[j]));
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&dempty_bar[b]);
      ++drained;
    };
    int s = 0, ph = 0;
    for (int c = 0; ok && c < nchunks; ++c) {
      ok = __all_sync(0xffffffffu, mbar_wait(&full_bar[s], ph, p.status, 106));   // (also: the stage's last products are done)
      if (!ok) break;
      unsigned char* st = smem + s * kHtStageBytes;
      if (conv) {
        const float4 wa = *reinterpret_cast<const float4*>(st + woff + wsw0), wb = *reinterpret_cast<const float4*>(st + woff + wsw1);
        const float w[8] = {wa.x, wa.y, wa.z, wa.w, wb.x, wb.y, wb.z, wb.w};
        uint32_t hi[4], mid[4], lo[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          hi[j] = pack_bf16x2(w[2 * j], w[2 * j + 1]);
          const float a = w[2 * j] - __uint_as_float(hi[j] << 16), b = w[2 * j + 1] - __uint_as_float(hi[j] & 0xffff0000u);
          mid[j] = pack_bf16x2(a, b);
          lo[j] = pack_bf16x2(a - __uint_as_float(mid[j] << 16), b - __uint_as_float(mid[j] & 0xffff0000u));
        }
        *reinterpret_cast<uint4*>(st + boff) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
        *reinterpret_cast<uint4*>(st + boff + 32 * 128) = make_uint4(mid[0], mid[1], mid[2], mid[3]);
        *reinterpret_cast<uint4*>(st + boff + 64 * 128) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint4 v = *reinterpret_cast<const uint4*>(st + xoff + ((((e & 1) * 4 + j) ^ (xr & 7)) << 4));
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const float a = __uint_as_float(w[k] << 16), b = __uint_as_float(w[k] & 0xffff0000u);
          sq0 = fmaf(a, a, sq0);
          sq1 = fmaf(b, b, sq1);
        }
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bfull_bar[s]);
      if (++s == kHtStages) { s = 0; ph ^= 1; }
      if (c >= kHtSeg && c % kHtSeg == kHtDrainLag) drain();
    }
    while (ok && drained < segs) drain();
    if (!ok) {   // a wait ran out (the status word has it): the sums are not to be taken for results
      sq0 = acc[0] = __int_as_float(0x7fc00000);
#pragma unroll
      for (int j = 1; j < 16; ++j) acc[j] = acc[0];
    }
    {
      float* part = p.partial + static_cast<size_t>(split) * p.t * kHcPartLd;
      const int tok = t0 + quarter * 32 + lane;
      if (tok < p.t) {
        float4* dst = reinterpret_cast<float4*>(part + static_cast<size_t>(tok) * kHcPartLd + half * 16);
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (half == 0 || j < 2) dst[j] = make_float4(acc[4 * j], acc[4 * j + 1], acc[4 * j + 2], acc[4 * j + 3]);
      }
      float sq = sq0 + sq1;
      sq += __shfl_xor_sync(0xffffffffu, sq, 1);
      if ((e & 1) == 0 && t0 + xr < p.t) part[static_cast<size_t>(t0 + xr) * kHcPartLd + kHtMix] = sq;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem_base, 256);
  }
}

// Splits of the reduction: every SM a CTA, none with fewer than four chunks.
int hc_pre_tc_splits(int t) {
  const int tiles = (t + 127) / 128, s = sm_count() / tiles;
  return s < 1 ? 1 : (s > kHtChunks / 4 ? kHtChunks / 4 : s);
}

int launch_hc_pre_dots_tc(const HcPreParams& p, cudaStream_t stream) {
  CUtensorMap x, w;
  int rc = make_tensor_map_2d_u8(&x, p.x, p.t, kHtK * 2, 128, 128);
  if (rc == DSV32_OK) rc = make_tensor_map_2d_u8(&w, p.hc_fn, kHtMix, kHtK * 4, kHtMix, 128);
  if (rc != DSV32_OK) return rc;
  cudaFuncSetAttribute(hc_pre_dots_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kHtSmemBytes));
  const int splits = hc_pre_tc_splits(p.t);
  launch_ex(hc_pre_dots_tc_kernel, dim3(splits, (p.t + 127) / 128), kHtThreads, kHtSmemBytes, stream, true, 1, x, w, p, splits);
  count_launch();
  return check_launch("hc_pre_dots_tc_kernel");
}

}  // namespace dsv32
