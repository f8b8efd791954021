// Per-head second halves of the V3.2 prologs and of the V4 indexer prolog on tcgen05, one persistent kernel:
//   MLA head      q_b = int32(q_norm . w_uq_qr[:, 192 of the head]) dequantised to bf16; its 128 nope dims times w_uk[head]
//                 -> query_nope, its 64 rope dims through the de-interleaving rotary embedding -> query_rope
//                 (models/deepseek_v32_exp/mla_prolog_quant_impl.py:480, 499-509, 223-247, 283-361)
//   indexer head  q = int32(q_norm . w_qb[:, 128 of the head]) dequantised to bf16, rotary embedding, times the hadamard
//                 matrix, per-row int8 quantisation -> q_int8, q_scale
//                 (models/deepseek_v32_exp/lightning_indexer_prolog_quant_impl.py:423-480; V4 form, reduction 1024 and the
//                 interleaved inverse rotary embedding on the last 64 dims:
//                 models/deepseek_v4/lightning_indexer_prolog_quant_v4_impl.py:118-252)
//
// An item is (head, tile of 128 tokens).  Its first product (kind::i8) accumulates in tensor memory, eight epilogue warps turn
// it into the bf16 left operand of the second product, also in tensor memory, and the second product is drained 128 columns at
// a time.  The intermediate q_b (33 KB per token) never leaves the SM, and one launch streams all of the weights: at 128 tokens
// the previous four launches (q_b, w_uk, indexer q) took 50 us for 67 MB, at 4096 tokens they wrote and read q_b once more and
// took 746 us.  Tensor memory: D1 192 columns, left operand 64, two output buffers of 128.
//
// Warp roles: 0 = TMA producer, 1 = MMA issuer (one elected lane), 2..9 = epilogue (tensor-memory lane quarter x column half).
// The kernel is launched dependent on the one that writes q_norm: the first ring slots' weights are on their way before that
// one has finished.
#include "kernels.cuh"
#include "tc_common.cuh"

namespace dsv32 {

namespace {

constexpr int kHdThreads = 320;
constexpr int kHdSlots = 4;
constexpr int kHdSlotBytes = 40960;                         // D1: A 16 KB | nope columns 16 KB | rope columns 8 KB; D2: 32 KB
constexpr int kHdOffStore = kHdSlots * kHdSlotBytes;        // one 4 KB store buffer per epilogue warp
constexpr int kHdOffRed = kHdOffStore + 8 * 4096;           // float[2][4 quarters][2 halves][32]
constexpr int kHdOffScale = kHdOffRed + 2 * 4 * 2 * 32 * 4; // float[2][192]: column scales of an item
constexpr int kHdOffBars = kHdOffScale + 2 * 192 * 4;
constexpr int kHdNumBars = 2 * kHdSlots + 2 + 4;            // full, empty, d1_full, a2_full, d2_full[2], d2_empty[2]
constexpr int kHdOffTmem = kHdOffBars + kHdNumBars * 8;
constexpr size_t kHdSmemBytes = kHdOffTmem + 16;
static_assert(kHdSmemBytes <= 232448, "shared memory of one CTA");
constexpr uint32_t kColD1 = 0, kColA2 = 192, kColD2 = 256;

__device__ __forceinline__ float bf16_round(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }
__device__ __forceinline__ float bf_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf_hi(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }
// 16 consecutive bf16 of a rotary table row as pairs; 16-byte loads where the table allows them.  A lane reads its own token's
// row, so a load instruction touches 32 lines: eight wide loads an item, issued before the accumulator is waited for
// (32 narrow ones after it kept the load/store unit busy for half of the kernel).
__device__ __forceinline__ void rope16(const __nv_bfloat16* row, bool vec, uint32_t (&w)[8]) {
  if (vec) {
    const uint4 a = __ldg(reinterpret_cast<const uint4*>(row)), b = __ldg(reinterpret_cast<const uint4*>(row) + 1);
    w[0] = a.x; w[1] = a.y; w[2] = a.z; w[3] = a.w;
    w[4] = b.x; w[5] = b.y; w[6] = b.z; w[7] = b.w;
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) w[i] = __ldg(reinterpret_cast<const uint32_t*>(row) + i);
  }
}
__device__ __forceinline__ void pair_barrier(int id) { asm volatile("bar.sync %0, 64;" ::"r"(id) : "memory"); }

}  // namespace

struct HeadParams {
  const float* row_scale;          // [t] scale of the int8 activations
  const float* w_uq_scale;         // [128 * 192]
  const float* w_qb_scale;         // [64 * 128]
  const __nv_bfloat16* cos;        // [t, 64], MLA heads
  const __nv_bfloat16* sin;
  const __nv_bfloat16* cos_idx;    // [t, 64], indexer heads
  const __nv_bfloat16* sin_idx;
  __nv_bfloat16* q_rope;           // [t, 128, 64]
  int8_t* q_int8;                  // [t, 64, 128]
  __half* q_scale;                 // [t, 64]
  uint32_t* status;
  int t, m_tiles;
  int vec_rope;                    // the rotary tables are 16-byte aligned
  int independent;                 // the activations do not come from the kernel before this one
  int mla_items, items;            // items [0, mla_items) are MLA heads, the rest indexer heads; token tile fastest
};

template <bool kV4>
__global__ void __launch_bounds__(kHdThreads, 1)
heads_tc_kernel(const __grid_constant__ CUtensorMap a_map, const __grid_constant__ CUtensorMap wuq_map,
                const __grid_constant__ CUtensorMap wuq64_map, const __grid_constant__ CUtensorMap wuk_map,
                const __grid_constant__ CUtensorMap out_map, const __grid_constant__ CUtensorMap wqb_map,
                const __grid_constant__ CUtensorMap had_map, HeadParams p) {
  extern __shared__ __align__(1024) unsigned char smem[];
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + kHdOffBars);
  uint64_t* empty_bar = full_bar + kHdSlots;
  uint64_t* d1_bar = empty_bar + kHdSlots;
  uint64_t* a2_bar = d1_bar + 1;
  uint64_t* d2full_bar = a2_bar + 1;     // [2]
  uint64_t* d2empty_bar = d2full_bar + 2;
  uint32_t* tmem_ptr_s = reinterpret_cast<uint32_t*>(smem + kHdOffTmem);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if ((smem_u32(smem) & 1023u) != 0u) {
    if (tid == 0) report_status(p.status, DSV32_STATUS_INTERNAL, 70, smem_u32(smem));
    return;
  }
  constexpr int kSteps = (kV4 ? 1024 : 1536) / 128;   // reduction steps of the first product
  if (warp == 0) {
    if (lane == 0) {
      tma_prefetch_desc(&a_map);
      tma_prefetch_desc(&wqb_map);
      tma_prefetch_desc(&had_map);
      if constexpr (!kV4) {
        tma_prefetch_desc(&wuq_map);
        tma_prefetch_desc(&wuq64_map);
        tma_prefetch_desc(&wuk_map);
        tma_prefetch_desc(&out_map);
      }
      for (int i = 0; i < kHdSlots; ++i) {
        mbar_init(&full_bar[i], 1);
        mbar_init(&empty_bar[i], 1);
      }
      mbar_init(d1_bar, 1);
      mbar_init(a2_bar, 8);
      for (int i = 0; i < 2; ++i) {
        mbar_init(&d2full_bar[i], 1);
        mbar_init(&d2empty_bar[i], 8);
      }
      mbar_fence_init();
    }
  } else if (warp == 1) {
    tmem_alloc(tmem_ptr_s, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_ptr_s;
  pdl_trigger();

  if (warp == 0) {
    // ---- TMA producer --------------------------------------------------------------------------------------------
    if (lane == 0) {
      auto load_b = [&](bool mla, int head, int c, unsigned char* st, uint64_t* bar) {   // weights of one D1 step
        if (mla) {
          mbar_arrive_expect_tx(bar, 40960);
          tma_load_2d(st + 16384, &wuq_map, head * 192, c * 128, bar);
          tma_load_2d(st + 32768, &wuq64_map, head * 192 + 128, c * 128, bar);
        } else {
          mbar_arrive_expect_tx(bar, 32768);
          tma_load_2d(st + 16384, &wqb_map, head * 128, c * 128, bar);
        }
      };
      bool ok = true;
      int s = 0, ph = 1;
      for (int item = blockIdx.x; ok && item < p.items; item += gridDim.x) {
        const bool mla = !kV4 && item < p.mla_items;
        const int local = mla ? item : item - p.mla_items;
        const int head = local / p.m_tiles, m = local % p.m_tiles;
        int c = 0;
        if (item == static_cast<int>(blockIdx.x)) {   // the ring is empty: weights first, activations once they exist
          for (; c < kHdSlots; ++c) load_b(mla, head, c, smem + c * kHdSlotBytes, &full_bar[c]);
          if (!p.independent) pdl_wait();
          for (c = 0; c < kHdSlots; ++c) tma_load_2d(smem + c * kHdSlotBytes, &a_map, c * 128, m * 128, &full_bar[c]);
          ph = 0;   // every slot has been used once
        }
        for (; c < kSteps; ++c) {
          if (!mbar_wait(&empty_bar[s], ph, p.status, 71)) { ok = false; break; }
          load_b(mla, head, c, smem + s * kHdSlotBytes, &full_bar[s]);
          tma_load_2d(smem + s * kHdSlotBytes, &a_map, c * 128, m * 128, &full_bar[s]);
          if (++s == kHdSlots) { s = 0; ph ^= 1; }
        }
        for (int j = 0; ok && j < (mla ? 4 : 1); ++j) {   // right operand of the second product: 128 x 128 bf16
          if (!mbar_wait(&empty_bar[s], ph, p.status, 72)) { ok = false; break; }
          unsigned char* st = smem + s * kHdSlotBytes;
          mbar_arrive_expect_tx(&full_bar[s], 32768);
          if (mla) {
            tma_load_2d(st, &wuk_map, j * 256, head * 128, &full_bar[s]);
            tma_load_2d(st + 16384, &wuk_map, j * 256 + 128, head * 128, &full_bar[s]);
          } else {
            tma_load_2d(st, &had_map, 0, 0, &full_bar[s]);
            tma_load_2d(st + 16384, &had_map, 128, 0, &full_bar[s]);
          }
          if (++s == kHdSlots) { s = 0; ph ^= 1; }
        }
      }
    }
  } else if (warp == 1) {
    // ---- MMA issuer ------------------------------------------------------------------------------------------------
    constexpr uint32_t idesc_nope = umma_idesc_i8(128, 128, true), idesc_rope = umma_idesc_i8(128, 64, true);
    constexpr uint32_t idesc2 = umma_idesc_bf16(128, 128, false, true);
    const uint32_t tbase = __shfl_sync(0xffffffffu, tmem_base, 0);
    bool ok = true;
    int s = 0, ph = 0, q = 0, i = 0;
    for (int item = blockIdx.x; ok && item < p.items; item += gridDim.x, ++i) {
      const bool mla = !kV4 && item < p.mla_items;
      for (int c = 0; c < kSteps; ++c) {
        ok = __all_sync(0xffffffffu, mbar_wait(&full_bar[s], ph, p.status, 73));
        if (!ok) break;
        tc_fence_after();
        const uint32_t st = smem_u32(smem + s * kHdSlotBytes);
        const uint64_t ad = umma_smem_desc_sw128(st, 16, 1024);
        const uint64_t bd = umma_smem_desc_sw128(st + 16384, 16384, 1024), rd = umma_smem_desc_sw64_mn(st + 32768);
        if (elect_one()) {
#pragma unroll
          for (int ks = 0; ks < 4; ++ks)   // 32 reduction elements: 32 bytes of A's row, 32 weight rows
            umma_i8_ss(tbase + kColD1, ad + 2 * ks, bd + 256 * ks, idesc_nope, (c > 0 || ks > 0) ? 1u : 0u);
          if (mla) {
#pragma unroll
            for (int ks = 0; ks < 4; ++ks)
              umma_i8_ss(tbase + kColD1 + 128, ad + 2 * ks, rd + 128 * ks, idesc_rope, (c > 0 || ks > 0) ? 1u : 0u);
          }
          umma_commit(&empty_bar[s]);
          if (c == kSteps - 1) umma_commit(d1_bar);
        }
        __syncwarp();
        if (++s == kHdSlots) { s = 0; ph ^= 1; }
      }
      // the left operand is in place (and D1 has been read: the next item may overwrite it)
      if (ok) ok = __all_sync(0xffffffffu, mbar_wait(a2_bar, i & 1, p.status, 74));
      for (int j = 0; ok && j < (mla ? 4 : 1); ++j, ++q) {
        const int b = q & 1;
        ok = __all_sync(0xffffffffu, mbar_wait(&full_bar[s], ph, p.status, 75) &&
                                         mbar_wait(&d2empty_bar[b], ((q >> 1) & 1) ^ 1, p.status, 76));
        if (!ok) break;
        tc_fence_after();
        const uint64_t bd = umma_smem_desc_sw128(smem_u32(smem + s * kHdSlotBytes), 16384, 1024);
        if (elect_one()) {
#pragma unroll
          for (int ks = 0; ks < 8; ++ks)   // 16 dims per product
            umma_f16_ts(tbase + kColD2 + b * 128, tbase + kColA2 + ks * 8, bd + 128 * ks, idesc2, ks > 0 ? 1u : 0u);
          umma_commit(&empty_bar[s]);
          umma_commit(&d2full_bar[b]);
        }
        __syncwarp();
        if (++s == kHdSlots) { s = 0; ph ^= 1; }
      }
    }
  } else {
    // ---- epilogue ----------------------------------------------------------------------------------------------------
    if (!p.independent) pdl_wait();   // the row scales are the predecessor's
    const int quarter = warp & 3, half = (warp - 2) >> 2;
    const uint32_t lane_base = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
    unsigned char* buf = smem + kHdOffStore + (warp - 2) * 4096;
    float* red = reinterpret_cast<float*>(smem + kHdOffRed);
    float* scale_s = reinterpret_cast<float*>(smem + kHdOffScale);
    const uint32_t sw = static_cast<uint32_t>(lane & 7);
    int q = 0, i = 0;
    for (int item = blockIdx.x; item < p.items; item += gridDim.x, ++i) {
      const bool mla = !kV4 && item < p.mla_items;
      const int local = mla ? item : item - p.mla_items;
      const int head = local / p.m_tiles, row0 = (local % p.m_tiles) * 128 + quarter * 32;
      const int tok = row0 + lane;
      const bool live = tok < p.t;
      const int tk = live ? tok : p.t - 1;   // clamp for loads
      const bool warp_live = row0 < p.t;
      // Everything the item needs from global memory is fetched before its accumulator is waited for: the next head's
      // scales and a token tile's factors are never in L1, and a miss on the way from D1 to the left operand idles the
      // tensor core for as long.
      const float qs = p.row_scale[tk];
      uint32_t cl[8], ch[8], sl[8], sh[8];   // rotary factors of dims 16 half .. and 32 + 16 half .. (V4: 32 half .. and 16 further)
      {
        const __nv_bfloat16* cr = (mla ? p.cos : p.cos_idx) + static_cast<size_t>(tk) * 64 + half * (kV4 ? 32 : 16);
        const __nv_bfloat16* sr = (mla ? p.sin : p.sin_idx) + static_cast<size_t>(tk) * 64 + half * (kV4 ? 32 : 16);
        const bool vec = p.vec_rope != 0;
        rope16(cr, vec, cl);
        rope16(cr + (kV4 ? 16 : 32), vec, ch);
        rope16(sr, vec, sl);
        rope16(sr + (kV4 ? 16 : 32), vec, sh);
      }
      float* ws = scale_s + (i & 1) * 192;
      {
        const int e = (warp - 2) * 32 + lane;
        if (mla ? e < 192 : e < 128) ws[e] = __ldg(mla ? p.w_uq_scale + head * 192 + e : p.w_qb_scale + head * 128 + e);
      }
      asm volatile("bar.sync 5, 256;" ::: "memory");   // (two buffers: the one before last has been read by everybody)
      if (!__all_sync(0xffffffffu, mbar_wait(d1_bar, i & 1, p.status, 77))) break;
      tc_fence_after();
      // dequantised value of an accumulator column with scale w
      auto dq = [&](uint32_t v, float w) { return __fmul_rn(__fmul_rn(__int2float_rn(static_cast<int>(v)), qs), w); };
      if (warp_live) {
        if (mla) {
          const float* w = ws + half * 64;
          uint32_t r[32], pk[32];
#pragma unroll
          for (int c = 0; c < 2; ++c) {   // nope dims 64 half + 32 c ..
            tmem_ld_32x32b_x32(lane_base + kColD1 + half * 64 + c * 32, r);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 32; j += 4) {
              const float4 w4 = *reinterpret_cast<const float4*>(w + c * 32 + j);
              pk[c * 16 + (j >> 1)] = pack_bf16x2(dq(r[j], w4.x), dq(r[j + 1], w4.y));
              pk[c * 16 + (j >> 1) + 1] = pack_bf16x2(dq(r[j + 2], w4.z), dq(r[j + 3], w4.w));
            }
          }
          tmem_st_32x32b_x32(lane_base + kColA2 + half * 32, pk);
          // rope inputs 32 half .. 32 half + 31 = pairs 16 half ..: de-interleave and rotate
          const float* wr = ws + 128 + half * 32;
          tmem_ld_32x32b_x32(lane_base + kColD1 + 128 + half * 32, r);
          tmem_ld_wait();
          uint32_t lo[8], hi[8];
#pragma unroll
          for (int jp = 0; jp < 8; ++jp) {   // output pairs (16 half + 2 jp, + 1) and 32 further
            const float4 w4 = *reinterpret_cast<const float4*>(wr + 4 * jp);
            const float e0 = bf16_round(dq(r[4 * jp], w4.x)), o0 = bf16_round(dq(r[4 * jp + 1], w4.y));
            const float e1 = bf16_round(dq(r[4 * jp + 2], w4.z)), o1 = bf16_round(dq(r[4 * jp + 3], w4.w));
            lo[jp] = pack_bf16x2(__fadd_rn(__fmul_rn(e0, bf_lo(cl[jp])), __fmul_rn(-o0, bf_lo(sl[jp]))),
                                 __fadd_rn(__fmul_rn(e1, bf_hi(cl[jp])), __fmul_rn(-o1, bf_hi(sl[jp]))));
            hi[jp] = pack_bf16x2(__fadd_rn(__fmul_rn(o0, bf_lo(ch[jp])), __fmul_rn(e0, bf_lo(sh[jp]))),
                                 __fadd_rn(__fmul_rn(o1, bf_hi(ch[jp])), __fmul_rn(e1, bf_hi(sh[jp]))));
          }
          if (live) {
            uint4* dst = reinterpret_cast<uint4*>(p.q_rope + (static_cast<size_t>(tok) * 128 + head) * 64 + half * 16);
            dst[0] = make_uint4(lo[0], lo[1], lo[2], lo[3]);
            dst[1] = make_uint4(lo[4], lo[5], lo[6], lo[7]);
            dst[4] = make_uint4(hi[0], hi[1], hi[2], hi[3]);
            dst[5] = make_uint4(hi[4], hi[5], hi[6], hi[7]);
          }
        } else if constexpr (!kV4) {
          // dims 16 half .. and 32 + 16 half ..: rotate-half pairs (d, d + 32); dims 64 + 32 half ..: plain
          uint32_t a[16], b[16], r[32];
          tmem_ld_32x32b_x16(lane_base + kColD1 + half * 16, a);
          tmem_ld_32x32b_x16(lane_base + kColD1 + 32 + half * 16, b);
          tmem_ld_32x32b_x32(lane_base + kColD1 + 64 + half * 32, r);
          tmem_ld_wait();
          uint32_t lo[8], hi[8], pk[16];
#pragma unroll
          for (int jp = 0; jp < 8; ++jp) {
            const float2 wl = *reinterpret_cast<const float2*>(ws + half * 16 + 2 * jp);
            const float2 wh = *reinterpret_cast<const float2*>(ws + 32 + half * 16 + 2 * jp);
            const float x0 = bf16_round(dq(a[2 * jp], wl.x)), x1 = bf16_round(dq(a[2 * jp + 1], wl.y));
            const float y0 = bf16_round(dq(b[2 * jp], wh.x)), y1 = bf16_round(dq(b[2 * jp + 1], wh.y));
            lo[jp] = pack_bf16x2(__fadd_rn(__fmul_rn(x0, bf_lo(cl[jp])), __fmul_rn(-y0, bf_lo(sl[jp]))),
                                 __fadd_rn(__fmul_rn(x1, bf_hi(cl[jp])), __fmul_rn(-y1, bf_hi(sl[jp]))));
            hi[jp] = pack_bf16x2(__fadd_rn(__fmul_rn(y0, bf_lo(ch[jp])), __fmul_rn(x0, bf_lo(sh[jp]))),
                                 __fadd_rn(__fmul_rn(y1, bf_hi(ch[jp])), __fmul_rn(x1, bf_hi(sh[jp]))));
          }
#pragma unroll
          for (int j = 0; j < 32; j += 4) {
            const float4 w4 = *reinterpret_cast<const float4*>(ws + 64 + half * 32 + j);
            pk[j >> 1] = pack_bf16x2(dq(r[j], w4.x), dq(r[j + 1], w4.y));
            pk[(j >> 1) + 1] = pack_bf16x2(dq(r[j + 2], w4.z), dq(r[j + 3], w4.w));
          }
          tmem_st_32x32b_x8(lane_base + kColA2 + half * 8, lo);
          tmem_st_32x32b_x8(lane_base + kColA2 + 16 + half * 8, hi);
          tmem_st_32x32b_x16(lane_base + kColA2 + 32 + half * 16, pk);
        } else {
          // dims 32 half ..: plain; dims 64 + 32 half ..: interleaved inverse rotary embedding
          uint32_t r[32], x[32], pk[16];
          tmem_ld_32x32b_x32(lane_base + kColD1 + half * 32, r);
          tmem_ld_32x32b_x32(lane_base + kColD1 + 64 + half * 32, x);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 32; j += 4) {
            const float4 w4 = *reinterpret_cast<const float4*>(ws + half * 32 + j);
            pk[j >> 1] = pack_bf16x2(dq(r[j], w4.x), dq(r[j + 1], w4.y));
            pk[(j >> 1) + 1] = pack_bf16x2(dq(r[j + 2], w4.z), dq(r[j + 3], w4.w));
          }
          tmem_st_32x32b_x16(lane_base + kColA2 + half * 16, pk);
#pragma unroll
          for (int j = 0; j < 32; j += 2) {
            const float2 w2 = *reinterpret_cast<const float2*>(ws + 64 + half * 32 + j);
            const uint32_t cw = j < 16 ? cl[(j >> 1) & 7] : ch[(j >> 1) & 7], sn = j < 16 ? sl[(j >> 1) & 7] : sh[(j >> 1) & 7];
            const float xe = bf16_round(dq(x[j], w2.x)), xo = bf16_round(dq(x[j + 1], w2.y));
            pk[j >> 1] = pack_bf16x2(__fadd_rn(__fmul_rn(xe, bf_lo(cw)), __fmul_rn(xo, bf_lo(sn))),
                                     __fadd_rn(__fmul_rn(xo, bf_hi(cw)), __fmul_rn(-xe, bf_hi(sn))));
          }
          tmem_st_32x32b_x16(lane_base + kColA2 + 32 + half * 16, pk);
        }
        tmem_st_wait();
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(a2_bar);

      // ---- second product -----------------------------------------------------------------------------------------
      bool ok = true;
      for (int j = 0; ok && j < (mla ? 4 : 1); ++j, ++q) {
        const int b = q & 1;
        ok = __all_sync(0xffffffffu, mbar_wait(&d2full_bar[b], (q >> 1) & 1, p.status, 78));
        if (!ok) break;
        tc_fence_after();
        uint32_t r[2][32];
        if (warp_live) {
          tmem_ld_32x32b_x32(lane_base + kColD2 + b * 128 + half * 64, r[0]);
          tmem_ld_32x32b_x32(lane_base + kColD2 + b * 128 + half * 64 + 32, r[1]);
          tmem_ld_wait();
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&d2empty_bar[b]);
        if (mla) {
          if (warp_live) {
            if (lane == 0) tma_store_wait_read<0>();   // the store before has read the buffer
            __syncwarp();
            unsigned char* dst = buf + lane * 128;
#pragma unroll
            for (int u = 0; u < 8; ++u) {
              const uint32_t* v = &r[u >> 2][(u & 3) * 8];
              *reinterpret_cast<uint4*>(dst + ((u ^ sw) << 4)) =
                  make_uint4(pack_bf16x2(__uint_as_float(v[0]), __uint_as_float(v[1])), pack_bf16x2(__uint_as_float(v[2]), __uint_as_float(v[3])),
                             pack_bf16x2(__uint_as_float(v[4]), __uint_as_float(v[5])), pack_bf16x2(__uint_as_float(v[6]), __uint_as_float(v[7])));
            }
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
              tma_store_2d(&out_map, buf, (head * 512 + j * 128 + half * 64) * 2, row0);
              tma_store_commit();
            }
          }
        } else {
          // row maximum of the bf16-rounded hadamard output over both halves, then int8
          float amax = 0.f;
          if (warp_live) {
#pragma unroll
            for (int e = 0; e < 64; ++e) {
              const float v = bf16_round(__uint_as_float(r[e >> 5][e & 31]));
              r[e >> 5][e & 31] = __float_as_uint(v);
              amax = fmaxf(amax, fabsf(v));
            }
          }
          float* slot = red + (((i & 1) * 4 + quarter) * 2) * 32;
          slot[half * 32 + lane] = amax;
          pair_barrier(1 + quarter);
          amax = fmaxf(amax, slot[(half ^ 1) * 32 + lane]);
          const float sq = __fdiv_rn(127.0f, amax);
          if (live) {
            uint4* dst = reinterpret_cast<uint4*>(p.q_int8 + (static_cast<size_t>(tok) * 64 + head) * 128 + half * 64);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              uint32_t o[4];
#pragma unroll
              for (int x = 0; x < 4; ++x) {
                const int e = u * 16 + x * 4;
                uint32_t w = 0;
#pragma unroll
                for (int y = 0; y < 4; ++y) {
                  const int v = static_cast<int>(rintf(__fmul_rn(__uint_as_float(r[(e + y) >> 5][(e + y) & 31]), sq)));
                  w |= static_cast<uint32_t>(v & 0xff) << (8 * y);
                }
                o[x] = w;
              }
              dst[u] = make_uint4(o[0], o[1], o[2], o[3]);
            }
            if (half == 0) p.q_scale[static_cast<size_t>(tok) * 64 + head] = __float2half_rn(__fdiv_rn(1.0f, sq));
          }
        }
      }
      if (!ok) break;
    }
    if (lane == 0) tma_store_wait_all();
    pdl_wait();   // this kernel does not complete before its predecessor
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

template <bool kV4>
static int launch_heads(const CUtensorMap (&maps)[7], const HeadParams& p, cudaStream_t stream, int ctas = 0) {
  auto kernel = heads_tc_kernel<kV4>;
  cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kHdSmemBytes));
  if (ctas <= 0) ctas = sm_count();
  launch_ex(kernel, dim3(p.items < ctas ? p.items : ctas), kHdThreads, kHdSmemBytes, stream, true, 1, maps[0], maps[1], maps[2], maps[3],
            maps[4], maps[5], maps[6], p);
  count_launch();
  return check_launch("heads_tc_kernel");
}

// The heads of the V3.2 prologs: MLA heads (m given), indexer heads (ip given), or both, which then share t and q_norm.
// Launched dependent on the kernel before it in the stream; `independent`: q_norm is not that kernel's output.
int launch_prolog_heads(const MlaParams* m, const PrologParams* ip, bool independent, cudaStream_t stream, int ctas) {
  HeadParams p{};
  p.t = m != nullptr ? m->t : ip->t;
  p.m_tiles = (p.t + 127) / 128;
  p.independent = independent ? 1 : 0;
  p.row_scale = m != nullptr ? m->q_norm_scale : ip->q_norm_scale;
  p.status = m != nullptr ? m->status : ip->status;
  CUtensorMap maps[7];
  int rc = make_tensor_map_2d_u8(&maps[0], m != nullptr ? m->q_norm : ip->q_norm, p.t, 1536, 128, 128);
  uintptr_t ralign = 0;
  if (m != nullptr) {
    p.w_uq_scale = m->w_qb_scale;
    p.cos = m->cos;
    p.sin = m->sin;
    ralign |= reinterpret_cast<uintptr_t>(m->cos) | reinterpret_cast<uintptr_t>(m->sin);
    p.q_rope = m->q_rope;
    p.mla_items = 128 * p.m_tiles;
    if (rc == DSV32_OK) rc = make_tensor_map_2d_u8(&maps[1], m->w_uq_qr, 1536, 24576, 128, 128);
    if (rc == DSV32_OK) rc = make_tensor_map_2d_sw64(&maps[2], m->w_uq_qr, 1536, 24576, 128);
    if (rc == DSV32_OK) rc = make_tensor_map_2d_u8(&maps[3], m->w_uk, 128 * 128, 1024, 128, 128);
    if (rc == DSV32_OK) rc = make_tensor_map_2d_u8(&maps[4], m->q_nope, p.t, 128 * 1024, 32, 128);
  }
  p.items = p.mla_items;
  if (ip != nullptr) {
    p.w_qb_scale = ip->w_qb_scale;
    p.cos_idx = ip->cos;
    p.sin_idx = ip->sin;
    ralign |= reinterpret_cast<uintptr_t>(ip->cos) | reinterpret_cast<uintptr_t>(ip->sin);
    p.q_int8 = ip->q_int8;
    p.q_scale = ip->q_scale;
    p.items += 64 * p.m_tiles;
    if (rc == DSV32_OK) rc = make_tensor_map_2d_u8(&maps[5], ip->w_qb, 1536, 8192, 128, 128);
    if (rc == DSV32_OK) rc = make_tensor_map_2d_u8(&maps[6], ip->had_q, 128, 256, 128, 128);
  }
  if (rc != DSV32_OK) return rc;
  p.vec_rope = ralign % 16 == 0 ? 1 : 0;
  for (int i = 1; i < 5; ++i)
    if (m == nullptr) maps[i] = maps[0];
  for (int i = 5; i < 7; ++i)
    if (ip == nullptr) maps[i] = maps[0];
  return launch_heads<false>(maps, p, stream, ctas);
}

// The query heads of the V4 indexer prolog.
int launch_prolog_v4_heads(const PrologParams& ip, cudaStream_t stream) {
  HeadParams p{};
  p.t = ip.t;
  p.m_tiles = (p.t + 127) / 128;
  p.independent = 1;
  p.row_scale = ip.q_norm_scale;
  p.w_qb_scale = ip.w_qb_scale;
  p.cos_idx = ip.cos;
  p.sin_idx = ip.sin;
  p.vec_rope = (reinterpret_cast<uintptr_t>(ip.cos) | reinterpret_cast<uintptr_t>(ip.sin)) % 16 == 0 ? 1 : 0;
  p.q_int8 = ip.q_int8;
  p.q_scale = ip.q_scale;
  p.status = ip.status;
  p.items = 64 * p.m_tiles;
  CUtensorMap maps[7];
  int rc = make_tensor_map_2d_u8(&maps[0], ip.q_norm, p.t, 1024, 128, 128);
  if (rc == DSV32_OK) rc = make_tensor_map_2d_u8(&maps[5], ip.w_qb, 1024, 8192, 128, 128);
  if (rc == DSV32_OK) rc = make_tensor_map_2d_u8(&maps[6], ip.had_q, 128, 256, 128, 128);
  if (rc != DSV32_OK) return rc;
  for (int i = 1; i < 5; ++i) maps[i] = maps[0];
  return launch_heads<true>(maps, p, stream);
}

}  // namespace dsv32
