// Page-grouped lightning-indexer prolog with 8-bit float formats (MXFP8 E4M3 with E8M0 block scales, and HiF8).
// Follows python/tests/st/operator/pg/lightning_indexer_prolog_quant_mxfp8_impl.py:230-401 and
// lightning_indexer_prolog_quant_hif8_impl.py:230-406 (golden: test_pg_lightning_indexer_prolog_quant_mxfp8.py:272-345).
//
//   proj_tc_kernel     x . [wk | w_proj] (launch_proj_bf16, fp32 partial sums)
//   pg_unpack_kernel   beside it: the 8-bit operands of q_norm . w_qb widened to bf16 -- exactly: an E4M3 or HiF8 value has at
//                      most four significant bits and an E8M0 scale is a power of two -- so that the product runs on bf16
//                      tensor cores with fp32 accumulation: the sum the golden forms in fp32
//   pg_heads_kernel    (head, 128-token tile) items: the product in tensor memory, (HiF8: x token scale x column scale,) bf16,
//                      rotate-half rotary embedding of dims 0..63, x hadamard_q as a second product with the left operand in
//                      tensor memory, per-row dynamic quantisation to the 8-bit format with an fp32 scale.  Its first CTAs
//                      finish the keys instead, a token per warp: bf16, RMSNorm, rotary embedding, x hadamard_k, quantisation,
//                      scatter of the code row and of its scale into the page-grouped caches; and the head weights
// At 300 tokens and 24 heads one CTA per (token, head) for the query tail took 26 of 62 us, the GEMM between it and the
// unpacking wrote and read 15 MB of partial sums; now the three launches overlap and take 24 us.
// Every bf16 rounding sits where the operator puts it; products and sums of the rotary embedding are rounded
// separately (no fused multiply-add), as the operator's separate vector instructions do.
#include <cuda_fp8.h>

#include "finish.cuh"
#include "kernels.cuh"
#include "tc_common.cuh"

namespace dsv32 {

constexpr int kPgDim = 128, kPgRope = 64, kPgXwCols = 256;

__device__ __forceinline__ float pg_bf16r(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }

// ---- HiF8 (bit layout: framework/src/interface/machine/device/tilefwk/aicore_print_base.h:361-484) -----------------
// sign | prefix-coded exponent width | sign-magnitude exponent with an implied leading one | mantissa:
//   0000mmm 2^(m-23) (m = 0: zero, or NaN with the sign bit)   0001mmm e = 0   001emmm e = +-1   01semmm e = +-(2+e)
//   10seemm e = +-(4+ee)   11seeem e = +-(8+eee), e = +15 with mantissa 1 is infinity
__device__ __forceinline__ float pg_pow2(int e) { return __int_as_float((e + 127) << 23); }  // -126 <= e <= 127

__device__ __forceinline__ float hif8_to_float(uint32_t code) {
  const uint32_t low = code & 0x7Fu;
  const float sign = (code & 0x80u) ? -1.f : 1.f;
  if ((low >> 3) == 0u) {
    const int m = static_cast<int>(low & 7u);
    if (m == 0) return (code & 0x80u) ? __int_as_float(0x7fc00000) : 0.f;
    return sign * pg_pow2(m - 23);
  }
  int ev, mant, bits;
  if ((low >> 3) == 1u) {
    ev = 0; mant = low & 7; bits = 3;
  } else if ((low >> 4) == 1u) {
    ev = ((low >> 3) & 1u) ? -1 : 1; mant = low & 7; bits = 3;
  } else if ((low >> 5) == 1u) {
    const int eb = (low >> 3) & 3;
    ev = (2 + (eb & 1)) * ((eb >> 1) ? -1 : 1); mant = low & 7; bits = 3;
  } else if ((low >> 5) == 2u) {
    const int eb = (low >> 2) & 7;
    ev = (4 + (eb & 3)) * ((eb >> 2) ? -1 : 1); mant = low & 3; bits = 2;
  } else {
    const int eb = (low >> 1) & 15;
    ev = (8 + (eb & 7)) * ((eb >> 3) ? -1 : 1); mant = low & 1; bits = 1;
    if (ev == 15 && mant == 1) return sign * __int_as_float(0x7f800000);
  }
  return sign * pg_pow2(ev) * (1.f + static_cast<float>(mant) * pg_pow2(-bits));
}
// Nearest representable value, a tie to the larger magnitude, magnitudes above 2^15 to 2^15; NaN to the NaN code.  Without a
// branch: the lanes of a warp meet all exponent ranges, and the code of a branch each is long.
__device__ __forceinline__ uint32_t float_to_hif8(float x) {
  const uint32_t u = __float_as_uint(x), mag = min(u & 0x7fffffffu, 0x47000000u);   // 2^15
  const int ae = abs(static_cast<int>(mag >> 23) - 127);
  const int bits = ae <= 3 ? 3 : (ae <= 7 ? 2 : (ae <= 15 ? 1 : 0));   // mantissa bits at this exponent
  // half a step is added and the rest cut off; a carry runs into the exponent and leaves no mantissa.  Below 2^-15 there are
  // only powers of two down to 2^-22, which takes everything from 2^-23 on; what is below is nearer to zero, which has no sign
  const uint32_t r = mag + (0x400000u >> bits);
  const int e = max(static_cast<int>(r >> 23) - 127, -22), a = abs(e);
  const uint32_t m = (r >> (23 - bits)) & ((1u << bits) - 1u), es = e < 0 ? 1u : 0u;
  const int k = 31 - __clz(a | 1);                                     // prefix of the exponent's width
  uint32_t code = (static_cast<uint32_t>(k) << 5) | (es << 4) | (static_cast<uint32_t>(a - (1 << k)) << (4 - k));
  code = a <= 1 ? (a == 0 ? 0x08u : 0x10u | (es << 3)) : code;
  code = e <= -16 ? static_cast<uint32_t>(e + 23) : code | m;
  code |= (u >> 24) & 0x80u;
  code = mag < 0x34000000u ? 0u : code;                                // 2^-23
  return (u & 0x7fffffffu) > 0x7f800000u ? 0x80u : code;
}

__device__ __forceinline__ float e8m0_to_float(uint32_t code) {  // 2^(code - 127); code 255 is NaN
  if (code == 255u) return __int_as_float(0x7fc00000);
  return code == 0u ? __int_as_float(0x00400000) : __int_as_float(static_cast<int>(code << 23));
}

// ---- operands to bf16 ----------------------------------------------------------------------------------------------
// grid-stride over the regions, eight elements per thread; the hadamard matrices are copied to where TMA and vector loads can
// read them whatever their alignment
struct PgOperands {
  __nv_bfloat16* q;      // [t, q_lora]
  __nv_bfloat16* w;      // [q_lora, n]
  __nv_bfloat16* had;    // hadamard_q, hadamard_k
  __nv_bfloat16* xw;     // [h, 256] = [wk | w_proj | 0], or NULL: the projection reads wk and w_proj themselves
};

__global__ void __launch_bounds__(256) pg_unpack_kernel(PgPrologParams p, PgOperands o, int vec_scale) {
  const long long nq = static_cast<long long>(p.t) * p.q_lora / 8;
  const long long nw = static_cast<long long>(p.q_lora) * p.n / 8;
  const long long nh = 2 * kPgDim * kPgDim / 8;
  const long long nx = o.xw != nullptr ? static_cast<long long>(p.h) * kPgXwCols / 8 : 0;
  const bool mx = p.format == DSV32_PG_FORMAT_MXFP8;
  pdl_trigger();
  for (long long i = blockIdx.x * 256ll + threadIdx.x; i < nq + nw + nh + nx; i += static_cast<long long>(gridDim.x) * 256) {
    if (i < nq + nw) {
      const bool is_q = i < nq;
      const long long e0 = (is_q ? i : i - nq) * 8;                // first of eight consecutive elements of a row
      const uint2 raw = __ldcs(reinterpret_cast<const uint2*>((is_q ? p.q_norm : p.w_qb) + e0));
      float scale[8];
      if (!mx) {
#pragma unroll
        for (int j = 0; j < 8; ++j) scale[j] = 1.f;
      } else if (is_q) {                                           // one scale per 32 reduction elements of the row
        const float s = e8m0_to_float(p.q_norm_scale_e8[e0 / 32]);
#pragma unroll
        for (int j = 0; j < 8; ++j) scale[j] = s;
      } else {                                                     // block kb of column c: [kb / 2][c][kb % 2]
        const int k = static_cast<int>(e0 / p.n), c0 = static_cast<int>(e0 % p.n), odd = (k / 32) & 1;
        const uint8_t* sp = p.w_qb_scale_e8 + (static_cast<size_t>(k / 64) * p.n + c0) * 2;
        if (vec_scale) {
          const uint4 v = __ldg(reinterpret_cast<const uint4*>(sp));
          const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
          for (int j = 0; j < 8; ++j) scale[j] = e8m0_to_float((w[j >> 1] >> (16 * (j & 1) + 8 * odd)) & 0xffu);
        } else {
#pragma unroll
          for (int j = 0; j < 8; ++j) scale[j] = e8m0_to_float(sp[2 * j + odd]);
        }
      }
      uint32_t w[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint32_t two = ((j < 2 ? raw.x : raw.y) >> (16 * (j & 1))) & 0xffffu;
        float a, b;
        if (mx) {
          const __half2_raw h = __nv_cvt_fp8x2_to_halfraw2(static_cast<__nv_fp8x2_storage_t>(two), __NV_E4M3);
          const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&h));
          a = f.x;
          b = f.y;
        } else {
          a = hif8_to_float(two & 0xffu);
          b = hif8_to_float(two >> 8);
        }
        w[j] = pack_bf16x2(a * scale[2 * j], b * scale[2 * j + 1]);
      }
      *reinterpret_cast<uint4*>((is_q ? o.q : o.w) + e0) = make_uint4(w[0], w[1], w[2], w[3]);
    } else if (i < nq + nw + nh) {
      const int e0 = static_cast<int>(i - nq - nw) * 8;
      const __nv_bfloat16* src = e0 < kPgDim * kPgDim ? p.hadamard_q + e0 : p.hadamard_k + (e0 - kPgDim * kPgDim);
      __nv_bfloat16 v[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = src[j];
      *reinterpret_cast<uint4*>(o.had + e0) = *reinterpret_cast<const uint4*>(v);
    } else {
      const long long e0 = (i - nq - nw - nh) * 8;
      const long long k = e0 / kPgXwCols;
      const int c0 = static_cast<int>(e0 % kPgXwCols);
      __nv_bfloat16 v[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int c = c0 + j;
        v[j] = c < kPgDim ? p.wk[k * kPgDim + c]
                          : (c < kPgDim + p.heads ? p.w_proj[k * p.heads + (c - kPgDim)] : __float2bfloat16_rn(0.f));
      }
      *reinterpret_cast<uint4*>(o.xw + e0) = *reinterpret_cast<const uint4*>(v);
    }
  }
  pdl_wait();   // this kernel does not complete before the projection it runs beside
}

// ---- 8-bit code of a value, and the scale of a row with maximum `amax` ----------------------------------------------
template <bool kMx>
__device__ __forceinline__ float pg_row_scale(float amax) {
  return __fmul_rn(amax, kMx ? (1.0f / 448.0f) : (1.0f / 32768.0f));
}
template <bool kMx>
__device__ __forceinline__ uint32_t pg_code(float v, float scale) {
  const float y = __fdiv_rn(v, scale);
  if constexpr (kMx) return static_cast<uint32_t>(__nv_cvt_float_to_fp8(y, __NV_SATFINITE, __NV_E4M3));
  else return float_to_hif8(y);
}

// ---- keys and head weights: one token per warp, four dims per lane --------------------------------------------------
template <bool kMx>
__device__ __forceinline__ void pg_finish_key(const PgPrologParams& p, const ProjSums& src, const __nv_bfloat16* had, float* vec,
                                              int tok, int lane) {
  // head weights: bf16, x heads^-0.5 -> bf16, x 128^-0.5 -> bf16
  for (int j = lane; j < p.heads; j += 32) {
    float w = pg_bf16r(proj_sum(src, tok, kPgDim + j));
    w = pg_bf16r(__fmul_rn(w, p.heads_rsqrt));
    p.weights_out[static_cast<size_t>(tok) * p.heads + j] = __float2bfloat16_rn(__fmul_rn(w, 0.08838834764831845f));
  }
  // RMSNorm: x / sqrt(sum(x^2 / 128) + eps) * gamma
  float4 v[1];
  proj_sum4(src, tok, 4 * lane, v);
  float k[4] = {pg_bf16r(v[0].x), pg_bf16r(v[0].y), pg_bf16r(v[0].z), pg_bf16r(v[0].w)};
  float sq = 0.f;
#pragma unroll
  for (int j = 0; j < 4; ++j) sq += __fmul_rn(__fmul_rn(k[j], k[j]), 1.0f / 128.0f);
  const float rms = __fsqrt_rn(warp_sum(sq) + p.eps);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    k[j] = pg_bf16r(__fmul_rn(__fdiv_rn(k[j], rms), __bfloat162float(p.gamma_k[4 * lane + j])));
    const float other = __shfl_xor_sync(0xffffffffu, k[j], 8);   // rotate-half pairs (d, d + 32) sit eight lanes apart
    if (lane < 16) {
      const size_t at = static_cast<size_t>(tok) * kPgRope + 4 * lane + j;
      k[j] = pg_bf16r(__fadd_rn(__fmul_rn(k[j], __bfloat162float(p.cos[at])),
                                __fmul_rn(lane < 8 ? -other : other, __bfloat162float(p.sin[at]))));
    }
  }
  *reinterpret_cast<float4*>(vec + 4 * lane) = make_float4(k[0], k[1], k[2], k[3]);
  __syncwarp();
  float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 16
  for (int i = 0; i < kPgDim; ++i) {
    const float f = vec[i];
    const uint2 h = __ldcg(reinterpret_cast<const uint2*>(had + i * kPgDim + 4 * lane));
    acc[0] = fmaf(f, __uint_as_float(h.x << 16), acc[0]);
    acc[1] = fmaf(f, __uint_as_float(h.x & 0xffff0000u), acc[1]);
    acc[2] = fmaf(f, __uint_as_float(h.y << 16), acc[2]);
    acc[3] = fmaf(f, __uint_as_float(h.y & 0xffff0000u), acc[3]);
  }
  float amax = 0.f;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    acc[j] = pg_bf16r(acc[j]);
    amax = fmaxf(amax, fabsf(acc[j]));
  }
  const float scale = pg_row_scale<kMx>(warp_max(amax));
  // scatter into the page-grouped caches: row r lives in page r / block_size at slot r % block_size
  const long long r = p.k_cache_index[tok], rs = p.k_scale_cache_index[tok];
  if (r < 0 || r >= p.cache_rows || rs < 0 || rs >= p.cache_rows) {
    if (lane == 0) report_status(p.status, DSV32_STATUS_BAD_INDEX, tok, static_cast<uint32_t>(r < 0 || r >= p.cache_rows ? r : rs));
    return;
  }
  uint32_t w = 0;
#pragma unroll
  for (int j = 0; j < 4; ++j) w |= pg_code<kMx>(acc[j], scale) << (8 * j);
  store_bytes4(reinterpret_cast<int8_t*>(p.k_cache + (r / p.block_size) * p.k_block_stride + (r % p.block_size) * kPgDim + 4 * lane), w);
  if (lane == 0)
    *reinterpret_cast<float*>(reinterpret_cast<unsigned char*>(p.k_scale_cache) + (rs / p.block_size) * p.k_scale_block_stride +
                              (rs % p.block_size) * sizeof(float)) = scale;
}

// ---- query heads (and, in the first CTAs, the keys) -------------------------------------------------------------------
namespace {
constexpr int kPhThreads = 320, kPhWarps = kPhThreads / 32;
constexpr int kPhSlots = 6;
constexpr int kPhSlotBytes = 32768;                            // A 128 x 64 bf16 | B 64 x 128 bf16; hadamard_q: 128 x 128 bf16
constexpr int kPhOffRed = kPhSlots * kPhSlotBytes;             // float[2][4 quarters][2 halves][32]
constexpr int kPhOffScale = kPhOffRed + 2 * 4 * 2 * 32 * 4;    // float[2][128]: column scales (HiF8)
constexpr int kPhOffBars = kPhOffScale + 2 * kPgDim * 4;
constexpr int kPhNumBars = 2 * kPhSlots + 2 + 4;               // full, empty, d1_full, a2_full, d2_full[2], d2_empty[2]
constexpr int kPhOffTmem = kPhOffBars + kPhNumBars * 8;
constexpr size_t kPhSmemBytes = kPhOffTmem + 16;
static_assert(kPhSmemBytes <= 232448, "shared memory of one CTA");
constexpr uint32_t kPhColD1 = 0, kPhColA2 = 128, kPhColD2 = 256;

// 16 consecutive bf16 of a rotary table row as pairs
__device__ __forceinline__ void pg_rope16(const __nv_bfloat16* row, bool vec, uint32_t (&w)[8]) {
  if (vec) {
    const uint4 a = __ldg(reinterpret_cast<const uint4*>(row)), b = __ldg(reinterpret_cast<const uint4*>(row) + 1);
    w[0] = a.x; w[1] = a.y; w[2] = a.z; w[3] = a.w;
    w[4] = b.x; w[5] = b.y; w[6] = b.z; w[7] = b.w;
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i)
      w[i] = __ldg(reinterpret_cast<const uint16_t*>(row) + 2 * i) |
             (static_cast<uint32_t>(__ldg(reinterpret_cast<const uint16_t*>(row) + 2 * i + 1)) << 16);
  }
}
__device__ __forceinline__ float pg_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float pg_hi(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }
}  // namespace

// The structure of heads_tc_kernel with bf16 operands: warp 0 = TMA producer, 1 = MMA issuer, 2..9 = epilogue.  What bounds it at
// decode sizes is the chain product -> tail -> product -> tail of a tile, 24 heads x ceil(t / 128) tiles wide.
template <bool kMx>
__global__ void __launch_bounds__(kPhThreads, 1)
pg_heads_kernel(const __grid_constant__ CUtensorMap a_map, const __grid_constant__ CUtensorMap b_map,
                const __grid_constant__ CUtensorMap had_map, PgPrologParams p, ProjSums src, const __nv_bfloat16* had_k, int key_ctas,
                int m_tiles, int vec_rope, int vec_out) {
  extern __shared__ __align__(1024) unsigned char smem[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (static_cast<int>(blockIdx.x) < key_ctas) {
    pdl_trigger();
    pdl_wait();
    const int tok = blockIdx.x * kPhWarps + warp;
    if (tok < p.t) pg_finish_key<kMx>(p, src, had_k, reinterpret_cast<float*>(smem) + warp * kPgDim, tok, lane);
    return;
  }
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + kPhOffBars);
  uint64_t* empty_bar = full_bar + kPhSlots;
  uint64_t* d1_bar = empty_bar + kPhSlots;
  uint64_t* a2_bar = d1_bar + 1;
  uint64_t* d2full_bar = a2_bar + 1;     // [2]
  uint64_t* d2empty_bar = d2full_bar + 2;
  uint32_t* tmem_ptr_s = reinterpret_cast<uint32_t*>(smem + kPhOffTmem);
  if ((smem_u32(smem) & 1023u) != 0u) {
    if (tid == 0) report_status(p.status, DSV32_STATUS_INTERNAL, 90, smem_u32(smem));
    return;
  }
  const int first = blockIdx.x - key_ctas, step = gridDim.x - key_ctas, items = p.heads * m_tiles, ksteps = p.q_lora / 64;
  if (warp == 0) {
    if (lane == 0) {
      tma_prefetch_desc(&a_map);
      tma_prefetch_desc(&b_map);
      tma_prefetch_desc(&had_map);
      for (int i = 0; i < kPhSlots; ++i) {
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
  pdl_wait();   // the operands are the unpacking kernel's

  if (warp == 0) {
    if (lane == 0) {
      bool ok = true;
      int s = 0, ph = 1;
      for (int item = first; ok && item < items; item += step) {
        const int head = item / m_tiles, m = item % m_tiles;
        for (int c = 0; c <= ksteps; ++c) {
          if (!mbar_wait(&empty_bar[s], ph, p.status, 91)) { ok = false; break; }
          unsigned char* st = smem + s * kPhSlotBytes;
          mbar_arrive_expect_tx(&full_bar[s], kPhSlotBytes);
          if (c < ksteps) {
            tma_load_2d(st, &a_map, c * 128, m * 128, &full_bar[s]);
            tma_load_2d(st + 16384, &b_map, head * 256, c * 64, &full_bar[s]);
            tma_load_2d(st + 16384 + 8192, &b_map, head * 256 + 128, c * 64, &full_bar[s]);
          } else {   // right operand of the second product
            tma_load_2d(st, &had_map, 0, 0, &full_bar[s]);
            tma_load_2d(st + 16384, &had_map, 128, 0, &full_bar[s]);
          }
          if (++s == kPhSlots) { s = 0; ph ^= 1; }
        }
      }
    }
  } else if (warp == 1) {
    constexpr uint32_t idesc = umma_idesc_bf16(128, 128, false, true);
    const uint32_t tbase = __shfl_sync(0xffffffffu, tmem_base, 0);
    bool ok = true;
    int s = 0, ph = 0, i = 0;
    for (int item = first; ok && item < items; item += step, ++i) {
      for (int c = 0; c < ksteps; ++c) {
        ok = __all_sync(0xffffffffu, mbar_wait(&full_bar[s], ph, p.status, 92));
        if (!ok) break;
        tc_fence_after();
        const uint32_t st = smem_u32(smem + s * kPhSlotBytes);
        const uint64_t ad = umma_smem_desc_sw128(st, 16, 1024), bd = umma_smem_desc_sw128(st + 16384, 8192, 1024);
        if (elect_one()) {
#pragma unroll
          for (int ks = 0; ks < 4; ++ks)
            umma_f16_ss(tbase + kPhColD1, ad + 2 * ks, bd + 128 * ks, idesc, (c > 0 || ks > 0) ? 1u : 0u);
          umma_commit(&empty_bar[s]);
          if (c == ksteps - 1) umma_commit(d1_bar);
        }
        __syncwarp();
        if (++s == kPhSlots) { s = 0; ph ^= 1; }
      }
      const int b = i & 1;
      // the left operand is in place (and D1 has been read: the next item may overwrite it)
      if (ok)
        ok = __all_sync(0xffffffffu, mbar_wait(a2_bar, i & 1, p.status, 93) && mbar_wait(&full_bar[s], ph, p.status, 94) &&
                                         mbar_wait(&d2empty_bar[b], ((i >> 1) & 1) ^ 1, p.status, 95));
      if (!ok) break;
      tc_fence_after();
      const uint64_t bd = umma_smem_desc_sw128(smem_u32(smem + s * kPhSlotBytes), 16384, 1024);
      if (elect_one()) {
#pragma unroll
        for (int ks = 0; ks < 8; ++ks)
          umma_f16_ts(tbase + kPhColD2 + b * 128, tbase + kPhColA2 + ks * 8, bd + 128 * ks, idesc, ks > 0 ? 1u : 0u);
        umma_commit(&empty_bar[s]);
        umma_commit(&d2full_bar[b]);
      }
      __syncwarp();
      if (++s == kPhSlots) { s = 0; ph ^= 1; }
    }
  } else {
    const int quarter = warp & 3, half = (warp - 2) >> 2;
    const uint32_t lane_base = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
    float* red = reinterpret_cast<float*>(smem + kPhOffRed);
    float* scale_s = reinterpret_cast<float*>(smem + kPhOffScale);
    int i = 0;
    for (int item = first; item < items; item += step, ++i) {
      const int head = item / m_tiles, row0 = (item % m_tiles) * 128 + quarter * 32;
      const int tok = row0 + lane;
      const bool live = tok < p.t, warp_live = row0 < p.t;
      const int tk = live ? tok : p.t - 1;   // clamp for loads
      float qs = 1.f;
      float* ws = scale_s + (i & 1) * kPgDim;
      if constexpr (!kMx) {
        qs = p.q_norm_scale_f32[tk];
        const int e = (warp - 2) * 32 + lane;
        if (e < kPgDim) ws[e] = __ldg(p.w_qb_scale_f32 + head * kPgDim + e);
        asm volatile("bar.sync 5, 256;" ::: "memory");
      }
      uint32_t cl[8], ch[8], sl[8], sh[8];   // rotary factors of dims 16 half .. and 32 + 16 half ..
      {
        const __nv_bfloat16* cr = p.cos + static_cast<size_t>(tk) * kPgRope + half * 16;
        const __nv_bfloat16* sr = p.sin + static_cast<size_t>(tk) * kPgRope + half * 16;
        pg_rope16(cr, vec_rope != 0, cl);
        pg_rope16(cr + 32, vec_rope != 0, ch);
        pg_rope16(sr, vec_rope != 0, sl);
        pg_rope16(sr + 32, vec_rope != 0, sh);
      }
      auto val = [&](uint32_t v, int col) {
        const float f = __uint_as_float(v);
        return kMx ? f : __fmul_rn(__fmul_rn(f, qs), ws[col]);
      };
      if (!__all_sync(0xffffffffu, mbar_wait(d1_bar, i & 1, p.status, 96))) break;
      tc_fence_after();
      if (warp_live) {
        // dims 16 half .. and 32 + 16 half ..: rotate-half pairs (d, d + 32); dims 64 + 32 half ..: plain
        uint32_t a[16], b[16], r[32];
        tmem_ld_32x32b_x16(lane_base + kPhColD1 + half * 16, a);
        tmem_ld_32x32b_x16(lane_base + kPhColD1 + 32 + half * 16, b);
        tmem_ld_32x32b_x32(lane_base + kPhColD1 + 64 + half * 32, r);
        tmem_ld_wait();
        uint32_t lo[8], hi[8], pk[16];
#pragma unroll
        for (int jp = 0; jp < 8; ++jp) {
          const float x0 = pg_bf16r(val(a[2 * jp], half * 16 + 2 * jp)), x1 = pg_bf16r(val(a[2 * jp + 1], half * 16 + 2 * jp + 1));
          const float y0 = pg_bf16r(val(b[2 * jp], 32 + half * 16 + 2 * jp)), y1 = pg_bf16r(val(b[2 * jp + 1], 33 + half * 16 + 2 * jp));
          lo[jp] = pack_bf16x2(__fadd_rn(__fmul_rn(x0, pg_lo(cl[jp])), __fmul_rn(-y0, pg_lo(sl[jp]))),
                               __fadd_rn(__fmul_rn(x1, pg_hi(cl[jp])), __fmul_rn(-y1, pg_hi(sl[jp]))));
          hi[jp] = pack_bf16x2(__fadd_rn(__fmul_rn(y0, pg_lo(ch[jp])), __fmul_rn(x0, pg_lo(sh[jp]))),
                               __fadd_rn(__fmul_rn(y1, pg_hi(ch[jp])), __fmul_rn(x1, pg_hi(sh[jp]))));
        }
#pragma unroll
        for (int j = 0; j < 32; j += 2)
          pk[j >> 1] = pack_bf16x2(val(r[j], 64 + half * 32 + j), val(r[j + 1], 65 + half * 32 + j));
        tmem_st_32x32b_x8(lane_base + kPhColA2 + half * 8, lo);
        tmem_st_32x32b_x8(lane_base + kPhColA2 + 16 + half * 8, hi);
        tmem_st_32x32b_x16(lane_base + kPhColA2 + 32 + half * 16, pk);
        tmem_st_wait();
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(a2_bar);
      // ---- hadamard product: row maximum of the bf16-rounded values over both halves, then the codes --------------------
      const int b = i & 1;
      if (!__all_sync(0xffffffffu, mbar_wait(&d2full_bar[b], (i >> 1) & 1, p.status, 97))) break;
      tc_fence_after();
      const uint32_t d2 = lane_base + kPhColD2 + b * 128 + half * 64;
      uint8_t* dst = p.q_out + (static_cast<size_t>(tk) * p.heads + head) * kPgDim + half * 64;
      float* slot = red + (((i & 1) * 4 + quarter) * 2) * 32;
      auto row_scale = [&](float amax) {   // of both halves
        slot[half * 32 + lane] = amax;
        asm volatile("bar.sync %0, 64;" ::"r"(1 + quarter) : "memory");
        return pg_row_scale<kMx>(fmaxf(amax, slot[(half ^ 1) * 32 + lane]));
      };
      auto release = [&] {   // D2 has been read
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&d2empty_bar[b]);
      };
      auto store16 = [&](int u, const uint32_t* r, float scale) {   // columns 16 u .. of this half
        uint32_t o[4] = {0u, 0u, 0u, 0u};
#pragma unroll
        for (int e = 0; e < 16; ++e) o[e >> 2] |= pg_code<kMx>(__uint_as_float(r[e]), scale) << (8 * (e & 3));
        if (vec_out) {
          reinterpret_cast<uint4*>(dst)[u] = make_uint4(o[0], o[1], o[2], o[3]);
        } else {
#pragma unroll
          for (int x = 0; x < 4; ++x) store_bytes4(reinterpret_cast<int8_t*>(dst + u * 16 + x * 4), o[x]);
        }
      };
      float scale, amax = 0.f;
      if constexpr (kMx) {
        uint32_t r[64];
        if (warp_live) {
          tmem_ld_32x32b_x32(d2, *reinterpret_cast<uint32_t(*)[32]>(r));
          tmem_ld_32x32b_x32(d2 + 32, *reinterpret_cast<uint32_t(*)[32]>(r + 32));
          tmem_ld_wait();
        }
        release();
        if (warp_live) {
#pragma unroll
          for (int e = 0; e < 64; ++e) {
            const float v = pg_bf16r(__uint_as_float(r[e]));
            r[e] = __float_as_uint(v);
            amax = fmaxf(amax, fabsf(v));
          }
        }
        scale = row_scale(amax);
        if (live) {
#pragma unroll
          for (int u = 0; u < 4; ++u) store16(u, r + 16 * u, scale);
        }
      } else {
        // The columns are read twice, for the maximum and then sixteen at a time in a loop that stays one: the code of 64 of these
        // conversions in a row is fetched anew by every call (45 KB without a branch in them, 100 with: 27, 44 and 59 us a call at
        // one token).  For the other format, whose conversion is one instruction, the second reading costs 1.5 us of 33 at 1024.
        uint32_t r[32];
        if (warp_live) {
#pragma unroll
          for (int g = 0; g < 2; ++g) {
            tmem_ld_32x32b_x32(d2 + g * 32, r);
            tmem_ld_wait();
#pragma unroll
            for (int e = 0; e < 32; ++e) amax = fmaxf(amax, fabsf(pg_bf16r(__uint_as_float(r[e]))));
          }
        }
        scale = row_scale(amax);
        if (warp_live) {
#pragma unroll 1
          for (int u = 0; u < 4; ++u) {
            uint32_t q[16];
            tmem_ld_32x32b_x16(d2 + u * 16, q);
            tmem_ld_wait();
            if (live) {   // (rows past the last token hold zeros: zero by zero would take the division's slow path)
#pragma unroll
              for (int e = 0; e < 16; ++e) q[e] = __float_as_uint(pg_bf16r(__uint_as_float(q[e])));
              store16(u, q, scale);
            }
            __syncwarp();   // the whole warp loads
          }
        }
        release();
      }
      if (live && half == 0) p.q_scale_out[static_cast<size_t>(tok) * p.heads + head] = scale;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

__global__ void __launch_bounds__(256) hif8_convert_kernel(int direction, const void* in, void* out, long long n) {
  for (long long i = blockIdx.x * 256ll + threadIdx.x; i < n; i += static_cast<long long>(gridDim.x) * 256) {
    if (direction == 0) static_cast<uint8_t*>(out)[i] = static_cast<uint8_t>(float_to_hif8(static_cast<const float*>(in)[i]));
    else static_cast<float*>(out)[i] = hif8_to_float(static_cast<const uint8_t*>(in)[i]);
  }
}

int launch_hif8_convert(int direction, const void* in, void* out, long long n, cudaStream_t stream) {
  if (n <= 0) return DSV32_OK;
  const long long blocks = (n + 255) / 256;
  hif8_convert_kernel<<<static_cast<int>(blocks < 148 * 8 ? blocks : 148 * 8), 256, 0, stream>>>(direction, in, out, n);
  count_launch();
  return check_launch("hif8_convert_kernel");
}

static size_t pg_align(size_t b) { return (b + 255) / 256 * 256; }

// The projection reads wk and w_proj themselves where TMA can: rows and bases of 16-byte multiples.  Otherwise both are packed.
static bool pg_direct(const PgPrologParams& p) {
  return p.heads % 8 == 0 && (reinterpret_cast<uintptr_t>(p.wk) | reinterpret_cast<uintptr_t>(p.w_proj)) % 16 == 0;
}

size_t pg_prolog_workspace_bytes(int t, int h, int q_lora, int heads) {
  if (t <= 0 || h <= 0 || q_lora <= 0 || heads <= 0) return 0;
  const size_t n = static_cast<size_t>(heads) * kPgDim;
  const size_t direct = proj_partial_bytes(t, h, kPgDim + proj_ld(heads)), packed = proj_partial_bytes(t, h, kPgXwCols);
  return pg_align(static_cast<size_t>(t) * q_lora * 2) + pg_align(static_cast<size_t>(q_lora) * n * 2) +
         pg_align(2 * kPgDim * kPgDim * 2) + pg_align(static_cast<size_t>(h) * kPgXwCols * 2) + (direct > packed ? direct : packed);
}

template <bool kMx>
static int launch_pg_heads(const PgPrologParams& p, const PgOperands& o, const ProjSums& src, cudaStream_t stream) {
  CUtensorMap a, b, had;
  int rc = make_tensor_map_2d_u8(&a, o.q, p.t, static_cast<uint64_t>(p.q_lora) * 2, 128, 128);
  if (rc == DSV32_OK) rc = make_tensor_map_2d_u8(&b, o.w, p.q_lora, static_cast<uint64_t>(p.n) * 2, 64, 128);
  if (rc == DSV32_OK) rc = make_tensor_map_2d_u8(&had, o.had, kPgDim, 2 * kPgDim, 128, 128);
  if (rc != DSV32_OK) return rc;
  auto kernel = pg_heads_kernel<kMx>;
  cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kPhSmemBytes));
  const int m_tiles = (p.t + 127) / 128, items = p.heads * m_tiles, keys = (p.t + kPhWarps - 1) / kPhWarps, sms = sm_count();
  const int vec_rope = (reinterpret_cast<uintptr_t>(p.cos) | reinterpret_cast<uintptr_t>(p.sin)) % 16 == 0 ? 1 : 0;
  const int vec_out = reinterpret_cast<uintptr_t>(p.q_out) % 16 == 0 ? 1 : 0;
  launch_ex(kernel, dim3(keys + (items < sms ? items : sms)), kPhThreads, kPhSmemBytes, stream, true, 1, a, b, had, p, src,
            static_cast<const __nv_bfloat16*>(o.had + kPgDim * kPgDim), keys, m_tiles, vec_rope, vec_out);
  count_launch();
  return check_launch("pg_heads_kernel");
}

int launch_pg_prolog(const PgPrologParams& p, void* workspace, cudaStream_t stream) {
  if (p.t <= 0) return DSV32_OK;
  char* ws = static_cast<char*>(workspace);
  PgOperands o{};
  o.q = reinterpret_cast<__nv_bfloat16*>(ws);
  ws += pg_align(static_cast<size_t>(p.t) * p.q_lora * 2);
  o.w = reinterpret_cast<__nv_bfloat16*>(ws);
  ws += pg_align(static_cast<size_t>(p.q_lora) * p.n * 2);
  o.had = reinterpret_cast<__nv_bfloat16*>(ws);
  ws += pg_align(2 * kPgDim * kPgDim * 2);
  const bool direct = pg_direct(p);
  if (!direct) o.xw = reinterpret_cast<__nv_bfloat16*>(ws);
  ws += pg_align(static_cast<size_t>(p.h) * kPgXwCols * 2);
  float* part_x = reinterpret_cast<float*>(ws);

  const ProjSegment segs[2] = {{p.wk, kPgDim}, {p.w_proj, p.heads}}, packed{o.xw, kPgXwCols};
  const int ld = direct ? kPgDim + proj_ld(p.heads) : kPgXwCols;
  auto project = [&] { return launch_proj_bf16(p.x, p.t, p.h, direct ? segs : &packed, direct ? 2 : 1, false, part_x, p.status, stream); };
  const ProjSums src{part_x, p.t, ld, proj_plan(p.t, ld, p.h / 64).splits};
  int rc = direct ? project() : DSV32_OK;
  if (rc != DSV32_OK) return rc;
  const long long items = (static_cast<long long>(p.t) * p.q_lora + static_cast<long long>(p.q_lora) * p.n + 2 * kPgDim * kPgDim +
                           (direct ? 0ll : static_cast<long long>(p.h) * kPgXwCols)) / 8;
  const long long blocks = (items + 255) / 256, most = static_cast<long long>(sm_count()) * 8;
  const int vec_scale = reinterpret_cast<uintptr_t>(p.w_qb_scale_e8) % 16 == 0 ? 1 : 0;
  // beside the projection where that does not read its output
  launch_ex(pg_unpack_kernel, dim3(static_cast<unsigned>(blocks < most ? blocks : most)), 256, 0, stream, direct, 1, p, o, vec_scale);
  count_launch();
  rc = check_launch("pg_unpack_kernel");
  if (rc == DSV32_OK && !direct) rc = project();
  if (rc != DSV32_OK) return rc;
  return p.format == DSV32_PG_FORMAT_MXFP8 ? launch_pg_heads<true>(p, o, src, stream) : launch_pg_heads<false>(p, o, src, stream);
}

}  // namespace dsv32
