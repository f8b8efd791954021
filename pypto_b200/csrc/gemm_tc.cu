// Products of activations with weight matrices on tcgen05: the first projections of every prolog (x times two to four
// weight matrices side by side), the compressor's two projections and the public bf16 / int8 GEMM entries.
//
//   partial[s][token, 64 j .. 64 j + 63] = A[token, k range s] x B_j[k range s, :]         fp32 (int32)
//
// The output columns are chunks of 64 (128 for int8) that may come from up to four weight matrices (`ProjSegment`), so one
// launch reads x once for all of them.  Weights are [k, n] row-major (MN-major operand) or [n, k] (K-major).
//
// Persistent CTAs, one per SM, walk (token tile of 128, column tile of kN, split of the reduction) with the token tile
// fastest, so that CTAs that run together share a column tile.  Warp 0 keeps a ring of TMA loads full, warp 1 issues the
// products (one elected lane), warps 2..9 take the accumulator -- double-buffered in tensor memory -- and leave through shared
// memory with TMA stores, 32 rows x 128 bytes a warp and step: a thread owns a token row, so storing from registers would
// touch 32 lines per instruction (the first form of these kernels did; at 128 tokens it cost as much as the weights).
//
// The reduction is accumulated in segments of at most 14 chunks (896 elements): tensor memory holds one segment, the epilogue
// adds the segments in fp32 registers, in order, under the products of the next one.  A single accumulation over a
// hidden size of 7168 drifts by the tensor core's truncation of small addends (the rounding to bf16 that follows then flips
// ten times as often); short segments keep the result at every token count where it is for small ones.
//
// Two tile widths.  Up to 128 tokens the call streams weights, and kN = 128 with the reduction split over all SMs keeps 192 KB
// in flight on each.  Beyond that the products matter: kN = 256 halves the reads of A from L2 per product (96 bytes a
// cycle at full rate, about what L2 delivers), and the reduction is only split while tiles are fewer than SMs.
// 4096 tokens x 7168 x 2304 columns: 100 us = 1350 TFLOP/s (the previous kernel, 128 columns and eight splits: 325 us).
#include "kernels.cuh"
#include "tc_common.cuh"

namespace dsv32 {

constexpr int kProjThreads = 320;
constexpr int kProjSegChunks = 14;   // longest segment, in reduction chunks

struct ProjParams {
  uint32_t* status;
  int t, m_tiles, n_tiles, splits;
  int k_chunks;          // reduction chunks (of 128 bytes of A's row)
  int segments;          // accumulated apart; a split takes segments [segments * s / splits, segments * (s + 1) / splits)
  int n_chunks;          // output column chunks in all
  int seg_end[4];        // first chunk past each weight matrix
};

template <int kN, bool kInt8>
struct ProjShape {
  static constexpr int kChunkCols = kInt8 ? 128 : 64;      // output columns of a chunk: 128 bytes of an MN-major weight row
  static constexpr int kKRows = kInt8 ? 128 : 64;          // reduction elements per stage (128 bytes of A)
  static constexpr int kChunks = kN / kChunkCols;
  static constexpr int kABytes = 128 * 128;
  static constexpr int kBChunk = kKRows * 128;
  static constexpr int kStageBytes = kABytes + kChunks * kBChunk;           // 32 or 48 KB
  static constexpr int kStages = kN == 128 ? 6 : 4;
  static constexpr int kOffStore = kStages * kStageBytes;                   // one 4 KB store buffer per epilogue warp
  static constexpr int kOffBars = kOffStore + 8 * 4096;
  static constexpr int kOffTmem = kOffBars + (2 * kStages + 4) * 8;
  static constexpr size_t kSmemBytes = kOffTmem + 16;
  static constexpr uint32_t kTmemCols = 2 * kN;
  static_assert(kSmemBytes <= 232448, "shared memory of one CTA");
};

template <int kN, bool kInt8, bool kKMajor>
__global__ void __launch_bounds__(kProjThreads, 1)
proj_tc_kernel(const __grid_constant__ CUtensorMap a_map, const __grid_constant__ CUtensorMap b0, const __grid_constant__ CUtensorMap b1,
               const __grid_constant__ CUtensorMap b2, const __grid_constant__ CUtensorMap b3,
               const __grid_constant__ CUtensorMap c_map, ProjParams p) {
  using Sh = ProjShape<kN, kInt8>;
  extern __shared__ __align__(1024) unsigned char smem[];   // no static shared memory: the window is 1024-byte aligned
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + Sh::kOffBars);
  uint64_t* empty_bar = full_bar + Sh::kStages;
  uint64_t* tfull_bar = empty_bar + Sh::kStages;    // [2]
  uint64_t* tempty_bar = tfull_bar + 2;             // [2]
  uint32_t* tmem_ptr_s = reinterpret_cast<uint32_t*>(smem + Sh::kOffTmem);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if ((smem_u32(smem) & 1023u) != 0u) {
    if (tid == 0) report_status(p.status, DSV32_STATUS_INTERNAL, 60, smem_u32(smem));
    return;
  }
  if (warp == 0) {
    if (lane == 0) {
      tma_prefetch_desc(&a_map);
      tma_prefetch_desc(&b0);
      tma_prefetch_desc(&c_map);
      for (int i = 0; i < Sh::kStages; ++i) {
        mbar_init(&full_bar[i], 1);
        mbar_init(&empty_bar[i], 1);
      }
      for (int i = 0; i < 2; ++i) {
        mbar_init(&tfull_bar[i], 1);
        mbar_init(&tempty_bar[i], 8);
      }
      mbar_fence_init();
    }
  } else if (warp == 1) {
    tmem_alloc(tmem_ptr_s, Sh::kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_ptr_s;
  pdl_wait();     // (first kernel of an operator: everything it reads may come from the kernel before)
  pdl_trigger();
  const int items = p.m_tiles * p.n_tiles * p.splits;
  // item -> (token tile, column tile, split = segments [g0, g1)); segment g = reduction chunks [chunk_of(g), chunk_of(g + 1))
  auto decode = [&](int item, int& m, int& n, int& split, int& g0, int& g1) {
    m = item % p.m_tiles;
    const int r = item / p.m_tiles;
    n = r % p.n_tiles;
    split = r / p.n_tiles;
    g0 = p.segments * split / p.splits;
    g1 = p.segments * (split + 1) / p.splits;
  };
  auto chunk_of = [&](int g) { return p.k_chunks * g / p.segments; };
  int m, n, split, g0, g1;

  if (warp == 0) {
    if (lane == 0) {
      bool ok = true;
      int s = 0, ph = 1;
      for (int item = blockIdx.x; ok && item < items; item += gridDim.x) {
        decode(item, m, n, split, g0, g1);
        // source of every column chunk of this tile
        const CUtensorMap* src[Sh::kChunks];
        int at[Sh::kChunks], live = 0;
#pragma unroll
        for (int j = 0; j < Sh::kChunks; ++j) {
          const int q = n * Sh::kChunks + j;
          src[j] = nullptr;
          at[j] = 0;
          if (q < p.n_chunks) {
            const int seg = q < p.seg_end[0] ? 0 : q < p.seg_end[1] ? 1 : q < p.seg_end[2] ? 2 : 3;
            src[j] = seg == 0 ? &b0 : seg == 1 ? &b1 : seg == 2 ? &b2 : &b3;
            at[j] = (q - (seg == 0 ? 0 : p.seg_end[seg - 1])) * (kKMajor ? Sh::kChunkCols : 128);
            ++live;
          }
        }
        const int c1 = chunk_of(g1);
        for (int c = chunk_of(g0); c < c1; ++c) {
          if (!mbar_wait(&empty_bar[s], ph, p.status, 61)) { ok = false; break; }
          unsigned char* st = smem + s * Sh::kStageBytes;
          mbar_arrive_expect_tx(&full_bar[s], Sh::kABytes + live * Sh::kBChunk);
          tma_load_2d(st, &a_map, c * 128, m * 128, &full_bar[s]);
#pragma unroll
          for (int j = 0; j < Sh::kChunks; ++j)
            if (src[j] != nullptr) {
              if constexpr (kKMajor) tma_load_2d(st + Sh::kABytes + j * Sh::kBChunk, src[j], c * 128, at[j], &full_bar[s]);
              else tma_load_2d(st + Sh::kABytes + j * Sh::kBChunk, src[j], at[j], c * Sh::kKRows, &full_bar[s]);
            }
          if (++s == Sh::kStages) {
            s = 0;
            ph ^= 1;
          }
        }
      }
    }
  } else if (warp == 1) {
    constexpr uint32_t idesc = kInt8 ? umma_idesc_i8(128, kN, !kKMajor) : umma_idesc_bf16(128, kN, false, !kKMajor);
    const uint32_t tbase = __shfl_sync(0xffffffffu, tmem_base, 0);
    bool ok = true;
    int s = 0, ph = 0, i = 0;
    for (int item = blockIdx.x; ok && item < items; item += gridDim.x) {
      decode(item, m, n, split, g0, g1);
      for (int g = g0; ok && g < g1; ++g, ++i) {
        const int a = i & 1, c0 = chunk_of(g), c1 = chunk_of(g + 1);
        ok = __all_sync(0xffffffffu, mbar_wait(&tempty_bar[a], ((i >> 1) & 1) ^ 1, p.status, 62));
        for (int c = c0; ok && c < c1; ++c) {
          ok = __all_sync(0xffffffffu, mbar_wait(&full_bar[s], ph, p.status, 63));
          if (!ok) break;
          tc_fence_after();
          const uint32_t a_s = smem_u32(smem + s * Sh::kStageBytes), b_s = a_s + Sh::kABytes;
          const uint64_t ad = umma_smem_desc_sw128(a_s, 16, 1024);
          const uint64_t bd = kKMajor ? umma_smem_desc_sw128(b_s, 16, 1024) : umma_smem_desc_sw128(b_s, Sh::kBChunk, 1024);
          constexpr int kBStep = kKMajor ? 2 : (kInt8 ? 4096 : 2048) / 16;   // 32 bytes of a K-major row, or 32 / 16 k rows
          if (elect_one()) {
#pragma unroll
            for (int ks = 0; ks < 4; ++ks) {   // 32 bytes of A's row per product
              if constexpr (kInt8) umma_i8_ss(tbase + a * kN, ad + 2 * ks, bd + kBStep * ks, idesc, (c > c0 || ks > 0) ? 1u : 0u);
              else umma_f16_ss(tbase + a * kN, ad + 2 * ks, bd + kBStep * ks, idesc, (c > c0 || ks > 0) ? 1u : 0u);
            }
            umma_commit(&empty_bar[s]);
            if (c == c1 - 1) umma_commit(&tfull_bar[a]);
          }
          __syncwarp();
          if (++s == Sh::kStages) {
            s = 0;
            ph ^= 1;
          }
        }
      }
    }
  } else {
    constexpr int kCols = kN / 2;                     // accumulator columns of this warp
    const int quarter = warp & 3, half = (warp - 2) >> 2;
    unsigned char* buf = smem + Sh::kOffStore + (warp - 2) * 4096;
    const uint32_t sw = static_cast<uint32_t>(lane & 7);
    const int lim = p.n_chunks * Sh::kChunkCols;      // columns past the last chunk hold nothing
    int i = 0;
    bool ok = true;
    for (int item = blockIdx.x; ok && item < items; item += gridDim.x) {
      decode(item, m, n, split, g0, g1);
      const int row0 = m * 128 + quarter * 32, col0 = n * kN + half * kCols;
      const bool live = row0 < p.t && col0 < lim;
      uint32_t acc[kCols];
#pragma unroll
      for (int j = 0; j < kCols; ++j) acc[j] = 0u;
      for (int g = g0; g < g1; ++g, ++i) {
        const int a = i & 1;
        ok = __all_sync(0xffffffffu, mbar_wait(&tfull_bar[a], (i >> 1) & 1, p.status, 64));
        if (!ok) break;
        tc_fence_after();
        if (live) {
          const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + a * kN + half * kCols;
#pragma unroll
          for (int c = 0; c < kCols; c += 16) {   // (sixteen at a time: 128 sums and 32 more would not fit 168 registers)
            uint32_t r[16];
            tmem_ld_32x32b_x16(taddr + c, r);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 16; ++j)
              acc[c + j] = kInt8 ? acc[c + j] + r[j] : __float_as_uint(__uint_as_float(acc[c + j]) + __uint_as_float(r[j]));
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&tempty_bar[a]);
      }
      if (ok && live) {
#pragma unroll
        for (int c = 0; c < kCols; c += 32) {
          if (col0 + c < lim) {
            if (lane == 0) tma_store_wait_read<0>();    // the store before has read the buffer
            __syncwarp();
#pragma unroll
            for (int u = 0; u < 8; ++u)
              *reinterpret_cast<uint4*>(buf + lane * 128 + ((u ^ sw) << 4)) =
                  make_uint4(acc[c + 4 * u], acc[c + 4 * u + 1], acc[c + 4 * u + 2], acc[c + 4 * u + 3]);
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
              tma_store_3d(&c_map, buf, (col0 + c) * 4, row0, split);
              tma_store_commit();
            }
          }
        }
      }
    }
    if (lane == 0) tma_store_wait_all();
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem_base, Sh::kTmemCols);
  }
}

// ---- host ------------------------------------------------------------------------------------------------------------
// Column tile and split of the reduction for a product of t tokens, `cols` output columns and `k_chunks` reduction chunks.
ProjPlan proj_plan(int t, int cols, int k_chunks, int ctas) {
  ProjPlan pl;
  pl.wide = t > 128;
  const int kn = pl.wide ? 256 : 128;
  pl.m_tiles = (t + 127) / 128;
  pl.n_tiles = (cols + kn - 1) / kn;
  int s = sm_count() / (pl.m_tiles * pl.n_tiles);
  // every split costs a write and a read of the partial sums, and below four chunks a CTA does not fill its ring
  s = s < k_chunks / 4 ? s : k_chunks / 4;
  s = s < 1 ? 1 : (s > 16 ? 16 : s);
  const int seg = (k_chunks + kProjSegChunks - 1) / kProjSegChunks;
  pl.segments = seg > s ? seg : s;
  // (fewer CTAs take the same segments, several each: how the sum is cut, and with it its error, does not depend on them)
  const int fit = ctas / (pl.m_tiles * pl.n_tiles);
  pl.splits = ctas <= 0 || s <= fit ? s : (fit < 1 ? 1 : fit);
  return pl;
}

template <int kN, bool kInt8, bool kKMajor>
static int launch_proj(const ProjPlan& pl, const CUtensorMap& a, const CUtensorMap* b, const CUtensorMap& c, const ProjParams& p,
                       cudaStream_t stream) {
  using Sh = ProjShape<kN, kInt8>;
  auto kernel = proj_tc_kernel<kN, kInt8, kKMajor>;
  cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(Sh::kSmemBytes));
  const int items = pl.m_tiles * pl.n_tiles * p.splits, sms = sm_count();
  launch_ex(kernel, dim3(items < sms ? items : sms), kProjThreads, Sh::kSmemBytes, stream, true, 1, a, b[0], b[1], b[2], b[3], c, p);
  count_launch();
  return check_launch("proj_tc_kernel");
}

// partial [splits][t][ldc] fp32 with ldc = proj_ld(columns of all segments); rows of x and w multiples of 16 bytes.
int launch_proj_bf16(const __nv_bfloat16* x, int t, int k, const ProjSegment* segs, int nsegs, bool k_major, float* partial,
                     uint32_t* status, cudaStream_t stream, int ctas) {
  if (t <= 0) return DSV32_OK;
  ProjParams p{};
  p.status = status;
  p.t = t;
  p.k_chunks = (k + 63) / 64;   // past the end both operands read as zero
  CUtensorMap a, b[4], c;
  int rc = make_tensor_map_2d_u8(&a, x, t, static_cast<uint64_t>(k) * 2, 128, 128);
  for (int i = 0; i < 4 && rc == DSV32_OK; ++i) {
    const ProjSegment& s = segs[i < nsegs ? i : 0];
    if (i < nsegs) p.n_chunks += (s.cols + 63) / 64;
    p.seg_end[i] = p.n_chunks;
    if (i >= nsegs) b[i] = b[0];
    else if (k_major) rc = make_tensor_map_2d_u8(&b[i], s.w, s.cols, static_cast<uint64_t>(k) * 2, 64, 128);
    else rc = make_tensor_map_2d_u8(&b[i], s.w, k, static_cast<uint64_t>(s.cols) * 2, 64, 128);
  }
  const int ldc = p.n_chunks * 64;
  const ProjPlan pl = proj_plan(t, ldc, p.k_chunks, ctas);
  if (rc == DSV32_OK) rc = make_tensor_map_3d_u8(&c, partial, pl.splits, t, static_cast<uint64_t>(ldc) * 4, 32);
  if (rc != DSV32_OK) return rc;
  p.m_tiles = pl.m_tiles; p.n_tiles = pl.n_tiles; p.splits = pl.splits; p.segments = pl.segments;
  if (pl.wide) return k_major ? launch_proj<256, false, true>(pl, a, b, c, p, stream) : launch_proj<256, false, false>(pl, a, b, c, p, stream);
  return k_major ? launch_proj<128, false, true>(pl, a, b, c, p, stream) : launch_proj<128, false, false>(pl, a, b, c, p, stream);
}

// int32 C[t, n] = int8 A[t, k] (row-major) x int8 B[k, n] (row-major): k a multiple of 128, n of 256.
int launch_i8_gemm(const int8_t* a8, int t, int k, const int8_t* b8, int n, int32_t* out, uint32_t* status, cudaStream_t stream) {
  if (t <= 0) return DSV32_OK;
  if (k <= 0 || k % 128 != 0 || n <= 0 || n % 256 != 0) {
    set_error("int8 gemm: k=%d must be a positive multiple of 128 and n=%d of 256", k, n);
    return DSV32_ERR_INVALID_ARG;
  }
  ProjParams p{};
  p.status = status;
  p.t = t;
  p.k_chunks = k / 128;
  p.n_chunks = n / 128;
  for (int& e : p.seg_end) e = p.n_chunks;
  const ProjPlan pl = proj_plan(t, n, 0);
  p.m_tiles = pl.m_tiles; p.n_tiles = pl.n_tiles;
  p.splits = p.segments = 1;   // exact sums, straight to the result
  CUtensorMap a, b[4], c;
  int rc = make_tensor_map_2d_u8(&a, a8, t, k, 128, 128);
  if (rc == DSV32_OK) rc = make_tensor_map_2d_u8(&b[0], b8, k, n, 128, 128);
  if (rc == DSV32_OK) rc = make_tensor_map_3d_u8(&c, out, 1, t, static_cast<uint64_t>(n) * 4, 32);
  if (rc != DSV32_OK) return rc;
  b[1] = b[2] = b[3] = b[0];
  return pl.wide ? launch_proj<256, true, false>(pl, a, b, c, p, stream) : launch_proj<128, true, false>(pl, a, b, c, p, stream);
}

// out[t, n] (fp32, or bf16 with one rounding) = sum over the reduction splits, in order, of the fp32 slabs [t, ldp]
__global__ void __launch_bounds__(256) gemm_reduce_kernel(const float* partial, int splits, int t, int ldp, int n, void* out,
                                                          int out_bf16) {
  pdl_wait();
  const long long total = static_cast<long long>(t) * n;
  for (long long i = blockIdx.x * 256ll + threadIdx.x; i < total; i += static_cast<long long>(gridDim.x) * 256) {
    const long long row = i / n, col = i % n;
    float acc = 0.f;
    for (int s = 0; s < splits; ++s) acc += partial[(static_cast<size_t>(s) * t + row) * ldp + col];
    if (out_bf16) static_cast<__nv_bfloat16*>(out)[i] = __float2bfloat16_rn(acc);
    else static_cast<float*>(out)[i] = acc;
  }
}

size_t proj_partial_bytes(int t, int k, int cols) {
  const int ldc = proj_ld(cols);
  return (static_cast<size_t>(proj_plan(t, ldc, (k + 63) / 64).splits) * t * ldc * sizeof(float) + 255) / 256 * 256;
}

size_t bf16_gemm_workspace_bytes(int t, int k, int n) {
  if (t <= 0 || k <= 0 || n <= 0 || k % 64 != 0) return 0;
  return proj_partial_bytes(t, k, n);
}

int launch_bf16_gemm(const __nv_bfloat16* a, int t, int k, const __nv_bfloat16* b, int n, bool b_kmajor, void* out,
                     bool out_bf16, void* workspace, uint32_t* status, cudaStream_t stream) {
  if (t <= 0) return DSV32_OK;
  float* partial = static_cast<float*>(workspace);
  const ProjSegment seg{b, n};
  int rc = launch_proj_bf16(a, t, k, &seg, 1, b_kmajor, partial, status, stream);
  if (rc != DSV32_OK) return rc;
  const long long blocks = (static_cast<long long>(t) * n + 255) / 256, most = sm_count() * 8;
  launch_ex(gemm_reduce_kernel, dim3(static_cast<unsigned>(blocks < most ? blocks : most)), 256, 0, stream, true, 1, partial,
            proj_plan(t, proj_ld(n), k / 64).splits, t, proj_ld(n), n, out, out_bf16 ? 1 : 0);
  count_launch();
  return check_launch("gemm_reduce_kernel");
}

}  // namespace dsv32
