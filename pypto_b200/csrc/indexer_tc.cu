// Lightning-indexer scores on the 5th-generation tensor cores (tcgen05, int8 -> int32 in tensor memory).
//
//   D[key, (token, head)] = K_block[128 keys x 128] . Q[(token, head) x 128]^T          (kind::i8, exact)
//   score[token, key]     = ( sum_h ws[token,h] * fp16( relu(D) * 2^-11 ) ) * k_scale[key]
//
// Keys are the M dimension: a 128-key cache block is one 16 KB TMA tile (128-byte swizzle) and one M=128 MMA tile, and an
// epilogue warp owns 32 keys of one token: all 64 heads of a key lie in the four lanes that hold its row.
// Follows models/deepseek_v32_exp/lightning_indexer_quant_impl.py:114-177 (golden:
// deepseekv32_lightning_indexer_quant.py:209-242).
//
// Warp roles: warp 0 = TMA producer, warp 1 = MMA issuer + tensor-memory owner, then the epilogue warps (one per TMEM
// lane quarter and token).  Key blocks go through a ring of shared-memory stages; the accumulator is double-buffered in
// tensor memory so the epilogue of block i overlaps the MMA of i+1.
#include <atomic>
#include <mutex>

#include "kernels.cuh"
#include "tc_common.cuh"

namespace dsv32 {

constexpr int kTcBlocksPerCta = 512;  // upper bound (page table in shared memory); the launcher or tc_share picks the count
constexpr int kKeyTileBytes = 128 * 128;

// Shared memory of one CTA (offsets from the 1024-byte aligned base).  The ring of key blocks is what keeps
// bytes in flight: with up to two tokens the query tile is 16 KB and five stages fit twice per SM.
template <int TOK>
struct TcSmemLayout {
  static constexpr int stages = TOK <= 2 ? 5 : 4;
  static constexpr int keys = 0;                               // stages x 16 KB
  static constexpr int q = stages * kKeyTileBytes;             // 64 * TOK rows x 128 B
  static constexpr int ws = q + 64 * TOK * 128;                // 64 * TOK fp16 weights (1 KB reserved)
  static constexpr int phys = ws + 256 * 4;                    // kTcBlocksPerCta ints
  static constexpr int bars = phys + ((kTcBlocksPerCta * 4 + 7) / 8) * 8;  // 8-byte aligned
  static constexpr int nbars = 2 * stages + 4 + 1;
  static constexpr int tmem_ptr = bars + nbars * 8;
  static constexpr int total = tmem_ptr + 16;
  static constexpr size_t bytes = total + 1024;                // slack for manual 1024-byte alignment
  static_assert(bars % 8 == 0 && q % 1024 == 0, "shared-memory layout alignment");
};

template <int TOK>
struct TcShape {
  static constexpr int kEpilogueWarps = 4 * TOK;      // one warp per TMEM lane quarter and token
  static constexpr int kThreads = 64 + 32 * kEpilogueWarps;
};

// D[16 x 8] += A[16 x 16] B[16 x 8], fp16 operands, fp32 sums (warp-level fragments)
__device__ __forceinline__ void mma_m16n8k16_f16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                                 uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// Key blocks of a request inside [key_begin, key_end).  A sequence length beyond what the request's page-table row can describe
// is reported and clamped: nothing is read past the row of the page table or written past the row of the score buffer.
__device__ __forceinline__ int tc_blocks(const IndexerParams& p, int b, bool report, int& hi) {
  int L = p.act_seq[b];
  if (L > p.max_blocks * 128) {
    if (report) report_status(p.status, DSV32_STATUS_BAD_INDEX, b, static_cast<uint32_t>(L));
    L = p.max_blocks * 128;
  }
  hi = min(L, p.key_end);
  return hi > p.key_begin ? (hi + 127) / 128 - p.key_begin / 128 : 0;
}

// Share of a CTA of a batch (one-dimensional grid): the lengths, which may differ a hundredfold and live on the device, set how
// many blocks a CTA takes, so that the whole batch makes `r` rounds of CTAs, and a request is cut into equal pieces.  With
// a number chosen on the host for the longest request, 256 requests of 1K to 128K left half of each request's last CTA idle.
// One warp; false: nothing to do.
__device__ __forceinline__ bool tc_share(const IndexerParams& p, int& b, int& begin, int& end) {
  const int lane = threadIdx.x & 31;
  int total = 0, longest = 0, hi, own[4];   // (the lengths of up to 128 requests stay in registers; loads in flight together)
#pragma unroll
  for (int k = 0; k < 4; ++k) own[k] = lane + 32 * k < p.b ? p.act_seq[lane + 32 * k] : 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    if (own[k] > p.max_blocks * 128 && blockIdx.x == 0) report_status(p.status, DSV32_STATUS_BAD_INDEX, lane + 32 * k, own[k]);
    own[k] = max((min(min(own[k], p.max_blocks * 128), p.key_end) + 127) / 128 - p.key_begin / 128, 0);
    total += own[k];
    longest = max(longest, own[k]);
  }
  for (int i = lane + 128; i < p.b; i += 32) {
    const int n = tc_blocks(p, i, blockIdx.x == 0, hi);
    total += n;
    longest = max(longest, n);
  }
  longest = __reduce_max_sync(0xffffffffu, longest);
  total = __reduce_add_sync(0xffffffffu, total);
  // about 56 blocks a piece, and no more pieces than `r` rounds hold: a few CTAs of a further round would cost as much as all
  const int half = p.b / 2, r = min(max((total / 56 + half + p.slots / 2) / p.slots, 1), p.rounds);
  int c = max((total + p.slots * r - 1) / (p.slots * r), 2);
  if (total == longest * p.b && total > 0) {   // all alike: no scans (2 us of a CTA's start)
    while (p.b * ((longest + c - 1) / c) > p.slots * r && c < longest && c < kTcBlocksPerCta) ++c;
    const int k = (longest + c - 1) / c, j = blockIdx.x % k;
    b = blockIdx.x / k;
    begin = p.key_begin / 128 + longest * j / k;
    end = p.key_begin / 128 + longest * (j + 1) / k;
    return b < p.b;
  }
  for (int k = 0; k < 8; ++k) {
    int pieces = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) pieces += static_cast<int>(static_cast<unsigned>(own[j] + c - 1) / static_cast<unsigned>(c));
    for (int i = lane + 128; i < p.b; i += 32) pieces += (tc_blocks(p, i, false, hi) + c - 1) / c;
    if (static_cast<int>(__reduce_add_sync(0xffffffffu, pieces)) <= p.slots * r) break;
    c = min(c + max(c >> 4, 1), kTcBlocksPerCta);
  }
  int first = 0;   // first piece of these 32 requests
  for (int b0 = 0; b0 < p.b; b0 += 32) {
    const int n = b0 + lane < p.b ? tc_blocks(p, b0 + lane, false, hi) : 0;
    const int k = (n + c - 1) / c;
    int inc = k;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += u;
    }
    const uint32_t past = __ballot_sync(0xffffffffu, first + inc > static_cast<int>(blockIdx.x));
    if (past != 0u) {
      const int l = __ffs(past) - 1;
      const int nb = __shfl_sync(0xffffffffu, n, l), kb = __shfl_sync(0xffffffffu, k, l);
      const int j = static_cast<int>(blockIdx.x) - __shfl_sync(0xffffffffu, first + inc - k, l);
      b = b0 + l;
      begin = p.key_begin / 128 + static_cast<int>(static_cast<long long>(nb) * j / kb);
      end = p.key_begin / 128 + static_cast<int>(static_cast<long long>(nb) * (j + 1) / kb);
      return true;
    }
    first += __shfl_sync(0xffffffffu, inc, 31);
  }
  return false;
}

// kDots: also store the raw dot products (verification; an instantiation of its own because its addresses cost registers)
template <int TOK, bool kDots>
__global__ void __launch_bounds__(TcShape<TOK>::kThreads, TOK <= 2 ? 2 : 1) indexer_scores_tc_kernel(const __grid_constant__ CUtensorMap key_map,
                                                                      const __grid_constant__ CUtensorMap q_map,
                                                                      IndexerParams p) {
  constexpr int N = 64 * TOK;
  constexpr int kEpThreads = 32 * TcShape<TOK>::kEpilogueWarps;
  constexpr uint32_t kTmemCols = 2 * N < 32 ? 32 : 2 * N;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  using Lay = TcSmemLayout<TOK>;
  constexpr int kTcStages = Lay::stages;
  unsigned char* k_s = smem + Lay::keys;
  unsigned char* q_s = smem + Lay::q;
  uint32_t* ws_s = reinterpret_cast<uint32_t*>(smem + Lay::ws);  // fp16 pairs
  int* phys_s = reinterpret_cast<int*>(smem + Lay::phys);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Lay::bars);
  uint64_t* full_bar = bars;                       // [kTcStages]
  uint64_t* empty_bar = bars + kTcStages;          // [kTcStages]
  uint64_t* tfull_bar = bars + 2 * kTcStages;      // [2]
  uint64_t* tempty_bar = bars + 2 * kTcStages + 2; // [2]
  uint64_t* q_bar = bars + 2 * kTcStages + 4;
  uint32_t* tmem_ptr_s = reinterpret_cast<uint32_t*>(smem + Lay::tmem_ptr);

  pdl_wait();     // (first kernel of an operator: everything it reads may come from the kernel before)
  pdl_trigger();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 64) {   // (by a warp that has nothing else to do yet)
    tma_prefetch_desc(&key_map);
    tma_prefetch_desc(&q_map);
    for (int i = 0; i < kTcStages; ++i) {
      mbar_init(&full_bar[i], 1);
      mbar_init(&empty_bar[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&tfull_bar[i], 1);
      mbar_init(&tempty_bar[i], TcShape<TOK>::kEpilogueWarps);   // one arrival per warp
    }
    mbar_init(q_bar, 1);
    mbar_fence_init();
  }
  const int tok0 = blockIdx.z * TOK;
  const int ntok = min(TOK, p.s1 - tok0);
  const int bs = 128;
  int b = blockIdx.y, blk_begin, blk_end, hi;
  if constexpr (TOK > 2) {   // three tokens or more a request: always the host's number of blocks, chosen for the longest request
    blk_begin = p.key_begin / bs + blockIdx.x * p.blocks_per_cta;
    blk_end = min(blk_begin + p.blocks_per_cta, p.key_begin / bs + tc_blocks(p, b, blockIdx.x == 0 && tid == 0, hi));
    if (blk_begin >= blk_end) return;   // uniform for the CTA
  } else {
    // (by one warp, and through shared memory in both cases: all warps at it take 2 us longer to start, and where the values can
    // come from two places the loops below are compiled worse, 5 % of the kernel)
    int* share_s = reinterpret_cast<int*>(smem + Lay::tmem_ptr) + 1;
    if (warp == 0) {
      int sb = b, s0, s1, h;
      if (p.blocks_per_cta > 0) {
        s0 = p.key_begin / bs + blockIdx.x * p.blocks_per_cta;
        s1 = min(s0 + p.blocks_per_cta, p.key_begin / bs + tc_blocks(p, sb, blockIdx.x == 0 && tid == 0, h));
      } else if (!tc_share(p, sb, s0, s1)) {
        sb = s0 = s1 = 0;
      }
      if (lane == 0) {
        share_s[0] = sb;
        share_s[1] = s0;
        share_s[2] = s1;
      }
    }
    __syncthreads();
    b = share_s[0];
    blk_begin = share_s[1];
    blk_end = share_s[2];
    if (blk_begin >= blk_end) return;   // uniform for the CTA
    (void)tc_blocks(p, b, false, hi);
  }
  const int nblk = blk_end - blk_begin;
  const size_t row0 = static_cast<size_t>(b) * p.s1 + tok0;

  // ---- setup ----------------------------------------------------------------------------------------
  if (warp == 0) {
    for (int j = lane; j < nblk; j += 32) {
      int phys = p.block_table[static_cast<size_t>(b) * p.max_blocks + blk_begin + j];
      if (phys < 0 || phys >= p.num_blocks) {
        report_status(p.status, DSV32_STATUS_BAD_PAGE, b, blk_begin + j);
        phys = 0;
      }
      phys_s[j] = phys;
    }
  } else if (warp == 1) {
    tmem_alloc(tmem_ptr_s, kTmemCols);
    tmem_relinquish();
  } else {
    __half* ws_h = reinterpret_cast<__half*>(ws_s);  // ws = fp16(q_scale * weight), one per (token, head)
    for (int i = tid - 64; i < N; i += kEpThreads)
      ws_h[i] = (i < ntok * 64) ? __hmul(p.q_scale[row0 * 64 + i], p.weight[row0 * 64 + i]) : __float2half(0.f);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_ptr_s;

  if (warp == 0) {
    // ---- TMA producer ----------------------------------------------------------------------------------
    if (lane == 0) {
      // With one group of tokens the key cache is read once per call and is far larger than L2: mark it evict-first so
      // that the score rows written below stay in L2 for the top-k that follows.  Further groups find it in L2.
      const bool once = gridDim.z == 1;
      const uint64_t evict_first = l2_policy_evict_first();
      mbar_arrive_expect_tx(q_bar, N * 128);
      tma_load_2d(q_s, &q_map, 0, static_cast<int>(row0 * 64), q_bar);
      for (int i = 0; i < nblk; ++i) {
        const int s = i % kTcStages;
        if (!mbar_wait(&empty_bar[s], ((i / kTcStages) & 1) ^ 1, p.status, 1)) break;
        mbar_arrive_expect_tx(&full_bar[s], kKeyTileBytes);
        if (once) tma_load_2d_hint(k_s + s * kKeyTileBytes, &key_map, 0, phys_s[i] * 128, &full_bar[s], evict_first);
        else tma_load_2d(k_s + s * kKeyTileBytes, &key_map, 0, phys_s[i] * 128, &full_bar[s]);
      }
    }
  } else if (warp == 1) {
    // ---- MMA issuer: the whole warp runs the loop, one elected lane issues ---------------------------------------------
    constexpr uint32_t idesc = umma_idesc_i8(128, N);
    const uint64_t b_desc0 = umma_smem_desc_sw128(smem_u32(q_s), 16, 1024);
    const uint32_t tbase = __shfl_sync(0xffffffffu, tmem_base, 0);
    bool ok = __all_sync(0xffffffffu, mbar_wait(q_bar, 0, p.status, 2));
    int s = 0, s_phase = 0;
    for (int i = 0; ok && i < nblk; ++i) {
      const int a = i & 1;
      ok = __all_sync(0xffffffffu, mbar_wait(&full_bar[s], s_phase, p.status, 3) &&
                                       mbar_wait(&tempty_bar[a], ((i >> 1) & 1) ^ 1, p.status, 4));
      if (!ok) break;
      tc_fence_after();
      const uint64_t a_desc0 = umma_smem_desc_sw128(smem_u32(k_s + s * kKeyTileBytes), 16, 1024);
      if (elect_one()) {
#pragma unroll
        for (int ks = 0; ks < 4; ++ks)  // K = 32 int8 per instruction: advance 32 B inside the swizzle atom
          umma_i8_ss(tbase + a * N, a_desc0 + 2 * ks, b_desc0 + 2 * ks, idesc, ks > 0 ? 1u : 0u);
        umma_commit(&empty_bar[s]);   // the stage may be refilled once these MMAs have read it
        umma_commit(&tfull_bar[a]);   // the accumulator is complete
      }
      __syncwarp();
      if (++s == kTcStages) {
        s = 0;
        s_phase ^= 1;
      }
    }
  } else {
    // ---- epilogue: warp = (TMEM lane quarter = 32 keys of the block, token) ----------------------------------------------
    // The head sum  sum_h ws[h] * fp16(relu(dot) 2^-11)  is a 64-long contraction whose left operand already lies in
    // registers: read in fragment layout, the rounded fp16 pairs are the A fragments of warp-level m16n8k16 products, and
    // the token's weights, the same in all eight columns of B, stay in eight registers for the whole CTA.  Four such
    // products stand for 256 unpack-unpack-multiply-add triples a lane group (6.1 -> 3.0 instructions a dot); fp16
    // products are exact and the sum is fp32, as before.  64 requests x 64K, two tokens each: 142 -> 123 us, of which the
    // keys take 84 at copy bandwidth; 4096 tokens x 128K: 8.7 -> 5.9 ms, where the int8 products alone take 2.6 at the
    // clock the chip holds under them and share the tensor pipe with the fragments' products.
    const int quarter = warp & 3;
    const int t = (warp - 2) >> 2;                      // token within the CTA
    const int g = lane >> 2, tq = lane & 3;
    uint32_t wb[8];                                     // B fragments: heads 8 j + tq and 8 j + 4 + tq
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const uint16_t* w = reinterpret_cast<const uint16_t*>(ws_s) + t * 64 + 8 * j + tq;
      wb[j] = w[0] | (static_cast<uint32_t>(w[4]) << 16);
    }
    // every lane ends up with the sums of four keys, in columns that are all alike: it keeps one of them
    const int key_in_blk = quarter * 32 + (tq >> 1) * 16 + (tq & 1) * 8 + g;
    // the key scale of a block is fetched one block ahead so that its latency is not exposed
    __half ks_next = p.key_scale[static_cast<size_t>(phys_s[0]) * bs + key_in_blk];
    const uint64_t scale2 = f2_pack(0x3A000000u, 0x3A000000u);    // 2^-11 twice
    const uint64_t bias2 = f2_pack(0xC5C00000u, 0xC5C00000u);     // -6144 = -(2^23 + 2^22) 2^-11 twice
    float* srow = p.scores + (row0 + t) * static_cast<size_t>(p.ld) + static_cast<size_t>(blk_begin) * bs + key_in_blk;
    const uint32_t taddr0 = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + t * 64;
    for (int i = 0; i < nblk; ++i) {
      const int a = i & 1;
      const float ks = __half2float(ks_next);
      if (i + 1 < nblk) ks_next = p.key_scale[static_cast<size_t>(phys_s[i + 1]) * bs + key_in_blk];
      if (!__all_sync(0xffffffffu, mbar_wait(&tfull_bar[a], (i >> 1) & 1, p.status, 5))) break;
      tc_fence_after();
      uint32_t r[2][32];                                // the two halves of 16 keys; the second is loaded under the first
      float sum[2][2];                                  // [half][row g / g + 8]
      tmem_ld_16x128b_x16(taddr0 + a * N, r[0]);
      tmem_ld_wait();
      tmem_ld_16x128b_x16(taddr0 + a * N + (16u << 16), r[1]);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        if (h == 1) {   // the warp's part of this accumulator is in registers: hand it back to the MMA warp
          tmem_ld_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&tempty_bar[a]);
        }
        if (kDots && t < ntok) {
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            const int dpos = (blk_begin + i) * bs + quarter * 32 + h * 16 + g + (j & 1) * 8;
            const int head = 4 * (j >> 1) + tq;
            if (dpos < hi && dpos >= p.key_begin)
              p.dots[((row0 + t) * 64 + head) * static_cast<size_t>(p.ld) + dpos] = static_cast<int32_t>(r[h][j]);
          }
        }
        uint32_t pk[16];   // fp16 pairs of two heads (round-to-nearest-even with ReLU): [2 m] of row g, [2 m + 1] of row g + 8
#pragma unroll
        for (int m = 0; m < 8; ++m) {
          // dot * 2^-11 exactly, half of them in each of two ways that load different pipes: (2^23 + 2^22 + dot) as a
          // float, then one FMA, or the conversion instruction and one product
          float lo_g, lo_g8, hi_g, hi_g8;
          f2_unpack(f2_fma(f2_pack(r[h][4 * m] + 0x4B400000u, r[h][4 * m + 1] + 0x4B400000u), scale2, bias2), lo_g, lo_g8);
          f2_unpack(f2_mul(f2_pack(__float_as_uint(__int2float_rn(static_cast<int>(r[h][4 * m + 2]))),
                                   __float_as_uint(__int2float_rn(static_cast<int>(r[h][4 * m + 3])))), scale2), hi_g, hi_g8);
          asm("cvt.rn.relu.f16x2.f32 %0, %1, %2;" : "=r"(pk[2 * m]) : "f"(hi_g), "f"(lo_g));
          asm("cvt.rn.relu.f16x2.f32 %0, %1, %2;" : "=r"(pk[2 * m + 1]) : "f"(hi_g8), "f"(lo_g8));
        }
        float c0[4] = {0.f, 0.f, 0.f, 0.f}, c1[4] = {0.f, 0.f, 0.f, 0.f};   // two chains of two products
        mma_m16n8k16_f16(c0, pk[0], pk[1], pk[2], pk[3], wb[0], wb[1]);
        mma_m16n8k16_f16(c1, pk[4], pk[5], pk[6], pk[7], wb[2], wb[3]);
        mma_m16n8k16_f16(c0, pk[8], pk[9], pk[10], pk[11], wb[4], wb[5]);
        mma_m16n8k16_f16(c1, pk[12], pk[13], pk[14], pk[15], wb[6], wb[7]);
        sum[h][0] = c0[0] + c1[0];
        sum[h][1] = c0[2] + c1[2];
      }
      const int pos = (blk_begin + i) * bs + key_in_blk;
      if (pos < hi && pos >= p.key_begin && t < ntok) {
        const float s0 = (tq & 1) ? sum[0][1] : sum[0][0], s1 = (tq & 1) ? sum[1][1] : sum[1][0];
        srow[i * bs] = ((tq >> 1) ? s1 : s0) * ks;
      }
    }
  }

  // ---- teardown -----------------------------------------------------------------------------------------
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

// ---- host ------------------------------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn get_encode_fn() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* sym = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &qres) == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(sym);
  });
  return fn;
}

static int encode_map(CUtensorMap* map, const void* base, int rank, const cuuint64_t* dims, const cuuint64_t* strides,
                      const cuuint32_t* box, CUtensorMapSwizzle swizzle) {
  EncodeTiledFn fn = get_encode_fn();
  if (fn == nullptr) {
    set_error("cuTensorMapEncodeTiled is not available from this driver");
    return DSV32_ERR_CUDA;
  }
  const cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, rank, const_cast<void*>(base), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    set_error("cuTensorMapEncodeTiled failed with code %d (base %p rows %llu row_bytes %llu)", static_cast<int>(r), base,
              static_cast<unsigned long long>(dims[1]), static_cast<unsigned long long>(dims[0]));
    return DSV32_ERR_CUDA;
  }
  return DSV32_OK;
}
int make_tensor_map_2d_u8(CUtensorMap* map, const void* base, uint64_t rows, uint64_t row_bytes, uint32_t box_rows,
                          uint32_t box_bytes) {
  const cuuint64_t dims[2] = {row_bytes, rows}, strides[1] = {row_bytes};
  const cuuint32_t box[2] = {box_bytes, box_rows};
  return encode_map(map, base, 2, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
}
int make_tensor_map_2d_sw64(CUtensorMap* map, const void* base, uint64_t rows, uint64_t row_bytes, uint32_t box_rows) {
  const cuuint64_t dims[2] = {row_bytes, rows}, strides[1] = {row_bytes};
  const cuuint32_t box[2] = {64, box_rows};
  return encode_map(map, base, 2, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_64B);
}
int make_tensor_map_3d_u8(CUtensorMap* map, const void* base, uint64_t slabs, uint64_t rows, uint64_t row_bytes, uint32_t box_rows) {
  const cuuint64_t dims[3] = {row_bytes, rows, slabs}, strides[2] = {row_bytes, row_bytes * rows};
  const cuuint32_t box[3] = {128, box_rows, 1};
  return encode_map(map, base, 3, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
}

int sm_count() {
  static std::atomic<int> counts[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
  int n = counts[dev].load(std::memory_order_relaxed);
  if (n == 0) {
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
    counts[dev].store(n, std::memory_order_relaxed);
  }
  return n;
}

__global__ void __launch_bounds__(32) wait_selftest_kernel(uint32_t* status, long long budget) {
  __shared__ uint64_t bar;
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    mbar_fence_init();
  }
  __syncwarp();
  // nobody arrives: the wait gives up after `budget` cycles, records DSV32_STATUS_TIMEOUT (location 99), returns false
  if (threadIdx.x == 0) (void)mbar_wait(&bar, 0, status, 99, budget);
}

int launch_wait_selftest(uint32_t* status, long long budget_cycles, cudaStream_t stream) {
  wait_selftest_kernel<<<1, 32, 0, stream>>>(status, budget_cycles);
  count_launch();
  return check_launch("wait_selftest_kernel");
}

template <int TOK, bool kDots>
static int launch_tc(const IndexerParams& p, const CUtensorMap& key_map, dim3 grid, cudaStream_t stream) {
  CUtensorMap q_map;
  const uint64_t q_rows = static_cast<uint64_t>(p.b) * p.s1 * 64;
  int rc = make_tensor_map_2d_u8(&q_map, p.q, q_rows, 128, 64 * TOK, 128);
  if (rc != DSV32_OK) return rc;
  cudaFuncSetAttribute(indexer_scores_tc_kernel<TOK, kDots>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TcSmemLayout<TOK>::bytes);
  launch_ex(indexer_scores_tc_kernel<TOK, kDots>, grid, TcShape<TOK>::kThreads, TcSmemLayout<TOK>::bytes, stream, true, 1, key_map, q_map, p);
  count_launch();
  return check_launch("indexer_scores_tc_kernel");
}
template <int TOK>
static int launch_tc(const IndexerParams& p, const CUtensorMap& key_map, dim3 grid, cudaStream_t stream) {
  return p.dots != nullptr ? launch_tc<TOK, true>(p, key_map, grid, stream) : launch_tc<TOK, false>(p, key_map, grid, stream);
}

int launch_indexer_scores_tc(const IndexerParams& p, cudaStream_t stream) {
  const int nblk = p.max_blocks - p.key_begin / p.block_size;
  if (nblk <= 0 || p.b <= 0) return DSV32_OK;
  if (p.num_blocks <= 0) {
    set_error("indexer: empty key cache");
    return DSV32_ERR_INVALID_ARG;
  }
  CUtensorMap key_map;
  int rc = make_tensor_map_2d_u8(&key_map, p.keys, static_cast<uint64_t>(p.num_blocks) * 128, 128, 128, 128);
  if (rc != DSV32_OK) return rc;
  IndexerParams q = p;
  if (p.b > 1 && p.s1 <= 2 && p.b < (1 << 20)) {
    // A decode batch of up to two tokens a request: the CTAs share the blocks among themselves (tc_share; not built for TOK = 4,
    // where a ragged batch still runs the blocks of its longest request).  At most four rounds while no share outgrows a CTA's page
    // table: more would mostly be CTAs that find nothing to do.
    const long long slots = 2ll * sm_count(), most = static_cast<long long>(nblk) * p.b;
    long long rounds = (most / 56 + p.b / 2 + slots / 2) / slots;
    const long long need = most / (kTcBlocksPerCta - 1) / slots + 1;
    rounds = rounds > 4 ? (need > 4 ? need : 4) : (rounds < 1 ? 1 : rounds);
    if (most <= INT32_MAX / 2 && rounds * slots + p.b <= INT32_MAX / 2) {
      q.blocks_per_cta = 0;
      q.slots = static_cast<int>(slots);
      q.rounds = static_cast<int>(rounds);
      const dim3 grid(static_cast<unsigned>(rounds * slots + p.b));
      return p.s1 == 1 ? launch_tc<1>(q, key_map, grid, stream) : launch_tc<2>(q, key_map, grid, stream);
    }
  }
  // Otherwise a fixed number of key blocks per CTA.  The CTAs run in rounds of (resident CTAs per SM) x (SMs), and a CTA spends
  // about two block times filling its pipeline; pick the count that minimises rounds x (count + 2), so that the last
  // round is not mostly empty.  Context lengths live on the device, so the longest request stands for all of them.
  int dev = 0, sms = 148;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int tok_groups = p.s1 <= 2 ? 1 : (p.s1 + 3) / 4;
  const long long slots = static_cast<long long>(sms) * (p.s1 <= 2 ? 2 : 1);  // tensor memory: 512 columns per SM
  int best_chunk = 32;
  long long best_cost = -1;
  for (int chunk = 2; chunk <= kTcBlocksPerCta / 2; ++chunk) {
    const long long ctas = static_cast<long long>((nblk + chunk - 1) / chunk) * p.b * tok_groups;
    const long long rounds = (ctas + slots - 1) / slots;
    const long long cost = rounds * (chunk + 2);
    if (best_cost < 0 || cost < best_cost) {
      best_cost = cost;
      best_chunk = chunk;
    }
  }
  q.blocks_per_cta = best_chunk;
  dim3 grid((nblk + best_chunk - 1) / best_chunk, p.b, 1);
  if (p.s1 == 1) return launch_tc<1>(q, key_map, grid, stream);
  if (p.s1 == 2) return launch_tc<2>(q, key_map, grid, stream);
  grid.z = (p.s1 + 3) / 4;
  return launch_tc<4>(q, key_map, grid, stream);
}

}  // namespace dsv32
