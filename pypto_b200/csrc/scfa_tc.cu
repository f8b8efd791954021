// DeepSeek-V4 window / sparse compress attention on tcgen05
// (models/deepseek_v4/sparse_compress_flash_attention_impl.py:47-168, compress_flash_attention_impl.py:115-240,
// win_attention_impl.py): bf16 rows of 512 dims that are key and value at once, a key list made of the token's window rows
// of one cache followed by selected rows of a second (compressed) cache, up to 128 query heads, and one attention sink per
// head added to the softmax denominator.
//
// A pre-pass turns every token's keys into a list of cache rows.  An item of the attention kernel is (token or pair of
// tokens, half of the 512 value dims, part of the key list); M = 128 = the heads of the token(s).  Persistent CTAs of 16 warps:
//   0      issues all products: S(i + 1) is queued before PV(i), so the softmax of a tile runs under the next tile's scores
//   1..3   gather key rows with TMA (gather4: four rows by index, 128 bytes each) into three stages of 48 keys; sixteen
//          rows that lie one below the other come as tiled copies of sixteen
//   4..7   softmax, one head per thread, and the epilogue
//   8..15  bring Q dims 0..319 of the next item into registers under the current one, then into tensor memory; dims 320..511
//          come by TMA
// Tensor memory (512 columns): O 256 | S/P 2 x 48 | Q dims 0..319 as bf16 pairs 160.  Q from tensor memory costs 24 cycles per
// 16 dims of a 48-key tile, from shared memory 46 (its 4 KB are read anew each time), hence as much of it as fits.  Tiles of 48
// keys and not 64: three stages then fit beside Q, and a window of 128 + 1 keys (two tokens) is three tiles with 10 % padding
// instead of 49 %.
// Before, sixteen warps moved the rows through registers, a CTA per item: 6,500 cycles per 64 keys where the products take
// 1,800, and 5 us of setup and epilogue that nothing overlapped.
#include "kernels.cuh"
#include "tc_common.cuh"

namespace dsv32 {

// Request of a token and its token range: the last bi with seq_q[bi] <= tok, or an even split without seq_q.
__device__ __forceinline__ void token_request(const SfaParams& p, int tok, int& bi, int& q0, int& q1) {
  if (p.seq_q == nullptr) {
    const int s1 = p.t_total / p.b;
    bi = tok / s1;
    q0 = bi * s1;
    q1 = q0 + s1;
    return;
  }
  int lo = 0, hi = p.b;  // invariant: seq_q[lo] <= tok < seq_q[hi] for well-formed input
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (__ldg(p.seq_q + mid) <= tok) lo = mid; else hi = mid;
  }
  bi = lo;
  q0 = __ldg(p.seq_q + lo);
  q1 = __ldg(p.seq_q + lo + 1);
}

// Key list of every token for the sparse compress attention: first the window rows (the last
// min(cur_len, win_size) positions before cur_len = max(seq - s1 + 1 + i, 0), paged by block_table), then the
// rows of the compressed cache named by the first min(max(seq / cmp_ratio - s1 + 1 + i, 0), sel_topk) entries of
// the token's index row (paged by block_table2)  (sparse_compress_flash_attention_impl.py:83-131) -- or, with
// cmp_dense, every compressed position below cur_len / cmp_ratio (compress_flash_attention_impl.py:160-186).
// An entry is row + 1 in bits 0..28, bit 29 = "a key of this token", bit 31 = row of the compressed cache;
// 0 = no key.  The window part is padded with empty entries to a multiple of four: the attention kernel gathers four rows of
// one cache at a time.
// With p.pair (at most 64 heads, key lists that do not depend on an index tensor) the tokens 2k and 2k+1 of a
// request share one CTA: lanes 0..63 of the M = 128 tile are the heads of the first, lanes 64..127 those of the
// second.  The list is then the union of both lists -- they differ in one window position and at most one
// compressed position -- with bit 29 / bit 30 = member of the first / second token's list; it is stored in the
// first token's slot, and the second token's count is -1 ("done by the partner").
__global__ void __launch_bounds__(256) scfa_row_ids_kernel(SfaParams p) {
  const int tok = blockIdx.y;
  const int j = blockIdx.x * 256 + threadIdx.x;
  pdl_wait();     // (first kernel of an operator: everything it reads may come from the kernel before)
  pdl_trigger();
  if (j >= p.topk) return;
  int bi, q0, q1;
  token_request(p, tok, bi, q0, q1);
  uint32_t out = 0;
  int count = 0;
  if (tok < q0 || tok >= q1) {
    if (j == 0) report_status(p.status, DSV32_STATUS_BAD_INDEX, tok, bi);
  } else if (p.pair && ((tok - q0) & 1)) {
    count = -1;  // second token of a pair
  } else {
    const int s1 = q1 - q0, si = tok - q0;
    const int seq = __ldg(p.act_seq + bi);
    const bool has_b = p.pair && si + 1 < s1;
    // first token (a), second token (b = a + 1 position) of the pair; without pairing only a
    const int len_a = max(seq - s1 + 1 + si, 0), len_b = has_b ? max(seq - s1 + 2 + si, 0) : len_a;
    const int win_a = min(len_a, p.win_size), win_b = min(len_b, p.win_size);
    const int sel_a = p.cmp_dense ? min(len_a / p.cmp_ratio, p.sel_topk)
                                  : min(max(seq / p.cmp_ratio - s1 + 1 + si, 0), p.sel_topk);
    const int sel_b = has_b ? min(len_b / p.cmp_ratio, p.sel_topk) : sel_a;   // pairs only exist with cmp_dense / no index
    const int w_start = len_a - win_a;              // first window position of the union (b's window starts later or equal)
    const int w_len = len_b - w_start;              // union window: [w_start, len_b)
    const int w_pad = (w_len + 3) & ~3;
    const int sel_u = max(sel_a, sel_b);
    count = w_pad + sel_u;
    if (j < w_len) {
      const int pos = w_start + j;
      const uint32_t mem = (pos < len_a ? 1u : 0u) | ((has_b && pos >= len_b - win_b) ? 2u : 0u);
      const int lb = pos / p.block_size;
      if (lb >= p.max_blocks) {
        report_status(p.status, DSV32_STATUS_BAD_INDEX, tok, pos);
      } else {
        const int pb = __ldg(p.block_table + static_cast<size_t>(bi) * p.max_blocks + lb);
        const long long row = static_cast<long long>(pb) * p.block_size + pos % p.block_size;
        if (pb < 0 || row >= p.rows) report_status(p.status, DSV32_STATUS_BAD_PAGE, tok, pos);
        else out = (static_cast<uint32_t>(row) + 1u) | (mem << 29);
      }
    } else if (j >= w_pad && j < count) {
      const int e = j - w_pad;
      const int idx = (p.cmp_dense || p.topk_idx == nullptr) ? e : __ldg(p.topk_idx + static_cast<size_t>(tok) * p.sel_topk + e);
      const uint32_t mem = (e < sel_a ? 1u : 0u) | ((has_b && e < sel_b) ? 2u : 0u);
      if (idx >= 0) {
        const int lb = idx / p.block_size;
        if (lb >= p.max_blocks2) {
          report_status(p.status, DSV32_STATUS_BAD_INDEX, tok, idx);
        } else {
          const int pb = __ldg(p.block_table2 + static_cast<size_t>(bi) * p.max_blocks2 + lb);
          const long long row = static_cast<long long>(pb) * p.block_size + idx % p.block_size;
          if (pb < 0 || row >= p.rows2) report_status(p.status, DSV32_STATUS_BAD_PAGE, tok, idx);
          else out = (static_cast<uint32_t>(row) + 1u) | (mem << 29) | 0x80000000u;
        }
      }
    }
  }
  p.row_ids[static_cast<size_t>(tok) * p.topk + j] = static_cast<int>(out);
  if (j == 0) p.key_counts[tok] = count;
}

// The same for the operator whose compressed keys come from an index tensor (p.pair == 2): one CTA per token.
// The CTA of the first token of a pair builds the union of both tokens' selections: two bitmaps over the compressed
// positions (shared memory) say which token selected what; the list is the union window, then the first token's
// entries (bit 30 set as well where the second token selected the same position), then the second token's
// entries that the first did not select, compacted in their original order by a block-wide scan (deterministic).
constexpr int kPairBitmapWords = 4096;   // 131,072 compressed positions per request at most

__global__ void __launch_bounds__(256) scfa_pair_ids_kernel(SfaParams p) {
  __shared__ uint32_t bm_a[kPairBitmapWords], bm_b[kPairBitmapWords];
  __shared__ int warp_cnt[8];
  const int tok = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  pdl_wait();     // (first kernel of an operator: everything it reads may come from the kernel before)
  pdl_trigger();
  int bi, q0, q1;
  token_request(p, tok, bi, q0, q1);
  int32_t* list = p.row_ids + static_cast<size_t>(tok) * p.topk;
  if (tok < q0 || tok >= q1) {
    if (tid == 0) {
      report_status(p.status, DSV32_STATUS_BAD_INDEX, tok, bi);
      p.key_counts[tok] = 0;
    }
    return;
  }
  const int s1 = q1 - q0, si = tok - q0;
  if (si & 1) {
    if (tid == 0) p.key_counts[tok] = -1;  // second token of a pair
    return;
  }
  const int seq = __ldg(p.act_seq + bi);
  const bool has_b = si + 1 < s1;
  const int len_a = max(seq - s1 + 1 + si, 0), len_b = has_b ? max(seq - s1 + 2 + si, 0) : len_a;
  const int win_a = min(len_a, p.win_size), win_b = min(len_b, p.win_size);
  const int sel_a = min(max(seq / p.cmp_ratio - s1 + 1 + si, 0), p.sel_topk);
  const int sel_b = has_b ? min(max(seq / p.cmp_ratio - s1 + 2 + si, 0), p.sel_topk) : 0;
  const int w_start = len_a - win_a, w_len = len_b - w_start, w_pad = (w_len + 3) & ~3;
  const int cap = p.max_blocks2 * p.block_size;   // compressed positions of a request (<= 32 * kPairBitmapWords)
  auto resolve = [&](int idx, uint32_t mem) -> uint32_t {   // entry of compressed position idx, 0 if it cannot be used
    if (idx < 0) return 0u;
    if (idx >= cap) {
      report_status(p.status, DSV32_STATUS_BAD_INDEX, tok, idx);
      return 0u;
    }
    const int pb = __ldg(p.block_table2 + static_cast<size_t>(bi) * p.max_blocks2 + idx / p.block_size);
    const long long row = static_cast<long long>(pb) * p.block_size + idx % p.block_size;
    if (pb < 0 || row >= p.rows2) {
      report_status(p.status, DSV32_STATUS_BAD_PAGE, tok, idx);
      return 0u;
    }
    return (static_cast<uint32_t>(row) + 1u) | (mem << 29) | 0x80000000u;
  };
  // window
  for (int j = tid; j < w_pad; j += 256) {
    if (j >= w_len) {
      list[j] = 0;
      continue;
    }
    const int pos = w_start + j;
    const uint32_t mem = (pos < len_a ? 1u : 0u) | ((has_b && pos >= len_b - win_b) ? 2u : 0u);
    uint32_t out = 0;
    const int lb = pos / p.block_size;
    if (lb >= p.max_blocks) {
      report_status(p.status, DSV32_STATUS_BAD_INDEX, tok, pos);
    } else {
      const int pb = __ldg(p.block_table + static_cast<size_t>(bi) * p.max_blocks + lb);
      const long long row = static_cast<long long>(pb) * p.block_size + pos % p.block_size;
      if (pb < 0 || row >= p.rows) report_status(p.status, DSV32_STATUS_BAD_PAGE, tok, pos);
      else out = (static_cast<uint32_t>(row) + 1u) | (mem << 29);
    }
    list[j] = static_cast<int>(out);
  }
  // bitmaps of both selections
  const int words = (cap + 31) / 32;
  for (int i = tid; i < words; i += 256) { bm_a[i] = 0u; bm_b[i] = 0u; }
  __syncthreads();
  const int32_t* ia = p.topk_idx + static_cast<size_t>(tok) * p.sel_topk;
  const int32_t* ib = ia + p.sel_topk;   // the next token's index row
  for (int e = tid; e < sel_a; e += 256) {
    const int idx = __ldg(ia + e);
    if (idx >= 0 && idx < cap) atomicOr(&bm_a[idx >> 5], 1u << (idx & 31));
  }
  for (int e = tid; e < sel_b; e += 256) {
    const int idx = __ldg(ib + e);
    if (idx >= 0 && idx < cap) atomicOr(&bm_b[idx >> 5], 1u << (idx & 31));
  }
  __syncthreads();
  // the first token's entries, in place
  for (int e = tid; e < sel_a; e += 256) {
    const int idx = __ldg(ia + e);
    const bool in_b = idx >= 0 && idx < cap && ((bm_b[idx >> 5] >> (idx & 31)) & 1u);
    list[w_pad + e] = static_cast<int>(resolve(idx, in_b ? 3u : 1u));
  }
  // the second token's entries that the first did not select, compacted in order
  int base = w_pad + sel_a;
  for (int e0 = 0; e0 < sel_b; e0 += 256) {
    const int e = e0 + tid;
    int idx = -1;
    if (e < sel_b) idx = __ldg(ib + e);
    const bool take = idx >= 0 && !(idx < cap && ((bm_a[idx >> 5] >> (idx & 31)) & 1u));
    const uint32_t ballot = __ballot_sync(0xffffffffu, take);
    if (lane == 0) warp_cnt[warp] = __popc(ballot);
    __syncthreads();
    int before = 0, total = 0;
#pragma unroll
    for (int w = 0; w < 8; ++w) {
      if (w < warp) before += warp_cnt[w];
      total += warp_cnt[w];
    }
    if (take) list[base + before + __popc(ballot & ((1u << lane) - 1u))] = static_cast<int>(resolve(idx, 2u));
    base += total;
    __syncthreads();
  }
  if (tid == 0) p.key_counts[tok] = base;
}

namespace {
constexpr int kScThreads = 512;
constexpr int kScTile = 48;                              // keys per tile
constexpr int kScGatherWarps = 3, kScWarpQuads = kScTile / 4 / kScGatherWarps;
constexpr int kScChunk = kScTile * 128;                  // one 64-dim chunk of a stage (6 KB)
constexpr int kScStage = 8 * kScChunk;                   // 49,152
constexpr int kScStages = 3;
constexpr int kScOffQ = kScStages * kScStage;            // Q dims 320..511: three 128 x 64 chunks
constexpr int kScOffStore = kScOffQ + 3 * 16384;         // one 4 KB store buffer per softmax warp
constexpr int kScOffTurn = kScOffStore + 4 * 4096;       // 2 KB per Q warp
constexpr int kScOffValid = kScOffTurn + 8 * 2048;       // int[3][48] membership bits of the staged keys
constexpr int kScOffBars = kScOffValid + kScStages * kScTile * 4;
constexpr int kScNumBars = 2 * kScStages + 2 + 2 + 4;    // full, empty, s_full[2], p_ready[2], q_full, q_free, o_full, o_free
constexpr int kScOffTmem = kScOffBars + kScNumBars * 8;
constexpr size_t kScSmemBytes = kScOffTmem + 16;
static_assert(kScSmemBytes <= 232448, "shared memory of one CTA");
constexpr uint32_t kScColO = 0, kScColS = 256, kScColQ = 352;
constexpr float kScRescale = 8.0f;                       // log2 units: the running maximum is raised beyond this only

__device__ __forceinline__ float sc_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// One warp's walk over the CTA's items: (token, value half, key range in tiles).  The list lengths of 32 items are read at once,
// one per lane; read item by item, they cost every role a trip to L2 each time.
struct ScWalk {
  const SfaParams& p;
  int items, base, lane;
  int raw, raw1;      // lengths of the list of this lane's item's token and of the next token
  uint32_t pending;   // lanes whose item has something to do
  int tok, half, split, live_rows, k_lo, k_hi, ntiles;

  __device__ __forceinline__ ScWalk(const SfaParams& p_, int items_, int lane_)
      : p(p_), items(items_), base(blockIdx.x), lane(lane_), raw(-1), raw1(0), pending(0) {
    load();
  }
  __device__ __forceinline__ void load() {
    const int it = base + lane * gridDim.x;
    raw = -1;
    raw1 = 0;
    if (it < items) {
      const int t = (it >> 1) % p.t_total;
      raw = __ldcg(p.key_counts + t);
      if (t + 1 < p.t_total) raw1 = __ldcg(p.key_counts + t + 1);
    }
    pending = __ballot_sync(0xffffffffu, raw >= 0);   // (negative: second token of a pair, lanes n_q .. of the partner's item)
  }
  // next item with something to do (empty: or zeros to write)
  __device__ __forceinline__ bool next(bool empty) {
    while (true) {
      if (pending == 0u) {
        base += 32 * gridDim.x;
        if (base >= items) return false;
        load();
        continue;
      }
      const int l = __ffs(pending) - 1;
      pending &= pending - 1u;
      const int c = __shfl_sync(0xffffffffu, raw, l), c1 = __shfl_sync(0xffffffffu, raw1, l), it = base + l * gridDim.x;
      half = it & 1;
      tok = (it >> 1) % p.t_total;
      split = (it >> 1) / p.t_total;
      live_rows = (p.pair && c1 < 0) ? 2 * p.nq : p.nq;
      const int cnt = min(c, p.topk);
      const int per = ((cnt + p.splits - 1) / p.splits + kScTile - 1) / kScTile * kScTile;
      k_lo = split * per;
      k_hi = min(cnt, k_lo + per);
      ntiles = k_hi > k_lo ? (k_hi - k_lo + kScTile - 1) / kScTile : 0;
      if (ntiles > 0 || empty) return true;
    }
  }
};
}  // namespace

__global__ void __launch_bounds__(kScThreads, 1)
scfa_tc_kernel(const __grid_constant__ CUtensorMap q_map, const __grid_constant__ CUtensorMap kv_map,
               const __grid_constant__ CUtensorMap kv2_map, const __grid_constant__ CUtensorMap run_map,
               const __grid_constant__ CUtensorMap run2_map, SfaParams p, int items) {
  extern __shared__ __align__(1024) unsigned char smem[];
  if ((smem_u32(smem) & 1023u) != 0u) {
    if (threadIdx.x == 0) report_status(p.status, DSV32_STATUS_INTERNAL, 110, smem_u32(smem));
    return;
  }
  int* valid_s = reinterpret_cast<int*>(smem + kScOffValid);
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + kScOffBars);   // [3] keys in place -> products
  uint64_t* empty_bar = full_bar + kScStages;                            // [3] PV of the stage's tile complete
  uint64_t* sfull_bar = empty_bar + kScStages;                           // [2] S complete -> softmax
  uint64_t* pready_bar = sfull_bar + 2;                                  // [2] P stored -> products
  uint64_t* qfull_bar = pready_bar + 2;                                  //     Q of an item in place
  uint64_t* qfree_bar = qfull_bar + 1;                                   //     last S of an item complete
  uint64_t* ofull_bar = qfull_bar + 2;                                   //     last PV of an item complete
  uint64_t* ofree_bar = qfull_bar + 3;                                   //     O has been read
  uint32_t* tmem_ptr_s = reinterpret_cast<uint32_t*>(smem + kScOffTmem);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (warp == 0) {
    if (lane == 0) {
      tma_prefetch_desc(&q_map);
      tma_prefetch_desc(&kv_map);
      tma_prefetch_desc(&kv2_map);
      tma_prefetch_desc(&run_map);
      tma_prefetch_desc(&run2_map);
      for (int i = 0; i < kScStages; ++i) {
        mbar_init(&full_bar[i], kScGatherWarps);
        mbar_init(&empty_bar[i], 1);
      }
      for (int i = 0; i < 2; ++i) {
        mbar_init(&sfull_bar[i], 1);
        mbar_init(&pready_bar[i], 4);
      }
      mbar_init(qfull_bar, 9);    // Q's TMA and the eight warps that fill tensor memory
      mbar_init(qfree_bar, 1);
      mbar_init(ofull_bar, 1);
      mbar_init(ofree_bar, 4);
      mbar_fence_init();
    }
    __syncwarp();
    tmem_alloc(tmem_ptr_s, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_ptr_s;
  pdl_trigger();
  pdl_wait();   // the key lists are the pre-pass'
  ScWalk w(p, items, lane);

  if (warp == 0) {
    // ---- products ---------------------------------------------------------------------------------------------------
    constexpr uint32_t idesc_s = umma_idesc_bf16(128, kScTile, false, false), idesc_pv = umma_idesc_bf16(128, 256, false, true);
    const uint32_t tbase = __shfl_sync(0xffffffffu, tmem_base, 0);
    bool ok = true;
    int g = 0, n = 0;   // tiles and items so far
    while (ok && w.next(false)) {
      ok = __all_sync(0xffffffffu, mbar_wait(qfull_bar, n & 1, p.status, 111));
      for (int k = 0; ok && k <= w.ntiles; ++k) {
        if (k < w.ntiles) {   // S of tile g + k
          const int t = g + k, s = t % kScStages, b = t & 1;
          ok = __all_sync(0xffffffffu, mbar_wait(&full_bar[s], (t / kScStages) & 1, p.status, 112));
          if (!ok) break;
          tc_fence_after();
          // (PV of the tile before last, which reads P from this buffer, is ahead in the tensor core's queue)
          const uint32_t d = tbase + kScColS + b * kScTile;
          const uint64_t kd = umma_smem_desc_sw128(smem_u32(smem + s * kScStage), 16, 1024);
          const uint64_t qd = umma_smem_desc_sw128(smem_u32(smem + kScOffQ), 16, 1024);
          if (elect_one()) {
#pragma unroll
            for (int ks = 0; ks < 20; ++ks)
              umma_f16_ts(d, tbase + kScColQ + ks * 8, kd + (((ks >> 2) * kScChunk + (ks & 3) * 32) >> 4), idesc_s, ks > 0 ? 1u : 0u);
#pragma unroll
            for (int ks = 20; ks < 32; ++ks)
              umma_f16_ss(d, qd + ((((ks >> 2) - 5) * 16384 + (ks & 3) * 32) >> 4), kd + (((ks >> 2) * kScChunk + (ks & 3) * 32) >> 4),
                          idesc_s, 1u);
            umma_commit(&sfull_bar[b]);
            if (k == w.ntiles - 1) umma_commit(qfree_bar);
          }
          __syncwarp();
        }
        if (k > 0) {          // PV of tile g + k - 1
          const int t = g + k - 1, s = t % kScStages, b = t & 1;
          ok = __all_sync(0xffffffffu, mbar_wait(&pready_bar[b], (t >> 1) & 1, p.status, 113) &&
                                           (k > 1 || mbar_wait(ofree_bar, (n & 1) ^ 1, p.status, 114)));
          if (!ok) break;
          tc_fence_after();
          const uint64_t vd = umma_smem_desc_sw128(smem_u32(smem + s * kScStage) + 4 * w.half * kScChunk, kScChunk, 1024);
          if (elect_one()) {
#pragma unroll
            for (int kk = 0; kk < kScTile / 16; ++kk)   // V = this item's four 64-dim chunks, MN-major
              umma_f16_ts(tbase + kScColO, tbase + kScColS + b * kScTile + kk * 8, vd + 128 * kk, idesc_pv, (k > 1 || kk > 0) ? 1u : 0u);
            umma_commit(&empty_bar[s]);
            if (k == w.ntiles) umma_commit(ofull_bar);
          }
          __syncwarp();
        }
      }
      g += w.ntiles;
      ++n;
    }
  } else if (warp <= kScGatherWarps) {
    // ---- keys: four quads of a tile per warp ------------------------------------------------------------------------------
    // The rows of a quad are the same in all lanes when one of them issues its eight copies: copies issued by different lanes
    // with rows of their own take 90 cycles each, a loop over the lanes that the hardware's uniform operands force.
    const int quad0 = (warp - 1) * kScWarpQuads;
    bool ok = true;
    int g = 0;
    while (ok && w.next(false)) {
      const int32_t* ids = p.row_ids + static_cast<size_t>(w.tok) * p.topk;   // (slots of a list: a multiple of four)
      auto fetch = [&](int k) {   // lane = key of the warp's quads
        const int j = w.k_lo + k * kScTile + 4 * quad0 + lane;
        return lane < 4 * kScWarpQuads && j < w.k_hi ? __ldcg(ids + j) : 0;
      };
      int next = fetch(0);
      for (int k = 0; k < w.ntiles; ++k, ++g) {
        const int v = next;
        if (k + 1 < w.ntiles) next = fetch(k + 1);
        const int s = g % kScStages;
        ok = __all_sync(0xffffffffu, mbar_wait(&empty_bar[s], ((g / kScStages) & 1) ^ 1, p.status, 115));
        if (!ok) break;
        if (lane < 4 * kScWarpQuads) valid_s[s * kScTile + 4 * quad0 + lane] = (v >> 29) & 3;
        __syncwarp();
        if (lane == 0) mbar_arrive_expect_tx(&full_bar[s], kScWarpQuads * 4 * 1024);
        __syncwarp();
        // bits 0..28: row + 1, 0 = no key (row -1 is outside the tensor: zeros); bit 31: the second cache, alike in a quad
        const uint32_t second = __ballot_sync(0xffffffffu, v < 0);
        const int row = (v & 0x1fffffff) - 1, row0 = __shfl_sync(0xffffffffu, row, 0);
        // sixteen rows one below the other in one cache (a window, dense compressed keys): eight tiled copies
        const bool run = __all_sync(0xffffffffu, lane >= 4 * kScWarpQuads || (row >= 0 && row == row0 + lane)) &&
                         ((second & 0xffffu) == 0u || (second & 0xffffu) == 0xffffu);
        if (run) {
          const CUtensorMap* map = second != 0u ? &run2_map : &run_map;
          unsigned char* dst = smem + s * kScStage + quad0 * 512;
          if (elect_one()) {
#pragma unroll
            for (int c = 0; c < 8; ++c) tma_load_2d(dst + c * kScChunk, map, c * 128, row0, &full_bar[s]);
          }
          __syncwarp();
          continue;
        }
#pragma unroll
        for (int q = 0; q < kScWarpQuads; ++q) {
          const int r0 = __shfl_sync(0xffffffffu, row, 4 * q), r1 = __shfl_sync(0xffffffffu, row, 4 * q + 1);
          const int r2 = __shfl_sync(0xffffffffu, row, 4 * q + 2), r3 = __shfl_sync(0xffffffffu, row, 4 * q + 3);
          const CUtensorMap* map = ((second >> (4 * q)) & 15u) != 0u ? &kv2_map : &kv_map;
          unsigned char* dst = smem + s * kScStage + (quad0 + q) * 512;
          if (elect_one()) {
#pragma unroll
            for (int c = 0; c < 8; ++c) tma_gather4(dst + c * kScChunk, map, c * 128, r0, r1, r2, r3, &full_bar[s]);
          }
          __syncwarp();
        }
      }
    }
  } else if (warp >= 8) {
    // ---- Q: dims 0..319 -> tensor memory, the rest by TMA -----------------------------------------------------------------------------------
    const int quarter = warp & 3, part = (warp - 8) >> 2;   // 160 dims = 80 columns each
    unsigned char* turn = smem + kScOffTurn + (warp - 8) * 2048;
    bool ok = true;
    int n = 0;
    while (ok && w.next(false)) {
      // Loaded with four lanes to 64 bytes of a row and turned in shared memory to a row per lane: loads of a row per lane
      // (32 lines each) kept the load/store unit busy for longer than an item's products take.
      const __nv_bfloat16* rows = p.q_nope + (static_cast<size_t>(w.tok) * p.nq + quarter * 32) * kKvLora + part * 160;
      uint4 v[20];
#pragma unroll
      for (int j = 0; j < 20; ++j) {   // step j / 4: dims 32 (j / 4) ..; rows 8 (j % 4) + lane / 4
        const int r = 8 * (j & 3) + (lane >> 2);
        v[j] = make_uint4(0u, 0u, 0u, 0u);
        if (quarter * 32 + r < w.live_rows)
          v[j] = __ldg(reinterpret_cast<const uint4*>(rows + static_cast<size_t>(r) * kKvLora + (j >> 2) * 32) + (lane & 3));
      }
#pragma unroll
      for (int st = 0; st < 5; ++st) {
        __syncwarp();
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int r = 8 * j + (lane >> 2);
          *reinterpret_cast<uint4*>(turn + r * 64 + (((lane & 3) ^ ((r >> 1) & 3)) << 4)) = v[4 * st + j];
        }
        __syncwarp();
#pragma unroll
        for (int j = 0; j < 4; ++j) v[4 * st + j] = *reinterpret_cast<const uint4*>(turn + lane * 64 + ((j ^ ((lane >> 1) & 3)) << 4));
      }
      uint32_t a[32], b[32], c[16];
#pragma unroll
      for (int j = 0; j < 20; ++j) {
        uint32_t* d = j < 8 ? a + 4 * j : j < 16 ? b + 4 * (j - 8) : c + 4 * (j - 16);
        d[0] = v[j].x; d[1] = v[j].y; d[2] = v[j].z; d[3] = v[j].w;
      }
      ok = __all_sync(0xffffffffu, mbar_wait(qfree_bar, (n & 1) ^ 1, p.status, 117));
      if (!ok) break;
      if (warp == 8 && lane == 0) {   // dims 320..511 -> shared memory
        mbar_arrive_expect_tx(qfull_bar, 3 * 16384);
        for (int c = 0; c < 3; ++c) tma_load_2d(smem + kScOffQ + c * 16384, &q_map, (5 + c) * 128, w.tok * p.nq, qfull_bar);
      }
      __syncwarp();
      tc_fence_after();
      const uint32_t dst = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + kScColQ + part * 80;
      tmem_st_32x32b_x32(dst, a);
      tmem_st_32x32b_x32(dst + 32, b);
      tmem_st_32x32b_x16(dst + 64, c);
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(qfull_bar);
      ++n;
    }
  } else if (warp >= 4) {
    // ---- softmax and epilogue -----------------------------------------------------------------------------------------------
    const int quarter = warp & 3, head = quarter * 32 + lane;
    const uint32_t lane_base = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
    unsigned char* buf = smem + kScOffStore + (warp - 4) * 4096;
    const uint32_t sw = static_cast<uint32_t>(lane & 7);
    const float sc2 = p.scale * 1.4426950408889634f;   // softmax scale in log2 units
    const uint64_t sc22 = f2_pack(__float_as_uint(sc2), __float_as_uint(sc2));
    bool ok = true;
    int g = 0, n = 0;
    while (ok && w.next(true)) {
      const int tok2 = w.tok + (head >= p.nq ? 1 : 0), head2 = head >= p.nq ? head - p.nq : head;   // this lane's token and head
      const bool live = head < w.live_rows;
      const size_t prow = (static_cast<size_t>(tok2) * p.splits + w.split) * p.nq + head2;
      if (w.ntiles == 0) {   // nothing to attend to
        if (live) {
          if (p.splits == 1) {
            uint4* o = reinterpret_cast<uint4*>(p.out + (static_cast<size_t>(tok2) * p.nq + head2) * kKvLora + w.half * 256);
            for (int i = 0; i < 32; ++i) o[i] = make_uint4(0u, 0u, 0u, 0u);
          } else {
            float4* o = reinterpret_cast<float4*>(p.part_o + prow * kKvLora + w.half * 256);
            for (int i = 0; i < 64; ++i) o[i] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (w.half == 0) p.part_lse[prow] = -INFINITY;
          }
        }
        continue;
      }
      // whose keys this lane's head takes: bit 0 = the first token's, bit 1 the second's; idle lanes take all
      const int hb = head < p.nq ? 1 : (live ? 2 : 3);
      float m_run = -INFINITY, l_run = 0.f;
      for (int k = 0; k < w.ntiles; ++k, ++g) {
        const int b = g & 1, s = g % kScStages;
        ok = __all_sync(0xffffffffu, mbar_wait(&sfull_bar[b], (g >> 1) & 1, p.status, 118));
        if (!ok) break;
        tc_fence_after();
        const uint32_t s_addr = lane_base + kScColS + b * kScTile;
        const int* vm = valid_s + s * kScTile;
        // this lane's keys of the tile as a bit mask
        const int f0 = vm[lane], f1 = lane < 16 ? vm[32 + lane] : 3;
        const uint32_t a0 = __ballot_sync(0xffffffffu, f0 & 1), a1 = __ballot_sync(0xffffffffu, f1 & 1);
        const uint32_t b0 = __ballot_sync(0xffffffffu, f0 & 2), b1 = __ballot_sync(0xffffffffu, f1 & 2);
        const uint32_t m0 = hb == 1 ? a0 : hb == 2 ? b0 : 0xffffffffu, m1 = hb == 1 ? a1 : hb == 2 ? b1 : 0xffffffffu;
        uint32_t r[32], q[16];
        tmem_ld_32x32b_x32(s_addr, r);
        tmem_ld_32x32b_x16(s_addr + 32, q);
        tmem_ld_wait();
        if (!__all_sync(0xffffffffu, (m0 & m1) == 0xffffffffu)) {
#pragma unroll
          for (int j = 0; j < 32; ++j)
            if (!((m0 >> j) & 1u)) r[j] = 0xff800000u;   // -inf
#pragma unroll
          for (int j = 0; j < 16; ++j)
            if (!((m1 >> j) & 1u)) q[j] = 0xff800000u;
        }
        float m_raw = -INFINITY;
#pragma unroll
        for (int j = 0; j < 32; j += 2) m_raw = fmaxf(m_raw, fmaxf(__uint_as_float(r[j]), __uint_as_float(r[j + 1])));
#pragma unroll
        for (int j = 0; j < 16; j += 2) m_raw = fmaxf(m_raw, fmaxf(__uint_as_float(q[j]), __uint_as_float(q[j + 1])));
        const float m_tile = m_raw * sc2;
        const bool need = m_tile > m_run + kScRescale;   // also true on the first non-empty tile (m_run = -inf)
        if (__any_sync(0xffffffffu, need)) {
          const float m_new = need ? m_tile : m_run;
          const float alpha = (m_new == -INFINITY) ? 1.f : exp2f(m_run - m_new);   // m_run = -inf -> 0
          l_run *= alpha;
          m_run = m_new;
          if (k > 0) {   // O holds data: scale this head's row (the previous PV must have finished)
            ok = __all_sync(0xffffffffu, mbar_wait(&empty_bar[(g - 1) % kScStages], ((g - 1) / kScStages) & 1, p.status, 119));
            if (!ok) break;
            tc_fence_after();
#pragma unroll 1
            for (int c = 0; c < 8; ++c) {
              uint32_t o[32];
              tmem_ld_32x32b_x32(lane_base + kScColO + c * 32, o);
              tmem_ld_wait();
#pragma unroll
              for (int j = 0; j < 32; ++j) o[j] = __float_as_uint(__uint_as_float(o[j]) * alpha);
              tmem_st_32x32b_x32(lane_base + kScColO + c * 32, o);
            }
            tmem_st_wait();
          }
        }
        const float neg_m = (m_run == -INFINITY) ? 0.f : -m_run;
        const uint64_t negm2 = f2_pack(__float_as_uint(neg_m), __float_as_uint(neg_m));
        uint64_t lsum_a = 0ull, lsum_b = 0ull;
        auto exp4 = [&](const uint32_t* v, uint32_t& w0, uint32_t& w1) {
          float p0, p1, p2, p3;
          f2_unpack(f2_fma(f2_pack(v[0], v[1]), sc22, negm2), p0, p1);
          f2_unpack(f2_fma(f2_pack(v[2], v[3]), sc22, negm2), p2, p3);
          p0 = sc_exp2(p0); p1 = sc_exp2(p1); p2 = sc_exp2(p2); p3 = sc_exp2(p3);
          lsum_a = f2_add(lsum_a, f2_pack(__float_as_uint(p0), __float_as_uint(p1)));
          lsum_b = f2_add(lsum_b, f2_pack(__float_as_uint(p2), __float_as_uint(p3)));
          w0 = pack_bf16x2(p0, p1);
          w1 = pack_bf16x2(p2, p3);
        };
        uint32_t pa[16], pb[8];   // P as bf16 pairs over the first 24 columns of the S buffer
#pragma unroll
        for (int j = 0; j < 32; j += 4) exp4(r + j, pa[j >> 1], pa[(j >> 1) + 1]);
#pragma unroll
        for (int j = 0; j < 16; j += 4) exp4(q + j, pb[j >> 1], pb[(j >> 1) + 1]);
        tmem_st_32x32b_x16(s_addr, pa);
        tmem_st_32x32b_x8(s_addr + 16, pb);
        {
          float s0, s1, s2, s3;
          f2_unpack(lsum_a, s0, s1);
          f2_unpack(lsum_b, s2, s3);
          l_run += (s0 + s1) + (s2 + s3);
        }
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&pready_bar[b]);
      }
      // ---- O / l -> bf16 (or fp32 partial + log-sum-exp for a key split) --------------------------------------------------
      if (ok) ok = __all_sync(0xffffffffu, mbar_wait(ofull_bar, n & 1, p.status, 120));
      if (!ok) break;
      tc_fence_after();
      if (p.splits == 1 && live && m_run != -INFINITY)   // the sink joins the denominator only, in the units of m_run
        l_run += exp2f(fmaf(__ldg(p.sinks + head2), 1.4426950408889634f, -m_run));
      const float inv = (l_run > 0.f) ? 1.f / l_run : 0.f;
      const bool whole = quarter * 32 + 32 <= w.live_rows;   // every lane of the warp holds a head
      if (quarter * 32 < w.live_rows) {
#pragma unroll 1
        for (int c = 0; c < 4; ++c) {                        // 64 columns = 128 bytes of bf16
          uint32_t o[2][32];
          tmem_ld_32x32b_x32(lane_base + kScColO + c * 64, o[0]);
          tmem_ld_32x32b_x32(lane_base + kScColO + c * 64 + 32, o[1]);
          tmem_ld_wait();
          auto val = [&](int j) { return __uint_as_float(o[j >> 5][j & 31]) * inv; };
          if (p.splits > 1) {
            // 32 columns at a time, as below; a row's place depends on its token
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              __syncwarp();
#pragma unroll
              for (int u = 0; u < 8; ++u)
                *reinterpret_cast<float4*>(buf + lane * 128 + ((u ^ sw) << 4)) =
                    make_float4(val(h * 32 + 4 * u), val(h * 32 + 4 * u + 1), val(h * 32 + 4 * u + 2), val(h * 32 + 4 * u + 3));
              __syncwarp();
#pragma unroll
              for (int i = 0; i < 8; ++i) {
                const int row = 4 * i + (lane >> 3), u = lane & 7, hd = quarter * 32 + row;
                const size_t pr = (static_cast<size_t>(w.tok + (hd >= p.nq ? 1 : 0)) * p.splits + w.split) * p.nq + (hd >= p.nq ? hd - p.nq : hd);
                if (hd < w.live_rows)
                  reinterpret_cast<float4*>(p.part_o + pr * kKvLora + w.half * 256 + c * 64 + h * 32)[u] =
                      *reinterpret_cast<const float4*>(buf + row * 128 + ((u ^ (row & 7)) << 4));
              }
            }
          } else if (whole) {
            // through shared memory to whole lines, eight lanes a row (a TMA store would queue behind the gathers in flight)
            __syncwarp();
#pragma unroll
            for (int u = 0; u < 8; ++u)
              *reinterpret_cast<uint4*>(buf + lane * 128 + ((u ^ sw) << 4)) =
                  make_uint4(pack_bf16x2(val(8 * u), val(8 * u + 1)), pack_bf16x2(val(8 * u + 2), val(8 * u + 3)),
                             pack_bf16x2(val(8 * u + 4), val(8 * u + 5)), pack_bf16x2(val(8 * u + 6), val(8 * u + 7)));
            __syncwarp();
            __nv_bfloat16* dst = p.out + (static_cast<size_t>(w.tok) * p.nq + quarter * 32) * kKvLora + w.half * 256 + c * 64;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const int row = 4 * i + (lane >> 3), u = lane & 7;
              reinterpret_cast<uint4*>(dst + static_cast<size_t>(row) * kKvLora)[u] =
                  *reinterpret_cast<const uint4*>(buf + row * 128 + ((u ^ (row & 7)) << 4));
            }
          } else if (live) {
            uint4* dst = reinterpret_cast<uint4*>(p.out + (static_cast<size_t>(tok2) * p.nq + head2) * kKvLora + w.half * 256 + c * 64);
#pragma unroll
            for (int u = 0; u < 8; ++u)
              dst[u] = make_uint4(pack_bf16x2(val(8 * u), val(8 * u + 1)), pack_bf16x2(val(8 * u + 2), val(8 * u + 3)),
                                  pack_bf16x2(val(8 * u + 4), val(8 * u + 5)), pack_bf16x2(val(8 * u + 6), val(8 * u + 7)));
          }
        }
        if (p.splits > 1 && w.half == 0 && live)
          p.part_lse[prow] = (l_run > 0.f) ? (m_run + log2f(l_run)) * 0.6931471805599453f : -INFINITY;
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(ofree_bar);
      ++n;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// ---- host ------------------------------------------------------------------------------------------------------------
// Lists that share the CTAs: one per two tokens where every request has an even number of them and all are paired; otherwise one per
// token, since the item of a second token, which has nothing to do, takes its turn like the others.
int scfa_lists(int t, int b, int pair) { return pair && t % b == 0 && t / b % 2 == 0 ? t / 2 : t; }

// Most parts a key list of `slots` entries is split into: while the items leave SMs idle, and no part below two tiles.  More items
// than CTAs would be a second round: 74 requests of one token, once counted as 37 pairs and split in two, took 63.6 us with
// selected keys and 40.4 with ratio 128, unsplit 33.5 and 16.4; 20 requests of three tokens 47.1 and 30.9, unsplit 32.8 and 16.5.
int scfa_most_splits(int lists, int slots) {
  const int tiles = (slots + kScTile - 1) / kScTile;
  int s = sm_count() / (2 * (lists > 0 ? lists : 1));
  s = s < tiles / 2 ? s : tiles / 2;
  return s < 1 ? 1 : (s > 8 ? 8 : s);
}
// Of these the number that costs least: a tile takes about a microsecond, a split list the combine kernel and the partial results
// of every part, about 4.5 and lists * parts / 12 of them.  us unsplit / in 2, 3, 4 and 8 parts (ctx 128K at ratio 128 is 24 tiles,
// 64K 14, 8K 4, selected keys 14):
//   ratio 128   1 list of 8K: 14.7 / 16.1 17.3   16 of 8K: 14.8 / 19.5 20.9   16 of 64K: 26.2 / 25.6 24.9 24.3
//               1 of 128K: 36.3 / 27.6 23.6 21.2 18.8   16 of 128K: 37.1 / 31.3 28.7 26.7 26.8
//   selected    1: 27.1 / 24.3 21.7 20.6 19.1   8: 29.4 / 27.1 25.0 24.1 26.2   32 pairs: 35.6 / 38.2
int scfa_splits(int lists, int most_slots, int slots) {
  const int most = scfa_most_splits(lists, most_slots), tiles = (slots + kScTile - 1) / kScTile;
  int best = 1, best_cost = 12 * tiles;
  for (int s = 2; s <= most; ++s) {
    const int cost = 12 * tiles / s + 54 + lists * s;   // (not rounded to whole tiles: a list may be a tile longer than expected)
    if (cost < best_cost) {
      best_cost = cost;
      best = s;
    }
  }
  return best;
}

int launch_scfa_tc(const SfaParams& p, cudaStream_t stream) {
  if (p.nq < 1 || p.nq > 128) {
    set_error("scfa: n_q=%d must be in [1, 128] (the heads of a token are the rows of one M = 128 tile)", p.nq);
    return DSV32_ERR_UNSUPPORTED;
  }
  if (p.rows > 0x1ffffffeLL || p.rows2 > 0x1ffffffeLL) {
    set_error("scfa: at most 2^29-2 rows per cache can be addressed (got %lld / %lld)", static_cast<long long>(p.rows),
              static_cast<long long>(p.rows2));
    return DSV32_ERR_UNSUPPORTED;
  }
  const int t = p.t_total;
  CUtensorMap q, kv, kv2, run, run2;
  int rc = make_tensor_map_2d_u8(&q, p.q_nope, static_cast<uint64_t>(t) * p.nq, kKvLora * 2, 128, 128);
  if (rc == DSV32_OK) rc = make_tensor_map_2d_u8(&kv, p.k_nope, p.rows > 0 ? p.rows : 1, kKvLora * 2, 1, 128);
  if (rc == DSV32_OK) {
    if (p.k_nope2 != nullptr) {
      rc = make_tensor_map_2d_u8(&kv2, p.k_nope2, p.rows2 > 0 ? p.rows2 : 1, kKvLora * 2, 1, 128);
      if (rc == DSV32_OK) rc = make_tensor_map_2d_u8(&run2, p.k_nope2, p.rows2 > 0 ? p.rows2 : 1, kKvLora * 2, 4 * kScWarpQuads, 128);
    } else {
      kv2 = kv;
      run2 = kv;
    }
  }
  if (rc == DSV32_OK) rc = make_tensor_map_2d_u8(&run, p.k_nope, p.rows > 0 ? p.rows : 1, kKvLora * 2, 4 * kScWarpQuads, 128);
  if (rc != DSV32_OK) return rc;
  if (p.pair == 2) launch_ex(scfa_pair_ids_kernel, dim3(t), 256, 0, stream, true, 1, p);
  else launch_ex(scfa_row_ids_kernel, dim3((p.topk + 255) / 256, t), 256, 0, stream, true, 1, p);
  count_launch();
  rc = check_launch("scfa row list kernel");
  if (rc != DSV32_OK) return rc;
  cudaFuncSetAttribute(scfa_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kScSmemBytes));
  // Persistent CTAs step over (token, half) with a stride of an odd number of tokens where there are pairs: with an even one, CTAs
  // would see first tokens of pairs only, or none.
  const int items = 2 * t * p.splits, tokens = sm_count() / 2, most = 2 * (p.pair && t != p.b ? (tokens - 1) | 1 : tokens);
  launch_ex(scfa_tc_kernel, dim3(items < most ? items : most), kScThreads, kScSmemBytes, stream, true, 1, q, kv, kv2, run, run2, p, items);
  count_launch();
  rc = check_launch("scfa_tc_kernel");
  if (rc == DSV32_OK && p.splits > 1) rc = launch_sfa_combine(p, stream);
  return rc;
}

}  // namespace dsv32
