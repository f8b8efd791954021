// DeepSeek-V4 KV compressor.
// Follows models/deepseek_v4/compressor_impl.py:421-923 (golden golden_compress,
// models/deepseek_v4/test_compressor.py:76-187).  For request b and its token i at position pos = start_pos[b] + i:
//   kv    = x . wkv^T,  score = x . wgate^T + ape[pos % ratio]          (both products in one projection launch, fp32)
//   kv_state[page(pos), pos % 128] = kv;  score_state[...] = score        (paged fp32 state, 128 positions per page)
//   if (pos + 1) % ratio == 0, the ratio positions that end at pos are compressed into one row:
//     ratio 128: softmax over the 128 score rows of the page, per column; kv = sum_r kv_r * softmax_r
//     ratio 4 (overlapping windows, state rows are [first half | second half] of 2 d columns): the rows are the
//       FIRST halves of the previous window's 4 positions and the SECOND halves of this window's 4 positions; a
//       request whose start position is below the ratio has no previous window (weight 0)
//     then bf16 -> RMSNorm * weight -> bf16 -> interleaved rotary embedding on the last 64 dims [-> x hadamard] -> out[b]
//
// A request belongs to a cluster of CTAs that own 64 output columns each (with ratio 4: state columns c and d + c), so the
// state rows a closing window reads were written by the same CTA; only the RMSNorm sum -- and, for the hadamard product, the
// row -- crosses, through distributed shared memory.  A window that closes with ratio 128 reads 512 KB of state: one CTA took
// 53 us for it, eight take 10.  Tokens of a request are handled in order because a later token's window contains the rows of
// the earlier ones; between two windows that close nothing is read, and a token's partial sums are fetched under the one before
// it (1024 tokens of one request, d = 128, hadamard: 2253 us with a fetch, a barrier and look-ups per token and a hadamard product
// per window, 1326 now, 1452 as separate launches; d = 512: 1622 and 1272).  The kernel adds the projection's partial sums itself
// and is launched dependent on it.  (The operator for one request of two tokens was two GEMM calls, two reduce kernels, a fill
// and, rotated, a third GEMM: 115 us of host work.)
#include <type_traits>

#include "finish.cuh"
#include "kernels.cuh"
#include "tc_common.cuh"

namespace dsv32 {

namespace {
constexpr int kCompThreads = 256, kCompPage = 128, kCompRope = 64;
constexpr int kCompCols = 64;     // output columns of a CTA
constexpr int kCompMaxD = 512;
}  // namespace

// V: columns per thread in the walk over 128 rows (the state rows' alignment allows 16-byte loads if d is a multiple of 4)
template <int V>
__global__ void __launch_bounds__(kCompThreads, 2) compressor_update_kernel(CompressorParams p, int csize) {
  constexpr int kGroups = kCompThreads / (kCompCols / V);   // row groups
  constexpr int kRows = kCompPage / kGroups;                // rows of a thread
  __shared__ float merge_s[kGroups][kCompCols][3];          // (maximum, sum, weighted sum) of a row group, per column
  __shared__ float red_s[2];
  __shared__ float sum_x[2][8];                             // every CTA's sum of squares; two, as a peer may be a window ahead
  __shared__ float row_x[kCompMaxD];                        // the whole row, for the hadamard product
  const int rank = blockIdx.x % csize, b = blockIdx.x / csize, tid = threadIdx.x;
  const int d = p.d, cd = p.coff * p.d, ratio = p.ratio, c0 = rank * kCompCols;
  const int nc = min(kCompCols, d - c0), cc = tid & (kCompCols - 1), grp = tid >> 6;
  pdl_trigger();
  bool closed = false;
  if (b < p.b) {
    float row_v = 0.f;   // this thread's column of the request's last compressed row
    const int start = p.start_pos[b];
    int nclose = 0;
    pdl_wait();
    if (csize > 1) cluster_arrive_wait();   // the peers' shared memory exists
    // this thread's state column: groups of 64 threads take (first | second half) x (kv | score)
    const bool score = p.coff == 2 ? (grp >> 1) != 0 : grp != 0;
    const int col = (p.coff == 2 ? (grp & 1) * d : 0) + c0 + cc;
    const bool writes = cc < nc && grp < 2 * p.coff;
    const float* sums = (score ? p.score_total : p.kv_total) + static_cast<size_t>(b) * p.s1 * p.ld + col;
    const size_t split_step = static_cast<size_t>(p.b) * p.s1 * p.ld;
    float part[16];   // a token's partial sums (a projection is cut into at most 16 splits), fetched a token ahead
    auto fetch = [&](int i) {
#pragma unroll
      for (int k = 0; k < 16; ++k)
        part[k] = writes && i < p.s1 && k < p.splits ? sums[static_cast<size_t>(i) * p.ld + k * split_step] : 0.f;
    };
    fetch(0);
    // The tokens up to the one that closes a window are taken together: they lie in one page, and nothing is read before the last
    // of them.
    for (int i = 0, n; i < p.s1; i += n) {
      const int pos0 = start + i;
      const int lb = pos0 / kCompPage;
      if (start < 0 || lb >= p.kv_cols || lb >= p.score_cols) {
        if (tid == 0 && rank == 0) report_status(p.status, DSV32_STATUS_BAD_INDEX, b, pos0);
        break;
      }
      const long long kb = p.kv_table[static_cast<size_t>(b) * p.kv_cols + lb];
      const long long sb = p.score_table[static_cast<size_t>(b) * p.score_cols + lb];
      if (kb < 0 || kb >= p.kv_blocks || sb < 0 || sb >= p.score_blocks) {
        if (tid == 0 && rank == 0) report_status(p.status, DSV32_STATUS_BAD_PAGE, b, pos0);
        break;
      }
      n = min(p.s1 - i, ratio - pos0 % ratio);
      if (writes) {
        float* state = (score ? p.score_state + sb * kCompPage * cd : p.kv_state + kb * kCompPage * cd) + col;
        for (int q = 0; q < n; ++q) {
          float v = 0.f;
#pragma unroll
          for (int k = 0; k < 16; ++k) v += part[k];   // in split order
          fetch(i + q + 1);
          const int at = pos0 + q;
          state[(at % kCompPage) * cd] = score ? v + p.ape[static_cast<size_t>(at % ratio) * cd + col] : v;
        }
      }
      __syncthreads();  // the rows just written are read below by other threads of this CTA
      const int pos = pos0 + n - 1;
      if ((pos + 1) % ratio != 0) continue;

      // ---- per column: softmax over the rows, weighted sum --------------------------------------------------------
      float v = 0.f;
      if (p.coff == 2) {
        const int cur_start = (pos - 3) % kCompPage;
        const float* kv1 = p.kv_state + (kb * kCompPage + cur_start) * cd + d + c0;
        const float* sc1 = p.score_state + (sb * kCompPage + cur_start) * cd + d + c0;
        const float *kv0 = nullptr, *sc0 = nullptr;
        if (start >= 4) {
          const int p0 = pos - 7;                     // >= 0 here
          const int lbp = p0 / kCompPage;
          const long long pkb = p.kv_table[static_cast<size_t>(b) * p.kv_cols + lbp];
          const long long psb = p.score_table[static_cast<size_t>(b) * p.score_cols + lbp];
          if (pkb < 0 || pkb >= p.kv_blocks || psb < 0 || psb >= p.score_blocks) {
            if (tid == 0 && rank == 0) report_status(p.status, DSV32_STATUS_BAD_PAGE, b, p0);
            break;
          }
          kv0 = p.kv_state + (pkb * kCompPage + p0 % kCompPage) * cd + c0;
          sc0 = p.score_state + (psb * kCompPage + p0 % kCompPage) * cd + c0;
        }
        if (tid < nc) {
          float s[8], k[8], m = -INFINITY, sum = 0.f;
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            s[r] = sc0 != nullptr ? sc0[static_cast<size_t>(r) * cd + cc] : -INFINITY;
            k[r] = kv0 != nullptr ? kv0[static_cast<size_t>(r) * cd + cc] : 0.f;
            s[4 + r] = sc1[static_cast<size_t>(r) * cd + cc];
            k[4 + r] = kv1[static_cast<size_t>(r) * cd + cc];
          }
#pragma unroll
          for (int r = 0; r < 8; ++r) m = fmaxf(m, s[r]);
#pragma unroll
          for (int r = 0; r < 8; ++r) {
            s[r] = (r >= 4 || sc0 != nullptr) ? expf(s[r] - m) : 0.f;
            sum += s[r];
          }
#pragma unroll
          for (int r = 0; r < 8; ++r) v += k[r] * __fdiv_rn(s[r], sum);
        }
      } else {
        // 128 rows: threads = (V columns) x (kRows rows), all loads in flight together; the row groups are then merged
        const int cg = tid % (kCompCols / V), rg = tid / (kCompCols / V);
        if (cg * V < nc) {
          using Vec = typename std::conditional<V == 4, float4, float2>::type;
          const size_t at = static_cast<size_t>(rg * kRows) * cd + c0 + cg * V;
          const float* sp = p.score_state + sb * kCompPage * cd + at;
          const float* kp = p.kv_state + kb * kCompPage * cd + at;
          Vec s4[kRows], k4[kRows];
#pragma unroll
          for (int r = 0; r < kRows; ++r) {
            s4[r] = *reinterpret_cast<const Vec*>(sp + static_cast<size_t>(r) * cd);
            k4[r] = *reinterpret_cast<const Vec*>(kp + static_cast<size_t>(r) * cd);
          }
#pragma unroll
          for (int j = 0; j < V; ++j) {
            float m = -INFINITY, sm = 0.f, ac = 0.f;
#pragma unroll
            for (int r = 0; r < kRows; ++r) m = fmaxf(m, reinterpret_cast<const float*>(&s4[r])[j]);
#pragma unroll
            for (int r = 0; r < kRows; ++r) {
              const float e = expf(reinterpret_cast<const float*>(&s4[r])[j] - m);
              sm += e;
              ac += reinterpret_cast<const float*>(&k4[r])[j] * e;
            }
            float* q = merge_s[rg][cg * V + j];
            q[0] = m;
            q[1] = sm;
            q[2] = ac;
          }
        }
        __syncthreads();
        if (tid < nc) {
          float mm = -INFINITY, st = 0.f, at = 0.f;
#pragma unroll
          for (int g = 0; g < kGroups; ++g) mm = fmaxf(mm, merge_s[g][cc][0]);
#pragma unroll
          for (int g = 0; g < kGroups; ++g) {
            const float f = expf(merge_s[g][cc][0] - mm);
            st += merge_s[g][cc][1] * f;
            at += merge_s[g][cc][2] * f;
          }
          v = __fdiv_rn(at, st);
        }
      }
      v = bf16r(v);   // threads 0 .. nc - 1 hold the row's columns c0 .. from here on
      // ---- RMSNorm * weight -> bf16 ---------------------------------------------------------------------------
      const int par = nclose & 1;
      if (tid < kCompCols) {
        const float sq = warp_sum(tid < nc ? v * v : 0.f);
        if ((tid & 31) == 0) red_s[tid >> 5] = sq;
      }
      __syncthreads();
      if (csize > 1) {
        if (tid < csize) st_peer_f32(peer_addr(&sum_x[par][rank], tid), red_s[0] + red_s[1]);
        cluster_arrive_wait();
      } else {
        if (tid == 0) sum_x[par][0] = red_s[0] + red_s[1];
        __syncthreads();
      }
      float total = 0.f;
      for (int r = 0; r < csize; ++r) total += sum_x[par][r];
      const float rinv = __fdiv_rn(1.0f, sqrtf(total / static_cast<float>(d) + p.eps));
      // ---- rotary embedding on the last 64 dims (pairs 2i, 2i+1) ---------------------------------------------------
      if (tid < kCompCols) {
        v = tid < nc ? bf16r(p.weight[c0 + tid] * (v * rinv)) : 0.f;
        const float other = __shfl_xor_sync(0xffffffffu, v, 1);
        const int j = c0 + tid - (d - kCompRope);
        if (j >= 0 && tid < nc) {
          const float cs = __bfloat162float(p.cos[static_cast<size_t>(b) * kCompRope + j]);
          const float sn = __bfloat162float(p.sin[static_cast<size_t>(b) * kCompRope + j]);
          v = __fadd_rn(__fmul_rn(v, cs), __fmul_rn((j & 1) ? other : -other, sn));
        }
      }
      if (p.hadamard != nullptr) row_v = bf16r(v);
      else if (tid < nc) p.out[static_cast<size_t>(b) * d + c0 + tid] = __float2bfloat16_rn(v);
      closed = true;
      ++nclose;
      __syncthreads();  // merge_s / red_s are reused by the next window
    }
    if (p.hadamard != nullptr && closed) {   // (alike in all CTAs of the cluster)
      // Row x hadamard, of the row that stays: a request's later windows overwrite the row of its earlier ones.  Every CTA gets the
      // whole row and makes its 64 columns, the reduction over four groups of threads.
      if (tid < nc)
        for (int r = 0; r < csize; ++r) st_peer_f32(peer_addr(&row_x[c0 + tid], r), row_v);
      if (csize > 1) cluster_arrive_wait();
      else __syncthreads();
      float acc = 0.f;
      if (cc < nc) {
#pragma unroll 16
        for (int k = grp; k < d; k += 4)
          acc = fmaf(row_x[k], __bfloat162float(p.hadamard[static_cast<size_t>(k) * d + c0 + cc]), acc);
      }
      merge_s[grp][cc][0] = acc;
      __syncthreads();
      if (tid < nc)
        p.out[static_cast<size_t>(b) * d + c0 + tid] =
            __float2bfloat16_rn((merge_s[0][tid][0] + merge_s[1][tid][0]) + (merge_s[2][tid][0] + merge_s[3][tid][0]));
    }
  } else {
    pdl_wait();
  }
  // rows without a closed window read as zero
  if (p.zero_rows && !closed && tid < nc) p.out[static_cast<size_t>(b) * d + c0 + tid] = __float2bfloat16_rn(0.f);
}

// dependent: on the projection, which has waited for everything before it (the kernel reads start_pos without waiting)
int launch_compressor(const CompressorParams& p, bool dependent, cudaStream_t stream) {
  if (p.b <= 0 || p.s1 <= 0) return DSV32_OK;
  const int csize = (p.d + kCompCols - 1) / kCompCols, rows = p.zero_rows > p.b ? p.zero_rows : p.b;
  auto kernel = p.d % 4 == 0 ? compressor_update_kernel<4> : compressor_update_kernel<2>;
  launch_ex(kernel, dim3(static_cast<unsigned>(csize) * rows), kCompThreads, 0, stream, dependent, csize, p, csize);
  count_launch();
  return check_launch("compressor_update_kernel");
}

size_t compressor_workspace_bytes(int t, int h, int cd) { return t <= 0 || h <= 0 ? 0 : proj_partial_bytes(t, h, 2 * proj_ld(cd)); }

// The whole operator: x . [wkv^T | wgate^T], then the update on its partial sums.
int launch_compressor_op(CompressorParams p, const __nv_bfloat16* x, const __nv_bfloat16* wkv, const __nv_bfloat16* wgate, int h,
                         float* partial, cudaStream_t stream) {
  const int t = p.b * p.s1, cd = p.coff * p.d;
  if (t <= 0) return DSV32_OK;
  const ProjSegment segs[2] = {{wkv, cd}, {wgate, cd}};
  const int rc = launch_proj_bf16(x, t, h, segs, 2, true, partial, p.status, stream);
  if (rc != DSV32_OK) return rc;
  p.ld = 2 * proj_ld(cd);
  p.splits = proj_plan(t, p.ld, (h + 63) / 64).splits;
  p.kv_total = partial;
  p.score_total = partial + proj_ld(cd);
  return launch_compressor(p, true, stream);
}

}  // namespace dsv32
