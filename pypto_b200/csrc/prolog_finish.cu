// What follows the first projections of the V3.2 prologs, one launch: a token's projected row is finished in three sections,
// each adding its fp32 partial sums in split order first.
//   0  q_a  (1536): bf16 -> RMSNorm(gamma_cq) -> bf16 -> per-token int8 -> q_norm, q_norm_scale
//   1  kv_a (512 + 64): bf16 -> RMSNorm(gamma_ckv) of the first 512 -> four 128-dim int8 groups + fp32 scales, scattered into
//      the latent cache; last 64 -> de-interleave + rotary embedding -> rope cache
//   2  k (128) and head weights (64) of the indexer: LayerNorm -> bf16 -> rotary embedding of the first 64 dims -> bf16 ->
//      x hadamard_k -> bf16 -> int8 + fp16 scale, scattered into the index-key cache; weights -> bf16, scaled -> fp16
// Reference: models/deepseek_v32_exp/mla_indexer_prolog_quant_impl.py:112-211, mla_prolog_quant_impl.py:96-361,
// lightning_indexer_prolog_quant_impl.py:423-543 (goldens deepseekv32_mla_indexer_prolog_quant.py:395-539,
// deepseekv32_lightning_indexer_prolog_quant.py:220-288).
// Launched dependent on the projection kernel; what does not come from it is fetched before it has finished.
#include "finish.cuh"
#include "kernels.cuh"
#include "tc_common.cuh"

namespace dsv32 {

namespace {
constexpr int kFinThreads = 512;
}  // namespace

// Few tokens, where latency is what counts: a CTA of 512 threads per token and section.
__global__ void __launch_bounds__(kFinThreads) prolog_finish_kernel(PrologFinishParams p) {
  __shared__ float red[16];
  __shared__ float vec[128], part[4][128];
  const int tok = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int section = p.sections[blockIdx.y];
  const ProjSums src{p.partial, p.t, p.ld, p.splits};
  pdl_trigger();
  const size_t rope_at = static_cast<size_t>(tok) * 64 + (tid & 63);
  float gm[3] = {0.f, 0.f, 0.f}, cs = 0.f, sn = 0.f, had[32];
  long long row = 0;
  if (section == 0) {
#pragma unroll
    for (int i = 0; i < 3; ++i) gm[i] = __bfloat162float(p.gamma_cq[tid + i * kFinThreads]);
  } else if (section == 1) {
    gm[0] = __bfloat162float(p.gamma_ckv[tid]);
    row = p.kv_index[tok];
    cs = __bfloat162float(p.cos[rope_at]);
    sn = __bfloat162float(p.sin[rope_at]);
  } else {
    row = p.idx_index[tok];
    if (tid < 128) {
      gm[0] = __bfloat162float(p.ln_gamma[tid]);
      gm[1] = __bfloat162float(p.ln_beta[tid]);
    }
    cs = __bfloat162float(p.cos_idx[rope_at]);
    sn = __bfloat162float(p.sin_idx[rope_at]);
#pragma unroll
    for (int k = 0; k < 32; ++k) had[k] = __bfloat162float(p.had_k[((tid >> 7) * 32 + k) * 128 + (tid & 127)]);
  }
  pdl_wait();
  if (section == 0) {
    float x[3], ss = 0.f;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      x[i] = bf16r(proj_sum(src, tok, p.col_q + tid + i * kFinThreads));
      ss += __fmul_rn(__fmul_rn(x[i], x[i]), 1.0f / 1536.0f);
    }
    const float rms = sqrtf(block_reduce<16, false>(ss, red) + p.eps_cq);
    float amax = 0.f;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      x[i] = bf16r(__fmul_rn(__fdiv_rn(x[i], rms), gm[i]));
      amax = fmaxf(amax, fabsf(x[i]));
    }
    amax = block_reduce<16, true>(amax, red);
    const float sq = __fdiv_rn(127.0f, amax);
#pragma unroll
    for (int i = 0; i < 3; ++i)
      p.q_norm[static_cast<size_t>(tok) * 1536 + tid + i * kFinThreads] =
          static_cast<int8_t>(static_cast<int>(rintf(__fmul_rn(x[i], sq))));
    if (tid == 0) p.q_norm_scale[tok] = __fdiv_rn(1.0f, sq);
  } else if (section == 1) {
    const float x = bf16r(proj_sum(src, tok, p.col_kv + tid));
    if (tid < 64) vec[tid] = bf16r(proj_sum(src, tok, p.col_kv + 512 + tid));
    const float rms = sqrtf(block_reduce<16, false>(__fmul_rn(__fmul_rn(x, x), 1.0f / 512.0f), red) + p.eps_ckv);
    const float y = bf16r(__fmul_rn(__fdiv_rn(x, rms), gm[0]));
    float a = fabsf(y);   // maximum per 128-dim group (four warps)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) a = fmaxf(a, __shfl_xor_sync(0xffffffffu, a, o));
    if (lane == 0) red[warp] = a;
    __syncthreads();
    const int g = tid >> 7;
    const float sq = __fdiv_rn(127.0f, fmaxf(fmaxf(red[4 * g], red[4 * g + 1]), fmaxf(red[4 * g + 2], red[4 * g + 3])));
    if (row < 0 || row >= p.kv_rows) {
      if (tid == 0) report_status(p.status, DSV32_STATUS_BAD_INDEX, tok, 1);
      return;
    }
    p.kv_cache[row * 512 + tid] = static_cast<int8_t>(static_cast<int>(rintf(__fmul_rn(y, sq))));
    if ((tid & 127) == 0) p.kv_scale_cache[row * 4 + g] = __fdiv_rn(1.0f, sq);
    if (tid < 64) {
      // x' = [x0, x2, .., x62, x1, x3, .., x63];  out[j] = x'[j] cos[j] + rot(x')[j] sin[j]
      const float xj = (tid < 32) ? vec[2 * tid] : vec[2 * (tid - 32) + 1];
      const float xr = (tid < 32) ? -vec[2 * tid + 1] : vec[2 * (tid - 32)];   // rotate_half: (-x'[j + 32], x'[j - 32])
      p.kr_cache[row * 64 + tid] = __float2bfloat16_rn(__fadd_rn(__fmul_rn(xj, cs), __fmul_rn(xr, sn)));
    }
  } else {
    // threads 0..127 hold k, 128..191 the head weights
    const float v = tid < 192 ? proj_sum(src, tok, p.col_kw + tid) : 0.f;
    if (tid >= 128 && tid < 192)
      p.weights[static_cast<size_t>(tok) * 64 + (tid - 128)] =
          __float2half_rn(__fmul_rn(__fmul_rn(bf16r(v), 0.125f), 0.08838834764831845f));
    const float mean = block_reduce<4, false>(v, red) * (1.0f / 128.0f);
    const float dlt = v - mean;
    const float var = block_reduce<4, false>(dlt * dlt, red) * (1.0f / 128.0f);
    if (tid < 128) {
      const float y = __fdiv_rn(dlt, sqrtf(var + p.eps_ln));
      part[0][tid] = bf16r(__fadd_rn(__fmul_rn(y, gm[0]), gm[1]));
    }
    __syncthreads();
    if (tid < 128) {
      float y = part[0][tid];
      if (tid < 64) {   // rotate-half pairs (d, d + 32)
        const float r = (tid < 32) ? -part[0][tid + 32] : part[0][tid - 32];
        y = bf16r(__fadd_rn(__fmul_rn(y, cs), __fmul_rn(r, sn)));
      }
      vec[tid] = y;
    }
    __syncthreads();
    {   // x hadamard_k: the 128 rows over the four groups of 128 threads
      const int k0 = (tid >> 7) * 32;
      float acc = 0.f;
#pragma unroll
      for (int k = 0; k < 32; ++k) acc = fmaf(vec[k0 + k], had[k], acc);
      part[tid >> 7][tid & 127] = acc;
    }
    __syncthreads();
    float hv = 0.f;
    if (tid < 128) hv = bf16r((part[0][tid] + part[1][tid]) + (part[2][tid] + part[3][tid]));
    const float amax = block_reduce<4, true>(fabsf(hv), red);
    if (tid < 128) {
      if (row < 0 || row >= p.idx_rows) {
        if (tid == 0) report_status(p.status_idx, DSV32_STATUS_BAD_INDEX, tok, 0);
      } else {
        const float sq = __fdiv_rn(127.0f, amax);
        p.idx_cache[row * 128 + tid] = static_cast<int8_t>(static_cast<int>(rintf(__fmul_rn(hv, sq))));
        if (tid == 0) p.idx_scale_cache[row] = __float2half_rn(__fdiv_rn(1.0f, sq));
      }
    }
  }
}

// Many tokens: a warp takes a token's section, eight tokens a CTA, with 16-byte loads and shuffles only.  With a CTA per
// token the kernel spent its time in barriers (4096 tokens, 60 MB: 130 us).
__global__ void __launch_bounds__(256) prolog_finish_rows_kernel(PrologFinishParams p) {
  __shared__ float vec[8][128];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int tok = blockIdx.x * 8 + warp;
  const int section = p.sections[blockIdx.y];
  const ProjSums src{p.partial, p.t, p.ld, p.splits};
  pdl_trigger();
  pdl_wait();
  if (tok >= p.t) return;
  if (section == 0) {
    float4 x[12];
    float ss = 0.f;
    proj_sum4(src, tok, p.col_q + 4 * lane, x);
#pragma unroll
    for (int i = 0; i < 12; ++i) {
      x[i] = make_float4(bf16r(x[i].x), bf16r(x[i].y), bf16r(x[i].z), bf16r(x[i].w));
      ss += x[i].x * x[i].x * (1.0f / 1536.0f) + x[i].y * x[i].y * (1.0f / 1536.0f) + x[i].z * x[i].z * (1.0f / 1536.0f) +
            x[i].w * x[i].w * (1.0f / 1536.0f);
    }
    const float rms = sqrtf(warp_sum(ss) + p.eps_cq);
    float amax = 0.f;
#pragma unroll
    for (int i = 0; i < 12; ++i) {
      const float4 g = bf16x4(p.gamma_cq + 128 * i + 4 * lane);
      x[i] = make_float4(bf16r(__fmul_rn(__fdiv_rn(x[i].x, rms), g.x)), bf16r(__fmul_rn(__fdiv_rn(x[i].y, rms), g.y)),
                         bf16r(__fmul_rn(__fdiv_rn(x[i].z, rms), g.z)), bf16r(__fmul_rn(__fdiv_rn(x[i].w, rms), g.w)));
      amax = fmaxf(amax, fmaxf(fmaxf(fabsf(x[i].x), fabsf(x[i].y)), fmaxf(fabsf(x[i].z), fabsf(x[i].w))));
    }
    const float sq = __fdiv_rn(127.0f, warp_max(amax));
#pragma unroll
    for (int i = 0; i < 12; ++i)
      store_bytes4(p.q_norm + static_cast<size_t>(tok) * 1536 + 128 * i + 4 * lane, quant4(x[i].x, x[i].y, x[i].z, x[i].w, sq));
    if (lane == 0) p.q_norm_scale[tok] = __fdiv_rn(1.0f, sq);
  } else if (section == 1) {
    float4 x[4];
    float ss = 0.f;
    const long long row = p.kv_index[tok];
    // rope part: lane holds the pair (2 lane, 2 lane + 1), which makes outputs lane and 32 + lane
    const float e = bf16r(proj_sum(src, tok, p.col_kv + 512 + 2 * lane)), o = bf16r(proj_sum(src, tok, p.col_kv + 513 + 2 * lane));
    proj_sum4(src, tok, p.col_kv + 4 * lane, x);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      x[i] = make_float4(bf16r(x[i].x), bf16r(x[i].y), bf16r(x[i].z), bf16r(x[i].w));
      ss += x[i].x * x[i].x * (1.0f / 512.0f) + x[i].y * x[i].y * (1.0f / 512.0f) + x[i].z * x[i].z * (1.0f / 512.0f) +
            x[i].w * x[i].w * (1.0f / 512.0f);
    }
    const float rms = sqrtf(warp_sum(ss) + p.eps_ckv);
    if (row < 0 || row >= p.kv_rows) {
      if (lane == 0) report_status(p.status, DSV32_STATUS_BAD_INDEX, tok, 1);
      return;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {   // group i = columns 128 i .. 128 i + 127
      const float4 g = bf16x4(p.gamma_ckv + 128 * i + 4 * lane);
      const float y0 = bf16r(__fmul_rn(__fdiv_rn(x[i].x, rms), g.x)), y1 = bf16r(__fmul_rn(__fdiv_rn(x[i].y, rms), g.y));
      const float y2 = bf16r(__fmul_rn(__fdiv_rn(x[i].z, rms), g.z)), y3 = bf16r(__fmul_rn(__fdiv_rn(x[i].w, rms), g.w));
      const float sq = __fdiv_rn(127.0f, warp_max(fmaxf(fmaxf(fabsf(y0), fabsf(y1)), fmaxf(fabsf(y2), fabsf(y3)))));
      store_bytes4(p.kv_cache + row * 512 + 128 * i + 4 * lane, quant4(y0, y1, y2, y3, sq));
      if (lane == 0) p.kv_scale_cache[row * 4 + i] = __fdiv_rn(1.0f, sq);
    }
    const __nv_bfloat16 *cr = p.cos + static_cast<size_t>(tok) * 64, *sr = p.sin + static_cast<size_t>(tok) * 64;
    p.kr_cache[row * 64 + lane] = __float2bfloat16_rn(
        __fadd_rn(__fmul_rn(e, __bfloat162float(cr[lane])), __fmul_rn(-o, __bfloat162float(sr[lane]))));
    p.kr_cache[row * 64 + 32 + lane] = __float2bfloat16_rn(
        __fadd_rn(__fmul_rn(o, __bfloat162float(cr[32 + lane])), __fmul_rn(e, __bfloat162float(sr[32 + lane]))));
  } else {
    const long long row = p.idx_index[tok];
    const float w0 = proj_sum(src, tok, p.col_kw + 128 + lane), w1 = proj_sum(src, tok, p.col_kw + 160 + lane);
    p.weights[static_cast<size_t>(tok) * 64 + lane] = __float2half_rn(__fmul_rn(__fmul_rn(bf16r(w0), 0.125f), 0.08838834764831845f));
    p.weights[static_cast<size_t>(tok) * 64 + 32 + lane] = __float2half_rn(__fmul_rn(__fmul_rn(bf16r(w1), 0.125f), 0.08838834764831845f));
    float4 v[1];
    proj_sum4(src, tok, p.col_kw + 4 * lane, v);
    const float mean = warp_sum((v[0].x + v[0].y) + (v[0].z + v[0].w)) * (1.0f / 128.0f);
    float y[4] = {v[0].x - mean, v[0].y - mean, v[0].z - mean, v[0].w - mean};
    const float var = warp_sum((y[0] * y[0] + y[1] * y[1]) + (y[2] * y[2] + y[3] * y[3])) * (1.0f / 128.0f);
    const float dev = sqrtf(var + p.eps_ln);
    const float4 g = bf16x4(p.ln_gamma + 4 * lane), b = bf16x4(p.ln_beta + 4 * lane);
    const float gs[4] = {g.x, g.y, g.z, g.w}, bs[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      y[j] = bf16r(__fadd_rn(__fmul_rn(__fdiv_rn(y[j], dev), gs[j]), bs[j]));
      // rotate-half pairs (d, d + 32): the partner sits eight lanes away
      const float other = __shfl_xor_sync(0xffffffffu, y[j], 8);
      if (lane < 16) {
        const size_t at = static_cast<size_t>(tok) * 64 + 4 * lane + j;
        y[j] = bf16r(__fadd_rn(__fmul_rn(y[j], __bfloat162float(p.cos_idx[at])),
                               __fmul_rn(lane < 8 ? -other : other, __bfloat162float(p.sin_idx[at]))));
      }
    }
    *reinterpret_cast<float4*>(&vec[warp][4 * lane]) = make_float4(y[0], y[1], y[2], y[3]);
    __syncwarp();
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 8
    for (int k = 0; k < 128; ++k) {
      const float f = vec[warp][k];
      const uint2 h = __ldg(reinterpret_cast<const uint2*>(p.had_k + k * 128 + 4 * lane));
      acc[0] = fmaf(f, __uint_as_float(h.x << 16), acc[0]);
      acc[1] = fmaf(f, __uint_as_float(h.x & 0xffff0000u), acc[1]);
      acc[2] = fmaf(f, __uint_as_float(h.y << 16), acc[2]);
      acc[3] = fmaf(f, __uint_as_float(h.y & 0xffff0000u), acc[3]);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[j] = bf16r(acc[j]);
    const float amax = warp_max(fmaxf(fmaxf(fabsf(acc[0]), fabsf(acc[1])), fmaxf(fabsf(acc[2]), fabsf(acc[3]))));
    if (row < 0 || row >= p.idx_rows) {
      if (lane == 0) report_status(p.status_idx, DSV32_STATUS_BAD_INDEX, tok, 0);
    } else {
      const float sq = __fdiv_rn(127.0f, amax);
      store_bytes4(p.idx_cache + row * 128 + 4 * lane, quant4(acc[0], acc[1], acc[2], acc[3], sq));
      if (lane == 0) p.idx_scale_cache[row] = __float2half_rn(__fdiv_rn(1.0f, sq));
    }
  }
}

static int launch_prolog_finish(const PrologFinishParams& p, int nsections, bool rows, cudaStream_t stream) {
  if (!rows) launch_ex(prolog_finish_kernel, dim3(p.t, nsections), kFinThreads, 0, stream, true, 1, p);
  else launch_ex(prolog_finish_rows_kernel, dim3((p.t + 7) / 8, nsections), 256, 0, stream, true, 1, p);
  count_launch();
  return check_launch("prolog_finish_kernel");
}

// Workspace of the projections of either or both halves.
size_t prolog_partial_bytes(int t, bool mla, bool indexer) {
  return t <= 0 ? 0 : proj_partial_bytes(t, 7168, (mla ? 2112 : 0) + (indexer ? 192 : 0));
}

// How the indexer prolog on its own runs: its heads take q_norm as an input, so they can run beside projection and finish.  A
// heads CTA needs an SM to itself (200 KB of shared memory, 53,760 registers), and a finish CTA that was launched early and waits
// for the projection keeps it from one: with the finish always before the heads the call went from 16.7 to 22.5 us where a CTA
// per token and 64 heads' CTAs no longer fit the SMs.  Two forms in which nothing waits for an SM:
//   finish, heads     while finish and heads CTAs fit
//   heads, finish     while the heads make at most two rounds: they take the CTAs of whole rounds, and the projection the SMs they
//                     leave, in no more splits than it needs to be done with them
// us at 64, 128, 192, 256, 384 and 512 tokens, everything read from memory, called on a stream | inside a CUDA graph
//                                        16.2 18.6 20.1 20.5 28.0 28.8 | 17.0 20.7 21.1 21.8 29.2 30.3
//   the finish always before the heads   16.2 23.5 26.6 29.4 30.8 37.0 | 17.0 24.1 27.4 30.8 31.5 37.6
//   the heads on a second stream         19.8 23.1 24.1 27.5 31.8 38.3 | 15.7 18.6 25.2 28.9 31.5 41.2
// As a stage of the decode chain at 128 tokens: 24.5, 28.1 and 24.0.  Beyond two rounds every kernel fills the chip by itself
// (1024 tokens: 45 us in the first order, 62 on two streams).
struct IndexerPlan {
  bool finish_rows, finish_last;
  int proj_ctas, head_ctas;   // 0: one per SM
};
static IndexerPlan plan_indexer(int t) {
  const int sms = sm_count(), m_tiles = (t + 127) / 128, items = 64 * m_tiles, rounds = (items + sms - 1) / sms;
  if (rounds > 2 || t + items <= sms) return IndexerPlan{t > 192, false, 0, 0};
  const ProjPlan proj = proj_plan(t, 192, 7168 / 64);
  const int head_ctas = (items + rounds - 1) / rounds;
  const int room = sms - head_ctas, most = proj.m_tiles * proj.n_tiles * (10 / rounds);
  return IndexerPlan{false, true, room < most ? room : most, head_ctas};
}

// The V3.2 prologs: x times all weight matrices that take it (one launch), their finish (one), the heads (one).
int launch_prolog_v32(const MlaParams* m, const PrologParams* ip, float* partial, cudaStream_t stream) {
  const int t = m != nullptr ? m->t : ip->t;
  if (t <= 0) return DSV32_OK;
  ProjSegment segs[4];
  int n = 0;
  if (m != nullptr) {
    segs[n++] = {m->w_dq, 1536};
    segs[n++] = {m->w_dkv_kr, 576};
  }
  if (ip != nullptr) {
    segs[n++] = {ip->wk, 128};
    segs[n++] = {ip->w_proj, 64};
  }
  // with the MLA half a CTA per token while that many run at once (three sections of 512 threads on every SM)
  const IndexerPlan plan = m == nullptr ? plan_indexer(t) : IndexerPlan{t > 192, false, 0, 0};
  int rc = launch_proj_bf16(m != nullptr ? m->x : ip->x, t, 7168, segs, n, false, partial, m != nullptr ? m->status : ip->status, stream,
                            plan.proj_ctas);
  if (rc != DSV32_OK) return rc;
  PrologFinishParams f{};
  f.partial = partial;
  f.t = t;
  f.ld = (m != nullptr ? 2112 : 0) + (ip != nullptr ? 192 : 0);
  f.splits = proj_plan(t, f.ld, 7168 / 64, plan.proj_ctas).splits;
  n = 0;
  if (m != nullptr) {
    f.sections[n++] = 0;
    f.sections[n++] = 1;
    f.col_q = 0; f.col_kv = 1536;
    f.gamma_cq = m->gamma_cq; f.gamma_ckv = m->gamma_ckv; f.eps_cq = m->eps_cq; f.eps_ckv = m->eps_ckv;
    f.q_norm = m->q_norm; f.q_norm_scale = m->q_norm_scale;
    f.cos = m->cos; f.sin = m->sin;
    f.kv_index = m->cache_index; f.kv_rows = m->cache_rows;
    f.kv_cache = m->kv_cache; f.kr_cache = m->kr_cache; f.kv_scale_cache = m->k_scale_cache;
    f.status = m->status;
  }
  if (ip != nullptr) {
    f.sections[n++] = 2;
    f.col_kw = f.ld - 192;
    f.ln_gamma = ip->ln_gamma; f.ln_beta = ip->ln_beta; f.eps_ln = ip->eps; f.had_k = ip->had_k;
    f.cos_idx = ip->cos; f.sin_idx = ip->sin;
    f.idx_index = ip->cache_index; f.idx_rows = ip->cache_rows;
    f.idx_cache = ip->k_cache; f.idx_scale_cache = ip->k_scale_cache; f.weights = ip->weights;
    f.status_idx = ip->status;
  }
  if (!plan.finish_last) rc = launch_prolog_finish(f, n, plan.finish_rows, stream);
  if (rc == DSV32_OK) rc = launch_prolog_heads(m, ip, m == nullptr, stream, plan.head_ctas);
  if (rc == DSV32_OK && plan.finish_last) rc = launch_prolog_finish(f, n, plan.finish_rows, stream);
  return rc;
}

}  // namespace dsv32
