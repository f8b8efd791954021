"""The tensor-core kernels at the sizes where their tilings change: one token more or less than a token tile, the last token
count of a dispatch rule and the first of the next, column and reduction remainders, more items than CTAs, split and unsplit
key lists.  Every case runs the operator against the same oracle and bounds as its tests in test_gpu_parity.py."""
import pytest
import torch

import helpers
import test_gpu_gemm as gemm
import test_gpu_parity as parity
import test_gpu_pg_prolog as pg

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
BF = torch.bfloat16


# 128 / 129 tokens: narrow and wide column tiles; one reduction chunk, a split of 112, segments of 14 with a remainder
@pytest.mark.parametrize("t,k,n", [(127, 64, 136), (128, 7168, 200), (129, 960, 264), (257, 1856, 72)])
@pytest.mark.parametrize("layout", [0, 1])
def test_projection_tiles(t, k, n, layout):
    gemm.test_gemm_bf16_matches_a_float64_product(t, k, n, layout, torch.float32)


# finish kernels up to / past 192 tokens; heads with one, two and three token tiles, full and of a single token
@pytest.mark.parametrize("t", [2, 129, 192, 193, 257])
def test_fused_prolog_tiles(t):
    parity.test_mla_indexer_prolog_seeded_vs_oracle(t)


# the indexer prolog on its own: the last and first token counts of the orders in which its kernels are launched and share the SMs.
# With this many values some bf16 roundings fall the other way (2e-4 of the weights, at any of these counts): a weight, or the
# maximum that a scale is, then differs by one step of bf16, 2^-7 of itself at most, and by the fp16 rounding after it.  A weight
# near zero keeps the absolute error of its 7168-long sum: the 2.5e-5 of test_gpu_parity.py.
@pytest.mark.parametrize("t", [84, 85, 128, 129, 193, 257, 385, 513])
def test_indexer_prolog_orders(t, monkeypatch):
    def check(got, ref, cache_index):
        for name, a, b in zip(("q_int8", "q_scale", "k", "k_scale", "weights"), got, ref):
            a, b = a.double().reshape(-1), b.double().reshape(-1)
            diff = (a - b).abs()
            if name in ("q_int8", "k"):
                assert diff.max() <= 1, name
                share, allowed = (diff > 0).double().mean().item(), 0.02
            else:
                assert bool((diff <= (2.0 ** -7 + 2.0 ** -10) * b.abs() + 2.5e-5).all()), name
                share, allowed = (diff > 2.0 ** -10 * b.abs()).double().mean().item(), 0.01
            print(f"[indexer prolog t={t}] {name}: {share:.1e} of the values differ")
            assert share <= allowed, (name, share)
        others = torch.ones(got[2].numel() // 128, dtype=torch.bool)
        others[cache_index] = False
        assert torch.equal(got[2].reshape(-1, 128)[others], ref[2].reshape(-1, 128)[others])

    monkeypatch.setattr(parity, "_assert_prolog_close", check)
    parity.test_prolog_config1_distributions_vs_oracle(t)


# an odd number of (head, token tile) items, a hidden size that is not a multiple of a reduction chunk
@pytest.mark.parametrize("t,heads,h", [(128, 3, 1000), (129, 3, 1000), (193, 2, 64), (257, 5, 1024)])
@pytest.mark.parametrize("quant", [True, False])
def test_v4_mla_tiles(t, heads, h, quant):
    (parity.test_mla_v4_seeded_vs_oracle if quant else parity.test_mla_v4_bf16_seeded_vs_oracle)(t, heads, h)


# CUDA cores up to 64 tokens, tensor cores beyond; one and several token tiles, more than eight tokens per finish CTA's share
@pytest.mark.parametrize("t", [64, 65, 128, 129, 600])
def test_hc_pre_tiles(t):
    parity.test_hc_pre_seeded_vs_oracle(t, 20, 1e-6)


# clusters of 1, 2, 3, 5 and 8 CTAs; a last CTA of few columns; rows of 8 bytes; windows that close twice, never, and with rows past b
@pytest.mark.parametrize("ratio,rotate,d,starts,s1", [
    (4, True, 64, [0, 3, 5], 2), (4, True, 136, [4, 127], 8), (128, False, 72, [127, 1], 2), (128, True, 320, [255], 1),
    (4, False, 512, [1], 9), (128, False, 70, [127, 126], 3)])
def test_compressor_clusters(ratio, rotate, d, starts, s1):
    parity.test_compressor_seeded_vs_oracle(ratio, rotate, d, starts, s1)


# many windows of one request in a call: a row that is written over, across pages, from and to the middle of a window
@pytest.mark.parametrize("ratio,rotate,d,starts,s1", [(4, True, 128, [0, 3, 126], 41), (4, False, 200, [2], 130), (128, True, 128, [0, 77], 300)])
def test_compressor_windows(ratio, rotate, d, starts, s1):
    parity.test_compressor_seeded_vs_oracle(ratio, rotate, d, starts, s1)


# lists split over idle SMs (few tokens) and not; more items than CTAs; idle lanes; lists shorter than a tile and than a split;
# no pairs, pairs beside single tokens, requests of different numbers of tokens
@pytest.mark.parametrize("ori_seq,s1_list,nq,kw", [
    ([4000], [1], 64, {}), ([300, 20], [1, 2], 24, {"topk": 40}), ([700] * 37, [1] * 37, 64, {"topk": 100}),
    ([200] * 74, [1] * 74, 16, {"topk": 60}), ([900] * 12, [3] * 12, 64, {"topk": 100}), ([400] * 7, [1, 2, 3, 4, 5, 6, 7], 32, {"topk": 60}),
    ([2000] * 9, [4] * 9, 64, {"topk": 100}), ([60, 1], [2, 1], 128, {"topk": 8})])
def test_compressed_attention_splits(ori_seq, s1_list, nq, kw):
    d = helpers.gen_scfa_inputs(900 + len(ori_seq) + nq, ori_seq, s1_list, nq=nq, **kw)
    # (with few keys the rounding of the probabilities shows in more last bits)
    parity._assert_attention_close(parity._run_scfa(d), parity._scfa_oracle(d), strict_frac=0.35)


@pytest.mark.parametrize("ori_seq,s1_list,nq", [([700], [301], 64), ([200, 5000], [150, 77], 40), ([900], [150], 128)])
def test_window_attention_persistent(ori_seq, s1_list, nq):
    parity.test_win_attention_seeded_cases(910 + nq, ori_seq, s1_list, nq, 128)


# rows ordered as a whole (up to 8192 entries, by value; scores that crowd take the general path) and the first length beyond
@pytest.mark.parametrize("n,k", [(65, 64), (3001, 2048), (8192, 2048), (8193, 2048), (8192, 1)])
def test_topk_short_rows(n, k):
    parity.test_topk_random_rows_exact_order(n, k)
    parity.test_topk_exact_order_across_score_distributions(n, k)


# one CTA an SM up to 148 rows and two beyond, for rows ordered whole, selected from, and with explicit ids; empty rows among them
@pytest.mark.parametrize("rows", [148, 149])
@pytest.mark.parametrize("ld", [2100, 8200])
@pytest.mark.parametrize("with_ids", [False, True])
def test_topk_row_counts(rows, ld, with_ids):
    g = torch.Generator().manual_seed(rows + ld)
    scores = torch.randn((rows, ld), generator=g).bfloat16().float()   # (ties)
    counts = torch.randint(0, ld + 1, (rows,), generator=g, dtype=torch.int32)
    counts[:3] = torch.tensor([0, 1, ld])
    ids = torch.stack([torch.randperm(2 * ld, generator=g)[:ld] for _ in range(rows)]).int() if with_ids else None
    if with_ids:
        ids[:, ::7] = -1   # entries to skip
    idx, sc = parity._run_topk(scores, counts, 2048, ids=ids)
    for r in range(rows):
        n = int(counts[r])
        v, i = scores[r, :n], ids[r, :n] if with_ids else torch.arange(n, dtype=torch.int32)
        v, i = v[i >= 0], i[i >= 0]
        i, order = i.sort()
        best = v[order].sort(descending=True, stable=True)
        k = min(2048, i.numel())
        assert torch.equal(idx[r, :k], i[best.indices[:k]]) and torch.equal(sc[r, :k], best.values[:k]), r
        assert bool((idx[r, k:] == -1).all()), r


# decode batches share their key blocks among the CTAs: lengths alike and ragged, empty requests, more than 128 requests
@pytest.mark.parametrize("act_seq,s1", [([700] * 5, 2), ([0, 129, 9000, 1, 128, 3000], 1), ([2 + 97 * (i % 40) for i in range(150)], 2)])
def test_indexer_shares(act_seq, s1):
    parity.test_indexer_ragged_vs_oracle(act_seq, s1)


# token tiles of the 8-bit-float prolog, and the packed projection where TMA cannot read the weights in place
@pytest.mark.parametrize("fmt", ["mxfp8", "hif8"])
@pytest.mark.parametrize("t", [128, 129, 257])
def test_pg_prolog_tiles(fmt, t):
    inp = helpers.gen_pg_prolog_inputs(920 + t, t, fmt)
    # a head weight is rounded to bf16 three times; the first rounding may fall the other way (2^-7 of it at most) and take the last
    # one with it, and a weight near zero keeps the absolute error of its 2560-long sum
    pg._check(inp, fmt, pg._run(inp, fmt), weights_rtol=2 ** -6, weights_atol=1e-5)


def test_pg_prolog_unaligned_weights():
    inp = helpers.gen_pg_prolog_inputs(930, 5, "mxfp8")
    odd = torch.empty(inp["w_proj"].numel() + 1, dtype=BF, device=DEV)[1:].view(inp["w_proj"].shape)
    odd.copy_(inp["w_proj"])
    assert odd.data_ptr() % 16 != 0
    for a, b in zip(pg._run(inp, "mxfp8"), pg._run(dict(inp, w_proj=odd), "mxfp8")):
        assert torch.equal(a.view(torch.uint8), b.view(torch.uint8))
