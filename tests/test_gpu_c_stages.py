"""The C entries for callers that bring their own products: the stages of the V4 MLA prolog one by one and the compressor's state
update.  Each gets the products the oracle forms (or what it forms them from) and is held to the oracle's rows with the bounds of
the operators' own tests."""
import ctypes as C

import pytest
import torch

import test_gpu_parity as parity
from oracle import dsv32_oracle as orc
from pypto_b200 import _lib
from pypto_b200 import _runtime as rt

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
BF = torch.bfloat16
EPS = 1e-6


def _stage(stage, **fields):
    dev = torch.device(DEV)
    tensors = {k: v.to(DEV) for k, v in fields.items() if isinstance(v, torch.Tensor)}
    a = _lib.MlaV4StageArgs()
    a.eps = EPS
    for k, v in fields.items():
        setattr(a, k, rt.ptr(tensors[k]) if k in tensors else v)
    with torch.cuda.device(dev):
        rt.check(_lib.load().dsv32_mla_prolog_v4_stage(C.byref(a), stage, rt.stream_ptr(dev)), f"stage {stage}")
    torch.cuda.synchronize()
    return {k: v.cpu() for k, v in tensors.items()}


def _rotary(t, g):
    ang = (torch.rand((t, 32), generator=g) * 6.2831853).repeat_interleave(2, -1)
    return torch.cos(ang).to(BF), torch.sin(ang).to(BF)


def _rms(v, gamma=None):
    v = v.double()
    v = v / torch.sqrt((v * v).mean(-1, keepdim=True) + EPS)
    return v if gamma is None else v * gamma.double()


def _rotated(rows, cos, sin):
    """bf16 rows [t, .., 512] with their last 64 dims through the rotary embedding."""
    head = rows.reshape(rows.shape[0], -1, 512)
    pe = orc.rope_interleaved_inverse(head[:, :, -64:], cos, -sin)
    return torch.cat([head[:, :, :-64], pe], dim=-1).reshape(rows.shape)


def _close_bf16(got, want):
    # one rounding to bf16, or two where the rotary embedding adds two such values: a step of 2^-7 of the larger, rarely taken
    diff = (got.double() - want.double()).abs()
    assert bool((diff <= 2.0 ** -7 * want.double().abs() + 2.0 ** -8).all())
    assert (diff > 0).double().mean() <= 0.01


@pytest.mark.parametrize("quant", [True, False])
@pytest.mark.parametrize("t,heads,pad", [(1, 1, 0), (5, 3, 64), (130, 2, 0)])
def test_mla_prolog_v4_stages(quant, t, heads, pad):
    g = torch.Generator().manual_seed(2100 + t + heads)
    of = (lambda v: v.float()) if quant else (lambda v: v.to(BF))
    cos, sin = _rotary(t, g)
    gam_q, gam_kv = ((1 + 0.1 * torch.randn(n, generator=g)).to(BF) for n in (1024, 512))
    # stage 0: q_a -> qr
    q_a = of(torch.randn((t, 1024), generator=g))
    got = _stage(0, q_a=q_a, gamma_cq=gam_q, t=t, heads=heads, quant=int(quant),
                 qr=torch.empty((t, 1024), dtype=torch.int8 if quant else BF), qr_scale=torch.empty(t))
    want = _rms(q_a, gam_q)
    if quant:
        qr, scale = orc.quant_int8_rows(want.float())
        diff = (got["qr"].int() - qr.int()).abs()
        assert diff.max() <= 1 and (diff > 0).float().mean() <= 0.005
        assert torch.allclose(got["qr_scale"], scale.reshape(-1), rtol=1e-5, atol=0)
    else:
        _close_bf16(got["qr"], want.to(BF))
    # stage 1: q_b -> q, the product's rows longer than the heads
    ld = heads * 512 + pad
    scale, w_scale = torch.rand(t, generator=g) * 0.01 + 0.001, torch.rand(heads * 512, generator=g) * 0.01 + 0.001
    if quant:
        q_b = torch.randint(-200000, 200001, (t, ld), generator=g, dtype=torch.int32)
        x = q_b[:, :heads * 512].double() * scale.double()[:, None] * w_scale.double()
    else:
        q_b = torch.randn((t, ld), generator=g).to(BF)
        x = q_b[:, :heads * 512].double()
    got = _stage(1, q_b=q_b, qr_scale=scale, wq_b_scale=w_scale, cos=cos, sin=sin, t=t, heads=heads, q_b_ld=ld, quant=int(quant),
                 q_out=torch.empty((t, heads, 512), dtype=BF))
    _close_bf16(got["q_out"], _rotated(_rms(x.reshape(t, heads, 512)).to(BF), cos, sin))
    # stage 2: kv_a -> kv
    kv_a = of(torch.randn((t, 512), generator=g))
    got = _stage(2, kv_a=kv_a, gamma_ckv=gam_kv, cos=cos, sin=sin, t=t, heads=heads, quant=int(quant),
                 kv_out=torch.empty((t, 512), dtype=BF))
    _close_bf16(got["kv_out"], _rotated(_rms(kv_a, gam_kv).to(BF), cos, sin))


@pytest.mark.parametrize("ratio,d,starts,s1", [(4, 512, [0, 3, 126], 6), (128, 72, [127, 1], 2), (4, 70, [4], 1)])
def test_compressor_update_alone(ratio, d, starts, s1, monkeypatch):
    def update(inp):   # in the place of the operator: the products come from torch, rows without a closed window stay as they are
        c = parity._cuda(inp)
        dev = torch.device(DEV)
        x = inp["x"].reshape(-1, inp["x"].shape[-1]).double()
        kv, score = ((x @ inp[w].double().t()).float().to(DEV) for w in ("wkv", "wgate"))
        kv_state, score_state = c["kv_state"].clone(), c["score_state"].clone()
        b = len(starts)
        out = torch.zeros((min(b * s1, b * s1 // ratio + b), d), dtype=BF, device=DEV)
        a = _lib.CompressorArgs(
            rt.ptr(kv), rt.ptr(score), rt.ptr(c["ape"]), rt.ptr(c["weight"]), rt.ptr(kv_state), rt.ptr(score_state), rt.ptr(c["table"]),
            rt.ptr(c["table"]), rt.ptr(c["sin"]), rt.ptr(c["cos"]), rt.ptr(c["start_pos"]), rt.ptr(out), rt.ptr(rt.status_word(dev)),
            kv_state.shape[0], score_state.shape[0], b, s1, d, ratio, c["table"].shape[1], c["table"].shape[1], EPS)
        with torch.cuda.device(dev):
            rt.check(_lib.load().dsv32_compressor_update(C.byref(a), rt.stream_ptr(dev)), "compressor_update")
        import pypto_b200
        pypto_b200.check_status()
        return out.cpu(), kv_state.cpu(), score_state.cpu()

    monkeypatch.setattr(parity, "_run_compressor", update)
    parity.test_compressor_seeded_vs_oracle(ratio, False, d, starts, s1)
