"""The register-tiled backward where one CTA takes a whole row tile (1536 row tiles and more; fewer go to pairs of CTAs, as in the other
tests), over every form it takes: bias and its gradient, dropout, token-packed sequences, grouped heads, 16-bit types; in one launch and
in two (16-bit types of head dims above 64 from 4096 row tiles on); against the oracle, and equal bit for bit to the separate stages.

Tolerances: those of test_gpu_random_shapes.py (atol = rtol = 1e-2 fp16, 2e-2 bf16, 1e-4 fp32; dBias four times the absolute one).
"""
import pytest
import torch

from oracle import attention as A
from _util import ATOL, close, randn_inputs

pytestmark = pytest.mark.gpu
SEED, OFFSET = 0x1BF52, 11


def _row_tiles(B, Hq, Hk, Sq, Sk):
    return B * (Hq * -(-Sq // 32) + Hk * -(-Sk // 32))


def _run(q, k, v, do, bias, stages, **kw):
    from aotriton_b200 import cabi
    B, Hq, Sq, _ = q.shape
    nan = lambda t: torch.full_like(t, float("nan"))
    out, lse = nan(q), torch.empty(B * Hq, Sq, device="cuda")
    assert cabi.attn_fwd(q, k, v, out, lse, bias=bias, **kw) == 0
    dq, dk, dv, delta, db = nan(q), nan(k), nan(v), torch.empty_like(lse), nan(bias) if bias is not None else None
    n0 = cabi.lib().ab200_launch_count()
    for s in stages:
        assert cabi.attn_bwd(q, k, v, out, do, dq, dk, dv, lse, delta, bias=bias, dbias=db, stage=s, **kw) == 0
    assert cabi.lib().ab200_last_bwd_family() == 1
    return [dq, dk, dv] + ([db] if bias is not None else []), cabi.lib().ab200_launch_count() - n0


@pytest.mark.parametrize("dt,D,B,Hq,Hk,Sq,Sk,causal,bias,p", [
    (torch.float32, 64, 4, 64, 64, 97, 65, False, True, 0.3), (torch.float32, 128, 4, 80, 40, 66, 129, True, False, 0.2),
    (torch.float32, 33, 4, 96, 96, 33, 64, False, False, 0.0), (torch.float16, 60, 4, 64, 32, 131, 100, False, True, 0.2),
    (torch.bfloat16, 60, 4, 96, 96, 70, 70, True, False, 0.0), (torch.float16, 100, 4, 64, 64, 97, 97, False, True, 0.2),
    (torch.bfloat16, 124, 4, 96, 48, 65, 130, True, False, 0.1),
    # two launches
    (torch.float16, 100, 8, 96, 96, 65, 95, False, True, 0.3), (torch.bfloat16, 124, 8, 96, 96, 96, 96, True, False, 0.0)])
def test_dense(dt, D, B, Hq, Hk, Sq, Sk, causal, bias, p):
    tiles = _row_tiles(B, Hq, Hk, Sq, Sk)
    assert tiles >= 1536
    q, k, v, do = randn_inputs((B, Hq, Sq, D), (B, Hk, Sk, D), (B, Hk, Sk, D), dt, seed=Sq + D)
    b = torch.randn(B, Hq, Sq, Sk, generator=torch.Generator().manual_seed(1)).to(dt) if bias else None
    ct = (3, A.TOP_LEFT, A.TOP_LEFT) if causal else (0, 0, 0)
    ref = A.attention(q, k, v, sm_scale=D ** -0.5, bias=b, mask=A.window_mask(Sq, Sk, *ct), dropout_p=p, dout=do,
                      keep=A.keep_masks(SEED, OFFSET, B, Hq, Sq, Sk, p) if p > 0 else None)
    kw = dict(sm_scale=D ** -0.5, causal_type=ct[0], window_left=ct[1], window_right=ct[2])
    if p > 0:
        kw.update(dropout_p=p, philox_seed=torch.tensor([SEED], dtype=torch.uint64, device="cuda"), philox_offset2=OFFSET)
    ins = [t.cuda() for t in (q, k, v, do)] + [b.cuda() if bias else None]
    got, launches = _run(*ins, ("all",), **kw)
    assert launches == (3 if dt != torch.float32 and D > 64 and tiles >= 4096 else 2)
    want, _ = _run(*ins, ("preprocess", "dkdv", "dq"), **kw)
    for name, a, w in zip(("dq", "dk", "dv", "db"), got, want):
        assert torch.equal(a, w), name
        ok, err = close(a.cpu().float(), getattr(ref, name), ATOL[dt] * (4 if name == "db" else 1), ATOL[dt])
        assert ok, (name, err)


@pytest.mark.parametrize("dt,D,H", [(torch.float32, 64, 64), (torch.float16, 60, 64), (torch.float16, 100, 64), (torch.float16, 100, 160)])
def test_packed(dt, D, H):
    from _gpu_runner import run_fwd_bwd
    lens = [0, 97, 1, 64, 130, 33]
    cu = [0, 0, 97, 98, 162, 292, 325]
    assert _row_tiles(6, H, H, 130, 130) >= (1536 if H == 64 else 4096)
    mk = lambda s: torch.randn(1, 325, H, D, generator=torch.Generator().manual_seed(s)).to(dt).transpose(1, 2)
    q, k, v, do = (mk(i) for i in range(4))
    ct = (3, A.BOTTOM_RIGHT, A.BOTTOM_RIGHT)
    ref = A.attention_varlen(q, k, v, cu, cu, sm_scale=D ** -0.5, causal_type=ct[0], window_left=ct[1], window_right=ct[2], dropout_p=0.2,
                             seed=SEED, offset_base=OFFSET, max_sq=max(lens), max_sk=max(lens), dout=do)
    res = run_fwd_bwd(q, k, v, do, sm_scale=D ** -0.5, causal_type=ct[0], window_left=ct[1], window_right=ct[2], dropout_p=0.2, seed=SEED,
                      offset1=0, offset2=OFFSET, cu_q=cu, cu_k=cu, max_sq=max(lens), max_sk=max(lens),
                      keep_layout=lambda t: t.transpose(1, 2).contiguous().transpose(1, 2))
    assert res["bwd_family"] == 1
    for key in ("out", "dq", "dk", "dv"):
        ok, err = close(res[key].float(), getattr(ref, key), ATOL[dt])
        assert ok, (key, err)
