"""Forward with dropout: the keep bits are drawn by warps of their own, two blocks ahead.  Numbers of key blocks
around the two buffers, one and two query tiles per CTA, partial tiles, windows, bias; against the oracle
with the reference's counter scheme.

Tolerances: those of test_gpu_parity.py (atol = rtol = 2e-2 bf16, 1e-2 fp16; LSE 1e-3).
"""
import pytest
import torch

from oracle import attention as A
from _util import ATOL, LSE_ATOL, close, randn_inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("B,Hq,Hk,Sq,Sk,D,causal,bias", [
    (1, 2, 1, 128, 128, 64, (0, 0, 0), False),          # one tile, one block
    (1, 2, 2, 129, 127, 64, (0, 0, 0), False),          # a second tile of one row
    (2, 1, 1, 256, 256, 128, (0, 0, 0), False),
    (1, 2, 1, 300, 385, 128, (0, 0, 0), True),          # four blocks, the last of one key
    (1, 2, 1, 256, 384, 128, (0, 0, 0), True),
    (1, 1, 1, 17, 900, 80, (3, A.BOTTOM_RIGHT, A.BOTTOM_RIGHT), False),
    (1, 2, 1, 700, 700, 128, (3, 150, 20), False),      # blocks outside the window are skipped
    (1, 1, 1, 60, 40, 64, (3, A.BOTTOM_RIGHT, A.BOTTOM_RIGHT), False),      # rows without a key
    (1, 2, 2, 130, 260, 256, (0, 0, 0), True),          # one tile per CTA
    (1, 1, 1, 384, 384, 256, (3, A.TOP_LEFT, A.TOP_LEFT), False),
])
def test_vs_oracle(B, Hq, Hk, Sq, Sk, D, causal, bias, dt):
    from _gpu_runner import run_fwd_bwd
    q, k, v, _ = randn_inputs((B, Hq, Sq, D), (B, Hk, Sk, D), (B, Hk, Sk, D), dt, seed=Sq + Sk + D)
    b = torch.randn(B, Hq, Sq, Sk, generator=torch.Generator().manual_seed(5)).to(dt) if bias else None
    (ct, wl, wr), p, seed, off = causal, 0.37, 0x123456789AB, 0xFFFFFF00
    keep = A.keep_masks(seed, off + 9, B, Hq, Sq, Sk, p)
    mask = A.window_mask(Sq, Sk, ct, wl, wr) if ct else None
    ref = A.attention(q, k, v, sm_scale=D ** -0.5, bias=b, mask=mask, keep=keep, dropout_p=p)
    res = run_fwd_bwd(q, k, v, sm_scale=D ** -0.5, bias=b, causal_type=ct, window_left=wl, window_right=wr, dropout_p=p,
                      seed=seed, offset1=off, offset2=9)
    assert res["fwd_family"] == 2 and res["seed_out"] == seed and res["off_out"] == off + 9
    ok, err = close(res["out"].float(), ref.out.float(), ATOL[dt])
    assert ok, f"out max err {err}"
    ok, err = close(res["lse"].reshape(-1), ref.lse.reshape(-1).float(), LSE_ATOL)
    assert ok, f"lse max err {err}"
