"""Forward with few query rows (the split-key kernel of decoding), against the oracle: lengths on both
sides of its 16-key, 64-key and 8-piece boundaries, row counts up to and beyond one 32-row tile, windows
that miss whole pieces, packed sequences with a neighbour's non-finite tokens behind the last key; and, with the cut
of the keys, the warps and the ring stages asserted, calls whose CTAs go round their ring several times.

Tolerances: those of test_gpu_parity.py (atol = rtol = 2e-2 bf16, 1e-2 fp16; LSE 1e-3).
"""
import ctypes as C

import numpy as np
import pytest
import torch

from oracle import attention as A
from _util import ATOL, LSE_ATOL, close, randn_inputs

pytestmark = pytest.mark.gpu
TL, BR = A.TOP_LEFT, A.BOTTOM_RIGHT


def _plan(q, k, v, **kw):
    """(pieces of the keys, consumer warps, ring stages) of the split-key kernel; None: another kernel."""
    from aotriton_b200 import cabi
    a = cabi.make_fwd_args(q, k, v, q.new_empty(*q.shape[:3], v.shape[3]), None, sm_scale=1.0, **kw)
    n = cabi.lib().ab200_debug_split_keys(C.byref(a), None)
    assert n >= 0
    return (n & 0xff, n >> 8 & 0xff, n >> 16) if n else None


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,Hq,Hk,Sq,Sk,D,Dv,causal", [
    (1, 1, 1, 1, 1, 128, 128, (0, 0, 0)),
    (2, 8, 2, 1, 63, 128, 128, (0, 0, 0)),
    (1, 4, 4, 16, 64, 64, 64, (0, 0, 0)),             # 16 rows, one tile of keys
    (1, 16, 2, 5, 1025, 128, 128, (3, BR, BR)),       # 40 rows: two tiles of rows, several pieces
    (3, 6, 2, 3, 2047, 80, 96, (3, BR, BR)),          # padded and unequal head dims
    (1, 8, 1, 16, 700, 64, 64, (3, TL, TL)),          # 128 rows; most keys masked
    (1, 2, 1, 9, 1500, 128, 128, (3, 200, 0)),        # window: the last pieces see nothing
    (1, 4, 1, 12, 5, 128, 128, (3, BR, BR)),          # rows without a key
])
def test_few_queries_vs_oracle(B, Hq, Hk, Sq, Sk, D, Dv, causal, dt):
    from _gpu_runner import run_fwd_bwd
    q, k, v, _ = randn_inputs((B, Hq, Sq, D), (B, Hk, Sk, D), (B, Hk, Sk, Dv), dt, seed=Sk + Sq)
    ct, wl, wr = causal
    assert _plan(q.cuda(), k.cuda(), v.cuda()) is not None
    ref = A.attention(q, k, v, sm_scale=D ** -0.5, mask=A.window_mask(Sq, Sk, ct, wl, wr))
    res = run_fwd_bwd(q, k, v, sm_scale=D ** -0.5, causal_type=ct, window_left=wl, window_right=wr)
    assert res["fwd_family"] == 2
    ok, err = close(res["out"].float(), ref.out, ATOL[dt])
    assert ok, f"out max err {err}"
    ok, err = close(res["lse"].reshape(-1), ref.lse.reshape(-1).float(), LSE_ATOL)
    assert ok, f"lse max err {err}"


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,Hq,Hk,Sq,Sk,D,Dv,plan", [
    (1, 4, 1, 1, 8200, 128, 128, (8, 8, 6)),        # eight warps, 16 tiles a CTA through 6 stages
    (1, 2, 1, 1, 8000, 64, 64, (8, 8, 12)),
    (4, 32, 8, 1, 6007, 128, 128, (8, 4, 3)),       # two CTAs an SM: half the ring
    (4, 32, 8, 1, 6007, 64, 64, (8, 4, 6)),
    (1, 16, 2, 5, 8200, 128, 128, (8, 4, 6)),       # 32-row tiles
    (4, 32, 4, 5, 6007, 64, 64, (8, 4, 6)),
    (20, 8, 8, 1, 1000, 128, 128, (1, 4, 3)),       # more clusters than SMs: no cut
    (20, 8, 8, 1, 1100, 64, 64, (1, 4, 6)),
    (25, 4, 4, 1, 2000, 128, 128, (2, 4, 3)),
    (10, 4, 4, 2, 3001, 128, 128, (4, 4, 3)),
    (1, 4, 2, 1, 6000, 64, 128, (8, 8, 6)),         # the second box of K lies outside the tensor
    (1, 4, 2, 1, 6000, 128, 64, (8, 8, 6)),
])
def test_round_the_ring_vs_oracle(B, Hq, Hk, Sq, Sk, D, Dv, plan, dt):
    from aotriton_b200 import cabi
    q, k, v, _ = randn_inputs((B, Hq, Sq, D), (B, Hk, Sk, D), (B, Hk, Sk, Dv), dt, seed=Sk + Sq)
    kw = dict(sm_scale=D ** -0.5, causal_type=3, window_left=BR, window_right=BR)
    ref = A.attention(q, k, v, sm_scale=D ** -0.5, mask=A.window_mask(Sq, Sk, 3, BR, BR))
    qd, kd, vd = q.cuda(), k.cuda(), v.cuda()
    assert _plan(qd, kd, vd) == plan
    out, lse = torch.full((B, Hq, Sq, Dv), float("nan"), dtype=dt, device="cuda"), torch.full((B * Hq, Sq), float("nan"), device="cuda")
    assert cabi.attn_fwd(qd, kd, vd, out, lse, **kw) == 0
    again = torch.empty_like(out)
    assert cabi.attn_fwd(qd, kd, vd, again, lse, **kw) == 0
    ok, err = close(out.float().cpu(), ref.out, ATOL[dt])
    assert ok, f"out max err {err}"
    ok, err = close(lse.reshape(-1).cpu(), ref.lse.reshape(-1).float(), LSE_ATOL)
    assert ok, f"lse max err {err}"
    assert torch.equal(out, again)
    assert cabi.lib().ab200_kernel_status(0) == 0


def test_few_queries_packed_with_foreign_tokens():
    """Packed keys: each sequence's last tile is followed by a neighbour's tokens, here non-finite."""
    from aotriton_b200 import cabi
    dt, Hq, Hk, D = torch.bfloat16, 8, 2, 128
    len_q, len_k = [1, 3, 1], [130, 1, 777]
    g = torch.Generator().manual_seed(3)
    mk = lambda T, H: torch.randn(1, T, H, D, generator=g).to(dt).transpose(1, 2)
    q = mk(sum(len_q), Hq)
    starts = [0]
    for L in len_k:
        starts.append(starts[-1] + L + 40)
    k, v = mk(starts[-1], Hk), mk(starts[-1], Hk)
    for a, L, b in zip(starts, len_k, starts[1:]):
        k[:, :, a + L:b] = float("nan")
        v[:, :, a + L:b] = float("inf")
    cu_q, cu_k = ([0] + [int(x) for x in np.cumsum(t)] for t in (len_q, len_k))
    t32 = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")
    qd, kd, vd = q.cuda(), k.cuda(), v.cuda()
    out = torch.full_like(qd, float("nan"))
    assert cabi.attn_fwd(qd, kd, vd, out, None, sm_scale=D ** -0.5, causal_type=3, window_left=BR, window_right=BR,
                         cu_seqlens_q=t32(cu_q), cu_seqlens_k=t32(cu_k), max_seqlen_q=max(len_q), max_seqlen_k=max(len_k),
                         varlen_type=cabi.VARLEN_STRIDED, seq_strides_q=t32(cu_q), seq_strides_k=t32(starts)) == 0
    for z, (nq, nk) in enumerate(zip(len_q, len_k)):
        a, b = cu_q[z], starts[z]
        ref = A.attention(q[:, :, a:a + nq], k[:, :, b:b + nk], v[:, :, b:b + nk], sm_scale=D ** -0.5,
                          mask=A.window_mask(nq, nk, 3, BR, BR))
        ok, err = close(out[:, :, a:a + nq].float().cpu(), ref.out, ATOL[dt])
        assert ok, f"sequence {z}: max err {err}"
    torch.cuda.synchronize()
    assert cabi.lib().ab200_kernel_status(0) == 0
