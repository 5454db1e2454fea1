"""Dropout keep bits that pass from the dK/dV kernel to the dQ kernel through rows of dQ.

The oracle is the same backward in separate stage calls, where every kernel draws its own bits: the
arithmetic is the same, so the gradients must be equal bit for bit.
"""
import ctypes as C

import numpy as np
import pytest
import torch

TL, BR = -2147483647, -2147483646


def _keep_tiles(q, k, v, dq, **kw):
    from aotriton_b200 import cabi
    out, do = torch.empty_like(q), torch.empty_like(q)
    dk, dv = torch.empty_like(k), torch.empty_like(v)
    lse = torch.empty(q.shape[0] * q.shape[1], q.shape[2])
    for name in ("out", "do"):
        if kw.get("alias") == name:
            dq = {"out": out, "do": do}[name]
    if kw.get("alias") == "lse":
        lse = dq
    a = cabi.make_bwd_args(q, k, v, out, do, dq, dk, dv, lse, torch.empty_like(lse), sm_scale=1.0,
                           dropout_p=kw.get("p", 0.1))
    return cabi.lib().ab200_debug_keep_tiles(C.byref(a))


def test_rule():
    mk = lambda *s: torch.empty(*s, dtype=torch.float16)
    for d, sk, want in ((64, 4000, 32), (72, 4000, 32), (120, 1000, 32), (128, 4000, 64), (128, 391, 13), (200, 5000, 64),
                        (256, 5000, 128), (56, 400, 0), (32, 400, 0)):
        q, k = mk(2, 4, 300, d), mk(2, 2, sk, d)
        assert _keep_tiles(q, k, mk(2, 2, sk, d), torch.empty_like(q)) == want, (d, sk)
    q, k, v = mk(2, 4, 300, 128), mk(2, 2, 300, 128), mk(2, 2, 300, 128)
    full = _keep_tiles(q, k, v, torch.empty_like(q))
    assert full == 10
    assert _keep_tiles(q, k, v, torch.empty_like(q), p=0.0) == 0
    # storage orders without shared memory are taken
    assert _keep_tiles(q, k, v, mk(2, 300, 4, 128).transpose(1, 2)) == full
    assert _keep_tiles(q, k, v, mk(4, 300, 2, 128).permute(2, 0, 1, 3)) == full
    assert _keep_tiles(q, k, v, mk(2, 4, 300, 136)[..., :128]) == full
    # dQ in the place of something the kernels still read, rows that overlap, other extents
    assert _keep_tiles(q, k, v, q) == 0
    assert _keep_tiles(q, k, v, None, alias="do") == 0
    assert _keep_tiles(q, k, v, torch.empty_like(q), alias="lse") == 0
    pool = mk(4 * 2 * 4 * 300 * 128)
    view = lambda at, *s: pool[at:at + int(np.prod(s))].view(*s)
    assert _keep_tiles(q, view(0, 2, 2, 300, 128), v, view(2 * 2 * 300 * 128 - 128, 2, 4, 300, 128)) == 0
    assert _keep_tiles(q, view(0, 2, 2, 300, 128), v, view(2 * 2 * 300 * 128, 2, 4, 300, 128)) == full
    assert _keep_tiles(q, k, v, mk(1, 4, 300, 128).expand(2, 4, 300, 128)) == 0
    assert _keep_tiles(q, k, v, mk(2, 4, 300 * 128).as_strided((2, 4, 300, 128), (4 * 300 * 128, 300 * 128, 64, 1))) == 0
    assert _keep_tiles(q, k, v, mk(2, 4, 200, 128)) == 0
    assert _keep_tiles(q, k, v, mk(2, 4, 300, 132)[..., :128]) == 0           # rows off a 16-byte boundary


def test_rule_follows_the_kernels_that_run():
    """No bits are handed on where the general kernels or the fused backward take the call."""
    from aotriton_b200 import cabi
    L = cabi.lib()

    def ask(dt, d, dq_acc=None, family=0, **kw):
        mk = lambda h: torch.empty(2, h, 300, d, dtype=dt)
        q, k, v, out, do, dq, dk, dv = mk(4), mk(2), mk(2), mk(4), mk(4), mk(4), mk(2), mk(2)
        lse = torch.empty(8, 300)
        a = cabi.make_bwd_args(q, k, v, out, do, dq, dk, dv, lse, torch.empty_like(lse), sm_scale=1.0, dropout_p=0.1, **kw)
        if dq_acc:
            a.dq_acc = lse.data_ptr()
        old = L.ab200_set_kernel_family(family)
        try:
            return L.ab200_debug_keep_tiles(C.byref(a))
        finally:
            L.ab200_set_kernel_family(old)

    h = torch.bfloat16
    assert ask(h, 128) == 10 and ask(h, 128, family=2) == 10
    assert ask(torch.float32, 128) == 0                              # general kernels: single precision,
    assert ask(h, 100) == 0 and ask(h, 264) == 0                     # head dims outside the tcgen05 kernels',
    assert ask(h, 128, family=1) == 0                                # or by force
    assert ask(h, 100, family=2) == -801                             # refused
    assert ask(h, 128, dq_acc=True, family=3) == 0                   # fused
    assert ask(h, 128, dq_acc=True, family=3, deterministic=True) == 10
    assert ask(h, 128, dq_acc=True) == 10 and ask(h, 128, family=3) == 10
    assert ask(h, 64, dq_acc=True, family=3) == 10                   # no fused form for 64 and above 128
    assert ask(h, 256, dq_acc=True, family=3) == 10


CASES = [
    # B, Hq, Hk, Sq, Sk, D, causal (type, left, right), bias, packed lengths
    (2, 4, 4, 128, 128, 64, (0, 0, 0), False, None),
    (1, 2, 2, 33, 31, 64, (0, 0, 0), False, None),               # one whole row group, one partial key tile
    (1, 2, 1, 31, 400, 64, (0, 0, 0), False, None),              # no whole row group
    (1, 4, 2, 391, 1100, 72, (0, 0, 0), True, None),             # keys beyond the 32 tiles of a row group
    (1, 2, 2, 300, 2200, 128, (3, BR, BR), False, None),         # beyond 64 tiles, masked tiles
    (1, 4, 1, 640, 640, 128, (3, 130, 65), False, None),         # window: tiles masked on both sides
    (1, 2, 2, 320, 500, 192, (3, TL, TL), False, None),          # wide: 64-row streams against 128-row blocks
    (1, 2, 1, 257, 321, 256, (0, 0, 0), True, None),
    (0, 4, 2, 0, 0, 128, (3, TL, TL), False, [5, 32, 401, 2300, 64]),
    (0, 2, 2, 0, 0, 256, (3, 90, 10), False, [97, 700, 1]),
]


@pytest.mark.gpu
@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("order", ["bhsd", "bshd"])
@pytest.mark.parametrize("case", CASES)
def test_equal_to_separate_stages(case, order, dt):
    from aotriton_b200 import cabi
    B, Hq, Hk, Sq, Sk, D, (ct, wl, wr), with_bias, lens = case
    g = torch.Generator(device="cuda").manual_seed(Sq + Sk + D)

    def mk(b, h, s, d):
        t = torch.randn(b, s, h, d, generator=g, device="cuda").to(dt)
        return t.transpose(1, 2) if order == "bshd" or lens else t.transpose(1, 2).contiguous()

    kw = dict(sm_scale=D ** -0.5, causal_type=ct, window_left=wl, window_right=wr, dropout_p=0.3,
              philox_seed=torch.tensor([0x5ca1ab1e12345], dtype=torch.uint64, device="cuda"),
              philox_offset1=torch.tensor([0xfffffff0], dtype=torch.uint64, device="cuda"), philox_offset2=7)
    if lens:
        B, Sq, Sk = 1, sum(lens), sum(lens)
        cu = torch.tensor([0] + [int(x) for x in np.cumsum(lens)], dtype=torch.int32, device="cuda")
        kw.update(cu_seqlens_q=cu, cu_seqlens_k=cu, max_seqlen_q=max(lens), max_seqlen_k=max(lens))
    q, do, k, v = mk(B, Hq, Sq, D), mk(B, Hq, Sq, D), mk(B, Hk, Sk, D), mk(B, Hk, Sk, D)
    bias = mk(B, Hq, Sq, Sk + -Sk % 8)[..., :Sk] if with_bias else None
    out, lse = torch.empty_like(q), torch.empty(B * Hq, Sq, device="cuda")
    assert cabi.attn_fwd(q, k, v, out, lse, bias=bias, **kw) == 0

    def backward(*stages):
        grads = [torch.full_like(t, float("nan")) for t in (q, k, v)]
        db = torch.full_like(bias, float("nan")) if with_bias else None
        delta = torch.empty_like(lse)
        for stage in stages:
            assert cabi.attn_bwd(q, k, v, out, do, *grads, lse, delta, bias=bias, dbias=db, stage=stage, **kw) == 0
        return grads + ([db] if with_bias else [])

    got, want = backward("all"), backward("preprocess", "dkdv", "dq")
    torch.cuda.synchronize()
    assert cabi.lib().ab200_kernel_status(0) == 0
    for name, a, b in zip(("dq", "dk", "dv", "db"), got, want):
        assert not torch.isnan(b.float()).any() and torch.equal(a, b), f"{name}: {float((a.float() - b.float()).abs().max())}"
