"""dK formed from the bias gradient (dK = scale * dB^T Q), against the stage calls, in which the dK
kernel computes dS itself; and the calls that keep the dK kernel: a dBias whose rows no tile map can describe,
dQ in the place of Q.

The 16-bit dS values and the order of the sums (16 query rows at a time) are the same, so the results are equal
bit for bit.
"""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu
TL, BR = -2147483647, -2147483646


@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("p", [0.0, 0.2])
@pytest.mark.parametrize("B,Hq,Hk,Sq,Sk,D,causal,how", [
    (1, 1, 1, 64, 128, 256, (0, 0, 0), ""),
    (2, 2, 2, 65, 72, 136, (0, 0, 0), ""),
    (1, 4, 2, 257, 320, 256, (0, 0, 0), ""),
    (1, 2, 1, 384, 264, 192, (3, BR, BR), ""),           # bottom-right causal: rows without a key
    (1, 2, 2, 200, 512, 256, (3, TL, TL), ""),           # keys no query attends to
    (1, 2, 1, 512, 512, 208, (3, 100, 30), ""),
    (1, 2, 2, 130, 136, 256, (0, 0, 0), "bshd"),
    (1, 2, 2, 130, 131, 256, (0, 0, 0), "odd"),          # rows of dBias off a 16-byte boundary
    (2, 2, 2, 130, 136, 256, (0, 0, 0), "in place"),     # dQ over Q
])
def test_equal_to_separate_stages(B, Hq, Hk, Sq, Sk, D, causal, how, p, dt):
    from aotriton_b200 import cabi
    g = torch.Generator(device="cuda").manual_seed(Sq + Sk + D)

    def mk(b, h, s, d):
        t = torch.randn(b, s, h, d, generator=g, device="cuda").to(dt).transpose(1, 2)
        return t if how == "bshd" else t.contiguous()

    q, do, k, v, bias = mk(B, Hq, Sq, D), mk(B, Hq, Sq, D), mk(B, Hk, Sk, D), mk(B, Hk, Sk, D), mk(B, Hq, Sq, Sk)
    kw = dict(sm_scale=D ** -0.5, bias=bias, causal_type=causal[0], window_left=causal[1], window_right=causal[2], dropout_p=p)
    if p:
        kw.update(philox_seed=torch.tensor([77], dtype=torch.uint64, device="cuda"),
                  philox_offset1=torch.tensor([5], dtype=torch.uint64, device="cuda"))
    out, lse = torch.empty_like(q), torch.empty(B * Hq, Sq, device="cuda")
    assert cabi.attn_fwd(q, k, v, out, lse, **kw) == 0

    def backward(q, dq, *stages):
        grads = [dq] + [torch.full_like(t, float("nan")) for t in (k, v)]
        db, delta = torch.full_like(bias, float("nan")), torch.empty_like(lse)
        n0 = cabi.lib().ab200_launch_count()
        if stages == ("all",):
            args = cabi.make_bwd_args(q, k, v, out, do, *grads, lse, delta, dbias=db, **kw)
            assert cabi.lib().ab200_debug_dk_from_dbias(C.byref(args)) == (how in ("", "bshd"))
        for stage in stages:
            assert cabi.attn_bwd(q, k, v, out, do, *grads, lse, delta, dbias=db, stage=stage, **kw) == 0
        assert cabi.lib().ab200_launch_count() - n0 == 4      # preprocess, dV, dQ, and dK by either kernel
        return grads + [db]

    nan = torch.full_like(q, float("nan"))
    want = backward(q, nan.clone(), "preprocess", "dkdv", "dq")
    mine = q.clone()
    got = backward(mine, mine if how == "in place" else nan.clone(), "all")
    torch.cuda.synchronize()
    assert cabi.lib().ab200_kernel_status(0) == 0
    for name, a, b in zip(("dq", "dk", "dv", "db"), got, want):
        assert not torch.isnan(b.float()).any(), name
        assert torch.equal(a, b), f"{name}: {float((a.float() - b.float()).abs().max())}"
